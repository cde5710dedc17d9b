// Internal interface of the LU and triangular-solve kernels.
#pragma once

#include "common.cuh"

constexpr int kLuNb = 64;  // panel width

// FP64 LU in place, LAPACK's pivot choices (interchanges to piv[0, n)).  use_digits: the updates on the tensor cores, for
// a matrix whose rows and columns are scaled (gemm_tc64.cu says to what); else by FP64 multiply-adds, for any.
size_t lu_64_workspace_bytes(int n);
int lu_factor_64(int n, double* W, int64_t ld, int32_t* piv, void* ws, size_t ws_bytes, DeviceStatus* st,
                 cudaStream_t s, bool use_digits);

// The panel W[k:n, k:k+w] (w <= 64) factored in place on one thread-block cluster (panel.cu): interchanges to
// piv[k..k+w) and their net permutation to swap_map (257 ints, may be null).  UPDES_ERR_UNSUPPORTED when a thread
// would have more rows than its registers hold.  after_kernel: launched early, as by launch_next.
int panel_cluster(float* W, int64_t ld, int n, int k, int w, int32_t* piv, int32_t* swap_map, DeviceStatus* st,
                  cudaStream_t s, bool after_kernel);
int panel_cluster(double* W, int64_t ld, int n, int k, int w, int32_t* piv, int32_t* swap_map, DeviceStatus* st,
                  cudaStream_t s, bool after_kernel);

// mode: 0 = L, 1 = U, 2 = U^T, 3 = L^T (x overwritten in place); sync_ws: ceil(n/64)+2 ints.
// dinv (FP32 factors only, may be null): inverted diagonal blocks from diag_inverse, applied as matvecs
// instead of the substitution inside each block.
// xh, xl (n FP32 each, may be null): scratch planes that carry solved blocks in double-float between CTAs
// (used together with dinv).
// dinv128 (with dinv, xh, xl): inverted 128 x 128 diagonal blocks from diag_inverse128, for the 128-row solve.
// xtag (with dinv128, may be null): 2n 8-byte words through which the 128-row solve hands each solved block
// to the blocks after it, the double-float value and the block's tag in one word (no flag, no fence).
template <typename TF>
int trsv_impl(int n, const TF* F, int64_t ldf, double* x, int mode, int* sync_ws, DeviceStatus* st, cudaStream_t s,
              const float* dinv = nullptr, float* xh = nullptr, float* xl = nullptr, const float* dinv128 = nullptr,
              unsigned long long* xtag = nullptr);

// Inverses of the 64 x 64 diagonal blocks of FP32 LU factors, as double-float planes (diag_inverse_bytes).
size_t diag_inverse_bytes(int n);
int diag_inverse(int n, const float* F, int64_t ldf, float* dinv, cudaStream_t s);
// Inverses of the 128 x 128 diagonal blocks, composed from those of diag_inverse (diag_inverse128_bytes).
size_t diag_inverse128_bytes(int n);
int diag_inverse128(int n, const float* F, int64_t ldf, const float* dinv64, float* dinv128, cudaStream_t s);

// Mixed LU on a double-float working matrix (Whi, Wlo FP32 planes): factors in FP32 (overwriting Whi),
// every trailing update formed from digit products on the tensor cores (to 2^-31 of |L||U| where its entries are of one size,
// see gemm_tc3.cu) and accumulated in double-float.
size_t lu_df_workspace_bytes(int n);
int lu_factor_df(int n, float* Whi, float* Wlo, int64_t ld, int32_t* piv, void* ws, size_t ws_bytes, DeviceStatus* st,
                 cudaStream_t s);
