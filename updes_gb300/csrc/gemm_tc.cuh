// Tensor-core trailing update of the mixed-precision LU (see gemm_tc.cu).
#pragma once

#include "common.cuh"


// C (double-float planes hi/lo, ldc) -= A (m x K FP32, lda) * B (K x nc FP32, ldb), products exact.
int ozaki_update(float* Chi, float* Clo, int64_t ldc, const float* A, int64_t lda, const float* B, int64_t ldb,
                 int m, int nc, int K, DeviceStatus* st, cudaStream_t s);

// The persistent, warp-specialised version (gemm_tc3.cu), K <= 256: digits written once per update into `scratch`
// (ozaki3_scratch_bytes(m, nc, K) bytes, 256-byte aligned), 8 products of FP16 digits, fed by bulk copies.  The kernel keeps one
// CTA per SM; `max_ctas` > 0 caps its grid so that work on another stream keeps the remaining SMs.
size_t ozaki3_scratch_bytes(int mmax, int ncmax, int Kmax);
// a_digits_ready: the previous update on `scratch` had the same A (same m, K and values), whose digits and
// scales are still there; only B's are written.  early: as in launch_next.
int ozaki3_update(float* Chi, float* Clo, int64_t ldc, const float* A, int64_t lda, const float* B, int64_t ldb,
                  int m, int nc, int K, void* scratch, size_t scratch_bytes, DeviceStatus* st, cudaStream_t s,
                  int max_ctas = 0, bool a_digits_ready = false, bool early = false);

// C (FP64, ldc) -= A (m x K FP64, lda) * B (K x nc FP64, ldb), K <= 256, from exact products of 7 digits of each
// operand (gemm_tc64.cu); scratch, max_ctas and a_digits_ready as for ozaki3_update.
size_t ozaki64_scratch_bytes(int mmax, int ncmax, int Kmax);
int ozaki64_update(double* C, int64_t ldc, const double* A, int64_t lda, const double* B, int64_t ldb, int m, int nc,
                   int K, void* scratch, size_t scratch_bytes, DeviceStatus* st, cudaStream_t s, int max_ctas = 0,
                   bool a_digits_ready = false, bool early = false);

// A fixed FP64 matrix (m x n) times up to 64 columns on the same digits (gemm_tc64.cu).  rhs64_matrix writes the digits
// of rows [r0, r0 + rows) into `matrix` (rhs64_matrix_bytes(m, n) bytes), from FP64 rows (A, lda) or, with A null,
// from the sum of two FP32 planes.  rhs64_multiply leaves the product as `splits` partial sums, each m x 64 (row
// stride 64), to be added in order; `columns`: scratch of rhs64_columns_bytes(n).  rhs64_setup before a capture.
// skip (device, may be null): nothing is done when it holds something other than 0.
constexpr int kRhs64MaxSplits = 16;
size_t rhs64_matrix_bytes(int m, int n);
size_t rhs64_columns_bytes(int n);
int rhs64_splits(int m, int n);
int rhs64_setup();
int rhs64_matrix(const double* A, const float* hi, const float* lo, int64_t lda, int m, int n, int r0, int rows,
                 void* matrix, cudaStream_t s);
int rhs64_multiply(const void* matrix, int m, int n, const double* X, int64_t ldx, int R, void* columns,
                   double* partial, int splits, DeviceStatus* st, cudaStream_t s, const int32_t* skip = nullptr);
