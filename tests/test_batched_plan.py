"""CPU: which systems of a batch go to clusters (updes_solve_batched_plan), on a GPU of 152 SMs that holds 16 clusters.

A batch of equal systems that fill the SMs one CTA each is not put on clusters, of which 16 at a time take 8.5 ms a round
for 784 nodes where the single CTAs need 30 ms in all; a few systems, or large ones among small ones, are.
"""
import ctypes

import pytest

from updes_gb300 import _lib

NONE = 2 ** 31 - 1


def _plan(sizes, sms=152, teams=16):
    n = (ctypes.c_int32 * len(sizes))(*sizes)
    start, ms = ctypes.c_int32(), ctypes.c_double()
    _lib.check(_lib.load().updes_solve_batched_plan(n, len(sizes), sms, teams, ctypes.byref(start), ctypes.byref(ms)), "plan")
    return start.value, ms.value


@pytest.mark.parametrize("count,n", [(64, 787), (100, 787), (127, 787), (152, 787), (200, 787), (300, 403), (127, 1603),
                                     (152, 2028), (1000, 203), (5, 200)])
def test_full_sms_take_one_cta_a_system(count, n):
    start, ms = _plan([n] * count)
    assert start == NONE
    alone = _plan([n], teams=0)[1]
    assert ms == pytest.approx(alone * -(-count // 152))


@pytest.mark.parametrize("count,n", [(1, 787), (16, 787), (17, 787), (40, 787), (1, 403), (16, 4000), (60, 1603)])
def test_few_systems_go_to_clusters(count, n):
    start, ms = _plan([n] * count)
    assert start == n and ms < _plan([n] * count, teams=0)[1]


def test_large_systems_among_small_ones():
    sizes = [70 + 7 * k for k in range(150)] + [1800, 2000, 2028]
    start, ms = _plan(sizes)
    assert 384 <= start <= 1800
    assert ms < 0.5 * _plan(sizes, teams=0)[1]


def test_small_and_many():
    assert _plan([383] * 10)[0] == NONE
    assert _plan(list(range(64, 4097)))[1] > 0
    assert _plan([1])[1] > 0
    n = (ctypes.c_int32 * 1)(4097)
    start, ms = ctypes.c_int32(), ctypes.c_double()
    assert _lib.load().updes_solve_batched_plan(n, 1, 152, 16, ctypes.byref(start), ctypes.byref(ms)) == _lib.ERR_UNSUPPORTED
