"""CPU: which prepared pieces of a batch are launched at once and which wait for the next."""
import pytest

from updes_gb300.batched import _finish

PIECES = [(0, 30), (30, 60), (60, 85), (85, 100)]


def _launches(host, solve):
    """The pieces launched, when each 1 % of the batch takes ``host`` seconds to prepare, and the end."""
    out, first, now, gpu = [], 0, 1e6, 0.0  # a clock's reading, whose zero is anywhere
    for k, (a, b) in enumerate(PIECES):
        now += host * (b - a)
        later = PIECES[k + 1:]
        if _finish((first, b), later, [host * (q - p) for p, q in later], now, gpu, solve)[1]:
            out.append((first, b))
            gpu = max(now, gpu) + solve((first, b))
            first = b
    return out, gpu - 1e6


def test_systems_that_fill_the_gpu_once_are_launched_once():
    # any launch takes one round, however few systems it has
    assert _launches(0.1, lambda p: 30.0)[0] == [(0, 100)]


def test_a_slow_host_launches_every_piece():
    launches, end = _launches(1.0, lambda p: 0.4 * (p[1] - p[0]))
    assert launches == PIECES and end == pytest.approx(100.0 + 0.4 * 15)


def test_rounds_hidden_behind_the_host():
    # 10 s a round against 25 s of preparation: only the last launch is seen, so nothing waits for company in vain
    launches, end = _launches(1.0, lambda p: 10.0)
    assert end == pytest.approx(110.0) and launches[-1][1] == 100


@pytest.mark.parametrize("host", [0.0, 0.01, 0.1, 1.0, 10.0])
@pytest.mark.parametrize("a,b", [(0.0, 1.0), (5.0, 0.0), (5.0, 1.0), (50.0, 0.2)])
def test_never_later_than_one_launch_nor_than_four(host, a, b):
    solve = lambda p: a + b * (p[1] - p[0])
    launches, end = _launches(host, solve)
    assert launches[0][0] == 0 and launches[-1][1] == 100 and all(p[1] == q[0] for p, q in zip(launches, launches[1:]))
    one, now, gpu = host * 100 + solve((0, 100)), 0.0, 0.0
    for p in PIECES:
        now += host * (p[1] - p[0])
        gpu = max(now, gpu) + solve(p)
    assert end <= 1.04 * min(one, gpu) + 1e-6
