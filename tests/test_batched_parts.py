"""The parts of a batch: consecutive, complete, none empty."""
import pytest

from updes_gb300.batched import _parts


@pytest.mark.parametrize("sizes", [[5], [7] * 127, [7] * 128, [2000] + [16] * 200, [16] * 200 + [2000], [1] * 128,
                                   list(range(10, 400)), list(range(400, 10, -1))])
def test_parts(sizes):
    parts = _parts(sizes)
    assert parts[0][0] == 0 and parts[-1][1] == len(sizes)
    assert all(a < b for a, b in parts)
    assert all(p[1] == q[0] for p, q in zip(parts, parts[1:]))
    assert len(parts) == 1 if len(sizes) < 128 else 1 <= len(parts) <= 4
