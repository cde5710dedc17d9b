"""The scratch of a batch: nobody else is given it while the batch runs."""
import pytest

from updes_gb300 import batched as B


@pytest.fixture(autouse=True)
def _empty_cache(monkeypatch):
    torch = pytest.importorskip("torch")
    monkeypatch.setattr(B, "_torch", lambda: torch)  # buffers on the CPU here
    kept = dict(B._WS)
    B._WS.clear()
    yield
    B._WS.clear()
    B._WS.update(kept)


def _cpu():
    return B._torch().device("cpu", 0)


def test_a_batch_inside_another_has_its_own():
    outer, inner = B._Workspace(_cpu()), B._Workspace(_cpu())
    a, b = outer.of(100), inner.of(50)
    assert a.data_ptr() != b.data_ptr() and not B._WS
    inner.give_back()
    assert outer.of(80) is a and B._Workspace(_cpu()).of(10) is b


def test_the_larger_one_is_kept():
    outer, inner = B._Workspace(_cpu()), B._Workspace(_cpu())
    a, b = outer.of(100), inner.of(50)
    inner.give_back()
    outer.give_back()
    outer.give_back()  # a second time changes nothing
    assert list(B._WS.values()) == [a]
    assert B._Workspace(_cpu()).of(90) is a


def test_parts_share_it_and_it_grows():
    w = B._Workspace(_cpu())
    a = w.of(100)
    assert w.of(60) is a and w.of(200).numel() >= 200
    w.give_back()
    assert B._WS[0].numel() >= 200
