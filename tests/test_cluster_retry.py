"""Which cluster sizes a solve tries in turn: wider ones where a plan does not fit
the shared memory, and narrower ones where the rule's own choice cannot be
scheduled (a device with few SMs a partition), never for a size the caller gave.
The device calls are replaced by their answers."""
import types

import pytest

from tensorfox_gb300 import gauss_newton as gn

UNSUPPORTED = 5


def batch(monkeypatch, R, answer):
    tried = []

    def solve(*a):
        tried.append(a[5])
        return 0 if answer(a[5]) else UNSUPPORTED

    def check(status):
        if status:
            raise RuntimeError("status %d" % status)

    monkeypatch.setattr(gn._lib, "load", lambda: types.SimpleNamespace(tfx_dgn_solve=solve))
    monkeypatch.setattr(gn._lib, "check", check)
    monkeypatch.setattr(gn._dev, "stream", lambda: 0)
    b = gn._Batch.__new__(gn._Batch)
    b.precision, b.R, b.n, b.desc, b.d_desc, b.opts = "fp64", R, len(R), None, None, gn._lib.DgnOptions()
    return b, tried


@pytest.mark.parametrize("limit", [1, 2, 4, 8])
def test_unschedulable_choice_is_narrowed(monkeypatch, limit):
    b, tried = batch(monkeypatch, [10], lambda c: c <= limit)
    assert b.launch(10, auto=True) == limit
    assert tried[0] == 10


def test_choice_too_large_for_shared_memory_is_widened(monkeypatch):
    b, tried = batch(monkeypatch, [40], lambda c: c >= 12)
    assert b.launch(8, auto=True) == 12
    assert tried == [8, 12]


def test_choice_above_the_smallest_rank(monkeypatch):
    b, tried = batch(monkeypatch, [2, 9], lambda c: c == 2)   # one CTA does not fit
    assert b.launch(8, auto=True) == 2


def test_given_size_is_not_narrowed(monkeypatch):
    b, tried = batch(monkeypatch, [40], lambda c: c <= 4)
    with pytest.raises(RuntimeError):
        b.launch(8)
    assert tried == [8, 12, 16]


def test_nothing_fits(monkeypatch):
    b, tried = batch(monkeypatch, [40], lambda c: False)
    with pytest.raises(RuntimeError):
        b.launch(8, auto=True)
    assert sorted(tried) == [1, 2, 4, 8, 12, 16]


def test_other_errors_are_raised_at_once(monkeypatch):
    b, tried = batch(monkeypatch, [40], lambda c: True)
    monkeypatch.setattr(gn._lib, "load", lambda: types.SimpleNamespace(tfx_dgn_solve=lambda *a: tried.append(a[5]) or 3))
    with pytest.raises(RuntimeError, match="status 3"):
        b.launch(8, auto=True)
    assert tried == [8]


@pytest.mark.parametrize("c,R,cands", [(8, 40, [8, 12, 16]), (1, 3, [1, 2]), (16, 3, [1]), (3, 3, [3])])
def test_sizes_of_a_given_cluster(c, R, cands):
    assert gn._cluster_candidates(c, R) == cands
