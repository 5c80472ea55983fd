"""The one-thread LAPACK context used by several threads at once.

An OpenMP limit belongs to the thread that sets it, a BLAS pool's limit to the
process; whatever the order in which threads enter and leave, each must find
both as they were."""

from __future__ import annotations

import threading

import numpy as np
import scipy.linalg  # noqa: F401  (loads its own BLAS)
import pytest
from threadpoolctl import threadpool_info, threadpool_limits


def _threads(api):
    return {m["filepath"]: m["num_threads"] for m in threadpool_info() if m["user_api"] == api}


def _together(body):
    """Runs body(step) in two threads; step(name) waits for the other's turn."""
    order = ["a in", "b in", "a out", "b out"]
    done = {name: threading.Event() for name in order}
    failed = []

    def step(name):
        at = order.index(name)
        if at:
            assert done[order[at - 1]].wait(30)

    def run(who):
        try:
            body(who, step, done)
        except BaseException as exc:  # noqa: BLE001
            failed.append(exc)
            for e in done.values():
                e.set()

    threads = [threading.Thread(target=run, args=(w,)) for w in "ab"]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    if failed:
        raise failed[0]


def test_overlapping_users_restore_their_own_limits():
    import torch

    from aospectrum_b200.ciss import small_lapack

    np.linalg.eigh(np.eye(4))
    blas = _threads("blas")
    assert blas
    inside, after = {}, {}

    def body(who, step, done):
        torch.set_num_threads(3 if who == "a" else 2)
        mine = _threads("openmp")
        context = small_lapack()
        step(f"{who} in")
        context.__enter__()
        inside[who] = (set(_threads("blas").values()), set(_threads("openmp").values()))
        done[f"{who} in"].set()
        step(f"{who} out")
        context.__exit__(None, None, None)
        after[who] = (mine, _threads("openmp"))
        done[f"{who} out"].set()

    _together(body)
    for who in "ab":
        assert inside[who] == ({1}, {1})
        assert after[who][0] == after[who][1]
    assert _threads("blas") == blas


def test_limits_that_changed_between_two_uses_are_kept():
    from aospectrum_b200.ciss import small_lapack

    with small_lapack():
        pass
    with threadpool_limits(limits=2):
        before = _threads("blas"), _threads("openmp")
        with small_lapack():
            assert set(_threads("blas").values()) == {1}
        assert (_threads("blas"), _threads("openmp")) == before


def test_nested_use_restores_the_limits():
    from aospectrum_b200.ciss import small_lapack

    before = _threads("blas"), _threads("openmp")
    with small_lapack():
        with small_lapack():
            assert set(_threads("blas").values()) == {1}
        assert set(_threads("blas").values()) == {1}
        assert set(_threads("openmp").values()) <= {1}
    assert (_threads("blas"), _threads("openmp")) == before


@pytest.mark.parametrize("width,items,one", [(0, 1, True), (512, 1, True), (513, 1, False),
                                             (1024, 1, False), (1024, 2, True)])
def test_a_single_wide_problem_keeps_the_blas_pool(width, items, one):
    from aospectrum_b200.engine import BandEngine

    eng = BandEngine.__new__(BandEngine)   # host part only: no device state
    eng._lapack_pool = None
    with threadpool_limits(limits=4, user_api="blas"):
        pool = _threads("blas")
        got = eng._host_map(lambda _: _threads("blas"), list(range(items)), width)
    assert got == [dict.fromkeys(pool, 1) if one else pool] * items
    if eng._lapack_pool is not None:
        eng._lapack_pool.shutdown()
