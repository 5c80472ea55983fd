"""Bounded waits of the cluster solve, made to run out on purpose.

The factorization runs with the default limit; only aosb_solve is launched with
a limit of one poll, so the waits for factor tiles and for the cluster's other
CTAs give up within microseconds, in whatever lanes they do.  Every CTA must
leave its loops, drain its copies and meet its cluster: aosb_solve_check reports
AOSB_ERR_TIMEOUT (52), and with the default limit the same solve on the same
context gives the bits it gave before.  Nothing here faults, traps or hangs the
GPU."""

from __future__ import annotations

import numpy as np
import pytest

import bundles
from test_gpu_parity import _factor_solve, _pencil_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("adjoint", [0, 1])
@pytest.mark.parametrize("pencils,columns", [(1, 8), (12, 17), (40, 32)])
def test_cluster_solve_reports_timeout_and_context_survives(pencils, columns, adjoint,
                                                           monkeypatch):
    import torch

    from aospectrum_b200 import native
    from aospectrum_b200.errors import SolverError

    lib = native.library()
    dev, plan, h, s = _pencil_case(bundles.c1(), bundles.KPOINTS[1], torch, 128)
    call = native.call

    def hasty(name, *args):
        if name != "aosb_solve":
            return call(name, *args)
        before = lib.aosb_tc_set_wait_limit(1)
        try:
            return call(name, *args)
        finally:
            lib.aosb_tc_set_wait_limit(before)

    try:
        rng = np.random.default_rng(3)
        rhs = rng.standard_normal((dev.n, columns)) + 1j * rng.standard_normal((dev.n, columns))
        shifts = np.linspace(-2.6, 0.5, pencils) + 1j * np.linspace(0.05, 0.6, pencils)
        kw = dict(precision=native.PRECISION_BF16X3, adjoint=adjoint,
                  flags=native.SOLVE_TENSOR_CORES)
        ref = _factor_solve(dev, plan, h, s, shifts, rhs, torch, **kw)
        monkeypatch.setattr(native, "call", hasty)
        with pytest.raises(SolverError, match="status 52"):
            _factor_solve(dev, plan, h, s, shifts, rhs, torch, **kw)
        monkeypatch.undo()
        torch.cuda.synchronize()
        got = _factor_solve(dev, plan, h, s, shifts, rhs, torch, **kw)
        assert np.array_equal(got, ref)
    finally:
        dev.close()
        plan.close()
