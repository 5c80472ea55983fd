"""Launch-per-step form of the tensor-core solves (AOSB_SOLVE_PER_STEP).

Batches that the clusters serve never reach it by themselves, so its own
variants are compared here: lookahead, CTAs per SM and graph replay do the same
arithmetic in the same order (one reduce-add per X tile and step) and must give
the same bits.  Against the cluster form and the FP32 sweeps on the same factors
it is held to the 1e-3 of unrefined split-BF16 solves: the updates drop lo x lo
and round lo, 2^-16 relative per product, which the pencil's condition
amplifies.  Column counts: one, ragged strips, two strips."""

from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest

import bundles
from test_gpu_parity import _factor_solve, _pencil_case

pytestmark = pytest.mark.gpu


def _cubic6():
    from aospectrum_b200 import synth

    return synth.generate_bundle(replace(synth.SPEC_C2, name="cubic6", grid=(6, 6, 6),
                                         cell=(14.4, 14.4, 14.4), seed=17))


@pytest.mark.parametrize("case", ["c1", "cubic6"])
@pytest.mark.parametrize("adjoint", [0, 1])
@pytest.mark.parametrize("columns", [1, 17, 32, 40])
def test_variants_agree(case, adjoint, columns):
    import torch

    from aospectrum_b200 import native

    torch.cuda.set_device(0)
    lib = native.library()
    b = bundles.c1() if case == "c1" else _cubic6()
    dev, plan, h, s = _pencil_case(b, bundles.KPOINTS[2], torch, 128, "natural")
    rng = np.random.default_rng(columns)
    rhs = rng.standard_normal((dev.n, columns)) + 1j * rng.standard_normal((dev.n, columns))
    shifts = [-2.5 + 0.03j, -1.2 + 0.4j, 0.3 + 0.01j]

    def solve(flags):
        return _factor_solve(dev, plan, h, s, shifts, rhs, torch, adjoint=adjoint, flags=flags,
                             precision=native.PRECISION_BF16X3)

    steps = native.SOLVE_TENSOR_CORES | native.SOLVE_PER_STEP
    lookahead = lib.aosb_solve_set_lookahead(0)
    try:
        lib.aosb_solve_set_ctas_per_sm(1)
        one = solve(steps)
        lib.aosb_solve_set_ctas_per_sm(2)
        two = solve(steps)
        lib.aosb_solve_set_ctas_per_sm(0)
        lib.aosb_solve_set_lookahead(1)
        ahead = solve(steps)
        graph = solve(steps | native.SOLVE_GRAPH)
        again = solve(steps | native.SOLVE_GRAPH)
        simt = solve(0)
        cluster = solve(native.SOLVE_TENSOR_CORES)
    finally:
        lib.aosb_solve_set_lookahead(lookahead)
        lib.aosb_solve_set_ctas_per_sm(0)
        dev.close()
        plan.close()
    for same in (two, ahead, graph, again):
        assert np.array_equal(same, one)
    # the automatic form is another one here, or this test compares nothing
    assert not np.array_equal(cluster, one)
    for other in (simt, cluster):
        for p in range(len(shifts)):
            err = np.linalg.norm(one[p] - other[p]) / np.linalg.norm(other[p])
            assert err < 1e-3, (p, err)


def test_the_rule_gives_a_large_batch_to_this_form():
    """108 units on 75 steps, where it is 7 % ahead of the clusters: 18 pencils,
    six strips of which the last one is ragged."""
    import torch

    from aospectrum_b200 import native, synth

    torch.cuda.set_device(0)
    b = synth.generate_bundle(replace(synth.SPEC_C2, name="cubic9", grid=(9, 9, 9),
                                      cell=(21.6, 21.6, 21.6), seed=17))
    dev, plan, h, s = _pencil_case(b, bundles.KPOINTS[2], torch, 128, "natural")
    try:
        assert plan.info.n_tiles == 75
        rng = np.random.default_rng(5)
        rhs = rng.standard_normal((dev.n, 190)) + 1j * rng.standard_normal((dev.n, 190))
        shifts = np.linspace(-2.6, 0.5, 18) + 0.3j
        auto, steps = (_factor_solve(dev, plan, h, s, shifts, rhs, torch, flags=flags,
                                     precision=native.PRECISION_BF16X3)
                       for flags in (native.SOLVE_TENSOR_CORES,
                                     native.SOLVE_TENSOR_CORES | native.SOLVE_PER_STEP))
        assert np.array_equal(auto, steps)
    finally:
        dev.close()
        plan.close()
