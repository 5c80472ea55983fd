"""FP32 sweeps with programmatic launches against the word-wise kernels, which
serve the same factors when their storage starts off a 16-byte boundary (every
tile size, both directions, column counts at the edges of the strips of 32 and
odd ones, 8-byte accesses); and FP32 factorizations whose diagonal steps run
beside the updates.

Both add the same products in FP32 in another order: 2^-24 times the pencils'
condition, which at 0.05 eV and more from the real axis is below 10^3 (the
unrefined solves are good to 1e-4): 10^-4."""

from __future__ import annotations

import numpy as np
import pytest

import bundles
from test_gpu_parity import _pencil_case

pytestmark = pytest.mark.gpu


def _factor(plan, h, s, shifts, torch):
    from aospectrum_b200 import native

    P = len(shifts)
    factor = torch.empty(native.library().aosb_factor_bytes(plan.handle, P) // 4,
                         dtype=torch.float32, device="cuda")
    pivots = torch.empty((P, plan.info.n_pad), dtype=torch.int32, device="cuda")
    status = torch.zeros(P, dtype=torch.int32, device="cuda")
    row = torch.zeros(P, dtype=torch.int32, device="cuda")
    z = torch.tensor(np.asarray(shifts, np.complex128), device="cuda")
    fa = native.FactorArgs(native.ABI_VERSION, native.C.sizeof(native.FactorArgs), P,
                           native.PRECISION_PLAIN, h.data_ptr(), s.data_ptr(), row.data_ptr(),
                           z.data_ptr(), factor.data_ptr(), pivots.data_ptr(), status.data_ptr(),
                           None, torch.cuda.current_stream().cuda_stream)
    native.call("aosb_factor", plan.handle, native.C.byref(fa))
    torch.cuda.synchronize()
    assert status.abs().max().item() == 0
    return factor, pivots


def _solve(plan, factor, pivots, rhs, adjoint, torch):
    from aospectrum_b200 import native

    P, n_pad, L = rhs.shape
    lib = native.library()
    work = rhs.clone()
    scratch = torch.empty(max(16, lib.aosb_solve_scratch_bytes(plan.handle, P, L)),
                          dtype=torch.uint8, device="cuda")
    sa = native.SolveArgs(native.ABI_VERSION, native.C.sizeof(native.SolveArgs), P, L, adjoint, 0,
                          factor.data_ptr(), pivots.data_ptr(), work.data_ptr(),
                          scratch.data_ptr(), torch.cuda.current_stream().cuda_stream)
    native.call("aosb_solve", plan.handle, native.C.byref(sa))
    torch.cuda.synchronize()
    return work


@pytest.mark.parametrize("adjoint", [0, 1])
@pytest.mark.parametrize("tile", [32, 64, 128])
@pytest.mark.parametrize("pencils,columns", [(1, 1), (3, 2), (2, 15), (5, 32), (2, 33), (1, 63),
                                             (3, 64)])
def test_row_block_sweeps_match_word_wise_kernels(pencils, columns, tile, adjoint):
    import torch

    dev, plan, h, s = _pencil_case(bundles.small2d(), bundles.KPOINTS[1], torch, tile)
    try:
        z = np.linspace(-2.6, 0.5, pencils) + 1j * np.linspace(0.05, 0.6, pencils)
        factor, pivots = _factor(plan, h, s, z, torch)
        shifted = torch.empty(factor.numel() + 1, dtype=torch.float32, device="cuda")[1:]
        shifted.copy_(factor)
        assert factor.data_ptr() % 16 == 0 and shifted.data_ptr() % 16 == 4
        gen = torch.Generator(device="cuda").manual_seed(columns)
        rhs = torch.randn((pencils, plan.info.n_pad, columns), dtype=torch.complex64,
                          device="cuda", generator=gen)
        got = _solve(plan, factor, pivots, rhs, adjoint, torch)
        ref = _solve(plan, shifted, pivots, rhs, adjoint, torch)
        for p in range(pencils):
            err = (torch.linalg.vector_norm(got[p] - ref[p])
                   / torch.linalg.vector_norm(ref[p])).item()
            assert err < 1e-4, (p, err)
    finally:
        dev.close()
        plan.close()


@pytest.mark.parametrize("tile,pencils", [(32, 8), (64, 4), (128, 12)])
def test_diagonal_steps_beside_the_updates_change_nothing(tile, pencils):
    """A batch large enough for the side stream gives each pencil the bits of a
    single pencil, whose updates are too small for it."""
    import torch

    bundle = bundles.small2d() if tile == 32 else bundles.c1()
    dev, plan, h, s = _pencil_case(bundle, bundles.KPOINTS[1], torch, tile, "natural")
    try:
        z = np.linspace(-2.6, 0.5, pencils) + 1j * np.linspace(0.05, 0.6, pencils)
        blocks = (plan.info.n_tiles - 1) ** 2 * (4 if tile == 128 else 1)
        assert blocks < 300 <= blocks * pencils
        factor, pivots = _factor(plan, h, s, z, torch)
        each = factor.numel() // pencils
        for p in range(pencils):
            one, piv = _factor(plan, h, s, z[p:p + 1], torch)
            assert torch.equal(factor[p * each:(p + 1) * each], one), p
            assert torch.equal(pivots[p], piv[0]), p
    finally:
        dev.close()
        plan.close()
