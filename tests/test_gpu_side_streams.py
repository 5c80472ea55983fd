"""aosb_stream_release gives back the side streams of a caller's stream, after
which the stream can be used again with the same results (bit for bit): the FP32
factorization's (its updates are long enough here to run the diagonal LU beside
them), the tensor-core factorization's and the solve lookahead's."""

from __future__ import annotations

import numpy as np
import pytest

import bundles
from test_gpu_parity import _factor_solve, _pencil_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile,precision,flags,sides", [(64, 0, 0, 1), (128, 1, 1, 1),
                                                        (128, 1, 1 | 4, 2)])
def test_release_and_use_again(tile, precision, flags, sides):
    import torch

    from aospectrum_b200 import native

    lib = native.library()
    dev, plan, h, s = _pencil_case(bundles.c1(), bundles.KPOINTS[1], torch, tile, "natural")
    rng = np.random.default_rng(6)
    rhs = rng.standard_normal((dev.n, 5)) + 1j * rng.standard_normal((dev.n, 5))
    shifts = np.linspace(-2.5, 0.0, 12) + 0.2j
    lookahead = lib.aosb_solve_set_lookahead(1)
    stream = torch.cuda.Stream()
    try:
        torch.cuda.synchronize()
        lib.aosb_stream_release(stream.cuda_stream)   # handles come from a pool
        got = []
        for _ in range(2):
            with torch.cuda.stream(stream):
                got.append(_factor_solve(dev, plan, h, s, shifts, rhs, torch, precision=precision,
                                         flags=flags))
            assert lib.aosb_stream_release(stream.cuda_stream) == sides
            assert lib.aosb_stream_release(stream.cuda_stream) == 0
        assert np.array_equal(got[0], got[1])
    finally:
        lib.aosb_solve_set_lookahead(lookahead)
        dev.close()
        plan.close()
