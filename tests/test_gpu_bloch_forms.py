"""The two kernels of the Bloch sum give the same bits.

Which one sums a bundle depends on its windows and on the number of k points, and
a k point's matrices do not depend on the others summed with it: so the same
points are summed alone and among many, on bundles whose kernel changes in
between, in both directions, and on bundles with a few windows of several lattice
images among strips.  The small ones are also held against the numpy restatement
of the reference (bit for bit for real values, 2e-6 per image for complex ones,
whose products numpy may contract)."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import bloch_ref
from test_gpu_bloch_strips import _bundle

pytestmark = pytest.mark.gpu


def _cube(side, orbitals, complex_values):
    """A periodic cube's topology with the given orbitals (cycled over the atoms)
    and random block values (the sums project them on Hermitian matrices)."""
    from aospectrum_b200 import synth
    from aospectrum_b200.data import (LocalizedOperatorBlocks, LocalizedOperatorBundle,
                                      OrbitalBasisLayout)

    source = synth.generate_bundle(synth.SyntheticSpec(
        name=f"cube{side}", grid=(side,) * 3, spacing=(2.4,) * 3, cell=(2.4 * side,) * 3,
        periodic=(True,) * 3, cutoff=7.0, orbitals_per_atom=5))
    ops, atoms = source.operators, source.basis.n_atoms
    counts = np.resize(np.asarray(orbitals), atoms)
    shapes = np.stack((counts[ops.row_atom], counts[ops.col_atom]), axis=1).astype(np.int32)
    offsets = np.concatenate(([0], np.cumsum(shapes.prod(1)))).astype(np.int64)
    rng = np.random.default_rng(side)
    h, s = (rng.standard_normal(offsets[-1]).astype(np.float32) for _ in range(2))
    if complex_values:
        h, s = (v + 1j * rng.standard_normal(offsets[-1]).astype(np.float32) for v in (h, s))
        h, s = h.astype(np.complex64), s.astype(np.complex64)
    basis = OrbitalBasisLayout(
        n_atoms=atoms, orbital_atom=np.repeat(np.arange(atoms, dtype=np.int32), counts),
        local_index=np.concatenate([np.arange(c, dtype=np.int32) for c in counts]),
        basis_family="synthetic", basis_identity="forms",
        orbital_labels=("s",) * int(counts.sum()))
    blocks = LocalizedOperatorBlocks(ops.row_atom, ops.col_atom, ops.lattice_shift, offsets, shapes,
                                     h, s)
    return LocalizedOperatorBundle(source.structure, basis, blocks, None, {})


def _sums(dev, k):
    h, s = dev.apply(k)
    return h.cpu().numpy(), s.cpu().numpy()


@pytest.mark.parametrize("side,orbitals", [(5, [5]), (5, [13]), (6, [5]), (6, [1]), (6, [16]),
                                           (6, [4, 13]), (5, [5, 14, 25]), (5, [37, 1, 2])])
@pytest.mark.parametrize("complex_values", [False, True])
def test_a_point_alone_and_among_many(side, orbitals, complex_values):
    import torch

    from aospectrum_b200.engine import BlochDevice

    dev = BlochDevice(_cube(side, orbitals, complex_values), torch.device("cuda", 0))
    try:
        most = min(33, int(2e9 / (16 * dev.nnz)))
        k = np.random.default_rng(1).uniform(-0.5, 0.5, (most, 3))
        many = _sums(dev, k)
        for n in (1, 3, 5, 9, 17):
            if n >= most:
                break
            few = _sums(dev, k[:n])
            for a, b in zip(few, many):
                assert np.array_equal(a, b[:n]), n
    finally:
        dev.close()


@pytest.mark.parametrize("orbitals,images", [([40, 1, 13, 2, 37, 38], 1), ([13] * 20, 1),
                                             ([16] * 12, 1), ([5, 14, 25] * 4, 1), ([41] * 3, 1),
                                             ([1], 1), ([13] * 4, 3)])
@pytest.mark.parametrize("n_k", [1, 5, 33])
@pytest.mark.parametrize("complex_values", [False, True])
def test_small_bundles_match_reference_restatement(orbitals, images, n_k, complex_values):
    import torch

    from aospectrum_b200.engine import BlochDevice

    b = _bundle(orbitals, images, complex_values, 5)
    k = np.random.default_rng(n_k).uniform(-0.5, 0.5, (n_k, 3))
    dev = BlochDevice(b, torch.device("cuda", 0))
    try:
        got = _sums(dev, k)
    finally:
        dev.close()
    pattern = bloch_ref.build_pattern(b)
    for q in (0, n_k // 2, n_k - 1):
        for values, want in zip(got, bloch_ref.bloch_pair(pattern, b, k[q])):
            if complex_values:
                np.testing.assert_allclose(values[q], want, rtol=0, atol=2e-6 * images)
            else:
                assert np.array_equal(values[q], want)
