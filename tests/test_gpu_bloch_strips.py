"""Bloch sums of bundles whose strips of windows reach their limits.

Atoms with 1 to 40 orbitals (windows longer than a strip's value space, narrow
ones, several per strip), one or three lattice images per pair, real and
complex values, and k counts around the four-point chunks, against the numpy
restatement of the reference: bit for bit for real values, within 2e-6 for
complex ones, whose products numpy may contract."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import bloch_ref

pytestmark = pytest.mark.gpu


def _bundle(orbitals, images, complex_values, seed):
    from aospectrum_b200.data import (AtomicStructure, LocalizedOperatorBlocks,
                                      LocalizedOperatorBundle, OrbitalBasisLayout)

    rng = np.random.default_rng(seed)
    orbitals = np.asarray(orbitals)
    atoms = orbitals.size
    rows, cols, shifts, hb, sb = [], [], [], [], []

    def add(i, j, r, h, s):
        rows.append(i), cols.append(j), shifts.append(r)
        hb.append(h.reshape(-1)), sb.append(s.reshape(-1))

    def values(i, j):
        v = rng.standard_normal((orbitals[i], orbitals[j]))
        if complex_values:
            v = v + 1j * rng.standard_normal(v.shape)
        return v.astype(np.complex64 if complex_values else np.float32)

    for i in range(atoms):
        for j in range(i, atoms):
            for r in range(images if i != j else 1):
                shift = (r, -r, 0)
                h, s = values(i, j), values(i, j)
                if i == j:
                    h, s = (0.5 * (v + v.conj().T) for v in (h, s))
                    add(i, i, shift, h, s)
                else:
                    add(i, j, shift, h, s)
                    add(j, i, tuple(-x for x in shift), h.conj().T, s.conj().T)
    order = np.lexsort((np.asarray(shifts)[:, 0], cols, rows))
    take = [np.asarray(x, dtype=np.int32)[order] for x in (rows, cols, shifts)]
    shapes = np.stack((orbitals[take[0]], orbitals[take[1]]), axis=1).astype(np.int32)
    offsets = np.concatenate(([0], np.cumsum(shapes.prod(1)))).astype(np.int64)
    owner = np.repeat(np.arange(atoms, dtype=np.int32), orbitals)
    local = np.concatenate([np.arange(o, dtype=np.int32) for o in orbitals])
    structure = AtomicStructure(cell_angstrom=np.diag([9.0, 9.0, 9.0]),
                                positions_angstrom=rng.uniform(0, 9, (atoms, 3)),
                                atomic_numbers=np.full(atoms, 6, dtype=np.int32),
                                periodic=(True, True, False), label="strips")
    basis = OrbitalBasisLayout(n_atoms=atoms, orbital_atom=owner, local_index=local,
                               basis_family="synthetic", basis_identity="strips",
                               orbital_labels=("s",) * int(orbitals.sum()))
    blocks = LocalizedOperatorBlocks(*take, offsets, shapes,
                                     np.concatenate([hb[o] for o in order]),
                                     np.concatenate([sb[o] for o in order]))
    return LocalizedOperatorBundle(structure, basis, blocks, None, {})


@pytest.mark.parametrize("orbitals,images", [([40, 1, 13, 2, 37, 38], 1), ([1] * 19, 1),
                                             ([16] * 9, 1), ([13, 5] * 6, 1), ([13, 5, 40, 3], 3),
                                             ([4], 1)])
@pytest.mark.parametrize("n_k", [1, 4, 6])
@pytest.mark.parametrize("complex_values", [False, True])
def test_strips_match_reference_restatement(orbitals, images, n_k, complex_values):
    import torch

    from aospectrum_b200.engine import BlochDevice

    b = _bundle(orbitals, images, complex_values, 3)
    k = np.random.default_rng(n_k).uniform(-0.5, 0.5, (n_k, 3))
    dev = BlochDevice(b, torch.device("cuda", 0))
    try:
        h, s = (v.cpu().numpy() for v in dev.apply(k))
    finally:
        dev.close()
    pattern = bloch_ref.build_pattern(b)
    for q in range(n_k):
        ref = bloch_ref.bloch_pair(pattern, b, k[q])
        for got, want in zip((h[q], s[q]), ref):
            if complex_values:
                np.testing.assert_allclose(got, want, rtol=0, atol=2e-6 * images)
            else:
                assert np.array_equal(got, want)
