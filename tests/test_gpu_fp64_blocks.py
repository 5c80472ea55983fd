"""FP64 block products on matrix instructions against numpy.

Sizes at the edges of the 8 x 8 x 4 fragments, the 16- and 32-wide tiles, the
512-row Gram chunks and the eight-row matrix blocks, with strided operands.
A complex inner product of length K summed in any order is within 8 K u of its
exact value relative to sum |a| |b| (u = 2^-53)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _stream():
    import torch

    return torch.cuda.current_stream().cuda_stream


def _device(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _complex(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def _within(got, ref, scale, terms):
    assert np.all(np.abs(got - ref) <= 8 * terms * U * scale), np.max(np.abs(got - ref) / scale)


@pytest.mark.parametrize("n,p,q", [(1, 1, 1), (5, 8, 9), (511, 16, 17), (512, 33, 15),
                                   (513, 31, 64), (2049, 128, 40), (13000, 128, 128)])
def test_gram_matches_numpy(n, p, q):
    import torch

    from aospectrum_b200 import native

    rng = np.random.default_rng(n + p)
    x, y = _complex(rng, n, p + 3), _complex(rng, n, q + 1)
    xd, yd = _device(x), _device(y)
    g = torch.empty((p, q), dtype=torch.complex128, device="cuda")
    scratch = torch.empty(max(16, native.library().aosb_gram_scratch_bytes(n, p, q)),
                          dtype=torch.uint8, device="cuda")
    native.call("aosb_gram", n, p, q, xd.data_ptr(), p + 3, yd.data_ptr(), q + 1, g.data_ptr(),
                scratch.data_ptr(), _stream())
    x, y = x[:, :p], y[:, :q]
    _within(g.cpu().numpy(), x.conj().T @ y, np.abs(x).T @ np.abs(y), n)


@pytest.mark.parametrize("n,p,r", [(1, 1, 1), (15, 3, 9), (64, 4, 32), (65, 5, 33), (130, 31, 8),
                                   (1715, 96, 53), (13000, 128, 104)])
def test_dense_mul_matches_numpy(n, p, r):
    import torch

    from aospectrum_b200 import native

    rng = np.random.default_rng(n + r)
    x, t = _complex(rng, n, p + 2), _complex(rng, p, r)
    xd, td = _device(x), _device(t)
    y = torch.zeros((n, r + 1), dtype=torch.complex128, device="cuda")
    native.call("aosb_dense_mul", n, p, r, xd.data_ptr(), p + 2, td.data_ptr(), y.data_ptr(), r + 1,
                _stream())
    y = y.cpu().numpy()
    x = x[:, :p]
    _within(y[:, :r], x @ t, np.abs(x) @ np.abs(t), p)
    assert np.all(y[:, r] == 0)


@pytest.mark.parametrize("n,m", [(1, 1), (31, 7), (256, 8), (257, 9), (4459, 33), (13000, 104)])
def test_column_norms_match_numpy(n, m):
    import torch

    from aospectrum_b200 import native

    rng = np.random.default_rng(n + m)
    a, b, e = _complex(rng, n, m + 1), _complex(rng, n, m + 1), rng.standard_normal(m)
    ad, bd, ed = _device(a), _device(b), _device(e)
    out = torch.empty(m, dtype=torch.float64, device="cuda")
    native.call("aosb_column_norms", n, m, ad.data_ptr(), bd.data_ptr(), m + 1, ed.data_ptr(),
                out.data_ptr(), _stream())
    ref = np.linalg.norm(a[:, :m] - e * b[:, :m], axis=0)
    _within(out.cpu().numpy(), ref, ref + np.linalg.norm(e * b[:, :m], axis=0), n)


@pytest.mark.parametrize("rows,blocks,ncols", [(5, 7, 1), (5, 11, 33), (8, 5, 8), (9, 6, 31),
                                               (13, 10, 40), (16, 4, 9)])
@pytest.mark.parametrize("residual", [False, True])
def test_row_block_products_match_numpy(rows, blocks, ncols, residual):
    """Dense-in-blocks patterns (every block couples to a random set of blocks,
    so the nonzero counts are no multiples of four), the last block shorter."""
    import torch

    from aospectrum_b200 import native

    rng = np.random.default_rng(rows * blocks + ncols)
    starts = np.append(np.arange(blocks) * rows, blocks * rows - 2).astype(np.int32)
    n, nb = int(starts[-1]), blocks
    touch = rng.random((nb, nb)) < 0.4
    touch |= np.eye(nb, dtype=bool)
    mask = np.zeros((n, n), dtype=bool)
    for i in range(nb):
        for j in range(nb):
            mask[starts[i]:starts[i + 1], starts[j]:starts[j + 1]] = touch[i, j]
    indptr = np.concatenate(([0], np.cumsum(mask.sum(1)))).astype(np.int64)
    indices = np.nonzero(mask)[1].astype(np.int32)
    h, s = (np.where(mask, _complex(rng, n, n), 0).astype(np.complex64) for _ in range(2))
    args = (n, ncols)
    ip, ix, rb = _device(indptr), _device(indices), _device(starts)
    widest = int(np.diff(starts).max())
    if not residual:
        x = _complex(rng, n, ncols + 2)
        xd, hd = _device(x), _device(h[mask])
        y = torch.zeros((n, ncols + 2), dtype=torch.complex128, device="cuda")
        native.call("aosb_spmm_blocks", *args, nb, rb.data_ptr(), widest, ip.data_ptr(),
                    ix.data_ptr(), hd.data_ptr(), indices.size, xd.data_ptr(), ncols + 2,
                    y.data_ptr(), ncols + 2, _stream())
        y, a, x = y.cpu().numpy(), h.astype(np.complex128), x[:, :ncols]
        _within(y[:, :ncols], a @ x, np.abs(a) @ np.abs(x) + 1e-300, n)
        assert np.all(y[:, ncols:] == 0)
        return
    z = np.asarray([-2.0 + 0.1j, 0.5 + 0.01j, 1.0 - 1.0j])
    x, b = _complex(rng, 3, n, ncols), _complex(rng, 3, n, ncols)
    xd, bd, hd, sd, zd = (_device(v) for v in (x, b, h[mask], s[mask], z))
    pk = torch.zeros(3, dtype=torch.int32, device="cuda")
    r = torch.empty((3, n, ncols), dtype=torch.complex128, device="cuda")
    native.call("aosb_shifted_residual_blocks", *args, 3, nb, rb.data_ptr(), widest, ip.data_ptr(),
                ix.data_ptr(), hd.data_ptr(), sd.data_ptr(), indices.size, pk.data_ptr(),
                zd.data_ptr(), bd.data_ptr(), n * ncols, xd.data_ptr(), r.data_ptr(), _stream())
    r = r.cpu().numpy()
    for q in range(3):
        a = h.astype(np.complex128) - z[q] * s.astype(np.complex128)
        scale = (np.abs(h) + np.abs(z[q]) * np.abs(s)).astype(np.float64) @ np.abs(x[q])
        _within(r[q], b[q] - a @ x[q], scale + np.abs(b[q]), n + 4)
