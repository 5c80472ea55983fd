"""aosb_dense_mul on more columns than one launch covers (65535 blocks of 32)."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_fp64_blocks import _complex, _device, _stream, _within

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("columns", [65535 * 32, 65535 * 32 + 1, 2 * 65535 * 32 + 9])
def test_more_columns_than_a_launch(columns):
    import torch

    from aospectrum_b200 import native

    rng = np.random.default_rng(1)
    x, t = _complex(rng, 2, 3), _complex(rng, 3, columns)
    xd, td = _device(x), _device(t)
    y = torch.zeros((2, columns), dtype=torch.complex128, device="cuda")
    native.call("aosb_dense_mul", 2, 3, columns, xd.data_ptr(), 3, td.data_ptr(), y.data_ptr(),
                columns, _stream())
    _within(y.cpu().numpy(), x @ t, np.abs(x) @ np.abs(t), 3)
