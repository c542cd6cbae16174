"""Batched rows that one warp works on, with ties and dense spots: bins of more
keys than one lane orders, with none, one or many of the row's ks in them."""
import numpy as np
import pytest

import ggms_b200 as G
import ggms_oracle as orc
from conftest import to_device

pytestmark = pytest.mark.gpu

DATA = {
    "half zeros": lambda g, n: np.where(g.random(n) < 0.5, 0.0, g.standard_normal(n)),
    "two neighbours": lambda g, n: np.where(g.random(n) < 0.8, np.where(g.random(n) < 0.5, 7.0, np.nextafter(np.float32(7), np.float32(8))), g.standard_normal(n)),
    "hundredths": lambda g, n: np.round(g.standard_normal(n) * 100) / 100,
    "one heap": lambda g, n: np.where(g.random(n) < 0.01, 1e30, 1.0 + 1e-5 * g.random(n)),
    "equal": lambda g, n: np.full(n, -2.5),
}


@pytest.mark.parametrize("dtype", [np.float32, np.uint32])
@pytest.mark.parametrize("per", [1, 2, 7, 32, 33])
@pytest.mark.parametrize("data", DATA)
def test_rows_with_ties(ctx, data, per, dtype):
    import torch
    g = np.random.default_rng(12)
    lens = np.tile([65, 90, 257, 600, 1023, 1024, 1025, 2047, 2048], 70)  # enough rows for both lengths' kernels
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    v = DATA[data](g, off[-1]).astype(np.float32)
    if dtype is np.uint32:
        v = v.view(np.uint32)
    ks = np.concatenate([g.integers(1, n + 1, per) for n in lens]).astype(np.uint32)
    k_off = (np.arange(len(lens) + 1) * per).astype(np.int64)
    dv, dk, do, dko = to_device(v), to_device(ks), to_device(off), to_device(k_off)
    out = torch.empty(len(ks), dtype=torch.float32 if dtype is np.float32 else torch.int32, device="cuda")
    assert G.segmented(ctx, dv.data_ptr(), do.data_ptr(), len(lens), dk.data_ptr(), dko.data_ptr(), out.data_ptr(),
                       dtype) == 0
    assert ctx.status() == 0
    np.testing.assert_array_equal(orc.bits(out.cpu().numpy().view(dtype)), orc.bits(orc.select_segmented(v, off, ks, k_off)))
