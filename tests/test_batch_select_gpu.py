"""Batched segments of one CTA's sort with few ks, which are selected one by one:
lengths at the edges of the class and of the threads, one to six ks (both sides
of the rule), ties, both ends of the key range."""
import numpy as np
import pytest

import ggms_b200 as G
import ggms_oracle as orc
from conftest import to_device

pytestmark = pytest.mark.gpu

LENS = [257, 300, 1023, 1024, 1025, 2047, 2049, 3000, 4096, 7169, 8191, 8192]


def raw(u):
    return np.asarray(u).astype(np.uint32)


DATA = {
    "normal": lambda g, n: g.standard_normal(n).astype(np.float32).view(np.uint32),
    "16 bits": lambda g, n: g.standard_normal(n).astype(np.float16).astype(np.float32).view(np.uint32),
    "equal": lambda g, n: raw(np.full(n, 0x3F800000)),
    "ends": lambda g, n: raw(g.choice([0, 0x7FFFFFFF, 0x80000000, 0xFFFFFFFF, 0x7F800000], n)),
    "all bits": lambda g, n: raw(g.integers(0, 1 << 32, n)),
    "dense and far": lambda g, n: raw(np.where(g.random(n) < 0.9, g.integers(1000, 1100, n), g.integers(0, 1 << 32, n))),
}


@pytest.mark.parametrize("dtype", [np.float32, np.uint32])
@pytest.mark.parametrize("data", DATA)
def test_few_ks(ctx, data, dtype):
    import torch
    g = np.random.default_rng(5)
    lens = np.repeat(LENS, 6)
    nks = np.tile(np.arange(1, 7), len(LENS))
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    k_off = np.concatenate([[0], np.cumsum(nks)]).astype(np.int64)
    v = np.concatenate([DATA[data](g, n) for n in lens]).view(dtype)
    ks = np.concatenate([np.where(g.random(k) < 0.3, g.choice([1, n], k), g.integers(1, n + 1, k))
                         for n, k in zip(lens, nks)]).astype(np.uint32)
    dv, dk, do, dko = to_device(v), to_device(ks), to_device(off), to_device(k_off)
    out = torch.empty(len(ks), dtype=torch.float32 if dtype is np.float32 else torch.int32, device="cuda")

    def call():
        return G.segmented(ctx, dv.data_ptr(), do.data_ptr(), len(lens), dk.data_ptr(), dko.data_ptr(),
                           out.data_ptr(), dtype)
    assert call() == 0 and ctx.status() == 0
    exp = orc.select_segmented(v, off, ks, k_off)
    np.testing.assert_array_equal(orc.bits(out.cpu().numpy().view(dtype)), orc.bits(exp))
    bad = int(k_off[6 * LENS.index(3000) + 1])  # the first k of a segment with two
    dk[bad] = 0
    assert call() == 0 and ctx.status() == G.GGMS_E_INVALID_ARG
    got = orc.bits(out.cpu().numpy().view(dtype))
    keep = np.arange(len(ks)) != bad
    np.testing.assert_array_equal(got[keep], orc.bits(exp)[keep])
