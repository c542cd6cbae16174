"""Vectors with more buckets than keys in some places: a bucket that one key alone
can be in is answered from the map, beside buckets that hold several keys, at
both ends of the key range and for one CTA, a team and the whole grid."""
import numpy as np
import pytest

import ggms_b200 as G
import ggms_oracle as orc
from conftest import to_device

pytestmark = pytest.mark.gpu


def ints(g, n, lo, hi):
    return g.integers(lo, hi, n, endpoint=True)


DATA = {
    "u32 equal": (np.uint32, lambda g, n: np.full(n, 77)),
    "u32 zero": (np.uint32, lambda g, n: np.zeros(n)),
    "u32 ten": (np.uint32, lambda g, n: ints(g, n, 0, 9)),
    "u32 bytes at the top": (np.uint32, lambda g, n: ints(g, n, 0xFFFFFF00, 0xFFFFFFFF)),
    "u32 thousands": (np.uint32, lambda g, n: ints(g, n, 5, 4000)),
    "u32 both ends": (np.uint32, lambda g, n: np.where(g.random(n) < 0.5, ints(g, n, 0, 3), ints(g, n, 0xFFFFFFF0, 0xFFFFFFFF))),
    "u32 a few beyond": (np.uint32, lambda g, n: np.where(g.random(n) < 1e-4, ints(g, n, 0, 0xFFFFFFFF), ints(g, n, 1000, 1600))),
    "i32 around zero": (np.int32, lambda g, n: ints(g, n, -40, 40)),
    "f32 narrow": (np.float32, lambda g, n: 1000 + 0.01 * g.standard_normal(n)),
    "f32 zeros of both signs": (np.float32, lambda g, n: np.where(g.random(n) < 0.5, -0.0, 0.0)),
    "f64 narrow": (np.float64, lambda g, n: 1 + 2.0 ** -52 * ints(g, n, 0, 700)),
    "f64 equal": (np.float64, lambda g, n: np.full(n, -np.inf)),
}


@pytest.mark.parametrize("n", [8193, 100_003, 300_001, (1 << 21) + 5])
@pytest.mark.parametrize("data", DATA)
def test_one_vector(ctx, data, n):
    dtype, make = DATA[data]
    g = np.random.default_rng(n)
    v = make(g, n).astype(dtype)
    d = to_device(v)
    for nk in (1, 40, 3000):  # the focus (16 ks and more), and many ks
        ks = g.integers(1, n + 1, nk).astype(np.uint32)
        ks[:1] = n
        got = G.select(ctx, d.data_ptr(), n, ks, dtype)
        np.testing.assert_array_equal(orc.bits(got), orc.bits(orc.select(v, ks)))
    top = G.topk(ctx, d.data_ptr(), n, 500, dtype)
    np.testing.assert_array_equal(orc.bits(top), orc.bits(orc.select(v, np.arange(1, 501, dtype=np.uint32))))


@pytest.mark.parametrize("data", [d for d in DATA if d.startswith(("u32", "f32"))])
def test_batched(ctx, data):
    import torch
    dtype, make = DATA[data]
    g = np.random.default_rng(13)
    lens = np.array([700_003, 262_145, 262_144, 50_000, 9000, 8193])  # teams and single CTAs
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    v = make(g, off[-1]).astype(dtype)
    ks = np.concatenate([g.integers(1, n + 1, 50) for n in lens]).astype(np.uint32)
    k_off = (np.arange(len(lens) + 1) * 50).astype(np.int64)
    dv, dk, do, dko = to_device(v), to_device(ks), to_device(off), to_device(k_off)
    out = torch.empty(len(ks), dtype=torch.float32 if dtype is np.float32 else torch.int32, device="cuda")
    assert G.segmented(ctx, dv.data_ptr(), do.data_ptr(), len(lens), dk.data_ptr(), dko.data_ptr(), out.data_ptr(),
                       dtype) == 0
    assert ctx.status() == 0
    np.testing.assert_array_equal(orc.bits(out.cpu().numpy().view(dtype)), orc.bits(orc.select_segmented(v, off, ks, k_off)))
