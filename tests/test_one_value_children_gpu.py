"""Large children of one value (floats of 16-bit precision, a value that half of
the vector has), beside large children of several values, for one CTA, a team
and the whole grid: the first answer their ks at once, the levels refine the
others."""
import numpy as np
import pytest

import ggms_b200 as G
import ggms_oracle as orc
from conftest import to_device

pytestmark = pytest.mark.gpu


def half(g, n, a, b):
    return np.where(g.random(n) < 0.5, a, b)


def bits(u, dtype):
    return np.asarray(u).astype({4: np.uint32, 8: np.uint64}[np.dtype(dtype).itemsize]).view(dtype)


def f16(g, n):
    return g.standard_normal(n).astype(np.float16).astype(np.float32)


# heavy: values that half of the keys share, next to values that no bucket has for itself
DATA = {
    "f32 of 16 bits": (np.float32, f16),
    "f32 of 16 bits, half dense": (np.float32, lambda g, n: half(g, n, f16(g, n), 1 + 1e-6 * g.standard_normal(n))),
    "f32 largest key": (np.float32, lambda g, n: half(g, n, bits(np.full(n, 0x7FFFFFFF), np.float32), 1e30 * g.standard_normal(n))),
    "f32 smallest key": (np.float32, lambda g, n: half(g, n, bits(np.full(n, 0xFFFFFFFF), np.float32), 1e30 * g.standard_normal(n))),
    "u32 both ends": (np.uint32, lambda g, n: half(g, n, half(g, n, 0, 0xFFFFFFFF), g.integers(0, 1 << 32, n))),
    "f64 of 16 bits": (np.float64, lambda g, n: f16(g, n)),
    "f64 heavy": (np.float64, lambda g, n: half(g, n, 0.1, g.standard_normal(n))),
}


@pytest.mark.parametrize("n", [40_000, 300_001, (1 << 23) + 3])
@pytest.mark.parametrize("data", DATA)
def test_one_vector(ctx, data, n):
    dtype, make = DATA[data]
    g = np.random.default_rng(n)
    v = make(g, n).astype(dtype)
    d = to_device(v)
    for nk in (1, 300, 2500):
        ks = g.integers(1, n + 1, nk).astype(np.uint32)
        got = G.select(ctx, d.data_ptr(), n, ks, dtype)
        np.testing.assert_array_equal(orc.bits(got), orc.bits(orc.select(v, ks)))


@pytest.mark.parametrize("data", [d for d in DATA if not d.startswith("f64")])
def test_batched(ctx, data):
    import torch
    dtype, make = DATA[data]
    g = np.random.default_rng(13)
    lens = np.array([2_000_003, 700_003, 262_145, 262_144, 50_000, 20_000])  # teams and single CTAs
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    v = np.concatenate([make(g, n) for n in lens]).astype(dtype)
    ks = np.concatenate([g.integers(1, n + 1, 200) for n in lens]).astype(np.uint32)
    k_off = (np.arange(len(lens) + 1) * 200).astype(np.int64)
    dv, dk, do, dko = to_device(v), to_device(ks), to_device(off), to_device(k_off)
    out = torch.empty(len(ks), dtype=torch.float32 if dtype is np.float32 else torch.int32, device="cuda")
    assert G.segmented(ctx, dv.data_ptr(), do.data_ptr(), len(lens), dk.data_ptr(), dko.data_ptr(), out.data_ptr(),
                       dtype) == 0
    assert ctx.status() == 0
    np.testing.assert_array_equal(orc.bits(out.cpu().numpy().view(dtype)), orc.bits(orc.select_segmented(v, off, ks, k_off)))
