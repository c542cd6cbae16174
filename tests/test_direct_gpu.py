"""The one-launch path (calls that leave everything to the library, on vectors
that fit the L2 cache): bit-exact against the CPU oracle at the sizes where its
parts change -- one CTA's sort (32 KB of keys), one or more CTAs, the bucket
counts, the focus on clustered ks, ks located per CTA (over 2048) -- for every
type, with duplicates, special values, sorted and unaligned input.  The answers
are elements of the input, so the tolerance is none."""
import numpy as np
import pytest

import ggms_b200 as G
import ggms_oracle as orc
from ggms_b200 import datagen as D
from conftest import to_device

pytestmark = pytest.mark.gpu

DTYPES = [np.float32, np.float64, np.uint32, np.int32]


def values(kind, dtype, n, seed):
    g = np.random.default_rng(seed)
    fp = np.dtype(dtype).kind == "f"
    if kind == "random":
        if fp:
            return g.standard_normal(n).astype(dtype)
        return g.integers(np.iinfo(dtype).min, np.iinfo(dtype).max, n, dtype=dtype, endpoint=True)
    if kind == "narrow":  # a range far below the type's, with one outlier at each end
        v = (1000 + g.integers(0, 500, n)).astype(dtype)
        v[g.integers(0, n)] = 1 << 30
        v[g.integers(0, n)] = 0
        return v
    if kind == "atoms":  # a few values hold almost everything: refinement levels
        v = np.where(g.random(n) < 0.9, 7, 3).astype(dtype)
        v[g.integers(0, n, 100)] = g.integers(0, 1 << 20, 100).astype(dtype)
        return v
    if kind == "sorted":
        return np.sort(values("random", dtype, n, seed))
    if kind == "equal":
        return np.full(n, 5, dtype)
    v = values("random", dtype, n, seed)  # specials
    if fp:
        u = np.uint32 if dtype == np.float32 else np.uint64
        b = np.dtype(dtype).itemsize * 8
        inf = 0x7F800000 if b == 32 else 0x7FF0000000000000
        sign = 1 << (b - 1)
        s = np.array([inf, inf | sign, 0, sign, 1, 1 | sign, inf | 1, inf | 1 | sign, sign - 1, 2 * sign - 1],
                     dtype=u).view(dtype)
    else:
        s = np.array([np.iinfo(dtype).min, np.iinfo(dtype).max, 0], dtype)
    v[g.integers(0, n, max(4, n // 50))] = s[g.integers(0, len(s), max(4, n // 50))]
    return v


def ks_of(n, nk, seed, clustered=False):
    g = np.random.default_rng(seed)
    ks = g.integers(1, (max(2, n // 100) if clustered else n) + 1, nk).astype(np.uint32)
    ks[0] = 1
    ks[-1] = n
    return ks


def check(ctx, v, ks, ptr=None, d=None):
    d = to_device(v) if d is None else d
    got = G.select(ctx, d.data_ptr() if ptr is None else ptr, len(v), ks, v.dtype)
    np.testing.assert_array_equal(orc.bits(got), orc.bits(orc.select(v, ks)))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n", [2, 1023, 1025, 4095, 4096, 4097, 8191, 8192, 8193, 65537, (1 << 18) - 1, (1 << 18) + 3])
def test_direct_sizes(ctx, dtype, n):
    v = values("random", dtype, n, n)
    check(ctx, v, ks_of(n, 41, n))
    check(ctx, v, ks_of(n, 41, n, clustered=True))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("kind", ["narrow", "atoms", "sorted", "equal", "specials"])
@pytest.mark.parametrize("n", [4001, 70_001, (1 << 20) + 5])
def test_direct_distributions(ctx, dtype, kind, n):
    v = values(kind, dtype, n, 7)
    check(ctx, v, ks_of(n, 301, 8))
    check(ctx, v, ks_of(n, 64, 9, clustered=True))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("nk", [1, 15, 16, 2048, 2049, 20_000])
def test_direct_k_counts(ctx, dtype, nk):
    n = 600_011
    v = values("random", dtype, n, nk)
    ks = np.full(nk, n // 3, np.uint32) if nk == 15 else ks_of(n, nk, nk)  # 15: one k many times
    check(ctx, v, ks)


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.uint32])
def test_direct_wide_buckets(ctx, dtype):
    """2^23 keys and more get 16384 buckets; duplicates there need the levels."""
    n = (1 << 23) + 9
    for kind in ("random", "atoms"):
        v = values(kind, dtype, n, 3)
        ks = np.concatenate([ks_of(n, 700, 4), ks_of(n, 300, 5, clustered=True)])
        got = G.select(ctx, to_device(v).data_ptr(), n, ks, dtype)
        np.testing.assert_array_equal(orc.bits(got), orc.bits(orc.cpu_multiselect(v, ks)))


@pytest.mark.parametrize("off", [1, 2, 3])
def test_direct_unaligned(ctx, off):
    v = values("random", np.float32, 50_003 + off, 11)
    d = to_device(v)
    check(ctx, v[off:], ks_of(50_003, 33, off), ptr=d.data_ptr() + 4 * off, d=d)


@pytest.mark.parametrize("n", [3000, 300_000])
def test_direct_invalid_device_k(n):
    """A device-resident k outside [1, n] is reported; the other ks are answered."""
    import torch
    ctx = G.Context(0)
    v = values("random", np.float32, n, 1)
    ks = np.array([5, 0, n + 1, n], np.uint32)
    d, dk = to_device(v), to_device(ks)
    out = torch.empty(4, dtype=torch.float32, device="cuda")
    o = G.default_opts(ks_on_device=1, out_on_device=1)
    for _ in range(3):
        assert G.multiselect_ex(ctx, d.data_ptr(), n, dk.data_ptr(), 4, out.data_ptr(), np.float32, o) == G.GGMS_OK
        assert ctx.status() == G.GGMS_E_INVALID_ARG
        got = out.cpu().numpy()[[0, 3]]
        np.testing.assert_array_equal(orc.bits(got), orc.bits(orc.select(v, ks[[0, 3]])))
    ctx.close()


def test_direct_call_inside_a_caller_graph():
    """The launch can be captured into the caller's CUDA graph (a first call of
    its key; the workspace is there already) and replays on new data."""
    import torch
    ctx = G.Context(0)
    n = 200_003
    ks = ks_of(n, 100, 3)
    dk = to_device(ks)
    d = to_device(values("random", np.float32, n, 1))
    warm = torch.empty(len(ks), dtype=torch.float32, device="cuda")
    out = torch.empty(len(ks), dtype=torch.float32, device="cuda")
    o = G.default_opts(ks_on_device=1, out_on_device=1)
    assert G.multiselect_ex(ctx, d.data_ptr(), n, dk.data_ptr(), len(ks), warm.data_ptr(), np.float32, o) == 0
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        s = torch.cuda.current_stream().cuda_stream
        rc = G.multiselect_ex(ctx, d.data_ptr(), n, dk.data_ptr(), len(ks), out.data_ptr(), np.float32, o, s)
    assert rc == 0
    for seed in (2, 3):
        v = values("random", np.float32, n, seed)
        d.copy_(torch.from_numpy(v))
        g.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(orc.bits(out.cpu().numpy()), orc.bits(orc.select(v, ks)))
    del g
    ctx.close()
