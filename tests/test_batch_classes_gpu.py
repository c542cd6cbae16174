"""Batched selection where its classes of segments meet: rows (one warp) up to
256, 1024 or 2048 keys by their number, one CTA's sort up to 32 KB of keys, one
CTA or a team beyond.  Every length at, one below and one above an edge, alone
in a batch and among many rows; bit-exact against the CPU oracle (the answers
are elements of the input, so the tolerance is none)."""
import numpy as np
import pytest

import ggms_oracle as orc
from test_segmented_gpu import run_segmented

pytestmark = pytest.mark.gpu

EDGES = [1, 2, 31, 32, 33, 64, 256, 1024, 2048, 4096, 8192]


def batch(lens, dtype, kind, seed):
    g = np.random.default_rng(seed)
    n = int(lens.sum())
    if kind == "dups":
        v = g.integers(0, 9, n).astype(dtype)
    elif np.dtype(dtype).kind == "f":  # both signs, many octaves
        v = (g.standard_normal(n) * np.exp(4 * g.standard_normal(n))).astype(dtype)
        v[::97] = 0.0
        v[::101] = -0.0
        v[::103] = np.inf
    else:
        v = g.integers(0, 1 << 32, n, dtype=np.uint64).astype(dtype)
    nks = g.integers(1, 40, len(lens))
    ks = [np.concatenate([[1, l], g.integers(1, l + 1, c)]).astype(np.uint32) for l, c in zip(lens, nks)]
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    k_off = np.concatenate([[0], np.cumsum([len(k) for k in ks])]).astype(np.int64)
    return v, off, np.concatenate(ks), k_off


@pytest.mark.parametrize("dtype", [np.float32, np.uint32])
@pytest.mark.parametrize("kind", ["wide", "dups"])
@pytest.mark.parametrize("filler", [0, 700, 5000])  # further rows: few or many per SM
@pytest.mark.parametrize("long", [0, (1 << 17) + 1, (1 << 19) + 3])
def test_class_edges(ctx, dtype, kind, filler, long):
    lens = [max(1, e + d) for e in EDGES for d in (-1, 0, 1)]
    lens += [200 + i % 800 for i in range(filler)] + ([long, long // 2] if long else [])
    v, off, ks, k_off = batch(np.array(lens, dtype=np.int64), dtype, kind, 7)
    got = run_segmented(ctx, v, off, ks, k_off)
    np.testing.assert_array_equal(orc.bits(got), orc.bits(orc.select_segmented(v, off, ks, k_off)))


@pytest.mark.parametrize("length", [1, 256, 257, 2049, 8193])
def test_one_segment(ctx, length):
    v, off, ks, k_off = batch(np.array([length], dtype=np.int64), np.float32, "wide", 11)
    got = run_segmented(ctx, v, off, ks, k_off)
    np.testing.assert_array_equal(orc.bits(got), orc.bits(orc.select_segmented(v, off, ks, k_off)))
