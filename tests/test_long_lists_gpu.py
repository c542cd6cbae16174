"""Many ks in one bin of a refinement level: a warp answers the first ks of the
bin's list one by one and finds the others by a scan.  Bins of up to 64 keys
(ranked by comparison) and of more (sorted); runs of consecutive ranks, so that
every k has an answer of its own, among ks elsewhere.  Bit-exact against a sort."""
import numpy as np
import pytest

import ggms_b200 as G
from conftest import to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk", [63, 64, 65, 700, 20_000])
@pytest.mark.parametrize("lump", [0, 500])
def test_many_ks_in_one_bin(ctx, nk, lump):
    # 1024 buckets of 2^15 keys each take a level; its bins span 2^11 keys and
    # hold 16, and those with a lump of 500 keys within 4 values also hold it
    g = np.random.default_rng(nk)
    n = 1 << 25
    v = g.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    at = g.integers(0, 1 << 32, 300, dtype=np.uint64)
    for j in range(300 if lump else 0):
        v[j * lump:(j + 1) * lump] = np.minimum(at[j] + g.integers(0, 4, lump).astype(np.uint64), 0xFFFFFFFF)
    g.shuffle(v[:1 << 20])
    s = np.sort(v)
    c = n - int(np.searchsorted(s, at[7])) - lump  # ranks from the largest down, through the lump's bin
    run = np.clip(c + np.arange(nk) % 520, 1, n)
    same = np.full(nk, run[3])
    for ks in (run, same):
        ks = np.concatenate([ks, g.integers(1, n + 1, 50)]).astype(np.uint32)
        got = G.select(ctx, to_device(v).data_ptr(), n, ks, np.uint32, assigner=G.ASSIGNER_SAMPLED, num_buckets=1024)
        np.testing.assert_array_equal(got, s[n - ks.astype(np.int64)])
