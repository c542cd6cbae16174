"""Batched segments that teams of CTAs work on: every length mix the plan of the
teams has to split the CTAs for (one segment, as many as CTAs, lengths around a
CTA's share, equal and very unequal ones), beside segments of the other classes."""
import numpy as np
import pytest

import ggms_b200 as G
import ggms_oracle as orc
from conftest import to_device

pytestmark = pytest.mark.gpu

SHARE = 1 << 18  # the shortest a team works on is one key more
MIXES = {
    "one": [3_000_001],
    "two around the share": [SHARE, SHARE + 1],
    "as many as CTAs": [SHARE + 1 + i for i in range(147)],
    "more than half the CTAs": [SHARE + 1 + 977 * i for i in range(100)],
    "64": [300_000 + 11_003 * i for i in range(64)],
    "one long, many of a share": [1 << 24] + [SHARE + 5] * 40,
    "beside singles, sorts and rows": [700_001, 5_000_000, 400_003] + [100_000] * 20 + [5000] * 20 + [90] * 50,
}


@pytest.mark.parametrize("dtype", [np.float32, np.uint32])
@pytest.mark.parametrize("mix", MIXES)
def test_teams(ctx, mix, dtype):
    import torch
    g = np.random.default_rng(11)
    lens = g.permutation(np.array(MIXES[mix]))
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    if dtype is np.float32:
        v = g.standard_normal(off[-1], dtype=np.float32)
    else:
        v = g.integers(0, 1 << 32, off[-1], dtype=np.uint32)
    per = 7
    ks = np.concatenate([np.concatenate([[1, n], g.integers(1, n + 1, per - 2)]) for n in lens]).astype(np.uint32)
    k_off = (np.arange(len(lens) + 1) * per).astype(np.int64)
    dv, dk, do, dko = to_device(v), to_device(ks), to_device(off), to_device(k_off)
    out = torch.empty(len(ks), dtype=torch.float32 if dtype is np.float32 else torch.int32, device="cuda")
    assert G.segmented(ctx, dv.data_ptr(), do.data_ptr(), len(lens), dk.data_ptr(), dko.data_ptr(), out.data_ptr(),
                       dtype) == 0
    assert ctx.status() == 0
    got = out.cpu().numpy().view(np.uint32)
    for s, (a, b) in enumerate(zip(off[:-1], off[1:])):
        srt = np.sort(v[a:b])
        k = ks[s * per:(s + 1) * per].astype(np.int64)
        np.testing.assert_array_equal(got[s * per:(s + 1) * per], srt[(b - a) - k].view(np.uint32), err_msg=str(s))
