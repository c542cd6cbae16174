"""Calls on a stream that has 16 of the device's SMs (a green context): the
cooperative launches ask for fewer CTAs there."""
import numpy as np
import pytest

import ggms_b200 as G
import ggms_oracle as orc
from ggms_b200 import datagen as D
from conftest import to_device

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def stream():
    import torch
    d = pytest.importorskip("cuda.bindings.driver")
    torch.zeros(1, device="cuda")

    def ok(r):
        assert r[0] == d.CUresult.CUDA_SUCCESS, r
        return r[1]
    dev = ok(d.cuDeviceGet(0))
    sms = ok(d.cuDeviceGetDevResource(dev, d.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    group = ok(d.cuDevSmResourceSplitByCount(1, sms, 0, 16))[0]
    green = ok(d.cuGreenCtxCreate(ok(d.cuDevResourceGenerateDesc([group], 1)), dev,
                                  d.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    st = ok(d.cuGreenCtxStreamCreate(green, d.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield int(st)
    torch.cuda.synchronize()
    d.cuStreamDestroy(st)
    d.cuGreenCtxDestroy(green)


@pytest.mark.parametrize("kw", [{}, {"num_buckets": 1024, "assigner": G.ASSIGNER_SAMPLED}])
def test_one_vector(stream, kw):
    ctx = G.Context(0)
    n = (1 << 21) + 3
    v, ks = D.normal_f32(n, 9), D.ks_uniform(n, 101, 9)
    v[::2] = v[1]
    d, out = to_device(v), np.empty(101, np.float32)
    for _ in range(3):  # directly, captured, replayed
        assert G.multiselect_ex(ctx, d.data_ptr(), n, ks, 101, out, np.float32, G.default_opts(**kw), stream) == 0
        np.testing.assert_array_equal(orc.bits(out), orc.bits(orc.cpu_multiselect(v, ks)))
    ctx.close()


def test_batch_with_more_teams_than_ctas(stream):
    import torch
    ctx = G.Context(0)
    g = np.random.default_rng(10)
    lens = np.array([(1 << 18) + 1 + i for i in range(60)] + [50_000] * 20 + [5000] * 20 + [300] * 100)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    v = g.integers(0, 1 << 32, off[-1], dtype=np.uint32)
    ks = np.concatenate([g.integers(1, n + 1, 3) for n in lens]).astype(np.uint32)
    k_off = (np.arange(len(lens) + 1) * 3).astype(np.int64)
    dv, dk, do, dko = to_device(v), to_device(ks), to_device(off), to_device(k_off)
    out = torch.empty(len(ks), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for _ in range(3):
        assert G.segmented(ctx, dv.data_ptr(), do.data_ptr(), len(lens), dk.data_ptr(), dko.data_ptr(),
                           out.data_ptr(), np.uint32, stream=stream) == 0
        assert ctx.status() == 0
    exp = np.concatenate([np.sort(v[a:b])[(b - a) - ks[3 * s:3 * s + 3].astype(np.int64)]
                          for s, (a, b) in enumerate(zip(off[:-1], off[1:]))])
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), exp)
    ctx.close()
