"""A grid barrier that runs out ends the call with an error that the host sees.
The failure is made by a limit at which every wait gives up at once (no wait
is left without an end), so the kernels return and the GPU stays usable."""
import ctypes

import numpy as np
import pytest

import ggms_b200 as G
import ggms_oracle as orc
from ggms_b200 import datagen as D
from conftest import to_device

pytestmark = pytest.mark.gpu

N = 300_007
# which launch holds the barriers: the one-launch path, or the refinement
# levels of the two-pass path (atoms of two neighbouring values need levels)
PATHS = {"one launch": {}, "levels": {"num_buckets": 1024, "assigner": G.ASSIGNER_SAMPLED}}


def limit(ctx, cycles):
    fn = G.load().ggms_diag_barrier_limit
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int64]
    assert fn(ctx.ptr, cycles) == 0


def vector(seed):
    g = np.random.default_rng(seed)
    v = g.standard_normal(N).astype(np.float32)
    v[g.random(N) < 0.9] = 7.0
    v[g.random(N) < 0.4] = np.nextafter(np.float32(7.0), np.float32(8.0))
    return v


def host_call(ctx, d, ks, out, **kw):
    return G.multiselect_ex(ctx, d.data_ptr(), N, ks, len(ks), out, np.float32, G.default_opts(**kw))


@pytest.mark.parametrize("path", PATHS)
def test_the_host_sees_a_barrier_that_ran_out(path):
    ctx = G.Context(0)
    v = vector(1)
    d, ks = to_device(v), D.ks_uniform(N, 101, 2)
    good = np.empty(len(ks), np.float32)
    assert host_call(ctx, d, ks, good, **PATHS[path]) == 0
    np.testing.assert_array_equal(orc.bits(good), orc.bits(orc.select(v, ks)))
    limit(ctx, -1)
    out = np.full(len(ks), 123.0, np.float32)
    assert host_call(ctx, d, ks, out, **PATHS[path]) == G.GGMS_E_INTERNAL
    assert (out == 123.0).all()  # no answers of an earlier call
    ctx.close()


def device_call(ctx, d, dk, dout, **kw):
    o = G.default_opts(ks_on_device=1, out_on_device=1, **kw)
    assert G.multiselect_ex(ctx, d.data_ptr(), N, dk.data_ptr(), len(dk), dout.data_ptr(), np.float32, o) == 0


@pytest.mark.parametrize("cycles", [-1, 1, 2000])
@pytest.mark.parametrize("path", PATHS)
def test_calls_after_a_barrier_that_ran_out(path, cycles):
    """... and leaves the context as it was: the calls after it are exact.  With
    a limit of some cycles the CTAs give up at different barriers (or not at
    all: then the answers are exact)."""
    import torch
    ctx = G.Context(0)
    v = vector(3)
    d, ks = to_device(v), D.ks_uniform(N, 101, 4)
    dk, dout = to_device(ks), torch.empty(len(ks), dtype=torch.float32, device="cuda")
    exp = orc.bits(orc.select(v, ks))
    out = np.empty(len(ks), np.float32)
    for _ in range(4):  # run directly, captured, replayed
        limit(ctx, cycles)
        rc = host_call(ctx, d, ks, out, **PATHS[path])
        assert rc == G.GGMS_E_INTERNAL or (cycles > 0 and rc == 0 and (orc.bits(out) == exp).all())
        device_call(ctx, d, dk, dout, **PATHS[path])
        assert ctx.status() == G.GGMS_E_INTERNAL or cycles > 0
        device_call(ctx, d, dk, dout, **PATHS[path])  # nobody asks for this one's status
        limit(ctx, 0)
        device_call(ctx, d, dk, dout, **PATHS[path])
        assert ctx.status() == 0
        np.testing.assert_array_equal(orc.bits(dout.cpu().numpy()), exp)
        assert host_call(ctx, d, ks, out, **PATHS[path]) == 0
        np.testing.assert_array_equal(orc.bits(out), exp)
    ctx.close()


@pytest.mark.parametrize("cycles", [-1, 1, 2000])
def test_batched_calls_after_a_barrier_that_ran_out(cycles):
    """Teams of every size (a long segment among equal ones), then single CTAs, sorts and rows."""
    import torch
    ctx = G.Context(0)
    g = np.random.default_rng(5)
    lens = np.array([1 << 22] + [(1 << 19) + 7] * 6 + [100_003] * 5 + [5000] * 7 + [700] * 9)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    v = g.integers(0, 1 << 32, off[-1], dtype=np.uint64).astype(np.uint32)
    v[g.random(len(v)) < 0.3] = 12345
    v[g.random(len(v)) < 0.3] = 12346
    ks = np.concatenate([g.integers(1, n + 1, 30) for n in lens]).astype(np.uint32)
    k_off = (np.arange(len(lens) + 1) * 30).astype(np.int64)
    dv, dk, do, dko = to_device(v), to_device(ks), to_device(off), to_device(k_off)
    out = torch.empty(len(ks), dtype=torch.int32, device="cuda")

    def call():
        assert G.segmented(ctx, dv.data_ptr(), do.data_ptr(), len(lens), dk.data_ptr(), dko.data_ptr(),
                           out.data_ptr(), np.uint32) == 0
    exp = orc.select_segmented(v, off, ks, k_off)
    for _ in range(3):
        limit(ctx, cycles)
        call()
        st = ctx.status()
        assert st == G.GGMS_E_INTERNAL or (cycles > 0 and st == 0)
        call()
        limit(ctx, 0)
        call()
        assert ctx.status() == 0
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), exp)
    ctx.close()


def test_a_long_list_of_ks_between_barriers():
    """One refinement level's child holds all 8 M ks (the same k many times): one
    warp walks their list while the other CTAs wait at the barrier behind it, for
    longer than a wait without ks may take.  fp32, 2^25 keys in 1024 buckets:
    every bucket takes a level, its bins hold some 16 keys."""
    ctx = G.Context(0)
    n, nk = 1 << 25, 8_000_000
    v = D.normal_f32(n, 6)
    k = n // 3
    got = G.select(ctx, to_device(v).data_ptr(), n, np.full(nk, k, np.uint32), np.float32,
                   assigner=G.ASSIGNER_SAMPLED, num_buckets=1024)
    assert (orc.bits(got) == orc.bits(np.sort(v)[n - k:n - k + 1])[0]).all()
    ctx.close()
