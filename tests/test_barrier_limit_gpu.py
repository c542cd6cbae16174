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
