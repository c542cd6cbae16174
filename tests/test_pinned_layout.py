"""The pinned buffer of a call with host ks and host answers: kernels read the
ks and store the answers there, so every part lies inside the size the buffer
is allocated with, at every number of ks (its parts start at 64-byte
boundaries, which the size has to pay for)."""
import ctypes

import numpy as np
import pytest

import ggms_b200 as G
import ggms_oracle as orc
from ggms_b200 import datagen as D
from conftest import to_device


def layout(nk, elem, host_k, host_out):
    out = (ctypes.c_int64 * 4)()
    fn = G.load().ggms_diag_pinned_layout
    fn.argtypes = [ctypes.c_int64, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    assert fn(nk, elem, host_k, host_out, out) == 0
    return list(out)


@pytest.mark.parametrize("elem", [4, 8])
@pytest.mark.parametrize("host_k,host_out", [(1, 1), (1, 0), (0, 1), (0, 0)])
def test_parts_lie_inside_the_buffer(elem, host_k, host_out):
    for nk in range(1, 20_001):
        counters, ks, out, total = layout(nk, elem, host_k, host_out)
        assert 0 < counters <= ks and ks % 64 == 0 and out % 64 == 0
        assert ks + (4 * nk if host_k else 0) <= out
        assert out + (elem * nk if host_out else 0) <= total, nk


@pytest.mark.gpu
@pytest.mark.parametrize("entry", ["select", "topk"])
def test_many_host_ks_on_a_new_context(entry):
    """The call that sizes the buffer needs more than its 64 KB minimum, with a
    number of ks that is not a multiple of 16, on the two-pass path."""
    ctx = G.Context(0)
    n, nk = (12 << 20) + 4099, 8673
    v = D.half_normal_f32(n, 5)
    d = to_device(v)
    if entry == "select":
        ks = D.ks_uniform(n, nk, 6)
        got = G.select(ctx, d.data_ptr(), n, ks, np.float32)
    else:
        ks = np.arange(1, nk + 1, dtype=np.uint32)
        got = G.topk(ctx, d.data_ptr(), n, nk, np.float32, num_buckets=8192)
    np.testing.assert_array_equal(orc.bits(got), orc.bits(orc.cpu_multiselect(v, ks)))
    ctx.close()
