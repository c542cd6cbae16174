"""The host code's launches.  The library's own objects are linked to a CUDA
runtime without a GPU (tests/launch_shim/fake_cudart.cpp).  A launch that fails
makes the call return an error, whichever launch of the call it is."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import ggms_b200 as G

LIBDIR = os.path.dirname(G.LIB_PATH)
SHIM = os.path.join(os.path.dirname(os.path.abspath(__file__)), "launch_shim")
UNITS = ("f32", "f64", "u32", "i32", "direct", "batch", "refine", "context")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "libggms_fake.so")
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-fvisibility=hidden", "-I/usr/local/cuda/include",
                    os.path.join(SHIM, "fake_cudart.cpp"), *(os.path.join(LIBDIR, f"ggms_{u}.o") for u in UNITS),
                    "-Wl,-z,defs", "-o", so], check=True)
    return ctypes.CDLL(so)


def call(lib, entry, n=1 << 20, nk=100, **kw):
    """One call on a new context, over host memory; its status."""
    ctx = ctypes.c_void_p()
    assert lib.ggms_create(ctypes.byref(ctx), 0) == 0
    o = G.Opts()
    lib.ggms_default_opts(ctypes.byref(o))
    for k, x in dict(ks_on_device=1, out_on_device=1, **kw).items():
        setattr(o, k, x)
    v, out = np.zeros(n, np.float32), np.zeros(nk, np.float32)
    ks = np.ones(nk, np.uint32)
    off, k_off = np.array([0, n // 2, n], np.int64), np.array([0, 1, nk], np.int64)
    p = lambda a: ctypes.c_void_p(a.ctypes.data)
    i64 = ctypes.c_int64
    if entry.startswith("segmented"):
        rc = getattr(lib, "ggms_multi" + entry.replace("segmented", "select_segmented"))(
            ctx, p(v), p(off), i64(2), p(ks), p(k_off), p(out), ctypes.byref(o), None)
    elif entry.startswith("topk"):
        rc = getattr(lib, "ggms_" + entry)(ctx, p(v), i64(n), i64(nk), p(out), ctypes.byref(o), None)
    else:
        rc = getattr(lib, f"ggms_multi{entry}_ex")(ctx, p(v), i64(n), p(ks), i64(nk), p(out), ctypes.byref(o), None)
    lib.ggms_destroy(ctx)
    return rc


CALLS = [("segmented_f32", {}), ("segmented_u32", {}), ("select_f32", {}), ("select_f32", {"n": 5000}),
         ("select_u32", {"num_buckets": 8192}), ("select_i32", {"num_buckets": 1024, "sample_size": 2048}),
         ("select_f32", {"assigner": G.ASSIGNER_LEARNED_MLP}), ("select_f32", {"nk": 70_000}), ("topk_f32", {}),
         ("topk_f32", {"num_buckets": 8192})]


@pytest.mark.parametrize("entry,kw", CALLS)
def test_every_failing_launch_is_reported(lib, entry, kw):
    lib.fake_reset(-1, 0)
    assert call(lib, entry, **kw) == G.GGMS_OK
    launches = lib.fake_launches()
    assert launches >= 1
    for i in range(launches):
        lib.fake_reset(i, 0)
        assert call(lib, entry, **kw) == G.GGMS_E_CUDA, f"launch {i} of {launches}"


def test_the_one_launch_path_is_a_candidate_of_the_autotuner(lib):
    """With every candidate as fast (the runtime's clock says 1 ms each) the first
    one is kept: the call that the library makes without tuning."""
    lib.fake_reset(-1, 0)
    n, nk = 1 << 20, 100
    ctx = ctypes.c_void_p()
    assert lib.ggms_create(ctypes.byref(ctx), 0) == 0
    o = G.Opts()
    lib.ggms_default_opts(ctypes.byref(o))
    o.ks_on_device = o.out_on_device = o.autotune = 1
    v, out, ks = np.zeros(n, np.float32), np.zeros(nk, np.float32), np.ones(nk, np.uint32)
    p = lambda a: ctypes.c_void_p(a.ctypes.data)
    per_call = []
    for _ in range(2):
        before = lib.fake_launches()
        assert lib.ggms_multiselect_f32_ex(ctx, p(v), ctypes.c_int64(n), p(ks), ctypes.c_int64(nk), p(out),
                                           ctypes.byref(o), None) == G.GGMS_OK
        per_call.append(lib.fake_launches() - before)
    lib.ggms_destroy(ctx)
    assert per_call[0] > 100 and per_call[1] == 1  # tunes, then calls as tuned


@pytest.mark.parametrize("entry,kw", CALLS)
@pytest.mark.parametrize("ctas", [1, 16, 147])
def test_fewer_sms_than_the_device_has(lib, entry, kw, ctas):
    """Cooperative launches are refused where fewer CTAs can be resident: the call
    makes smaller ones."""
    lib.fake_reset(-1, ctas)
    assert call(lib, entry, **kw) == G.GGMS_OK
    assert lib.fake_coop_grid() <= ctas
    if kw.get("n", ctas) >= 1 << 20:
        assert lib.fake_coop_grid() > ctas * 3 // 4
