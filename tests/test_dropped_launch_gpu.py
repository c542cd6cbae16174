"""Batched calls: the ks of segments that no kernel has taken are reported, not
answered.  The library's objects are linked with a shim around the runtime's
launch calls that drops the launch of one class of segments."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import ggms_b200 as G
import ggms_oracle as orc
from conftest import to_device

LIBDIR = os.path.dirname(G.LIB_PATH)
SHIM = os.path.join(os.path.dirname(os.path.abspath(__file__)), "launch_shim", "drop_launch.cpp")
UNITS = ("f32", "f64", "u32", "i32", "direct", "batch", "refine", "context")
# the order of the batched path's launches; 0 sorts the segments into classes, 6 writes the answers
CLASSES = {"rows": 1, "longer rows": 2, "sorts": 3, "teams": 4, "singles": 5}


def link(out_dir):
    so = os.path.join(out_dir, "libggms_shim.so")
    wraps = [x for f in ("cudaLaunchKernel", "cudaLaunchKernelExC") for x in ("-Xlinker", f"--wrap={f}")]
    subprocess.run(["nvcc", "-shared", "-Xcompiler", "-fPIC,-fvisibility=hidden", *wraps, SHIM,
                    *(os.path.join(LIBDIR, f"ggms_{u}.o") for u in UNITS), "-o", so], check=True)
    return so


def test_shim_links(tmp_path):
    assert os.path.exists(link(str(tmp_path)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return ctypes.CDLL(link(str(tmp_path_factory.mktemp("shim"))))


@pytest.mark.gpu
@pytest.mark.parametrize("dropped", CLASSES)
def test_segments_without_a_kernel_are_reported(lib, dropped):
    import torch
    g = np.random.default_rng(7)
    lens = np.array([1 << 20] + [100_003] * 5 + [5000] * 5 + [1500] * 50 + [700] * 600)  # teams .. rows
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    v = g.standard_normal(off[-1]).astype(np.float32)
    ks = np.concatenate([g.integers(1, n + 1, 3) for n in lens]).astype(np.uint32)
    k_off = (np.arange(len(lens) + 1) * 3).astype(np.int64)
    dv, dk, do, dko = to_device(v), to_device(ks), to_device(off), to_device(k_off)
    out = torch.empty(len(ks), dtype=torch.float32, device="cuda")
    ctx = ctypes.c_void_p()
    assert lib.ggms_create(ctypes.byref(ctx), 0) == 0
    p = lambda t: ctypes.c_void_p(t.data_ptr())

    def status_of_a_call(drop):
        lib.shim_drop(drop)
        assert lib.ggms_multiselect_segmented_f32(ctx, p(dv), p(do), ctypes.c_int64(len(lens)), p(dk), p(dko), p(out),
                                                  None, None) == 0
        st = ctypes.c_int(-1)
        assert lib.ggms_context_status(ctx, None, ctypes.byref(st)) == 0
        return st.value
    assert status_of_a_call(CLASSES[dropped]) == G.GGMS_E_NOT_CONVERGED
    assert status_of_a_call(-1) == G.GGMS_OK
    np.testing.assert_array_equal(orc.bits(out.cpu().numpy()), orc.bits(orc.select_segmented(v, off, ks, k_off)))
    lib.ggms_destroy(ctx)
