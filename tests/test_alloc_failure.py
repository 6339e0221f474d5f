"""Calls after a failed device allocation, without a GPU: the library's own
objects linked against a CUDA runtime whose memory is host memory and whose
kernels do nothing (fake_cudart.cpp). Each allocation of a call fails in turn;
the call reports it, and the same call on the same context then runs with
workspaces that all stand."""
import ctypes as C
import glob
import os
import shutil
import subprocess

import numpy as np
import pytest

from hulktracer_b200 import build, scenes

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = build.nvcc()
SAH_RESORT = 2

pytestmark = pytest.mark.skipif(not (os.path.exists(NVCC) and shutil.which("g++")), reason="no CUDA toolkit")


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    build.build()
    out = str(tmp_path_factory.mktemp("fake") / "libhulk_fake.so")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(NVCC))), "include")
    subprocess.check_call(["g++", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I" + inc, "-o", out,
                           os.path.join(HERE, "fake_cudart.cpp")] + sorted(glob.glob(os.path.join(build.OBJ, "*.o"))) +
                          ["-ldl", "-lpthread"])
    L = C.CDLL(out)
    L.fake_live_bytes.restype = C.c_size_t
    for f in ("fake_allocs", "fake_bad_launches", "fake_scan_launches"):
        getattr(L, f).restype = C.c_long
    L.fake_fail_at.argtypes = [C.c_long]
    L.fake_fail_at.restype = None
    return L


def context(L):
    h = C.c_void_p()
    assert L.hk_create(C.byref(h), None) == 0
    return h


def p(a):
    return a.ctypes.data_as(C.c_void_p)


def test_resort_build_after_each_failed_allocation(fake):
    L = fake
    sc = scenes.random_soup(40_000, seed=2)   # the radix sort's scan needs more tiles than the first one's
    v, t = np.ascontiguousarray(sc.verts, np.float32), np.ascontiguousarray(sc.tris, np.uint32)

    def ready():
        h = context(L)
        assert L.hk_scene_upload(h, p(v), C.c_uint32(v.shape[0]), p(t), C.c_uint32(t.shape[0])) == 0
        return h
    h = ready()
    before = L.fake_allocs()
    assert L.hk_build(h, SAH_RESORT, None) == 0
    n = L.fake_allocs() - before
    assert n > 30 and L.fake_scan_launches() > 0 and L.fake_bad_launches() == 0
    L.hk_destroy(h)
    small = scenes.random_soup(20_000, seed=3)   # its arrays stand at sizes between the large scene's
    sv, s_t = np.ascontiguousarray(small.verts, np.float32), np.ascontiguousarray(small.tris, np.uint32)
    for k in range(1, n + 1):
        h = ready()
        L.fake_fail_at(k)
        assert L.hk_build(h, SAH_RESORT, None) != 0, "allocation %d" % k
        L.fake_fail_at(0)
        if k % 2:
            assert L.hk_scene_upload(h, p(sv), C.c_uint32(sv.shape[0]), p(s_t), C.c_uint32(s_t.shape[0])) == 0
            assert L.hk_build(h, SAH_RESORT, None) == 0
            assert L.hk_scene_upload(h, p(v), C.c_uint32(v.shape[0]), p(t), C.c_uint32(t.shape[0])) == 0
        assert L.hk_build(h, SAH_RESORT, None) == 0
        assert L.fake_bad_launches() == 0, "scan workspaces after allocation %d failed" % k
        L.hk_destroy(h)
    assert L.fake_live_bytes() == 0


@pytest.mark.parametrize("call", ["forward", "grad"])
def test_proposer_calls_give_large_buffers_back(fake, call):
    """Rows beyond the bound that a context keeps: nothing is held after the
    call, whether it succeeded or one of its allocations failed."""
    L = fake
    rows = 16_384 + 1
    x, y = np.zeros((rows, 200), np.float32), np.zeros(rows, np.int32)
    logits, grads = np.zeros((rows, 96), np.float32), np.zeros(1 << 20, np.float32)

    def run(h):
        if call == "forward":
            return L.hk_mlp_forward(h, p(x), C.c_uint32(rows), p(logits))
        return L.hk_mlp_grad(h, p(x), p(y), C.c_uint32(rows), p(grads), None)
    h = context(L)
    assert L.hk_mlp_init(h, C.c_uint64(1)) == 0
    held, before = L.fake_live_bytes(), L.fake_allocs()
    assert run(h) == 0
    n = L.fake_allocs() - before
    assert n >= 2 and L.fake_live_bytes() == held
    for k in range(1, n + 1):
        L.fake_fail_at(k)
        assert run(h) != 0
        L.fake_fail_at(0)
        assert L.fake_live_bytes() == held, "allocation %d" % k
    assert run(h) == 0
    L.hk_destroy(h)
