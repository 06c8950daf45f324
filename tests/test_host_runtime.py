"""The library's host code on a stand-in for the CUDA runtime (fake_cudart.c):
what it believes about the device after replays, failed allocations, failed
launches and a context reset.  Each case runs in a process of its own."""
from __future__ import annotations

import ctypes as C
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


class Total(C.Structure):  # the head of the control block (hpmc_device.cuh)
    _fields_ = [("total", C.c_ulonglong)] + [(n, C.c_uint) for n in (
        "reduce_done", "status", "written", "work_next", "work_done", "col_next", "col_done", "extracting",
        "mesh_edges", "mesh_done")]


def _handle(L, size=(40, 40, 40)):
    c = L.HPMCcreateConstants(4, 3)
    h = L.HPMCcreateHistoPyramid(c)
    L.HPMCsetLatticeSize(h, *size)
    field = C.create_string_buffer(4 * size[0] * size[1] * size[2] + 16)
    assert L.HPMCsetFieldDevice(h, (C.addressof(field) + 15) // 16 * 16, 0, 0, 0) == 0
    p = C.c_void_p()
    assert L.HPMCgetDeviceVertexCount(h, C.byref(p)) == 0
    return c, h, field, C.cast(p, C.POINTER(Total))[0]


def case_count_of_replays(L):
    """Every replay of a captured build may change the count."""
    _, h, field, ctrl = _handle(L)
    L.HPMCbuildHistopyramid(h, 0.0)
    L.fake_capture(1, None)
    L.HPMCbuildHistopyramid(h, 0.0)
    L.fake_capture(0, None)
    th = L.HPMCcreateTraversalHandle(h)
    for n in (300, 90, 600):
        ctrl.total = n  # a replay
        assert L.HPMCacquireNumberOfVertices(h) == n
        ctrl.total = n + 3  # another one
        nv, ni = C.c_uint64(), C.c_uint64()
        assert L.HPMCextractVerticesIndexed(th, None, None, 1 << 20, None, 1 << 20, C.byref(nv), C.byref(ni)) == 0
        assert ni.value == n + 3
        ctrl.total = n - 30  # and one whose vertices fit
        assert L.HPMCextractVerticesToBuffers(th, 16, None, n, C.byref(nv)) == 0
        assert nv.value == n - 30


def case_failed_setup(L):
    """A set-up that ran out of memory leaves nothing that could be read or extracted."""
    for size in ((400, 400, 400), (40, 40, 40)):  # the larger pyramid, then a smaller one
        _, h, field, ctrl = _handle(L)
        th = L.HPMCcreateTraversalHandle(h)
        L.HPMCbuildHistopyramid(h, 0.0)
        L.HPMCsetLatticeSize(h, 400, 400, 400)
        L.fake_limit(1 << 16)
        L.HPMCbuildHistopyramid(h, 0.0)
        L.fake_limit(1 << 30)
        assert L.HPMCgetLastError(h) == 6  # HPMC_ERR_OUT_OF_MEMORY
        launches = L.fake_launches()
        assert L.HPMCacquireNumberOfVertices(h) == 0
        assert L.HPMCextractVerticesToBuffers(th, 16, None, 1, None) == 8  # HPMC_ERR_NOT_BUILT
        assert L.HPMCextractVerticesAdjoint(th, None, None, 1, 16) == 8
        assert L.HPMCextractVerticesIndexed(th, None, None, 0, None, 0, None, None) == 8
        assert L.HPMCreadLevel(h, 5, 4096, 1 << 20) == 8
        assert L.fake_launches() == launches
        L.HPMCsetLatticeSize(h, *size)
        L.HPMCbuildHistopyramid(h, 0.0)
        p = C.c_void_p()
        assert L.HPMCgetDeviceVertexCount(h, C.byref(p)) == 0
        assert L.HPMCextractVerticesToBuffers(th, 16, None, 1, None) == 0
        assert L.HPMCgetLastError(h) == 0


def case_failed_weld(L):
    """A weld whose launches fail part-way leaves its counters behind; the next one starts from zero."""
    _, h, field, ctrl = _handle(L)
    th = L.HPMCcreateTraversalHandle(h)
    L.HPMCbuildHistopyramid(h, 0.0)
    L.HPMCbuildHistopyramid(h, 0.0)  # (the count of the first was not read: the second's is copied)
    ctrl.total = 100
    weld = lambda: L.HPMCextractVerticesIndexed(th, None, None, 1 << 20, None, 1 << 20, None, None)  # noqa: E731
    assert weld() == 0
    for after in range(6):  # mesh_edges .. mesh_indices
        L.fake_fail_launch(L.fake_launches() + after)
        assert weld() == 5  # HPMC_ERR_CUDA
        ctrl.mesh_edges, ctrl.mesh_done = 70, 1
        assert L.HPMCsetFieldDevice(h, 16, 0, 0, 0) == 0  # un-breaks the handle without a set-up
        assert weld() == 0
        assert (ctrl.total, ctrl.mesh_edges, ctrl.mesh_done) == (100, 0, 0)


def case_context_reset(L):
    """Host memory of a context that was reset is neither handed out nor read."""
    _, h, field, ctrl = _handle(L)
    L.HPMCbuildHistopyramid(h, 0.0)
    assert L.HPMCacquireNumberOfVertices(h) == 0
    L.HPMCdestroyHandle(h)
    allocs = L.fake_host_allocs()
    L.HPMCdestroyHandle(_handle(L)[1])
    assert L.fake_host_allocs() == allocs == 1  # kept for the next handle ...
    L.fake_new_context()  # ... of the same context
    _, h, field, ctrl = _handle(L)
    assert L.fake_host_allocs() == allocs + 1
    L.HPMCbuildHistopyramid(h, 0.0)
    ctrl.total = 50
    L.fake_new_context()
    assert L.HPMCacquireNumberOfVertices(h) == 50  # copied, as far as the runtime lets it


def case_static_scratch_after_reset(L):
    """The scratch array has an address per context."""
    field = C.create_string_buffer(4 * 20 * 20 * 20 + 16)
    count = C.c_uint()
    lookups = []
    for _ in range(2):
        for _ in range(2):
            assert L.HPMCextractStatic((C.addressof(field) + 15) // 16 * 16, 0, 20, 20, 20, 0, 0, 0.0, 0, None, None, None, 0,
                                       C.byref(count), None, None) == 0
        lookups.append(L.fake_symbol_lookups())
        L.fake_new_context()
    assert lookups == [1, 2]


def case_opt_in_per_device(L):
    """The classifiers' shared-memory opt-in holds for one device and until a reset: constants renew it."""
    set_up = []
    for _ in range(2):
        before = L.fake_attributes()
        L.HPMCdestroyConstants(L.HPMCcreateConstants(4, 3))
        set_up.append(L.fake_attributes() - before)
        L.fake_new_context()
    assert set_up[0] == set_up[1] > 0


CASES = {k[5:]: v for k, v in list(globals().items()) if k.startswith("case_")}


@pytest.fixture(scope="module")
def fake_library(hpmc, tmp_path_factory):
    from hpmc_b200 import build as B

    if not shutil.which("gcc"):
        pytest.skip("no C compiler")
    B.build()
    out = tmp_path_factory.mktemp("fake")
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(B.nvcc())))
    fake, lib = str(out / "fake_cudart.o"), str(out / "libhpmc_fake.so")
    subprocess.run(["gcc", "-O1", "-fPIC", "-I" + os.path.join(cuda, "include"), "-c",
                    os.path.join(HERE, "fake_cudart.c"), "-o", fake], check=True)
    objs = sorted(os.path.join(B.OBJ_DIR, os.path.basename(s)[:-3] + ".o") for s in B._sources())
    subprocess.run([B.nvcc(), *B.NVCC_FLAGS[:2], "-shared", "-cudart", "none", "-Xlinker", "-Bsymbolic", "-o", lib,
                    *objs, fake], check=True)
    return lib


@pytest.mark.parametrize("name", sorted(CASES))
def test_host_runtime(fake_library, name):
    r = subprocess.run([sys.executable, os.path.abspath(__file__), fake_library, name], capture_output=True, text=True,
                       cwd=ROOT, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]


if __name__ == "__main__":
    sys.path.insert(0, ROOT)
    from hpmc_b200 import _capi

    _capi.LIB_PATH = sys.argv[1]
    lib = _capi.lib()
    lib.fake_capture.argtypes = [C.c_int, C.c_void_p]
    lib.fake_limit.argtypes = [C.c_size_t]
    CASES[sys.argv[2]](lib)
