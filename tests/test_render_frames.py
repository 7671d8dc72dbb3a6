"""A renderer's frames share a depth buffer and a queue that each frame leaves empty for the next.  A
frame whose launches fail part way leaves marks in them: the frames after it must not see them.  The
renderer's host code runs here on a stand-in for the CUDA runtime (tests/cuda/fake_runtime.cpp), which
makes a chosen launch fail."""
import ctypes
import os
import subprocess

import pytest

import akuaengine_gb300 as ak
from akuaengine_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    d = tmp_path_factory.mktemp("frames")
    obj, fake, so = str(d / "splat.o"), str(d / "fake.o"), str(d / "frames.so")
    for cmd in (build.compile_command(os.path.join(build.CSRC, "splat.cu"), obj),
                ["g++", "-std=c++17", "-O1", "-fPIC", "-c", "-o", fake,
                 os.path.join(ROOT, "tests", "cuda", "fake_runtime.cpp")],
                ["g++", "-shared", "-Wl,-Bsymbolic", "-o", so, obj, fake]):
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
    return so


class Frames:
    def __init__(self, so):
        self.lib = ctypes.CDLL(so)
        self.lib.fake_reset()
        self.handle = ctypes.c_void_p()
        assert self.lib.akua_splat_create(8, 4, ctypes.byref(self.handle)) == 0
        self.camera = ak._abi.CCamera()
        self.lib.akua_camera_default(ctypes.byref(self.camera))

    def value(self, name):
        return ctypes.c_int.in_dll(self.lib, name)

    def render(self, n=100, fail=None):
        at = self.lib.fake_launches()
        self.value("fake_fail_launch").value = -1 if fail is None else at + fail
        records, image = ctypes.c_void_p(1 << 20), ctypes.c_void_p(1 << 21)  # never read
        return self.lib.akua_splat_render(self.handle, records, ctypes.c_size_t(108), n,
                                          ctypes.byref(self.camera), image, None)


@pytest.mark.parametrize("fail", [0, 1, 2])
def test_frame_after_a_failed_launch_starts_empty(built, fail):
    f = Frames(built)
    assert f.render() == 0 and f.render() == 0
    cleared = f.lib.fake_memsets()
    assert f.render() == 0 and f.lib.fake_memsets() == cleared  # no clearing of empty buffers
    assert f.render(fail=fail) == ak.AKUA_ERR_CUDA
    assert f.render() == 0 and f.render() == 0
    assert f.value("fake_dirty_frames").value == 0
    cleared = f.lib.fake_memsets()
    assert f.render() == 0 and f.lib.fake_memsets() == cleared


def test_clearing_that_was_only_captured_is_done_again(built):
    """A frame captured into a graph after a failed one clears when the graph runs, not now."""
    f = Frames(built)
    assert f.render(fail=2) == ak.AKUA_ERR_CUDA
    f.value("fake_capturing").value = 1
    assert f.render() == 0
    f.value("fake_capturing").value = 0
    assert f.render() == 0
    assert f.value("fake_dirty_frames").value == 0
