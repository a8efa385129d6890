"""The host transfers (csrc/host_stage.cu) against a fake of the CUDA runtime (host_stage_fake.cpp), on the
CPU: whole copies, and no processor time while a transfer waits for the work before it."""
from __future__ import annotations

import ctypes as C
import mmap
import os
import subprocess
import time

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "winds-master_b200", "csrc")


@pytest.fixture(scope="module")
def stage(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("stage") / "stage.so")
    # -Bsymbolic: the fake's functions, also after another test has loaded the CUDA runtime for all.
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I/usr/local/cuda/include",
                    "-I" + os.path.join(ROOT, "include"), "-I" + CSRC, "-x", "c++",
                    os.path.join(CSRC, "host_stage.cu"), os.path.join(ROOT, "tests", "host_stage_fake.cpp"),
                    "-o", so, "-lpthread", "-Wl,-Bsymbolic"], check=True, capture_output=True)
    L = C.CDLL(so)
    L.stage_download.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int, C.c_int, C.c_int]
    L.stage_upload.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
    yield L
    L.stage_release()


@pytest.mark.parametrize("mb", [0.001, 1.0, 1.5, 8.0, 40.0])
def test_download_is_whole(stage, mb):
    src = np.random.default_rng(0).integers(0, 255, int(mb * 2 ** 20), dtype=np.uint8)
    for wide in (0, 1):
        dst = np.ones_like(src)  # pages in place
        assert stage.stage_download(dst.ctypes.data, src.ctypes.data, src.nbytes, 0, 0, wide) == 0
        np.testing.assert_array_equal(dst, src)
        pages = mmap.mmap(-1, src.nbytes)  # none yet
        dst = np.frombuffer(pages, dtype=np.uint8)
        assert stage.stage_download(dst.ctypes.data, src.ctypes.data, src.nbytes, 0, 0, wide) == 0
        np.testing.assert_array_equal(dst, src)


@pytest.mark.parametrize("mb,there,wide,copies", [
    (0.5, True, 0, 1), (4.5, True, 0, 5), (15.5, True, 0, 16), (40.0, True, 0, 1),
    (0.5, False, 0, 1), (4.5, False, 0, 5), (15.5, False, 0, 16), (40.0, False, 0, 40),
    (4.5, True, 1, 5), (40.0, True, 1, 40), (40.0, False, 1, 40)])
def test_route(stage, mb, there, wide, copies):
    """Chunks of 1 MB, and one plain copy for large outputs into pages that are there."""
    src = np.ones(int(mb * 2 ** 20), dtype=np.uint8)
    pages = mmap.mmap(-1, src.nbytes)
    dst = np.frombuffer(pages, dtype=np.uint8)
    if there:
        pages.write(bytes(src.nbytes))
    assert stage.stage_download(dst.ctypes.data, src.ctypes.data, src.nbytes, 0, 0, wide) == 0
    assert stage.stage_copies() == copies
    np.testing.assert_array_equal(dst, src)


def test_copies_without_pinned_memory(stage):
    """A system that has no pinned memory to give: the driver's own staging, as for larger inputs."""
    stage.stage_release()
    src = np.random.default_rng(1).integers(0, 255, 3 * 2 ** 20, dtype=np.uint8)
    for n in (5, 2 ** 20, src.nbytes):
        dst = np.zeros(n, dtype=np.uint8)
        assert stage.stage_upload(src.ctypes.data, dst.ctypes.data, n, 1) == 0
        np.testing.assert_array_equal(dst, src[:n])
        dst[:] = 0
        assert stage.stage_download(dst.ctypes.data, src.ctypes.data, n, 0, 1, 0) == 0
        np.testing.assert_array_equal(dst, src[:n])
        assert stage.stage_last_error() == 0


def test_waiting_takes_no_processor_time(stage):
    """Eight threads copy 16 MB out once the first chunk has landed, 0.5 s after the call. The copies take
    some 10 ms of processor time; a tenth of the wait is far above that."""
    src = np.ones(16 * 2 ** 20, dtype=np.uint8)
    dst = np.zeros_like(src)
    stage.stage_download(dst.ctypes.data, src.ctypes.data, src.nbytes, 0, 0, 1)  # pages of both
    cpu, wall = time.process_time(), time.perf_counter()
    assert stage.stage_download(dst.ctypes.data, src.ctypes.data, src.nbytes, 500, 0, 1) == 0
    cpu, wall = time.process_time() - cpu, time.perf_counter() - wall
    assert wall >= 0.5
    assert cpu <= 0.1 * wall, (cpu, wall)
