"""The library's host side without a GPU: the CUDA runtime replaced by
fake_cudart.c, in a child process."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def child(tmp_path_factory):
    from chimera_b200 import build, gpu
    if not os.path.exists(gpu.LIB_PATH):
        build.build()
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    include = os.path.join(os.path.dirname(os.path.dirname(build._nvcc())), "include")
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-I" + include, "-o", so, os.path.join(HERE, "fake_cudart.c")],
                   check=True)
    head = f"""
import ctypes as C, sys
sys.path.insert(0, {ROOT!r})
from chimera_b200 import gpu
from chimera_b200.config import *
fake = C.CDLL(None)
fake.fake_live_bytes.restype = C.c_longlong
lib = gpu.lib()
def grid(nx, ny=None, **kw):
    return SolverConfig(nx=nx, ny=ny or nx, dx=1.0 / nx, dy=1.0 / nx, gamma=5.0 / 3.0, **kw)
"""

    def run(body):
        r = subprocess.run([sys.executable, "-c", head + body], env=dict(os.environ, LD_PRELOAD=so), capture_output=True,
                           text=True, timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr
    return run


def test_autotuned_choice_stays_with_its_shape(child):
    """A tile chosen for one problem is not taken for another one of as many cells: a
    mixed pair of sides, which has one tile, or another shape."""
    child("""
ms = (C.c_float * 64)(*([5.0] * 3 + [1.0] + [5.0] * 60))
fake.fake_elapsed(ms, 64)
with gpu.Solver(grid(64, bc=(BC_PERIODIC,) * 4)) as s:
    default = s.variant()["variant"]
    chosen, _ = s.autotune(1)
    assert chosen == 3 != default
with gpu.Solver(grid(64, bc=(BC_OUTFLOW,) * 4)) as s:
    assert s.variant()["variant"] == 3
with gpu.Solver(grid(64, bc=(BC_PERIODIC, BC_OUTFLOW, BC_PERIODIC, BC_PERIODIC))) as s:
    assert s.variant_count() == 1 and s.variant()["variant"] == 0
    s.step(1)
with gpu.Solver(grid(32, 128)) as s:
    assert s.variant()["variant"] == default
""")


@pytest.mark.parametrize("precision", ["FP64", "FP32_BULK", "FP32_MIXED"])
def test_state_and_time_with_another_device_current(child, precision):
    """set_state, get_state and set_time of a handle whose device is not the current one:
    done on the handle's device, the caller's choice left as it was."""
    child(f"""
with gpu.Solver(grid(16, precision={precision})) as s:
    dev = [C.c_void_p() for _ in range(6)]
    for d in dev:
        assert fake.cudaMalloc(C.byref(d), C.c_size_t(16 * 16 * 8)) == 0
    assert fake.cudaSetDevice(1) == 0
    assert lib.chimera_batch_set_state(s.handle, 0, *dev, 16, gpu.DEVICE) == 0
    assert lib.chimera_batch_get_state(s.handle, 0, *dev, 16, gpu.DEVICE) == 0
    assert fake.fake_launches(b"move_state_kernel") == 2
    assert lib.chimera_batch_set_time(s.handle, 0, 0.5, 2) == 0
    assert fake.fake_launches(b"set_time_kernel") == 1
    now = C.c_int()
    assert fake.cudaGetDevice(C.byref(now)) == 0 and now.value == 1
""")


def test_work_list_memory_follows_the_tiles(child):
    """A large grid holds partials and a work list for large tiles (52 bytes a tile of 256
    cells: 0.21 a cell); a small tile gets its own when it is chosen, or the choice is
    refused and the handle stays as it was."""
    child("""
cells = 1024 * 1024
with gpu.Solver(grid(1024, precision=FP32_BULK)) as s:
    state = 18 * 4 * cells + 8 * cells          # three buffer sets, the float64 staging
    other = fake.fake_live_bytes() - state
    assert 0 < other <= 0.21 * cells, other / cells
    before = s.variant()
    fake.fake_memory(C.c_longlong(fake.fake_live_bytes() + cells // 2))
    assert lib.chimera_set_variant(s.handle, 11) == -7      # 8 x 8 tiles: 0.8 bytes a cell
    assert s.variant() == before
    s.step(1)
    s.autotune(1)
    fake.fake_memory(C.c_longlong(1 << 60))
    s.set_variant(11)
    assert s.variant()["tile"] == (8, 8) and fake.fake_live_bytes() - state >= 52 * cells // 64
    s.step(1)
assert fake.fake_live_bytes() == 0
""")


def test_autotuner_times_a_kernel_once(child):
    """Two variants that name the same kernels are one candidate: each stage kernel runs in
    the warm-up step and in the timed one."""
    child("""
for precision in (FP64, FP32_BULK, FP32_MIXED):
    with gpu.Solver(grid(512, precision=precision)) as s:
        fake.fake_reset()
        s.autotune(1)
        assert fake.fake_most_launches() == 2, precision
""")


def test_capture_of_another_stream_refuses_state_and_time(child):
    """set_state, get_state and set_time while the thread captures a stream that forbids
    waiting: refused before anything is launched, and done again afterwards."""
    child("""
with gpu.Solver(grid(16)) as s:
    dev = [C.c_void_p() for _ in range(6)]
    for d in dev:
        assert fake.cudaMalloc(C.byref(d), C.c_size_t(16 * 16 * 8)) == 0
    def calls():
        return [lib.chimera_batch_set_state(s.handle, 0, *dev, 16, gpu.DEVICE),
                lib.chimera_batch_get_state(s.handle, 0, *dev, 16, gpu.DEVICE),
                lib.chimera_batch_set_time(s.handle, 0, 0.5, 2)]
    fake.fake_reset()
    fake.fake_capture(1)
    assert calls() == [-2, -2, -2]
    assert fake.fake_launches(b"") == 0
    fake.fake_capture(0)
    assert calls() == [0, 0, 0]
""")
