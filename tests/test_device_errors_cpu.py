"""When a kernel's bounded wait gives up, the next synchronisation says so: launched, or replayed from a graph.  device.cu over a
stand-in for the CUDA runtime (fake_cudart.cpp), where the host makes the wait give up."""
import ctypes as C
import os
import subprocess

import pytest

from denograd_b200 import build as B
from tests.util import ROOT

JG_ETIMEDOUT = 110
# what stands for the launch of a kernel with bounded waits, for one of them that ran out, and for the other parts of the library
HOOKS = """
#include "common.cuh"
#define API extern "C" __attribute__((visibility("default")))
API int fake_resets = 0;
API void fake_launch(jg_dev* dev) { dev->tc_pending = true; }
API void fake_give_up(jg_dev* dev) { *dev->err_word = 2; }
void jg_pair_reset(jg_dev*) { fake_resets++; }
int jg_peer_error(jg_dev*, int* code) { *code = 0; return JG_OK; }
int jg_peer_run_boundary(jg_dev*) { return JG_OK; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fake")
    (d / "hooks.cu").write_text(HOOKS)
    so = str(d / "libfake.so")
    subprocess.run([B.nvcc(), *B.ARCH, *B.FLAGS, "-I", B.CSRC, "-cudart", "none", "-shared", "-o", so, str(d / "hooks.cu"),
                    os.path.join(ROOT, "tests", "fake_cudart.cpp"), os.path.join(B.CSRC, "device.cu")], check=True)
    return C.CDLL(so)


@pytest.fixture
def dev(lib):
    h = C.c_void_p()
    assert lib.jg_device_open(0, C.byref(h)) == 0
    return h


def count(lib, what):
    return C.c_int.in_dll(lib, "fake_" + what).value


def capture(lib, dev, with_waits):
    g = C.c_void_p()
    assert lib.jg_graph_begin(dev) == 0
    if with_waits:
        lib.fake_launch(dev)
    assert lib.jg_graph_end(dev, C.byref(g)) == 0
    return g


def test_a_launch(lib, dev):
    lib.fake_launch(dev)
    assert lib.jg_device_sync(dev) == 0
    lib.fake_launch(dev)
    lib.fake_give_up(dev)
    before = count(lib, "resets")
    assert lib.jg_device_sync(dev) == JG_ETIMEDOUT
    assert count(lib, "resets") == before + 1  # flags that it left behind are cleared
    lib.fake_launch(dev)
    assert lib.jg_device_sync(dev) == 0


def test_a_replay(lib, dev):
    g, plain = capture(lib, dev, True), capture(lib, dev, False)
    assert lib.jg_device_sync(dev) == 0
    for _ in range(2):  # the first replay and a later one
        assert lib.jg_graph_launch(dev, g) == 0 and lib.jg_device_sync(dev) == 0
        assert lib.jg_graph_launch(dev, g) == 0
        lib.fake_give_up(dev)
        before = count(lib, "resets")
        assert lib.jg_device_sync(dev) == JG_ETIMEDOUT
        assert count(lib, "resets") == before + 1
        assert lib.jg_graph_launch(dev, plain) == 0 and lib.jg_device_sync(dev) == 0


def test_a_launch_ahead_of_a_capture(lib, dev):
    lib.fake_launch(dev)
    lib.fake_give_up(dev)
    capture(lib, dev, False)
    assert lib.jg_device_sync(dev) == JG_ETIMEDOUT
