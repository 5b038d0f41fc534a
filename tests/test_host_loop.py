"""The host side of the request loop and of the launch plans, without a GPU:
the engine's host sources are compiled against a stand-in for the CUDA runtime
(host/fake_runtime.cpp), whose solves only take time."""
import ctypes as C
import glob
import os
import subprocess
import threading

import numpy as np
import pytest

from svmb200.datagen import CSR
from svmb200.lib import Engine, Server, make_params

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "libsvm-cuda_b200")
CUDA = os.environ.get("CUDA", "/usr/local/cuda")


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("host") / "libsvm_b200_host.so")
    src = [s for s in glob.glob(os.path.join(PKG, "csrc", "*.cpp")) if not s.endswith("_main.cpp")]
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I" + os.path.join(PKG, "..", "include"),
                           "-I" + os.path.join(PKG, "csrc"), "-I" + os.path.join(CUDA, "include"),
                           os.path.join(HERE, "host", "fake_runtime.cpp"), *src, "-o", so, "-lpthread"])
    eng = Engine(so)
    eng.set_option("autotune", 0)
    eng.lib.fake_h2d_bytes.restype = C.c_longlong
    eng.lib.fake_us_per_row.argtypes = [C.c_longlong]
    yield eng
    eng.lib.fake_us_per_row(1)


def _rows(n, d=4):
    """n dense rows; the labels alternate."""
    return CSR(np.arange(n + 1, dtype=np.int64) * d, np.tile(np.arange(1, d + 1), n).astype(np.int64), np.ones(n * d),
               np.where(np.arange(n) % 2, 1.0, -1.0), d)


def test_launches_of_two_loops_and_a_call_fit_the_device(host):
    """Blocks of a general launch wait for one another, so launches at work
    together may not have more blocks than the device has SMs (148)."""
    p, prm = _rows(14000), make_params(gamma=1.0, cache_mb=10.0)
    host.lib.fake_peak_blocks()
    host.lib.fake_general_launches()
    loops = [Server(host, rows_per_block=100) for _ in range(2)]
    call = threading.Thread(target=host.solve_binary, args=(p, prm))
    try:
        tickets = [s.submit(p, prm) for s in loops]
        call.start()
        got = [s.wait(t) for s, t in zip(loops, tickets)]
        call.join()
    finally:
        for s in loops:
            s.close()
    assert [st["iters"] for _, st, _ in got] == [14000, 14000]
    assert host.lib.fake_general_launches() == 3
    assert host.lib.fake_peak_blocks() <= 148
