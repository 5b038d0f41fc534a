"""The host side of the request loop and of the launch plans, without a GPU:
the engine's host sources are compiled against a stand-in for the CUDA runtime
(host/fake_runtime.cpp), whose solves only take time."""
import ctypes as C
import glob
import os
import subprocess
import threading
import time

import numpy as np
import pytest

from svmb200.datagen import CSR
from svmb200.lib import Engine, EngineError, Server, make_params

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


@pytest.mark.parametrize("form", [0, 1, 3])
def test_a_request_that_waits_for_blocks_is_passed_and_uploaded_once(host, form):
    """140 of 148 blocks are at work; the next request's 60000 positions need
    more than the other 8.  A small request that comes later does not wait for
    it, and the waiting one's rows go to the device once."""
    long, wide, small = _rows(14000), _rows(60000), _rows(500)
    prm = make_params(gamma=1.0, cache_mb=10.0, form=form)
    host.lib.fake_us_per_row(30)
    loop = Server(host, max_inflight=4, rows_per_block=100, form=form)
    try:
        alone = 0
        for p in (long, wide, small):
            host.lib.fake_us_per_row(0)
            host.lib.fake_h2d_bytes()
            loop.wait(loop.submit(p, prm))
            alone += host.lib.fake_h2d_bytes()
        host.lib.fake_us_per_row(30)
        t_long = loop.submit(long, prm)
        while not host.lib.fake_h2d_bytes():
            time.sleep(0.001)
        t_wide = loop.submit(wide, prm)
        time.sleep(0.02)
        t_small = loop.submit(small, prm)
        loop.wait(t_small)
        assert not loop.done(t_long) and not loop.done(t_wide)
        host.lib.fake_us_per_row(0)
        assert loop.wait(t_wide)[1]["iters"] == 60000 and loop.done(t_long)
        loop.wait(t_long)
    finally:
        host.lib.fake_us_per_row(1)
        loop.close()
    assert host.lib.fake_h2d_bytes() <= alone


def test_a_request_too_large_for_the_device_fails_alone(host):
    first, huge, large = _rows(500), _rows(900000, 1), _rows(300000, 1)
    prm = make_params(gamma=1.0, cache_mb=10.0)
    host.lib.fake_us_per_row(100)
    loop = Server(host, max_inflight=1, policy=1)       # arrival order: the two that wait are taken together
    try:
        tickets = [loop.submit(p, prm) for p in (first, huge, large)]
        loop.wait(tickets[0])
        host.lib.fake_us_per_row(0)
        with pytest.raises(EngineError, match="too large"):
            loop.wait(tickets[1])
        assert loop.wait(tickets[2])[1]["iters"] == 300000
    finally:
        host.lib.fake_us_per_row(1)
        loop.close()


def test_a_request_too_large_for_the_device_fails_also_when_it_waited(host):
    p, huge = _rows(14000), _rows(900000, 1)
    prm = make_params(gamma=1.0, cache_mb=10.0)
    host.lib.fake_us_per_row(10)
    loop = Server(host, rows_per_block=100)
    try:
        t = loop.submit(p, prm)
        while loop.stats()["waves"] < 1:
            time.sleep(0.001)
        with pytest.raises(EngineError, match="too large"):
            loop.wait(loop.submit(huge, prm))
        assert loop.done(t) and loop.wait(t)[1]["iters"] == 14000
    finally:
        host.lib.fake_us_per_row(1)
        loop.close()


@pytest.mark.parametrize("form,inflight", [(0, 4), (0, 1), (3, 4), (4, 1)])
def test_the_loop_does_not_wait_for_the_device(host, form, inflight):
    """A call that waits (a synchronisation, or an allocation or a release that
    is not stream-ordered) would hold every request up behind whatever runs, and
    so would memory that becomes another request's only when a launch ends."""
    prm = make_params(gamma=1.0, cache_mb=10.0, form=form)
    loop = Server(host, max_inflight=inflight, form=form)
    host.lib.fake_us_per_row(5)
    try:
        host.lib.fake_waits()
        host.lib.fake_frees_behind_a_launch()
        tickets = [(n, loop.submit(_rows(n), prm)) for n in (500, 3000, 700, 9000, 1900, 12000)]
        for n, t in tickets:
            alpha, st, _ = loop.wait(t)
            assert st["iters"] == n and np.array_equal(np.abs(alpha), np.ones(n))
        assert host.lib.fake_waits() == 0
        assert host.lib.fake_frees_behind_a_launch() == 0
    finally:
        host.lib.fake_us_per_row(1)
        loop.close()


@pytest.mark.parametrize("form", [0, 1, 3])
def test_sparse_rows_of_every_width_are_taken(host, form):
    """The staging of sparse sources leaves room for a block's positions at every
    width between the ones that are scattered eight at a time and the table's."""
    refused = []
    for d in range(500, 30000, 250):
        p = CSR(np.arange(101, dtype=np.int64) * 2, np.tile(np.array([1, d]), 100), np.ones(200), np.where(np.arange(100) % 2, 1.0, -1.0), d)
        for cache_mb in (100.0, 0.001):     # evaluated ahead, and by row passes
            try:
                host.solve_binary(p, make_params(gamma=1.0, cache_mb=cache_mb, form=form))
            except EngineError as e:
                refused.append((d, cache_mb, str(e)))
    assert not refused


def test_instances_that_queue_stay_one_launch_of_clusters(host):
    """The matrices of 330 instances are weighed against the whole launch, in which
    they wait for room, not against the longest of them."""
    host.lib.fake_us_per_row(0)
    p = _rows(500, 64)
    inst = [np.arange(500, dtype=np.int32)] * 330
    host.lib.fake_cluster_launches()
    host.lib.fake_general_launches()
    _, st = host.solve_many(p, inst, [p.y] * 330, [make_params(gamma=1.0 / 64)] * 330)
    host.lib.fake_us_per_row(1)
    assert host.lib.fake_cluster_launches() == 1 and host.lib.fake_general_launches() == 0
    assert {s["launch"] for s in st} == {0}
