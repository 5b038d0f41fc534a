"""The request loop (svmb_server_*): continuous batching of independent
binary solves.  Requests submitted while others run are admitted next to
them (concurrent launches); every result must equal the same request solved
alone (the exact form is bit-reproducible, so the check is equality)."""
import subprocess
import sys
import time

import numpy as np
import pytest

from svmb200 import datagen
from svmb200.lib import PKG_DIR, EngineError, Server, make_params

pytestmark = pytest.mark.gpu


def _params(job, form=0):
    return make_params(svm_type=job.svm_type, kernel_type=job.kernel_type, gamma=job.gamma, degree=job.degree,
                       C_pos=job.C, nu=job.nu, cache_mb=40.0, form=form)


def test_results_equal_alone_and_in_the_mix(engine):
    jobs = datagen.serving_mix(n_jobs=14, rate=400.0, n_lo=300, n_hi=6000, seed=11)
    big, _ = datagen.dense_gauss(n=12000, n_test=0, d=64, seed=12, flip=0.05)
    big_prm = make_params(svm_type=0, kernel_type=2, gamma=1.0 / 64, C_pos=10.0, cache_mb=40.0)
    srv = Server(engine, max_inflight=4)
    try:
        t_big = srv.submit(big, big_prm)
        time.sleep(0.02)
        tickets = []
        t0 = time.perf_counter()
        for j in jobs:
            while time.perf_counter() - t0 < j.arrival:
                time.sleep(0.0005)
            tickets.append(srv.submit(j.problem, _params(j)))
        got = [srv.wait(t) for t in tickets]
        got_big = srv.wait(t_big)
        st = srv.stats()
    finally:
        srv.close()
    assert st["completed"] == len(jobs) + 1 and st["failed"] == 0, st
    assert st["max_concurrent_waves"] >= 2, st          # later requests ran next to the large one
    assert 0 < st["p50_s"] <= st["p99_s"] <= st["max_s"]
    for j, (alpha, stats, lat) in zip(jobs, got):
        want, st_want = engine.solve_binary(j.problem, _params(j))
        assert np.array_equal(alpha, want)
        assert stats["iters"] == st_want["iters"] and stats["rho"] == st_want["rho"]
        assert lat > 0
    want_big, _ = engine.solve_binary(big, big_prm)
    assert np.array_equal(got_big[0], want_big)


def test_rejects_a_request_larger_than_the_budget(engine):
    p, _ = datagen.dense_gauss(n=2000, n_test=0, d=16, seed=3)
    srv = Server(engine, mem_bytes=1 << 20)
    try:
        t = srv.submit(p, make_params(svm_type=0, kernel_type=2, gamma=1.0 / 16, C_pos=1.0))
        with pytest.raises(EngineError, match="budget"):
            srv.wait(t)
    finally:
        srv.close()


def test_a_request_waits_for_the_blocks_its_state_needs(engine):
    """A request whose positions need more blocks than the running launches
    leave free waits for them: 140 of the blocks are taken by the first, and the
    second's 60000 positions need more than the other 8."""
    long, _ = datagen.dense_gauss(n=14000, n_test=0, d=32, seed=21, flip=0.05)
    long_prm = make_params(svm_type=0, kernel_type=2, gamma=1.0 / 32, C_pos=10.0, cache_mb=40.0)
    wide, _ = datagen.dense_gauss(n=60000, n_test=0, d=4, seed=22, flip=0.05)
    wide_prm = make_params(svm_type=0, kernel_type=2, gamma=0.25, C_pos=0.01, eps=0.5, cache_mb=40.0)
    srv = Server(engine, max_inflight=4, rows_per_block=100)
    try:
        t_long = srv.submit(long, long_prm)
        time.sleep(0.1)
        t_wide = srv.submit(wide, wide_prm)
        got = srv.wait(t_wide), srv.wait(t_long)
        st = srv.stats()
    finally:
        srv.close()
    assert st["completed"] == 2 and st["failed"] == 0, st
    assert np.array_equal(got[0][0], engine.solve_binary(wide, wide_prm)[0])
    assert np.array_equal(got[1][0], engine.solve_binary(long, long_prm)[0])


FIRST_DENSE = """
import sys, time
sys.path.insert(0, sys.argv[1])
from svmb200 import datagen
from svmb200.lib import Engine, Server, make_params
eng = Engine()
form = int(sys.argv[2])
long, _ = datagen.sparse_text(n=12000 if form == 0 else 8000, n_test=0, d=2000, seed=31)
small, _ = datagen.dense_gauss(n=500, n_test=0, d=16, seed=32)
srv = Server(eng, form=form)
more = dict(C_pos=30.0, eps=1e-4) if form == 0 else dict(C_pos=4.0)     # several seconds
t_long = srv.submit(long, make_params(gamma=0.5, cache_mb=0.5, form=form, **more))
while srv.stats()["waves"] < 1:
    time.sleep(0.001)
time.sleep(0.02)
srv.wait(srv.submit(small, make_params(gamma=1.0 / 16, form=form)))
print("long one done:", srv.done(t_long))
srv.wait(t_long)
srv.close()
"""


@pytest.mark.parametrize("form", [0, 3])
def test_the_first_dense_request_does_not_wait_for_a_running_solve(engine, form):
    """In a new process: the kernels of the dense rows' upload are loaded when the
    loop is made, not by its first dense request (a load waits for what runs)."""
    out = subprocess.run([sys.executable, "-c", FIRST_DENSE, PKG_DIR, str(form)], capture_output=True, text=True, timeout=250)
    assert out.returncode == 0, out.stderr
    assert "long one done: False" in out.stdout


def test_dense_and_sparse_requests_of_both_formulations_in_one_launch(engine):
    """At the default cache size every one of these is resident; with one launch
    at a time, those that come during the first are taken into the second."""
    ps = [datagen.dense_gauss(n=900 + 37 * k, n_test=0, d=24, seed=50 + k)[0] if k % 2 else
          datagen.sparse_text(n=950 + 61 * k, n_test=0, d=300, nnz_mean=15.0, seed=60 + k)[0] for k in range(8)]
    prm = [make_params(svm_type=k // 2 % 2, kernel_type=1 + k // 4 % 2, gamma=0.3, nu=0.2) for k in range(8)]
    first, _ = datagen.dense_gauss(n=9000, n_test=0, d=64, seed=70)
    srv = Server(engine, max_inflight=1)
    try:
        t_first = srv.submit(first, make_params(gamma=1.0 / 64, C_pos=10.0, cache_mb=40.0))
        while srv.stats()["waves"] < 1:
            time.sleep(0.0005)
        got = [srv.wait(t) for t in [srv.submit(p, q) for p, q in zip(ps, prm)]]
        srv.wait(t_first)
        assert srv.stats()["waves"] == 2
    finally:
        srv.close()
    for p, q, (alpha, st, _) in zip(ps, prm, got):
        want, st_want = engine.solve_binary(p, q)
        assert np.array_equal(alpha, want) and st["iters"] == st_want["iters"] and st["rho"] == st_want["rho"]
        assert st["fills"] == 0
