"""Whole kernel matrices evaluated before the solve (a cache with a slot for
every variable) against rows evaluated during it (a cache too small for that).
Both evaluate the same expressions in the same order, so the coefficients and
the iteration counts must be identical, at tile edges, at widths with a partial
last slice, and for every kind of rows and form."""
import numpy as np
import pytest

from svmb200 import datagen
from svmb200.lib import FORM_EXACT, FORM_FP16X3, FORM_FP32, FORM_TF32, make_params

pytestmark = pytest.mark.gpu


def _same(engine, p, **more):
    n = p.n * (2 if more.get("svm_type") in (3, 4) else 1)
    small = make_params(cache_mb=4.0 * n * max(4, n // 3) / (1 << 20), **more)
    a, sa = engine.solve_binary(p, small)
    b, sb = engine.solve_binary(p, make_params(cache_mb=100.0, **more))
    assert sb["fills"] == 0 and sa["fills"] > 0
    assert sa["iters"] == sb["iters"]
    np.testing.assert_array_equal(a, b)
    assert sa["rho"] == sb["rho"] and sa["obj"] == sb["obj"]


@pytest.mark.parametrize("form", [FORM_EXACT, FORM_FP32, FORM_FP16X3, FORM_TF32])
@pytest.mark.parametrize("n,d", [(9, 1), (63, 4), (64, 16), (65, 17), (129, 70), (1030, 33)])
def test_dense(engine, n, d, form):
    p, _ = datagen.dense_gauss(n=n, n_test=0, d=d, seed=n + d)
    _same(engine, p, kernel_type=2, gamma=1.0 / d, C_pos=2.0, form=form)


@pytest.mark.parametrize("kernel", [0, 1, 2, 3])
@pytest.mark.parametrize("d", [150, 20000])
def test_sparse_rows_and_kernels(engine, d, kernel):
    p, _ = datagen.sparse_text(n=203, n_test=0, d=d, nnz_mean=12.0, seed=d + kernel)
    _same(engine, p, kernel_type=kernel, gamma=0.4, coef0=0.5, C_pos=2.0)


@pytest.mark.parametrize("svm_type", [1, 2, 3, 4])
def test_formulations(engine, svm_type):
    p, _ = (datagen.regression(n=150, n_test=0, d=7, seed=3) if svm_type >= 3 else
            datagen.dense_gauss(n=300, n_test=0, d=12, seed=4))
    _same(engine, p, svm_type=svm_type, kernel_type=2, gamma=0.1, nu=0.3, C_pos=2.0)


@pytest.mark.parametrize("n,kind,more", [
    (65, "dense", {}), (130, "dense", dict(form=FORM_FP32)), (1301, "dense", {}), (1024, "dense", dict(svm_type=1, nu=0.3)),
    (260, "sparse", dict(kernel_type=1)), (777, "wide", {}), (301, "wide", dict(svm_type=1, nu=0.2)), (90, "regression", dict(svm_type=3))])
def test_triangles(engine, n, kind, more):
    """A cache with room for half of the matrix: its lower triangle, against rows evaluated during the solve."""
    if kind == "dense":
        p, _ = datagen.dense_gauss(n=n, n_test=0, d=19, seed=n)
    elif kind == "regression":
        p, _ = datagen.regression(n=n, n_test=0, d=5, seed=n)
    else:
        p, _ = datagen.sparse_text(n=n, n_test=0, d=120 if kind == "sparse" else 20000, nnz_mean=15.0, seed=n)
    l = 2 * n if more.get("svm_type") == 3 else n
    prm = dict(kernel_type=2, gamma=0.2, C_pos=2.0)
    prm.update(more)
    mb = lambda rows: 4.0 * l * (rows + 0.5) / (1 << 20)
    a, sa = engine.solve_binary(p, make_params(cache_mb=mb(l // 3), **prm))
    b, sb = engine.solve_binary(p, make_params(cache_mb=mb((l + 2) // 2), **prm))
    assert sa["fills"] > 0 and sb["fills"] == 0
    assert sa["iters"] == sb["iters"]
    np.testing.assert_array_equal(a, b)
    assert sa["rho"] == sb["rho"] and sa["obj"] == sb["obj"]


def test_instances_of_one_launch(engine):
    """Uneven instances over shared rows: tiles of several matrices in one grid."""
    p, _ = datagen.dense_gauss(n=400, n_test=0, d=20, seed=9)
    rng = np.random.default_rng(1)
    rows = [np.sort(rng.choice(p.n, m, replace=False)).astype(np.int32) for m in (70, 64, 301, 9)]
    ys = [p.y[r] for r in rows]
    prm = make_params(kernel_type=2, gamma=0.05)
    got, _ = engine.solve_many(p, rows, ys, [prm] * len(rows))
    for r, y, a in zip(rows, ys, got):
        want, _ = engine.solve_binary(p.take(r), make_params(kernel_type=2, gamma=0.05, cache_mb=1e-3), y=y)
        np.testing.assert_array_equal(a, want)


@pytest.mark.parametrize("n,more", [(3001, dict(svm_type=1, nu=0.3)), (4001, {}), (5117, dict(svm_type=1, nu=0.2)),
                                    (4100, dict(form=FORM_FP16X3)), (2100, dict(svm_type=3, C_pos=1.0))])
def test_clusters_of_8_and_16_blocks(engine, n, more):
    p, _ = (datagen.regression(n=n, n_test=0, d=5, seed=n) if more.get("svm_type") == 3 else
            datagen.dense_gauss(n=n, n_test=0, d=10, seed=n))
    _same(engine, p, **dict(dict(kernel_type=2, gamma=0.1, C_pos=2.0), **more))


@pytest.mark.parametrize("n,more", [(7300, {}), (7001, dict(svm_type=1, nu=0.2))])
def test_triangles_on_16_blocks(engine, n, more):
    test_triangles(engine, n, "dense", more)


def test_more_blocks_than_positions(engine):
    """9 rows launched beside 5,000, on 16 blocks as these."""
    p, _ = datagen.dense_gauss(n=5000, n_test=0, d=20, seed=9)
    rows = [np.sort(np.random.default_rng(1).choice(p.n, 9, replace=False)).astype(np.int32), np.arange(p.n, dtype=np.int32)]
    ys = [p.y[r] for r in rows]
    prm = make_params(kernel_type=2, gamma=0.05)
    got, st = engine.solve_many(p, rows, ys, [prm] * 2)
    assert [s["launch"] for s in st] == [0, 0]
    for r, y, a in zip(rows, ys, got):
        want, _ = engine.solve_binary(p.take(r), make_params(kernel_type=2, gamma=0.05, cache_mb=0.1), y=y)
        np.testing.assert_array_equal(a, want)
