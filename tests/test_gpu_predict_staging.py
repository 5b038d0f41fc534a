"""Test rows go to the device through ordinary memory in a program's first call
of a size and through kept page-locked memory afterwards: the same values either
way, in either order of sizes, for dense, sparse and split rows."""
import numpy as np
import pytest

from svmb200 import cabi, datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,form", [("dense", 0), ("sparse", 0), ("dense", 3)])
def test_values_do_not_depend_on_the_staging(engine, rows, form):
    p, te = (datagen.dense_gauss(n=300, n_test=6000, d=40, seed=5) if rows == "dense" else
             datagen.sparse_text(n=300, n_test=6000, d=30000, nnz_mean=30.0, seed=5))
    model = engine.train(p, cabi.make_param(kernel_type=2, gamma=0.05, C_=1.0))
    engine.set_option("predict_form", form)
    try:
        want = np.concatenate([engine.predict(model, te.take(np.arange(k, k + 100)))[1] for k in range(0, te.n, 100)])
        for n in (3000, 3000, 1, 3000, 6000, 6000, 50, 6000):
            np.testing.assert_array_equal(engine.predict(model, te.take(np.arange(n)))[1], want[:n])
    finally:
        engine.set_option("predict_form", 0)
        model.free()
