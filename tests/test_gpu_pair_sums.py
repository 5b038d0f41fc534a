"""Decision values of a batch (a thread walks all SVs for a row) against those of
single rows (a block per sum): both add a pair's terms in model order, so they
are identical, for any number of classes and rows that fill no block."""
import numpy as np
import pytest

from svmb200 import cabi, datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("classes,n", [(2, 20001), (3, 9000), (5, 4000), (6, 4001), (10, 2100), (14, 1500), (12, 65)])
def test_batches_match_single_rows(engine, classes, n):
    tr, te, _ = datagen.multiclass_geo(n_classes=classes, largest=150, ratio=0.9, d=12, seed=classes, n_test_frac=0.3)
    model = engine.train(tr, cabi.make_param(kernel_type=2, gamma=0.2, C_=2.0))
    rows = te.take(np.arange(n) % te.n)
    label, dec = engine.predict(model, rows)
    for i in (0, 1, n // 2, n - 1):
        lab1, dec1 = engine.predict_one(model, rows, i)
        np.testing.assert_array_equal(dec1, dec[i])
        assert lab1 == label[i]
    np.testing.assert_array_equal(dec[te.n:], dec[:max(n - te.n, 0)])
    model.free()


def test_one_group_of_svs(engine):
    """Regression and one-class models: one group of SVs, longer than a piece."""
    p, te = datagen.regression(n=1500, n_test=20000, d=6, seed=5)
    for svm_type in (2, 3):
        model = engine.train(p, cabi.make_param(svm_type=svm_type, kernel_type=2, gamma=0.2, C_=4.0, p=0.01, nu=0.9))
        assert model.contents.l > 1024
        _, dec = engine.predict(model, te)
        for i in (0, 19999):
            _, one = engine.predict_one(model, te, i)
            np.testing.assert_array_equal(one, dec[i])
        model.free()
