"""Sparse rows declared wider than their last column: how sources are staged
depends on the width, results may not."""
import dataclasses

import numpy as np
import pytest

from svmb200 import datagen
from svmb200.lib import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [3200, 6500, 9000, 13500])    # four and two sources scattered, and the table
@pytest.mark.parametrize("cache_mb", [100.0, 0.5])          # evaluated ahead, and by row passes
def test_width_does_not_change_results(engine, d, cache_mb):
    p, _ = datagen.sparse_text(n=1300, n_test=0, d=2000, seed=41)
    prm = make_params(gamma=0.5, C_pos=4.0, cache_mb=cache_mb)
    want, st_want = engine.solve_binary(p, prm)
    got, st = engine.solve_binary(dataclasses.replace(p, d=d), prm)
    assert np.array_equal(got, want)
    assert st["iters"] == st_want["iters"] and st["rho"] == st_want["rho"]
