"""The cost model on more rows than 65,535 tiles of 32 hold."""

import numpy as np
import pytest

from bitstreamzoo_b200 import tuner

import mlp_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65_535 * 32 + 1, 2_500_000])
def test_predictions_of_millions_of_rows(ctx, n):
    m = tuner.CostModel(ctx, 5, hidden=8, layers=1, seed=3)
    rng = np.random.default_rng(n)
    x = rng.normal(0, 1, (n, 5)).astype(np.float32)
    ref = mlp_ref.forward(m.params(), mlp_ref.dims_of(5, 8, 1), x)[-1][:, 0]
    np.testing.assert_allclose(m.raw_predict(x), ref, rtol=1e-4, atol=1e-5)
