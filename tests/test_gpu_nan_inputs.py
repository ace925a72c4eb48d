"""The backward step of a cell whose input is not a number (GPU): what a Hill
response of it reaches is not a number either, and no other cell is touched."""
import numpy as np
import pytest

import cellweave_b200 as cw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["activated_by", "inhibited_by"])
@pytest.mark.parametrize("n", [2.0, 3.5])
def test_a_gradient_through_a_hill_response_of_nan_is_nan(kind, n):
    spec = {"nodes": [{"name": "a", "initial": 0.1, "terms": [
        {"kind": kind, "source": "egf", "rate": 0.7, "hill": {"n": n, "k": 0.5}}, {"kind": "decays", "rate": 0.3}]}],
        "roles": {"growth": "a", "survival": "a", "hypoxia_response": "a"},
        "mechanics": {"growth_coefficient": 1.0, "lambda_volume": 1.0}}
    net = cw.Network.from_spec(spec, 64)
    ins = np.zeros((3, 6))
    ins[:, 1] = 0.4, np.nan, 0.0
    back, _, d_rates = net.backward_batch(np.full((3, 1), 0.5), ins, 0.05, 2, np.ones((3, 1)), nrates=2)
    assert np.isnan(back[1, 0]) and np.isfinite(back[[0, 2], 0]).all()
    assert np.isnan(d_rates[0])
