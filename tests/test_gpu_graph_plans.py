"""A simulation whose steps are replayed from CUDA graphs and whose lattice is
given another contact order or copy neighbourhood between two steps (GPU): the
sweeps' plan and scratch are made anew, and the steps are those of a simulation
that captures nothing.
"""
import os
import tempfile

import numpy as np
import pytest

import cellweave_b200 as cw
from cellweave_b200 import synthetic

pytestmark = pytest.mark.gpu


def network():
    p = os.path.join(tempfile.mkdtemp(), "n.toml")
    open(p, "w").write(synthetic.network_toml(8, seed=8))
    return cw.Network.load(p, 49)


# order 1 has the most pixels a colour (and so the largest scratch), order 3 the fewest
@pytest.mark.parametrize("orders", [(3, 1), (2, 1), (1, 3), (2, "copies")])
def test_a_lattice_set_anew_between_captured_steps(orders):
    net = network()
    cfg = synthetic.campaign(per_size=2, sizes=(96, 128), base_seed=500)
    cfg.pop("S")
    cfg["omega"] = 1.9  # no tuning: the same factors on both
    cfg["contact_order"] = orders[0]
    sims = [cw.Simulation(net, **dict(cfg, use_graphs=g)) for g in (True, False)]
    for s in sims:
        s.step(5)
    assert sims[0].graph_info()[0] > 0
    for s in sims:
        if orders[1] == "copies":
            s.lattice().set_copy_neighbourhood(True)
        else:
            s.lattice().set_contact(cfg["J"], orders[1])
        s.step(12)
    for k in range(len(cfg["dims"])):
        np.testing.assert_array_equal(sims[0].grid(k), sims[1].grid(k))
        assert sims[0].records_match_grid(k)
