"""The RK4 step's split of a cell's nodes over warps (GPU): node counts and
batch sizes at the edges of the dispatch, every kind of term, squares and
powers, against the oracle; the same cells in batches of every split, and as
clones, to the bit.
"""
import numpy as np
import pytest

import cellweave_b200 as cw
from oracle import oracle as O

pytestmark = pytest.mark.gpu

KINDS = ["activated_by", "inhibited_by", "activated_by_absence_of", "produced_by", "damaged_below", "damaged_above"]
SOURCES = ["oxygen", "egf", "crowding", "stress", "waste", "necrotic_factor"]


def spec_of(S):
    rng = np.random.default_rng(S)
    nodes = []
    for i in range(S):
        terms = [{"kind": "decays", "rate": float(rng.uniform(0.1, 1.0))}]
        for q, kind in enumerate(KINDS):
            source = SOURCES[(i + q) % 6] if q % 2 else f"n{(i * 7 + q) % S}"
            t = {"kind": kind, "source": source, "rate": float(rng.uniform(0.1, 1.0))}
            if q < 2 and i % 3:
                t["hill"] = {"n": 2.0 if i % 3 == 1 else 3.5, "k": float(rng.uniform(0.2, 1.0))}
            if kind.startswith("damaged"):
                t["threshold"] = float(rng.uniform(0.2, 0.8))
            terms.append(t)
        terms.append({"kind": "relaxes_to", "rate": 0.3, "value": 0.4})
        nodes.append({"name": f"n{i}", "initial": 0.1, "terms": terms[i % 4:]})
    return {"nodes": nodes, "roles": {"growth": "n0", "survival": "n0", "hypoxia_response": "n0"},
            "mechanics": {"growth_coefficient": 1.0, "lambda_volume": 1.0}}


def cells_of(n, S):
    rng = np.random.default_rng(1)
    return rng.uniform(0, 1, (n, S)), rng.uniform(-0.5, 1.5, (n, 6))


# most cells: past 16 blocks of 32 an SM with up to 8 nodes, past 2 an SM above
@pytest.mark.parametrize("S,most", [(1, 76_000), (7, 76_000), (8, 76_001), (9, 9_600), (17, 9_473), (32, 9_500)])
def test_every_split_of_a_cells_nodes_gives_the_same_bits(S, most):
    spec = spec_of(S)
    net, ref = cw.Network.from_spec(spec, 64), O.compile_network(spec, 64)
    st, ins = cells_of(most, S)
    whole = st.copy()
    net.step_batch(whole, ins, 0.05, 3)
    for n in (1, 31, 33, 700):
        part = st[:n].copy()
        net.step_batch(part, ins[:n], 0.05, 3)
        np.testing.assert_array_equal(part.view(np.uint64), whole[:n].view(np.uint64))
        clones = st[:n].copy()
        cw.Network.step_clones([net, net], np.arange(n) % 2, clones, ins[:n], 0.05, 3)
        np.testing.assert_array_equal(clones.view(np.uint64), part.view(np.uint64))
    pick = np.r_[0:300, most - 300:most]
    want = st[pick].copy()
    O.network_step(ref, want, np.ascontiguousarray(ins[pick]), 0.05, 3)
    # CUDA's pow is within 2 ulp of libm's; three steps of four evaluations
    np.testing.assert_allclose(whole[pick], want, rtol=1e-12, atol=1e-14)
