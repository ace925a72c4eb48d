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


def torch_steps(spec, x, ins, rates, dt, steps):
    """rk4 of step_batch on torch float64 tensors, for autograd."""
    import torch

    read = {"oxygen": ins[:, 0].clamp(0, 1), "egf": ins[:, 1], "crowding": ins[:, 2].clamp(0, 1)}
    read.update({s: ins[:, q].clamp(min=0) for q, s in enumerate(SOURCES) if q > 2})

    def f(z):
        out, t = [], 0
        for i, node in enumerate(spec["nodes"]):
            own, rate = z[:, i], torch.zeros_like(z[:, 0])
            for term in node["terms"]:
                k, kind, src = rates[t], term["kind"], term.get("source")
                t += 1
                s = None if src is None else read[src] if src in read else z[:, int(src[1:])]
                if "hill" in term:
                    n, half = term["hill"]["n"], term["hill"]["k"]
                    sn = s.clamp(min=0) ** n
                    s = sn / (half ** n + sn)
                th = term.get("threshold", 1.0)
                rate = rate + {"activated_by": lambda: k * s * (1 - own), "inhibited_by": lambda: -k * s * own,
                               "activated_by_absence_of": lambda: k * (1 - s) * (1 - own),
                               "produced_by": lambda: k * s, "decays": lambda: -k * own,
                               "relaxes_to": lambda: -k * (own - term["value"]),
                               "damaged_below": lambda: -k * ((th - s) / th).clamp(min=0),
                               "damaged_above": lambda: -k * ((s - th) / th).clamp(min=0)}[kind]()
            out.append(rate)
        return torch.stack(out, 1)

    for _ in range(steps):
        k1 = f(x)
        k2 = f(x + 0.5 * dt * k1)
        k3 = f(x + 0.5 * dt * k2)
        k4 = f(x + dt * k3)
        x = (x + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)).clamp(0, 1)
    return x


# one cell, a block and one more; a block's last warp without a node (7), the
# oxygen's list on the first warp (8) and past the sixteenth (17)
@pytest.mark.parametrize("S,n,steps", [(1, 1, 1), (7, 33, 3), (8, 32, 2), (9, 65, 3), (17, 40, 2), (32, 31, 2)])
def test_the_backward_step_is_the_derivative_of_the_forward(S, n, steps):
    import torch

    spec = spec_of(S)
    net = cw.Network.from_spec(spec, 64)
    rng = np.random.default_rng(7)
    st, (_, ins) = rng.uniform(0.2, 0.8, (n, S)), cells_of(n, S)
    w = rng.normal(size=(n, S))
    flat = [t["rate"] for nd in spec["nodes"] for t in nd["terms"]]
    nr = min(len(flat), 32)
    adj, d_o2, d_rates = net.backward_batch(st, ins, 0.02, steps, w, nrates=nr)
    x, i, k = (torch.tensor(v, dtype=torch.float64, requires_grad=True) for v in (st, ins, flat))
    (torch_steps(spec, x, i, k, 0.02, steps) * torch.tensor(w)).sum().backward()
    # float64 throughout: a few hundred roundings of 1e-16 of numbers up to some tens
    np.testing.assert_allclose(adj, x.grad.numpy(), rtol=1e-10, atol=1e-12)
    np.testing.assert_allclose(d_o2, i.grad.numpy()[:, 0], rtol=1e-10, atol=1e-12)
    np.testing.assert_allclose(d_rates, k.grad.numpy()[:nr], rtol=1e-10, atol=1e-12 * n)


# the memory a network keeps: grown, shrunk into, past what is kept (64 MB), and
# taken by two threads at a time
def test_batches_of_any_size_share_a_networks_memory():
    import threading

    S = 8
    net = cw.Network.from_spec(spec_of(S), 64)
    st, ins = cells_of(650_000, S)

    def step(n):
        x = st[:n].copy()
        return net.step_batch(x, ins[:n], 0.05, 1)

    whole = step(650_000)
    for n in (10, 40_000, 1, 650_000, 33):
        np.testing.assert_array_equal(step(n).view(np.uint64), whole[:n].view(np.uint64))
    out = {}

    def many(k):
        out[k] = [step(2_000 * (k + 1)) for _ in range(10)]

    threads = [threading.Thread(target=many, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(4):
        for x in out[k]:
            np.testing.assert_array_equal(x.view(np.uint64), whole[:2_000 * (k + 1)].view(np.uint64))
