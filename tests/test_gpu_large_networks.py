"""Networks of thousands of terms (GPU): the forward and the backward step at the
counts where a block's shared memory takes another layout, and at the last that
are accepted, against the closed form of a linear network.
"""
import numpy as np
import pytest

import cellweave_b200 as cw

pytestmark = pytest.mark.gpu

DT, STEPS = 0.05, 2


def network(S, nterms):
    """Node i: produced by oxygen and by itself, decaying, a third of its terms each."""
    kinds = [{"kind": "produced_by", "source": "oxygen", "rate": 1e-4}, {"kind": "decays", "rate": 2e-4},
             {"kind": "produced_by", "source": None, "rate": 1e-4}]
    nodes, left = [], nterms
    for i in range(S):
        n = left // (S - i)
        left -= n
        terms = [dict(kinds[q % 3]) for q in range(n)]
        for t in terms:
            if t.get("source", 0) is None:
                t["source"] = f"n{i}"
        nodes.append({"name": f"n{i}", "initial": 0.1, "terms": terms})
    spec = {"nodes": nodes, "roles": {"growth": "n0", "survival": "n0", "hypoxia_response": "n0"},
            "mechanics": {"growth_coefficient": 1.0, "lambda_volume": 1.0}}
    return cw.Network.from_spec(spec, 64), spec


def expected(spec, x, o2, w):
    """x' = B o2 - A x a node: RK4's polynomials, their slopes in x, o2 and the rates."""
    out, back, d_o2, d_rates = np.empty_like(x), np.empty_like(x), np.zeros(len(x)), []
    for i, node in enumerate(spec["nodes"]):
        B = sum(t["rate"] for t in node["terms"] if t.get("source") == "oxygen")
        A = sum(t["rate"] * (1.0 if t["kind"] == "decays" else -1.0) for t in node["terms"]
                if t.get("source") != "oxygen")

        def step(A):
            z = -A * DT
            return 1 + z + z**2 / 2 + z**3 / 6 + z**4 / 24, DT * (1 + z / 2 + z**2 / 6 + z**3 / 24)

        R, Q = step(A)
        geo = sum(R**k for k in range(STEPS))
        out[:, i] = R**STEPS * x[:, i] + Q * B * o2 * geo
        back[:, i] = w[:, i] * R**STEPS
        d_o2 += w[:, i] * Q * B * geo
        # the first rates of a node's kinds; those of x by a central difference in A
        h = 1e-4
        def final(A):
            R, Q = step(A)
            return R**STEPS * x[:, i] + Q * B * o2 * sum(R**k for k in range(STEPS))
        dA = (w[:, i] * (final(A + h) - final(A - h)) / (2 * h)).sum()
        per = {"oxygen": (w[:, i] * Q * o2 * geo).sum(), None: dA, f"n{i}": -dA}
        d_rates += [per[t.get("source")] for t in node["terms"]]
    return out, back, d_o2, np.array(d_rates)


def cells(S, n=40):
    rng = np.random.default_rng(S)
    ins = np.zeros((n, 6))
    ins[:, 0] = rng.uniform(0.2, 0.8, n)
    return rng.uniform(0.2, 0.8, (n, S)), ins, rng.normal(size=(n, S))


# one node's terms in shared memory up to 4,789, where they are up to 4,799
@pytest.mark.parametrize("S,nterms", [(1, 4788), (1, 4789), (1, 4790), (1, 4799), (2, 4748), (32, 3400)])
def test_forward(S, nterms):
    net, spec = network(S, nterms)
    x, ins, w = cells(S)
    want = expected(spec, x, ins[:, 0], w)[0]
    # sums of a few thousand terms, float64
    np.testing.assert_allclose(net.step_batch(x.copy(), ins, DT, STEPS), want, rtol=1e-11)


# whole lists up to 4,238 (one node), 4,194 (two), 4,149 (three) terms with 32 rates
@pytest.mark.parametrize("S,nterms", [(1, 4237), (1, 4239), (1, 4394), (2, 4287), (3, 4180), (4, 4073), (32, 1080)])
def test_backward(S, nterms):
    net, spec = network(S, nterms)
    x, ins, w = cells(S)
    _, back, d_o2, d_rates = expected(spec, x, ins[:, 0], w)
    got = net.backward_batch(x, ins, DT, STEPS, w, nrates=32)
    np.testing.assert_allclose(got[0], back, rtol=1e-11)
    np.testing.assert_allclose(got[1], d_o2, rtol=1e-10, atol=1e-12)
    # (a central difference of 1e-4: 1e-8 of a third derivative near 1e-3, and rounding / 1e-4)
    np.testing.assert_allclose(got[2], d_rates[:32], rtol=1e-8, atol=1e-9)


def test_what_was_refused_is_refused():
    with pytest.raises(cw.ConfigError):
        network(1, 4800)
    net, _ = network(1, 4395)
    x, ins, w = cells(1)
    with pytest.raises(cw.ConfigError):
        net.backward_batch(x, ins, DT, STEPS, w, nrates=1)
