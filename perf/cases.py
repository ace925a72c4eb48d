"""The work a user of this framework has it do, as cases to be timed.

A case is a dict of plain values; ``prepare`` makes what a user's program
holds before the call, ``run`` is one pass through the public entry points,
``work`` the bytes and operations that the pass cannot do without and
``exact`` the same outputs from plain torch in 64 bits where they are computed
numbers.  Sizes are those of the benchmark's configurations (``synthetic``),
of the configuration runner's scenarios and of the tests, and odd sizes
between them.
"""
from __future__ import annotations

import math
import tomllib

import numpy as np
import torch

import cellweave_b200 as cw
from cellweave_b200 import _lib, config, synthetic

NODES = 8  # species of the plain and campaign networks


def listed():
    return [
        # one plain 2D history: 120 cells, the reference's FP64 solve every ten steps; the smallest launches count
        dict(name="plain-256", kind="plain", n=256, steps=10),
        # the configuration runner's step: tissue in a bath, FP64 solve on the largest change, four sub-sweeps
        dict(name="run-300", kind="run", w=300, h=300, radius=80, steps=4),
        # the batched campaign, the benchmark's workload: 64 histories of uneven sizes, two FP32 solves a step
        dict(name="campaign-64", kind="campaign", per_size=16, sizes="128,256,512,1024", steps=4),
        # the large tumour cord: one history, 40,000 cells, two fields, 16 species
        dict(name="cord-2048", kind="cord", n=2048, steps=4),
        # the 3D spheroid: 26-neighbour contact with surfaces, oxygen in the volume; the largest case
        dict(name="spheroid-256", kind="spheroid", n=256, steps=2),
        # ScalarField.relax as the reference has it: a first FP64 solve around a tissue, odd sides
        dict(name="relax-bath-301", kind="bath", w=301, h=287, d=1, tolerance=1e-8),
        # the same in a small volume
        dict(name="relax-ball-61", kind="bath", w=64, h=61, d=57, tolerance=1e-8),
        # a single FP32 defect-correction solve on a sheet whose rows are not 16-byte aligned
        dict(name="relax-sheet-1023", kind="sheet", w=1023, h=769, tolerance=1e-9),
        # a linear solve for a loss on the field, the backward direction
        dict(name="adjoint-1024", kind="adjoint", w=1024, h=1024, tolerance=1e-10),
        # Monte Carlo steps of a volume's lattice alone, surfaces on
        dict(name="sweeps-96", kind="sweeps", n=96, steps=4),
        # the networks of a cord's cells stepped from host arrays
        dict(name="networks-40k", kind="networks", cells=40000, species=16, substeps=8),
        # and their derivatives, the backward direction
        dict(name="networks-back-8k", kind="networks_back", cells=8192, species=8, substeps=40),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "run", "campaign", "cord", "spheroid", "bath", "ball", "sheet", "adjoint", "sweeps",
                       "networks", "networks_back"])
    if kind == "plain":
        return dict(kind=kind, n=_log(rng, 96, 640), steps=10)
    if kind == "run":
        w, h = _log(rng, 120, 480), _log(rng, 120, 480)
        return dict(kind=kind, w=w, h=h, radius=int(min(w, h) * rng.uniform(0.2, 0.35)), steps=rng.randint(1, 4))
    if kind == "campaign":
        sizes = [_log(rng, 96, 1024) for _ in range(3)]
        if rng.random() < 0.7:  # most campaigns have aligned rows
            sizes = [(s + 15) // 16 * 16 for s in sizes]
        return dict(kind=kind, per_size=rng.randint(1, 12), sizes=",".join(map(str, sizes)), steps=rng.randint(1, 4))
    if kind == "cord":
        n = _log(rng, 300, 2048)
        return dict(kind=kind, n=(n + 15) // 16 * 16 if rng.random() < 0.5 else n, steps=rng.randint(1, 4))
    if kind == "spheroid":
        return dict(kind=kind, n=_log(rng, 96, 256), steps=rng.randint(1, 2))
    if kind == "bath":
        return dict(kind=kind, w=_log(rng, 40, 640), h=_log(rng, 40, 640), d=1,
                    tolerance=10.0 ** -rng.randint(7, 10))
    if kind == "ball":
        return dict(kind="bath", w=_log(rng, 24, 110), h=_log(rng, 24, 110), d=_log(rng, 24, 110),
                    tolerance=10.0 ** -rng.randint(7, 9))
    if kind in ("sheet", "adjoint"):
        w, h = _log(rng, 100, 1400), _log(rng, 100, 1400)
        if rng.random() < 0.5:
            w = (w + 15) // 16 * 16
        return dict(kind=kind, w=w, h=h, tolerance=10.0 ** -rng.randint(8, 10))
    if kind == "sweeps":
        return dict(kind=kind, n=_log(rng, 40, 176), steps=rng.randint(1, 4))
    if kind == "networks":
        return dict(kind=kind, cells=_log(rng, 200, 120000), species=rng.randint(4, 20), substeps=rng.randint(4, 16))
    return dict(kind=kind, cells=_log(rng, 200, 16384), species=rng.randint(4, 16), substeps=rng.randint(10, 60))


# ------------------------------------------------------------------ preparation
def _network(species, refvol):
    return cw.Network.from_spec(tomllib.loads(synthetic.network_toml(species, species)), refvol)


def _pinned(n, dtype):
    t = torch.empty(n, dtype=dtype, pin_memory=True)
    return t, t.numpy()


def _with_buffers(sim, net, fields, steps, **more):
    """The simulation and the pinned host buffers its user reads it back into."""
    total = sum(w * h * d for w, h, d in sim.dims)
    return dict(sim=sim, net=net, steps=steps, grid=_pinned(total, torch.int32),
                fields=[_pinned(total, torch.float64) for _ in range(fields)], **more)


def _simulation(case, seed):
    kind = case["kind"]
    if kind == "plain":
        cfg = synthetic.plain_2d(seed)
        n = case["n"]
        cfg.update(dims=[(n, n, 1)], ncells=[max(4, 120 * n * n // (256 * 256))])
        warm = 10
    elif kind == "campaign":
        cfg = synthetic.campaign(case["per_size"], [int(s) for s in case["sizes"].split(",")],
                                 base_seed=1000 * (seed + 1))
        warm = 12
    elif kind == "cord":
        cfg = synthetic.tumour_cord(case["n"])
        cfg["seeds"] = [seed]
        warm = 12
    else:
        cfg = synthetic.spheroid_3d(case["n"])
        radius = min(40, case["n"] // 4)
        cfg.update(seeds=[seed], ncells=[int(4.0 / 3.0 * math.pi * radius ** 3 / 125)])
        warm = 10
    net = _network(cfg.pop("S"), cfg["target_volume"])
    sim = cw.Simulation(net, **cfg)
    sim.step(warm)  # past the autotuner's trials, as a run of hundreds of steps is
    return _with_buffers(sim, net, cfg["nfields"], case["steps"])


RUN_SIDE = 14   # a cell of the runner's tissue, about the seeded ball's 197 pixels
RUN_UPTAKE = 2e-5


def _run_simulation(case, seed):
    """A tissue as the runner's spheroid scenario grows it, laid out in place:
    squares within `radius` of the box's centre."""
    w, h, s = case["w"], case["h"], RUN_SIDE
    spots = [(x, y) for y in range(0, h - s, s) for x in range(0, w - s, s)
             if (x + s / 2 - w / 2) ** 2 + (y + s / 2 - h / 2) ** 2 <= case["radius"] ** 2]
    net = _network(NODES, s * s)
    sim = cw.Simulation(net, [(w, h, 1)], [len(spots)], [seed], temperature=10.0, J=config.CONTACT, contact_order=1,
                        target_volume=s * s, lambda_volume=1.0, seeding=1, seed_side=s, o2_dcoef=0.2,
                        o2_sink_by_type=(0.0, 0.0, 0.0, 0.0), o2_hold=3, o2_uptake=RUN_UPTAKE,
                        tolerance=0.01 * RUN_UPTAKE, precision=cw.FP64, stop_rule=cw.STOP_MAX_CHANGE, dt=0.05,
                        substeps=8, subsweeps=4, necrotic_type=config.NECROTIC, divide_every=20,
                        first_tolerance=1e-8)
    grid = np.zeros((1, h, w), np.int32)
    for k, (x, y) in enumerate(spots):
        grid[0, y:y + s, x:x + s] = k + 1
    sim.lattice().upload(grid)
    sim.step(8)
    return _with_buffers(sim, net, 1, case["steps"], measure=True)


def _shape(case):
    return case["w"], case["h"], case.get("d", 1)


def _bath_problem(case, seed):
    """A tissue (a disc or ball off the centre, a bite out of it) taking up
    oxygen in a bath held at one: (uptake, bath) as host arrays."""
    w, h, d = _shape(case)
    rng = np.random.default_rng(seed)
    z, y, x = np.ogrid[0:d, 0:h, 0:w]
    sides = [w, h] + ([d] if d > 1 else [])
    r = 0.35 * min(sides)
    cx, cy, cz = (v * (0.5 + 0.04 * float(rng.uniform(-1, 1))) for v in (w, h, d))
    if d == 1:
        cz = 0.0
    tissue = (x - cx) ** 2 + (y - cy) ** 2 + (z - cz) ** 2 <= r * r
    a = float(rng.uniform(0, 2 * math.pi))
    tissue &= (x - cx - r * math.cos(a)) ** 2 + (y - cy - r * math.sin(a)) ** 2 + (z - cz) ** 2 > (0.3 * r) ** 2
    # about a fifth of the supply is used at the centre; rates differ from cell to cell
    rate = (0.2 * (4 if d == 1 else 6) * 0.2 / (r * r)) * rng.uniform(0.5, 1.5, (d, h, w))
    return np.where(tissue, rate, 0.0).reshape(-1), ~tissue.reshape(-1)


def _sheet_problem(case, seed):
    """Cells over a plane as first-order sinks, row 0 held at one: (sink, held)."""
    w, h, _ = _shape(case)
    rng = np.random.default_rng(seed)
    cells = rng.uniform(size=(h // 7 + 1, w // 7 + 1)) < 0.3
    sink = np.kron(cells, np.ones((7, 7)))[:h, :w] * 0.01
    held = np.zeros((h, w), np.uint8)
    held[0] = 1
    return sink.reshape(-1), held.reshape(-1)


def _volume_lattice(case, seed):
    """5^3 cells packed in a ball, surfaces on, as the 3D spheroid's lattice."""
    n, s = case["n"], 5
    radius = 0.42 * n
    grid = np.zeros((n, n, n), np.int32)
    cid = 0
    for z in range(0, n - s + 1, s):
        for y in range(0, n - s + 1, s):
            for x in range(0, n - s + 1, s):
                if (x + 2.5 - n / 2) ** 2 + (y + 2.5 - n / 2) ** 2 + (z + 2.5 - n / 2) ** 2 <= radius * radius:
                    cid += 1
                    grid[z:z + s, y:y + s, x:x + s] = cid
    types = np.random.default_rng(seed).integers(1, 3, cid + 1).astype(np.int32)
    types[0] = 0
    volume = np.full(cid + 1, s ** 3, np.int32)
    volume[0] = 0
    lat = cw.CpmLattice([(n, n, n)], 20.0, [cid + 1], 3, synthetic.two_type_table())
    lat.upload(grid)
    lat.set_cells(types, volume, volume, np.where(volume > 0, 1.0, 0.0))
    lat.set_seed(seed)
    lat.set_surface(np.full(cid + 1, 150, np.int32), np.full(cid + 1, 0.2))
    lat.monte_carlo_step(2)
    return dict(lattice=lat, steps=case["steps"])


def _cells_problem(case, seed):
    rng = np.random.default_rng(seed)
    n, S = case["cells"], case["species"]
    state = rng.uniform(0.05, 0.95, (n, S))
    inputs = np.zeros((n, 6))
    inputs[:, 0] = rng.uniform(0.0, 1.0, n)
    inputs[:, 1] = 0.2
    return state, inputs, rng.normal(size=(n, S))


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("plain", "campaign", "cord", "spheroid"):
        st = _simulation(case, seed)
    elif kind == "run":
        st = _run_simulation(case, seed)
    elif kind == "bath":
        uptake, bath = _bath_problem(case, seed)
        f = cw.ScalarField([_shape(case)], 0.2, 0.0, 1.0)
        f.set_uptake_array(uptake)
        f.hold_bath(1.0, bath)
        st = dict(field=f, tolerance=case["tolerance"])
    elif kind == "sheet":
        sink, held = _sheet_problem(case, seed)
        f = cw.ScalarField([_shape(case)], 1.0, 0.0, 1.0)
        f.set_linear_sink(sink)
        f.set_held(held)
        st = dict(field=f, tolerance=case["tolerance"])
    elif kind == "adjoint":
        sink, held = _sheet_problem(case, seed)
        f = cw.ScalarField([_shape(case)], 1.0, 0.01, 1.0)
        f.set_linear_sink(sink)
        f.set_held(held)
        st = dict(field=f, tolerance=case["tolerance"], dl_dc=_loss_slope(case, seed))
    elif kind == "sweeps":
        st = _volume_lattice(case, seed)
    else:
        state, inputs, adjoint = _cells_problem(case, seed)
        st = dict(net=_network(case["species"], 64), state=state, inputs=inputs, adjoint=adjoint,
                  substeps=case["substeps"])
    st["kind"] = kind
    return st


def _loss_slope(case, seed):
    w, h, _ = _shape(case)
    return np.random.default_rng(seed + 1).normal(size=w * h)


# ------------------------------------------------------------------ one pass
def _read_back(st):
    """The lattice, every field and the histories' statistics, as a snapshot takes them."""
    sim, L = st["sim"], _lib.lib()
    _lib.check(L.cw_lattice_download_all(sim.lattice_handle(), _lib.ptr(st["grid"][1])))
    for which, (_, buf) in enumerate(st["fields"]):
        fh, at = sim.field_handle(which), 0
        for k, (w, h, d) in enumerate(sim.dims):
            n = w * h * d
            _lib.check(L.cw_field_download(fh, k, cw.VALUES, _lib.ptr(buf[at:at + n])))
            at += n
    return dict(grid=st["grid"][0], fields=[t for t, _ in st["fields"]])


def run(st):
    kind = st["kind"]
    if kind in ("plain", "campaign", "cord", "spheroid"):
        st["sim"].step(st["steps"])
        stats = st["sim"].stats()
        # living cells, mean oxygen, hypoxic fraction (the last column is the solve's residual, at rounding level)
        return dict(_read_back(st), living=stats[:, 0], oxygen=stats[:, 1], hypoxic=stats[:, 2],
                    levels=st["sim"].network_state(min(64, st["sim"].lattice().cell_count())))
    if kind == "run":
        measured = None
        for _ in range(st["steps"]):
            st["sim"].step(1)
            measured = st["sim"].measure()[0]
            st["sim"].touches_edge()
        return dict(_read_back(st), counts=[int(v) for v in measured.values() if isinstance(v, int)])
    if kind == "bath":
        f = st["field"]
        f.fill(1.0)
        sweeps = f.relax(st["tolerance"], 200_000)
        return dict(values=f.values(), sweeps=sweeps)
    if kind == "sheet":
        f = st["field"]
        f.fill(1.0)
        f.relax(st["tolerance"], 200_000, omega=1.9, stop=cw.STOP_RESIDUAL, precision=cw.FP32_DC, inner_sweeps=64,
                block_depth=8)
        return dict(values=f.values())
    if kind == "adjoint":
        lam = st["field"].relax_adjoint(st["dl_dc"], st["tolerance"], 200_000, omega=1.9, precision=cw.FP32_DC,
                                        inner_sweeps=32, block_depth=8)
        return dict(adjoint=lam)
    if kind == "sweeps":
        lat = st["lattice"]
        lat.monte_carlo_step(st["steps"])
        return dict(grid=lat.grid(), volume=lat.cells()["volume"], surface=lat.surfaces())
    if kind == "networks":
        state = st["state"].copy()
        return dict(state=st["net"].step_batch(state, st["inputs"], 0.01, st["substeps"]))
    back, d_oxygen, d_rates = st["net"].backward_batch(st["state"], st["inputs"], 0.01, st["substeps"],
                                                       st["adjoint"], nrates=8)
    return dict(back=back, d_oxygen=d_oxygen, d_rates=d_rates)


# ------------------------------------------------------------------ the work that cannot be left out
def _terms(species):
    return sum(len(n["terms"]) for n in tomllib.loads(synthetic.network_toml(species, species))["nodes"])


def work(case):
    """One pass.  A step reads and writes the grid (4 B a site) and each field
    (8 B), its solve reading the held mask and the sink once (9 B); a solve from
    scratch reads its problem and writes its field.  Operations: a cell's RK4
    steps, four evaluations of about eight operations a term (three times
    that backward); a solve's own count depends on how it is done and is left out."""
    kind = case["kind"]
    if kind in ("plain", "campaign", "cord", "spheroid", "run"):
        steps, fields, species = case["steps"], 1, NODES
        if kind == "campaign":
            sites = sum(case["per_size"] * int(s) ** 2 for s in case["sizes"].split(","))
            fields, cells = 2, sites * 0.3 / 49
        elif kind == "cord":
            sites, fields, species = case["n"] ** 2, 2, 16
            cells = sites / 105
        elif kind == "spheroid":
            sites, species = case["n"] ** 3, 12
            cells = 2144
        elif kind == "plain":
            sites = case["n"] ** 2
            cells = 120 * sites / 65536
        else:
            sites = case["w"] * case["h"]
            cells = math.pi * case["radius"] ** 2 / RUN_SIDE ** 2
        return dict(bytes=steps * sites * (8 + fields * (16 + 9)), flops=steps * cells * 8 * 4 * 8 * _terms(species))
    if kind == "bath":
        w, h, d = _shape(case)
        return dict(bytes=w * h * d * (8 + 1 + 8), flops=w * h * d * 9)
    if kind in ("sheet", "adjoint"):
        w, h, _ = _shape(case)
        return dict(bytes=w * h * (8 + 1 + 8 + (8 if kind == "adjoint" else 0)), flops=w * h * 9)
    if kind == "sweeps":
        return dict(bytes=case["steps"] * case["n"] ** 3 * 8, flops=case["steps"] * case["n"] ** 3 * 26)
    n, S, sub = case["cells"], case["species"], case["substeps"]
    back = kind == "networks_back"
    return dict(bytes=n * 8 * ((3 if back else 2) * S + 6 + (1 if back else 0)),
                flops=n * sub * 4 * 8 * _terms(S) * (3 if back else 1))


# ------------------------------------------------------------------ the same outputs in 64 bits
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _neighbours(c):
    """The sum of the real neighbours of every pixel of [d, h, w] and their count."""
    s, n = torch.zeros_like(c), torch.zeros_like(c)
    for axis in range(3):
        m = c.shape[axis]
        if m == 1:
            continue
        lo, hi = [slice(None)] * 3, [slice(None)] * 3
        lo[axis], hi[axis] = slice(0, m - 1), slice(1, m)
        s[tuple(hi)] += c[tuple(lo)]
        s[tuple(lo)] += c[tuple(hi)]
        n[tuple(hi)] += 1
        n[tuple(lo)] += 1
    return s, n


def _exact_bath(case, seed):
    """Red-black successive over-relaxation with the reference's factor and stop."""
    w, h, d = _shape(case)
    uptake, bath = (torch.from_numpy(a).to(_device()).reshape(d, h, w) for a in _bath_problem(case, seed))
    free = ~bath
    if d > 1:
        at = free.nonzero()
        span = int((at.max(0).values - at.min(0).values).max()) + 1
        omega = 2.0 / (1.0 + math.sin(math.pi / max(span, 2)))
    else:
        omega = min(2.0 / (1.0 + math.sin(math.pi / max(w, h))), 1.95)
    z, y, x = (torch.arange(m, device=free.device) for m in (d, h, w))
    parity = (x[None, None, :] + y[None, :, None] + z[:, None, None]) % 2
    c = torch.ones((d, h, w), dtype=torch.float64, device=free.device)
    real = _neighbours(c)[1]
    masks = [free & (parity == k) for k in (0, 1)]
    sweeps = 0
    while sweeps < 200_000:
        moved = []
        for mask in masks:
            s, _ = _neighbours(c)
            after = ((1.0 - omega) * c + omega * ((0.2 * s - uptake) / (real * 0.2))).clamp_min(0.0)
            after = torch.where(mask, after, c)
            moved.append((after - c).abs().max())
            c = after
        sweeps += 1
        if float(max(moved)) < case["tolerance"]:
            break
    return dict(values=c.reshape(-1).cpu(), sweeps=None)


def _conjugate_gradients(diagonal, free, b, dcoef):
    """A x = b on the free pixels of [1, h, w] (A = diagonal - dcoef neighbours), to rounding."""
    x = torch.zeros_like(b)
    r = torch.where(free, b, x)
    inv = torch.where(free, 1.0 / diagonal, x)
    p = inv * r
    rho = (r * p).sum()
    first = float(r.abs().max())
    for k in range(20_000):
        ap = torch.where(free, diagonal * p - dcoef * _neighbours(p)[0], torch.zeros_like(p))
        alpha = rho / (p * ap).sum()
        x = x + alpha * p
        r = r - alpha * ap
        q = inv * r
        new = (r * q).sum()
        p = q + (new / rho) * p
        rho = new
        if k % 20 == 0 and float(r.abs().max()) < 1e-15 * first:
            break
    return x


def _exact_plane(case, seed):
    w, h, _ = _shape(case)
    sink, held = (torch.from_numpy(a).to(_device()).reshape(1, h, w) for a in _sheet_problem(case, seed))
    free = held == 0
    decay = 0.01 if case["kind"] == "adjoint" else 0.0
    ones = torch.ones_like(sink)
    diagonal = _neighbours(ones)[1] + decay + sink
    if case["kind"] == "adjoint":
        b = torch.from_numpy(_loss_slope(case, seed)).to(_device()).reshape(1, h, w)
        return dict(adjoint=_conjugate_gradients(diagonal, free, b, 1.0).reshape(-1).cpu())
    rim = torch.where(free, torch.zeros_like(sink), ones)
    x = _conjugate_gradients(diagonal, free, _neighbours(rim)[0], 1.0)
    return dict(values=torch.where(free, x, ones).reshape(-1).cpu())


class _Network64:
    """The synthetic network's RK4 step on rows of [cells, species], in torch."""

    def __init__(self, species, rates):
        spec = tomllib.loads(synthetic.network_toml(species, species))
        self.index = {n["name"]: i for i, n in enumerate(spec["nodes"])}
        self.nodes, k = [], 0
        for node in spec["nodes"]:
            terms = []
            for t in node["terms"]:
                terms.append((t, rates[k]))
                k += 1
            self.nodes.append(terms)

    def slope(self, x, oxygen, egf):
        out = []
        for i, terms in enumerate(self.nodes):
            own, rate = x[i], 0.0
            for t, k in terms:
                src = t.get("source")
                s = oxygen.clamp(0.0, 1.0) if src == "oxygen" else egf if src == "egf" else \
                    None if src is None else x[self.index[src]]
                if t.get("hill"):
                    u = s.clamp_min(0.0) ** t["hill"]["n"]
                    s = u / (t["hill"]["k"] ** t["hill"]["n"] + u)
                kind = t["kind"]
                rate = rate + (k * s * (1.0 - own) if kind == "activated_by" else
                               -k * s * own if kind == "inhibited_by" else
                               k * (1.0 - s) * (1.0 - own) if kind == "activated_by_absence_of" else
                               -k * own if kind == "decays" else
                               -k * (own - t["value"]) if kind == "relaxes_to" else
                               -k * ((t["threshold"] - s) / t["threshold"]).clamp_min(0.0))
            out.append(rate)
        return torch.stack(out)

    def step(self, x, oxygen, egf, dt):
        k1 = self.slope(x, oxygen, egf)
        k2 = self.slope(x + 0.5 * dt * k1, oxygen, egf)
        k3 = self.slope(x + 0.5 * dt * k2, oxygen, egf)
        k4 = self.slope(x + dt * k3, oxygen, egf)
        return (x + (dt / 6.0) * (k1 + 2.0 * k2 + 2.0 * k3 + k4)).clamp(0.0, 1.0)


def _exact_cells(case, seed):
    state, inputs, adjoint = (torch.from_numpy(a).to(_device()) for a in _cells_problem(case, seed))
    spec = tomllib.loads(synthetic.network_toml(case["species"], case["species"]))
    rates = [torch.tensor(float(t["rate"]), dtype=torch.float64, device=state.device)
             for n in spec["nodes"] for t in n["terms"]]
    back = case["kind"] == "networks_back"
    oxygen, egf = inputs[:, 0].clone(), inputs[:, 1]
    if not back:
        with torch.no_grad():
            net, x = _Network64(case["species"], rates), state.t().contiguous()
            for _ in range(case["substeps"]):
                x = net.step(x, oxygen, egf, 0.01)
        return dict(state=x.t().cpu())
    # the chain rule step by step from the last, each step's own graph made anew
    xs = [state.t().contiguous()]
    net = _Network64(case["species"], rates)
    with torch.no_grad():
        for _ in range(case["substeps"]):
            xs.append(net.step(xs[-1], oxygen, egf, 0.01))
    lam = adjoint.t().contiguous()
    d_oxygen, d_rates = torch.zeros_like(oxygen), torch.zeros(8, dtype=torch.float64, device=state.device)
    lead = [r.clone().requires_grad_(True) for r in rates[:8]]
    net = _Network64(case["species"], lead + rates[8:])
    for x in reversed(xs[:-1]):
        x, o = x.clone().requires_grad_(True), oxygen.clone().requires_grad_(True)
        got = torch.autograd.grad(net.step(x, o, egf, 0.01), [x, o] + lead, lam)
        lam = got[0]
        d_oxygen += got[1]
        d_rates += torch.stack(got[2:])
    return dict(back=lam.t().cpu(), d_oxygen=d_oxygen.cpu(), d_rates=d_rates.cpu())


def exact(case, seed):
    kind = case["kind"]
    if kind == "bath":
        return _exact_bath(case, seed)
    if kind in ("sheet", "adjoint"):
        return _exact_plane(case, seed)
    if kind in ("networks", "networks_back"):
        return _exact_cells(case, seed)
    return None  # a stochastic trajectory: its lattice is compared with the start's, value by value
