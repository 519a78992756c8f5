"""The calls that a user of this framework makes, over the range of sizes they are made at.

A strong-strong simulation is a loop of turns: a beam-beam collision of an electron and a proton beam, the rings'
maps (or their lines) in between, and a row of beam moments now and then.  The listed cases are that loop with each
solver in earnest use, in both element types and from the smallest beams (where launches and latency count) to the
production size; the lines and the observer by themselves; a batch of independent collisions (a parameter scan); and
the learned correction's network, forward and in training.  ``draw`` gives other sizes of the same calls.

``exact`` restates each call in 64 bits with plain torch, from the published algorithm alone.
"""
import math
import os
import statistics
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "octopus.jl_b200"))

import octo_b200 as ob  # noqa: E402
from octo_b200 import learned  # noqa: E402

CLIGHT = 299792458.0
DEVICE = "cuda:0"
SY = 8.5e-6
# The two rings at the interaction point: optics, tunes, bunch length and energy spread, bunch population, energy.
RINGS = {
    "e": dict(beta=(0.55, 0.056, 0.7e-2 / 5.5e-4), tune=(0.08, 0.06, -0.069), sz=7e-3, charge=-1.0, mc2=ob.EMASS_EV,
              E0=10e9, r0=ob.RE, npart=1.7e11, crab_beta=(150.0, 30.0, 0.7e-2 / 5.5e-4), chromaticity=(1.0, 1.0),
              crab_frequency=394e6, crab=(math.tan(12.5e-3) / math.sqrt(150.0 * 0.55), 0.0, 0.0),
              damping_turns=(4000.0, 4000.0, 2000.0), rng_id=3),
    "p": dict(beta=(0.8, 0.072, 6e-2 / 6.6e-4), tune=(0.228, 0.210, -0.01), sz=6e-2, charge=1.0, mc2=ob.PMASS_EV,
              E0=275e9, r0=ob.RE * ob.ME0 / ob.PMASS_EV, npart=6.9e10, crab_beta=(1300.0, 30.0, 6e-2 / 6.6e-4),
              chromaticity=(2.0, 2.0), crab_frequency=197e6,
              crab=(math.tan(12.5e-3) / math.sqrt(1300.0 * 0.8) * 4.0 / 3.0,
                    -math.tan(12.5e-3) / math.sqrt(1300.0 * 0.8) / 3.0, 0.0), damping_turns=None, rng_id=0),
}
HALF_CROSSING = 12.5e-3


# ------------------------------------------------------------------------------------------------ the cases
def turn(solver, n1, n2, s1, s2, grid, ny=0, dtype="f64", aspect=95 / 8.5, tsc=False, fourth=False, quadratic=False):
    return {"kind": "turn", "solver": solver, "n1": n1, "n2": n2, "s1": s1, "s2": s2, "nx": grid, "ny": ny or grid,
            "dtype": dtype, "aspect": aspect, "tsc": tsc, "fourth": fourth, "quadratic": quadratic}


def listed():
    return [
        # the framework's reason to be: the production turn (2.56M electrons, 1.024M protons, 15 slices, 128 x 128
        # node meshes), and the same turn in the precision form
        {"name": "turn_production_f64", **turn("node", 2_560_000, 1_024_000, 15, 15, 128)},
        {"name": "turn_production_f32", **turn("node", 2_560_000, 1_024_000, 15, 15, 128, dtype="f32")},
        # the reference's default meshes at the size of a study on a workstation, round beams
        {"name": "turn_pair_f64", **turn("pair", 100_000, 100_000, 5, 5, 64, aspect=1.0)},
        # the higher-order options, on a mesh whose sides are not powers of two, and ragged particle counts
        {"name": "turn_high_order_f32", **turn("pair", 633_337, 250_001, 11, 9, 96, 64, dtype="f32", tsc=True,
                                               fourth=True, quadratic=True)},
        # set-up and debugging runs: a few thousand particles
        {"name": "turn_small_f64", **turn("pair", 4_001, 3_003, 3, 3, 32)},
        # the Gaussian-subtracted hybrid on its coarse mesh, and the soft-Gaussian solver
        {"name": "turn_hybrid_f64", **turn("hybrid", 1_280_000, 512_000, 15, 15, 48)},
        {"name": "turn_soft_f64", **turn("soft", 1_280_000, 512_000, 15, 15, 0)},
        # both rings' lines around the collision: crab cavities, boosts, maps, chromaticity, radiation
        {"name": "lines_production_f64", "kind": "lines", "n1": 2_560_000, "n2": 1_024_000, "dtype": "f64"},
        # a stretch of turns without collision, a row of moments of each beam every turn
        {"name": "monitor_f64", "kind": "monitor", "n1": 2_560_000, "n2": 1_024_000, "turns": 4, "dtype": "f64"},
        # a parameter scan: independent collisions of unequal sizes, together
        {"name": "scan_batch_f32", "kind": "scan", "scan": 7, "count": 5, "most": 1_000_000},
        # the correction network over the planes of a wavefront, and one training step
        {"name": "net_forward_20", "kind": "forward", "batch": 20},
        {"name": "net_train_64", "kind": "train", "batch": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["node", "node", "pair", "pair", "high", "hybrid", "soft", "lines", "monitor", "scan", "forward",
                       "train"])
    dtype = rng.choice(["f64", "f32"])
    n1 = _log(rng, 3_000, 2_560_000)
    n2 = max(2_000, min(2_560_000, int(n1 * rng.uniform(0.3, 1.2))))
    s1, s2 = rng.randint(3, 15), rng.randint(3, 15)
    aspect = math.exp(rng.uniform(0.0, math.log(25.0)))
    if kind in ("node", "pair"):
        return turn(kind, n1, n2, s1, s2, rng.choice([32, 48, 64, 96, 128]), dtype=dtype, aspect=aspect)
    if kind == "high":
        return turn("pair", min(n1, 1_280_000), min(n2, 1_280_000), s1, s2, rng.choice([32, 64, 96, 128]),
                    rng.choice([32, 48, 64, 128]), dtype, aspect, rng.random() < 0.7, rng.random() < 0.7,
                    rng.random() < 0.7)
    if kind == "hybrid":
        return turn("hybrid", min(n1, 1_280_000), min(n2, 512_000), s1, s2, rng.choice([32, 48, 64]), dtype=dtype,
                    aspect=max(2.0, aspect))
    if kind == "soft":
        return turn("soft", min(n1, 1_280_000), min(n2, 512_000), s1, s2, 0, dtype=dtype, aspect=max(2.0, aspect))
    if kind == "lines":
        return {"kind": "lines", "n1": n1, "n2": n2, "dtype": dtype}
    if kind == "monitor":
        return {"kind": "monitor", "n1": n1, "n2": n2, "turns": rng.randint(1, 8), "dtype": dtype}
    if kind == "scan":
        return {"kind": "scan", "scan": rng.randrange(1 << 20), "count": rng.randint(2, 5), "most": 600_000}
    return {"kind": kind, "batch": rng.randint(1, 64)}


def _scan_members(case):
    """The collisions of a scan: particles log-uniform per beam, slices, meshes and aspect ratios as they come."""
    r = np.random.default_rng(case["scan"])
    out = []
    for _ in range(case["count"]):
        n1, n2 = (int(np.exp(r.uniform(np.log(64_000), np.log(case["most"])))) for _ in range(2))
        s1, s2 = (int(r.integers(5, 16)) for _ in range(2))
        out.append(turn("pair", n1, n2, s1, s2, int(r.choice([64, 96, 128])), dtype="f32",
                        aspect=float(np.exp(r.uniform(0.0, np.log(25.0))))))
    return out


# ------------------------------------------------------------------------------------------------ what a user has
def _dtype(case):
    return torch.float32 if case["dtype"] == "f32" else torch.float64


def _beam(which, n, aspect, seed, dtype):
    """A matched Gaussian bunch, cut at five sigma."""
    r = RINGS[which]
    g = torch.Generator(device=DEVICE)
    g.manual_seed(2 * seed + (which == "p"))
    c = torch.randn(6, n, generator=g, device=DEVICE, dtype=torch.float64).clamp_(-5.0, 5.0)
    for k, s in enumerate((aspect * SY, SY, r["sz"])):
        c[2 * k] *= s
        c[2 * k + 1] *= s / r["beta"][k]
    return ob.Beam(c.to(dtype), ob.BeamParams(r["charge"], r["mc2"], r["E0"], r["r0"], r["npart"]))


def _solver(case):
    sl = dict(slicing1=ob.LongitudinalSlicing(nslices=case["s1"], method="normal_quantile"),
              slicing2=ob.LongitudinalSlicing(nslices=case["s2"], method="normal_quantile"))
    if case["solver"] == "soft":
        return ob.GaussianPoissonSolver(**sl)
    if case["solver"] == "hybrid":
        return ob.GaussianPICPoissonSolver(grid=(case["nx"], case["ny"]), **sl)
    return ob.PICPoissonSolver(grid=(case["nx"], case["ny"]), deposit_method="TSC" if case["tsc"] else "CIC",
                               field_derivative="fourth" if case["fourth"] else "second",
                               slice_interpolation="quadratic" if case["quadratic"] else "linear",
                               interaction_grid="node" if case["solver"] == "node" else "slice_pair", **sl)


def _segments(which):
    """The line elements of one ring before and after its collision."""
    r = RINGS[which]
    a = (0.0, 0.0, 0.0)
    to_ip = ob.Linear6DSpec(beta1=r["crab_beta"], beta2=r["beta"], alpha1=a, alpha2=a, dmu=(math.pi / 2, 0.0, 0.0))
    from_ip = ob.Linear6DSpec(beta1=r["beta"], beta2=r["crab_beta"], alpha1=a, alpha2=a, dmu=(math.pi / 2, 0.0, 0.0))
    crab = ob.ThinCrabCavitySpec(r["crab_frequency"], N=3, strengthX=r["crab"], strengthY=(0.0,) * 3, phase=(0.0,) * 3)
    ring = ob.Linear6DSpec(beta1=r["beta"], beta2=r["beta"], alpha1=a, alpha2=a,
                           dmu=tuple(2 * math.pi * t for t in r["tune"]))
    before = (to_ip.inverse(), crab, to_ip, ob.LorentzBoostSpec(HALF_CROSSING))
    after = [ob.RevLorentzBoostSpec(HALF_CROSSING), from_ip, crab, from_ip.inverse(), ring,
             ob.ChromaticityKickSpec(xi=r["chromaticity"], beta=r["beta"], alpha=a)]
    if r["damping_turns"]:
        after.append(ob.LumpedRadSpec(damping_turns=r["damping_turns"], beta=r["beta"], alpha=a,
                                      sigma=(95e-6, SY, r["sz"]), rng_id=r["rng_id"]))
    return before, tuple(after)


def _net_input(batch, seed):
    """Charge grids of Gaussian slices with the noise of a few thousand particles a cell, as the correction gets them."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    t = torch.linspace(-4.0, 4.0, 48, device=DEVICE)
    s = 0.6 + 0.8 * torch.rand(batch, 2, 1, generator=g, device=DEVICE)
    px, py = (torch.exp(-0.5 * (t / s[:, k]) ** 2) for k in range(2))
    q = py[:, :, None] * px[:, None, :] * 4000.0
    q = (q + q.sqrt() * torch.randn(q.shape, generator=g, device=DEVICE)).clamp_(min=0.0)
    x = torch.zeros(batch, 48, 48, 8, device=DEVICE)
    x[..., 0] = q / q.sum(dim=(1, 2), keepdim=True) * (48 * 48)
    x[..., 1] = -3.2 * torch.rand(batch, 1, 1, generator=g, device=DEVICE)
    target = 0.1 * torch.randn(batch, 48, 48, 2, generator=g, device=DEVICE)
    mask = torch.zeros(batch, 48, 48, device=DEVICE)
    mask[:, 2:-2, 2:-2] = 1.0
    return x.to(torch.bfloat16), target, mask


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("forward", "train"):
        net, _ = learned.load_net(max_batch=64, coarse="pic")
        x, target, mask = _net_input(case["batch"], seed)
        return {"kind": kind, "net": net, "x": x, "target": target, "mask": mask}
    if kind == "scan":
        members = _scan_members(case)
        beams = [(_beam("e", m["n1"], m["aspect"], seed + 100 * k, torch.float32),
                  _beam("p", m["n2"], m["aspect"], seed + 100 * k, torch.float32)) for k, m in enumerate(members)]
        return {"kind": kind, "contexts": [ob.Context(_solver(m), 0, torch.float32) for m in members],
                "e": [b[0] for b in beams], "p": [b[1] for b in beams], "turn": 0,
                "streams": [torch.cuda.Stream() for _ in members], "map_e": _maps("e"), "map_p": _maps("p")}
    aspect = case.get("aspect", 95 / 8.5)
    st = {"kind": kind, "turn": 0, "e": _beam("e", case["n1"], aspect, seed, _dtype(case)),
          "p": _beam("p", case["n2"], aspect, seed, _dtype(case))}
    st["rows"] = {b: list(st[b].coords.unbind()) for b in "ep"}  # views: the beams' own coordinates
    if kind == "lines":
        st["lines"] = {b: _segments(b) for b in "ep"}
        return st
    st["map_e"], st["map_p"] = _maps("e"), _maps("p")
    if kind == "monitor":
        st["turns"] = case["turns"]
        return st
    st["solver"], st["runtime"] = _solver(case), ob.StrongStrongRuntime()
    st["runtime"].context("ip", st["solver"], 0, _dtype(case))
    return st


def _maps(which):
    r = RINGS[which]
    return ob.Linear6D(r["beta"], (0.0, 0.0, 0.0), r["tune"])


# ------------------------------------------------------------------------------------------------ one pass
def run(st):
    kind = st["kind"]
    if kind == "forward":
        return st["net"].forward(st["x"])
    if kind == "train":
        loss, grads = st["net"].train_step(st["x"], st["target"], st["mask"], lr=1e-5, want_grads=True)
        return {"loss": loss, "grads": grads}
    if kind == "scan":
        lum = ob.collide_batch(st["contexts"], st["e"], st["p"], turn=st["turn"], streams=st["streams"])
        for e, p in zip(st["e"], st["p"]):
            st["map_e"].track(e)
            st["map_p"].track(p)
        st["turn"] += 1
        return {"luminosity": np.array(lum), "e": [row for b in st["e"] for row in b.coords.unbind()],
                "p": [row for b in st["p"] for row in b.coords.unbind()]}
    if kind == "lines":
        ctx = ob.TrackingContext(turn=st["turn"], seed=20261204, rng_method="philox")
        for b in "ep":
            ob.track(st[b], st["lines"][b][0], 1, ctx)
            ob.track(st[b], st["lines"][b][1], 1, ctx)
        st["turn"] += 1
        return st["rows"]
    if kind == "monitor":
        obs = {b: ob.MomentObserver(b, orders=(1, 2), capacity=64) for b in "ep"}
        for t in range(st["turns"]):
            for b in "ep":
                st["map_" + b].track(st[b])
                obs[b].observe(t, st[b])
        return {"rows": st["rows"], "moments": {b: _by_order(obs[b].rows()) for b in "ep"}}
    lum = ob.collide(st["solver"], st["e"], st["p"], ob.CUDABackend, ob.TrackingContext(turn=st["turn"]),
                     runtime=st["runtime"])
    st["map_e"].track(st["e"])
    st["map_p"].track(st["p"])
    st["turn"] += 1
    return {"luminosity": lum, "rows": st["rows"]}


def _by_order(rows):
    """A recorder's rows by the size of what they hold: the turns, the means, and the variances of the six
    coordinates with the covariances of each plane's pair."""
    pairs = [(i, j) for i in range(6) for j in range(i, 6)]
    own = [7 + k for k, (i, j) in enumerate(pairs) if i == j]
    cross = [7 + k for k, (i, j) in enumerate(pairs) if i != j]
    return {"turn": rows[:, 0], "mean_t": rows[:, [1, 2, 3, 4]], "mean_l": rows[:, [5, 6]],
            "var": {str(k): rows[:, c] for k, c in enumerate(own)}, "cov": rows[:, cross]}


# ------------------------------------------------------------------------------------------------ work and tolerance
def _planes(case):
    return 3 if case["solver"] == "node" or case["quadratic"] else 2


def work(case):
    """Each particle's six coordinates read once and written once.  Operations: per particle and pair visit, a drift
    and the taps of every plane it is deposited to, the luminosity plane's, and the gather and kick of a field
    particle; per directed pair the padded transforms of its planes, forward and back."""
    kind = case["kind"]
    if kind in ("forward", "train"):
        chans = [(8, 32, 0), (32, 32, 0), (32, 64, 1), (64, 64, 1), (64, 128, 2), (128, 128, 2), (128, 128, 3),
                 (256, 64, 2), (128, 32, 1), (64, 32, 0), (32, 8, 0)]
        macs = sum(9 * a * b * (48 >> lv) ** 2 for a, b, lv in chans) * case["batch"]
        params = sum(9 * a * b + b for a, b, _ in chans)
        io = case["batch"] * 48 * 48
        if kind == "forward":
            return {"bytes": io * (16 + 8) + 2 * params, "flops": 2 * macs}
        return {"bytes": io * (16 + 8 + 4) + params * (3 * 4 * 2 + 4), "flops": 6 * macs}
    if kind == "scan":
        parts = [work(m) for m in _scan_members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    size = 4 if case["dtype"] == "f32" else 8
    n = case["n1"] + case["n2"]
    if kind == "lines":
        return {"bytes": 2 * 2 * 6 * size * n, "flops": 900 * case["n1"] + 500 * case["n2"]}
    if kind == "monitor":
        return {"bytes": case["turns"] * 3 * 6 * size * n, "flops": case["turns"] * (72 + 60) * n}
    visits = case["n1"] * case["s2"] + case["n2"] * case["s1"]
    if case["solver"] == "soft":
        return {"bytes": 4 * 6 * size * n, "flops": visits * 400}
    taps = 9 if case["tsc"] else 4
    per = _planes(case) * (10 + 8 * taps) + 10 + 4 * taps + 60 + 6 * taps * _planes(case)
    cells = 4 * case["nx"] * case["ny"]
    fft = 2 * case["s1"] * case["s2"] * _planes(case) * 2 * 2.5 * cells * math.log2(cells)
    return {"bytes": 4 * 6 * size * n, "flops": visits * (per + (700 if case["solver"] == "hybrid" else 0)) + fft}


def tolerance(case):
    """About four times what the calls show against their 64-bit restatement, output by output (2-norms): the network
    7.5e-3 (bf16 operands and activations); lines 1e-15 and 3.6e-8 (one rounding to storage), moments 5.5e-15;
    collisions 5e-14 in float64 (more where slices are thin) and 4e-5 in float32, where each pair visit rounds the vertical coordinates to
    storage again and a particle at a slice's edge may fall to either side."""
    kind = case["kind"]
    if kind in ("forward", "train"):
        return {"rel": 2e-2, "max": 0.5}
    f32 = kind == "scan" or case["dtype"] == "f32"
    if kind in ("lines", "monitor"):
        return {"rel": 2e-7, "max": 2e-6} if f32 else {"rel": 3e-14, "max": 3e-12}
    return {"rel": 1.6e-4, "max": 2e-2} if f32 else {"rel": 1e-12, "max": 1e-9}


# ------------------------------------------------------------------------------------------------ 64-bit restatement
def exact(case, seed):
    kind = case["kind"]
    if kind in ("forward", "train"):
        return _exact_net(case, seed)
    if kind == "scan":
        lum, es, ps = [], [], []
        for k, m in enumerate(_scan_members(case)):
            e = _beam("e", m["n1"], m["aspect"], seed + 100 * k, torch.float32).coords.double()
            p = _beam("p", m["n2"], m["aspect"], seed + 100 * k, torch.float32).coords.double()
            lum.append(_exact_pic(m, e, p))
            es += list(_linear("e", e).unbind())
            ps += list(_linear("p", p).unbind())
        return {"luminosity": np.array(lum), "e": es, "p": ps}
    aspect = case.get("aspect", 95 / 8.5)
    b = {w: _beam(w, n, aspect, seed, _dtype(case)).coords.double() for w, n in (("e", case["n1"]), ("p", case["n2"]))}
    if kind == "lines":
        return {w: list(_exact_line(w, b[w]).unbind()) for w in "ep"}
    if kind == "monitor":
        rows = {"e": [], "p": []}
        for t in range(case["turns"]):
            for w in "ep":
                b[w] = _linear(w, b[w])
                c = b[w].to(_dtype(case)).double()
                m = c.mean(dim=1)
                d = c - m[:, None]
                cov = d @ d.T / c.shape[1]
                rows[w].append([float(t)] + m.tolist() + [float(cov[i, j]) for i in range(6) for j in range(i, 6)])
        return {"rows": {w: list(b[w].unbind()) for w in "ep"},
                "moments": {w: _by_order(np.array(rows[w])) for w in "ep"}}
    lum = (_exact_soft if case["solver"] == "soft" else _exact_pic)(case, b["e"], b["p"])
    return {"luminosity": lum, "rows": {w: list(_linear(w, b[w]).unbind()) for w in "ep"}}


def _rotation(beta, mu):
    """The 6x6 map of phase advances mu at equal optics, alpha = 0, or between optics beta = (from, to)."""
    b1, b2 = beta if isinstance(beta[0], tuple) else (beta, beta)
    m = np.zeros((6, 6))
    for k in range(3):
        s, c = math.sin(mu[k]), math.cos(mu[k])
        m[2 * k, 2 * k], m[2 * k, 2 * k + 1] = math.sqrt(b2[k] / b1[k]) * c, math.sqrt(b1[k] * b2[k]) * s
        m[2 * k + 1, 2 * k], m[2 * k + 1, 2 * k + 1] = -s / math.sqrt(b1[k] * b2[k]), math.sqrt(b1[k] / b2[k]) * c
    return m


def _linear(which, c):
    r = RINGS[which]
    return torch.from_numpy(_rotation(r["beta"], [2 * math.pi * t for t in r["tune"]])).to(c.device) @ c


def _splitmix(x):
    m = (1 << 64) - 1
    z = (x + 0x9E3779B97F4A7C15) & m
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return z ^ (z >> 31)


def _uniform(n, seed, t, rng_id, component):
    """Philox4x32-10 of (particle, turn) under the key of (seed, stream, component), as an open-interval uniform."""
    key = _splitmix(seed) ^ _splitmix(rng_id + 0x9E3779B97F4A7C15) ^ _splitmix(component + 0xBF58476D1CE4E5B9)
    k0, k1, low = key & 0xFFFFFFFF, key >> 32, 0xFFFFFFFF
    i = torch.arange(1, n + 1, device=DEVICE, dtype=torch.int64)
    c = [i & low, i >> 32, torch.full_like(i, t & low), torch.full_like(i, t >> 32)]
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57  # 64-bit products; they wrap, and only bits are used
        c = [((p1 >> 32) & low) ^ c[1] ^ k0, p1 & low, ((p0 >> 32) & low) ^ c[3] ^ k1, p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & low, (k1 + 0xBB67AE85) & low
    bits = (c[0] << 20) | (c[1] >> 12)  # the upper 52 of the 64 bits
    return (bits.double() + 0.5) * 2.0 ** -52


def _exact_line(which, c):
    r = RINGS[which]
    x, px, y, py, z, pz = c.unbind()
    m = lambda a, v: list((torch.from_numpy(a).to(c.device) @ torch.stack(v)).unbind())  # noqa: E731
    quarter = (math.pi / 2, 0.0, 0.0)
    to_ip = _rotation((r["crab_beta"], r["beta"]), quarter)
    from_ip = _rotation((r["beta"], r["crab_beta"]), quarter)

    def crab(v):
        x, px, y, py, z, pz = v
        k = 2 * math.pi * r["crab_frequency"] / CLIGHT
        for i, s in enumerate(r["crab"], 1):
            px, pz = px - s * torch.sin(i * k * z) / (i * k), pz - s * x * torch.cos(i * k * z)
        return [x, px, y, py, z, pz]

    ca, sa = math.cos(HALF_CROSSING), math.sin(HALF_CROSSING)
    x, px, y, py, z, pz = m(to_ip, crab(m(np.linalg.inv(to_ip), [x, px, y, py, z, pz])))
    h = 1.0 + pz - torch.sqrt((1.0 + pz) ** 2 - px ** 2 - py ** 2)
    h1, py1 = h / ca ** 2, py / ca
    px1 = px / ca - h1 * sa
    pz1 = pz - px1 * sa
    ps = 1.0 + pz1 - h1
    d = x * sa
    x, px, y, py, z, pz = (x + z * sa / ca + px1 / ps * d, px1, y + py1 / ps * d, py1, z / ca - h1 / ps * d, pz1)
    ps = torch.sqrt((1.0 + pz) ** 2 - px ** 2 - py ** 2)
    h = 1.0 + pz - ps
    x1 = (x - z * sa) / (1.0 + (px + h * sa) * sa / ps)
    v = [x1, (px + h * sa) * ca, y - py / ps * x1 * sa, py * ca, (z + h / ps * x1 * sa) * ca, pz + px * sa]
    v = m(np.linalg.inv(from_ip), crab(m(from_ip, v)))
    x, px, y, py, z, pz = m(_rotation(r["beta"], [2 * math.pi * t for t in r["tune"]]), v)
    (bx, by, _), (qx, qy) = r["beta"], r["chromaticity"]
    mx, my = 2 * math.pi * qx * pz, 2 * math.pi * qy * pz
    z = z + 2 * math.pi * (qx * 0.5 * (x * x / bx + bx * px * px) + qy * 0.5 * (y * y / by + by * py * py))
    x, px = x * torch.cos(mx) + px * bx * torch.sin(mx), px * torch.cos(mx) - x * torch.sin(mx) / bx
    y, py = y * torch.cos(my) + py * by * torch.sin(my), py * torch.cos(my) - y * torch.sin(my) / by
    v = [x, px, y, py, z, pz]
    if r["damping_turns"]:
        n = c.shape[1]
        for k, (tau, s) in enumerate(zip(r["damping_turns"], (95e-6, SY, r["sz"]))):
            u1, u2 = (_uniform(n, 20261204, 0, r["rng_id"], 2 * k + q) for q in (1, 2))
            rad, amp = torch.sqrt(-2.0 * torch.log(u1)), s * math.sqrt(-math.expm1(-2.0 / tau))
            v[2 * k] = v[2 * k] * math.exp(-1.0 / tau) + amp * rad * torch.cos(2 * math.pi * u2)
            v[2 * k + 1] = v[2 * k + 1] * math.exp(-1.0 / tau) + amp / r["beta"][k] * rad * torch.sin(2 * math.pi * u2)
    return torch.stack(v)


# ---------------------------------------------------------------- collisions
def _scales(case):
    e, p = RINGS["e"], RINGS["p"]
    q = e["charge"] * p["charge"]
    return q * e["r0"] * p["npart"] * e["mc2"] / e["E0"], q * p["r0"] * e["npart"] * p["mc2"] / p["E0"]


class _Slices:
    def __init__(self, c, ns):
        z = c[4]
        mu, sigma = float(z.mean()), float(z.std(correction=0))
        lo, hi = float(z.min()), float(z.max())
        q = statistics.NormalDist()
        self.edge = [lo] + [min(max(mu + sigma * q.inv_cdf(s / ns), lo), hi) for s in range(1, ns)] + [hi]
        inner = torch.tensor(self.edge[1:-1], device=z.device, dtype=torch.float64)
        which = torch.bucketize(z, inner, right=True)
        self.index = [(which == s).nonzero().squeeze(1) for s in range(ns)]
        self.state = [c[:, i].clone() for i in self.index]
        self.center = [float(s[4].mean()) if s.shape[1] else (a + b) / 2
                       for s, a, b in zip(self.state, self.edge, self.edge[1:])]

    def back(self, c):
        for i, s in zip(self.index, self.state):
            c[:, i] = s


def _pairs(a, b):
    order = [(-(ci + cj) / 2, i, j) for i, ci in enumerate(a.center) for j, cj in enumerate(b.center)]
    return [(i, j) for _, i, j in sorted(order, key=lambda o: o[0])]


def _box(*points):
    """((xmin, xmax), (ymin, ymax)) over pairs of coordinate tensors."""
    mm = [torch.stack([t.aminmax().min, t.aminmax().max]) for p in points for t in p]
    v = torch.stack(mm).tolist()
    xs, ys = v[0::2], v[1::2]
    return ((min(a for a, _ in xs), max(b for _, b in xs)), (min(a for a, _ in ys), max(b for _, b in ys)))


def _axis_grid(n, src, fld, growth):
    """One axis of an interaction's source and field meshes: a common cell, three cells of margin, origins moved to a
    whole-cell offset, grown about the middle where the mesh will be kept for later turns."""
    w = max(src[1] - src[0], fld[1] - fld[0])
    t = w / (n - 4)
    w += 3 * t
    s0, f0 = src[0] - 1.5 * t, fld[0] - 1.5 * t
    f1, f2 = s0 / t - math.floor(s0 / t), f0 / t - math.floor(f0 / t)
    k = (f2 - f1) / 2
    k = k - 0.5 if k > 0.5 else k + 0.5 if k < -0.5 else k
    s0, f0 = s0 + k * t, f0 - k * t
    more = w * growth
    return s0 - more / 2, f0 - more / 2, (w + more) / (n - 1)


class _Mesh:
    def __init__(self, case, src, fld, growth):
        self.nx, self.ny = case["nx"], case["ny"]
        self.sx, self.fx, self.hx = _axis_grid(self.nx, src[0], fld[0], growth)
        self.sy, self.fy, self.hy = _axis_grid(self.ny, src[1], fld[1], growth)
        i = torch.arange(2 * self.nx, device=DEVICE, dtype=torch.float64)
        j = torch.arange(2 * self.ny, device=DEVICE, dtype=torch.float64)
        x = self.fx - self.sx + torch.where(i < self.nx, i, i - 2 * self.nx) * self.hx
        y = self.fy - self.sy + torch.where(j < self.ny, j, j - 2 * self.ny) * self.hy

        def corner(a, b):
            X, Y = (x + a)[None, :], (y + b)[:, None]
            r2 = X * X + Y * Y
            at = lambda p, q: torch.where(q == 0, torch.sign(p) * (math.pi / 2), torch.atan(p / q))  # noqa: E731
            v = (torch.log(r2) - 3) * X * Y + at(Y, X) * X * X + at(X, Y) * Y * Y
            return torch.where(r2 == 0, 0.0, v)

        a, b = self.hx / 2, self.hy / 2
        g = corner(a, b) + corner(-a, -b) - corner(a, -b) - corner(-a, b)
        self.green = torch.fft.rfft2(-0.5 / (self.hx * self.hy) * g)

    def field(self, q, fourth):
        """(phi, Ex, Ey) of a charge grid [ny, nx]."""
        nx, ny = self.nx, self.ny
        f = torch.fft.rfft2(q, s=(2 * ny, 2 * nx)) * self.green
        phi = torch.fft.irfft2(f, s=(2 * ny, 2 * nx))[:ny, :nx].contiguous()
        ey = _derivative(phi, self.hy, fourth)
        return phi, _derivative(phi.T.contiguous(), self.hx, fourth).T, ey


def _derivative(p, h, fourth):
    """-d/dy along the first axis: one-sided of second order at the ends, central of order two or four inside."""
    d = torch.empty_like(p)
    d[0] = 1.5 * p[0] - 2 * p[1] + 0.5 * p[2]
    d[-1] = -1.5 * p[-1] + 2 * p[-2] - 0.5 * p[-3]
    d[1:-1] = 0.5 * (p[:-2] - p[2:])
    if fourth:
        d[2:-2] = ((p[4:] - p[:-4]) + 8 * (p[1:-3] - p[3:-1])) / 12
    return d / h


def _taps(u, n, tsc):
    """First node and weights [taps, N] of the cloud at u, zero outside the mesh."""
    ok = (u >= 0) & (u <= n - 1)
    f = torch.floor(u)
    if not tsc:
        base = f.clamp(0, n - 2)
        t = (u - base).clamp(0.0, 1.0)
        w = torch.stack([1 - t, t])
    else:
        near = torch.where(u - f < 0.5, f, f + 1)
        d = u - near
        w = torch.stack([0.5 * (0.5 - d) ** 2, 0.75 - d * d, 0.5 * (0.5 + d) ** 2])
        base = (near - 1).clamp(0, n - 3)
    return torch.where(ok, base, 0.0).long(), torch.where(ok, w, 0.0)


def _cloud(x, y, x0, y0, hx, hy, nx, ny, tsc):
    """Flat node numbers and weights [taps, N]."""
    ix, wx = _taps((x - x0) / hx, nx, tsc)
    iy, wy = _taps((y - y0) / hy, ny, tsc)
    k = range(wx.shape[0])
    return (torch.stack([(iy + b) * nx + ix + a for a in k for b in k]),
            torch.stack([wx[a] * wy[b] for a in k for b in k]))


def _deposit(x, y, x0, y0, hx, hy, nx, ny, tsc):
    at, w = _cloud(x, y, x0, y0, hx, hy, nx, ny, tsc)
    q = torch.zeros(ny * nx, device=x.device, dtype=torch.float64)
    return q.index_add_(0, at.reshape(-1), w.reshape(-1)).view(ny, nx)


def _gather(cloud, planes):
    at, w = cloud
    return [(p.reshape(-1)[at] * w).sum(0) for p in planes]


def _luminosity(case, p1, p2):
    nx, ny, tsc = case["nx"], case["ny"], case["tsc"]
    (xlo, xhi), (ylo, yhi) = _box(p1, p2)
    tx, ty = (xhi - xlo) / (nx - 1.1), (yhi - ylo) / (ny - 1.1)
    hx, hy = (xhi - xlo + 0.1 * tx) / (nx - 1), (yhi - ylo + 0.1 * ty) / (ny - 1)
    q1, q2 = (_deposit(x, y, xlo - 0.05 * tx, ylo - 0.05 * ty, hx, hy, nx + 1, ny + 1, tsc) for x, y in (p1, p2))
    return float((q1 * q2).sum()) / (hx * hy)


def _at(c, s):
    return c[0] + s * c[1], c[2] + s * c[3]


def _exact_pic(case, e, p):
    """Collides e and p (their coordinates are replaced) and returns the luminosity."""
    S = (_Slices(e, case["s1"]), _Slices(p, case["s2"]))
    n1, n2 = e.shape[1], p.shape[1]
    k1, k2 = _scales(case)
    kbb = (k1 / n2, k2 / n1)
    node = _node_meshes(case, S) if case["solver"] == "node" else None
    lum = 0.0
    for i, j in _pairs(*S):
        a, b = S[0].state[i], S[1].state[j]
        if not a.shape[1] or not b.shape[1]:
            continue
        new_b = _kicked(case, a, S[0].center[i], b, S[1].edge[j], S[1].edge[j + 1], kbb[1],
                        node and (node[0][i][j], node[0][i][j + 1]))
        new_a = _kicked(case, b, S[1].center[j], a, S[0].edge[i], S[0].edge[i + 1], kbb[0],
                        node and (node[1][j][i], node[1][j][i + 1]))
        lum += _luminosity(case, _at(a, 0.5 * (S[0].center[i] - S[1].center[j])),
                           _at(b, 0.5 * (S[1].center[j] - S[0].center[i])))
        S[0].state[i], S[1].state[j] = new_a, new_b
    S[0].back(e)
    S[1].back(p)
    return lum * RINGS["e"]["npart"] * RINGS["p"]["npart"] / (n1 * n2)


def _node_meshes(case, S):
    """A mesh for every source slice at every boundary of the other beam's slices, from the beams before the turn."""
    out = []
    for own, other in ((S[0], S[1]), (S[1], S[0])):
        rows = []
        for state, c in zip(own.state, own.center):
            if not state.shape[1]:
                rows.append([None] * len(other.edge))
                continue
            src = [_box(_at(state, 0.5 * (c - b))) for b in other.edge]
            fld = [_box(_at(f, 0.5 * (f[4] - c))) if f.shape[1] else None for f in other.state]
            row = []
            for b in range(len(other.edge)):
                near = [f for f in (fld[b - 1] if b else None, fld[b] if b < len(fld) else None) if f]
                both = [src[b], src[min(b + 1, len(src) - 1)]]
                join = lambda v: tuple((min(t[k][0] for t in v), max(t[k][1] for t in v)) for k in (0, 1))  # noqa: E731
                row.append(_Mesh(case, join(both), join(near), 0.0) if near else None)
            rows.append(row)
        out.append(rows)
    return out


def _kicked(case, src, center, fld, left, right, kbb, meshes):
    """The field slice after the source slice's kick: drifted to its collision points, kicked, drifted back."""
    x, px, y, py, z, pz = fld.unbind()
    tsc, fourth = case["tsc"], case["fourth"]
    sl, sr = 0.5 * (center - left), 0.5 * (center - right)
    s = 0.5 * (z - center)
    x, y, pz = x + s * px, y + s * py, pz - 0.25 * (px * px + py * py)
    h = 1.0 / (right - left) if right != left else 0.0
    zl = (-z * h + right * h if h else torch.full_like(z, 0.5)).clamp(0.0, 1.0)
    zr = 1.0 - zl
    hybrid = _gaussians(src, sl, sr) if case["solver"] == "hybrid" else None

    def solve(m, s, ref=None):
        q = _deposit(*_at(src, s), m.sx, m.sy, m.hx, m.hy, m.nx, m.ny, tsc)
        if ref:
            gx, gy = _profile(m.sx, m.hx, m.nx, ref[0], ref[2]), _profile(m.sy, m.hy, m.ny, ref[1], ref[3])
            q = q - q.sum() / (gx.sum() * gy.sum()) * gy[:, None] * gx[None, :]
        return m.field(q, fourth)

    def cloud(m):
        return _cloud(x, y, m.fx, m.fy, m.hx, m.hy, m.nx, m.ny, tsc)

    extra = None
    if meshes:
        ml, mr = meshes
        L, R, Z = solve(ml, sl), solve(mr, sr), solve(ml, sr)
        ex, ey, kz = _gather(cloud(ml), [L[1], L[2], L[0] - Z[0]])
        fx, fy = _gather(cloud(mr), R[1:])
        kx, ky = zl * ex + zr * fx, zl * ey + zr * fy
    else:
        box = _box(_at(src, sl), _at(src, sr))
        if hybrid:
            (L0, R0), mean, cov = hybrid
            box = tuple((min(box[k][0], *(g[k] - 5 * g[k + 2] for g in (L0, R0))),
                         max(box[k][1], *(g[k] + 5 * g[k + 2] for g in (L0, R0)))) for k in (0, 1))
        m = _Mesh(case, box, _box((x, y)), 0.25)
        L, R = solve(m, sl, hybrid and L0), solve(m, sr, hybrid and R0)
        if case["quadratic"]:
            M, t = solve(m, 0.5 * (sl + sr)), zr
            al, am, ar = 2 * t * t - 3 * t + 1, 4 * t - 4 * t * t, 2 * t * t - t
            bl, bm, br = 3 - 4 * t, 8 * t - 4, 1 - 4 * t
            g = _gather(cloud(m), [f[k] for f in (L, M, R) for k in range(3)])
            kz = bl * g[0] + bm * g[3] + br * g[6]
            kx, ky = (al * g[k] + am * g[3 + k] + ar * g[6 + k] for k in (1, 2))
        else:
            ex, ey, fx, fy, kz = _gather(cloud(m), [L[1], L[2], R[1], R[2], L[0] - R[0]])
            kx, ky = zl * ex + zr * fx, zl * ey + zr * fy
        if hybrid:
            half = 0.5 * src.shape[1]
            kl, kr = (_bassetti(g[2], g[3], x - g[0], y - g[1]) for g in (L0, R0))
            ax, ay = half * (zl * kl[0] + zr * kr[0]), half * (zl * kl[1] + zr * kr[1])
            kx, ky = kx + ax, ky + ay
            k = 2 * kbb
            cv = [k * half * 0.25 * (kk[2] * c[0] + kk[3] * c[1]) for kk, c in zip((kl, kr), cov)]
            extra = zl * cv[0] + zr * cv[1] + 0.5 * k * (ax * mean[0] + ay * mean[1])
    px, py, pz = px + 2 * kbb * kx, py + 2 * kbb * ky, pz + 2 * kbb * kz * h
    if extra is not None:
        pz = pz + extra
    return torch.stack([x - s * px, px, y - s * py, py, z, pz + 0.25 * (px * px + py * py)])


def _moments(c):
    """Means of x, px, y, py and per plane (variance, covariance, momentum variance)."""
    m = c[:4].mean(dim=1)
    d = c[:4] - m[:, None]
    v = (d @ d.T / c.shape[1]).tolist()
    return m.tolist(), (v[0][0], v[0][1], v[1][1]), (v[2][2], v[2][3], v[3][3])


def _gaussians(src, sl, sr):
    """The source's Gaussian drifted to both boundaries, its mean angles, and d(variance)/ds there."""
    (mx, mpx, my, mpy), vx, vy = _moments(src)
    ref, cov = [], []
    for s in (sl, sr):
        a, d = (v[0] + 2 * s * v[1] + s * s * v[2] for v in (vx, vy))
        ref.append((mx + mpx * s, my + mpy * s, math.sqrt(a), math.sqrt(d)))
        cov.append((2 * (vx[1] + s * vx[2]), 2 * (vy[1] + s * vy[2])))
    return ref, (mpx, mpy), cov


def _profile(x0, h, n, mu, s):
    """A unit Gaussian against the linear assignment function at every node."""
    x = x0 + h * torch.arange(n, device=DEVICE, dtype=torch.float64)
    m0 = lambda a, b: 0.5 * (torch.erf((b - mu) / (s * math.sqrt(2))) - torch.erf((a - mu) / (s * math.sqrt(2))))  # noqa: E731
    pdf = lambda t: torch.exp(-(t - mu) ** 2 / (2 * s * s)) / (s * math.sqrt(2 * math.pi))  # noqa: E731
    m1 = lambda a, b: (mu - x) * m0(a, b) - s * s * (pdf(b) - pdf(a))  # noqa: E731
    return m0(x - h, x + h) + (m1(x - h, x) - m1(x, x + h)) / h


def _faddeeva_coefficients(n):
    """Weideman's rational expansion of w(z) (SIAM J. Numer. Anal. 31, 1994)."""
    m = 2 * n
    L = math.sqrt(n / math.sqrt(2.0))
    t = L * np.tan(np.arange(-m + 1, m) * math.pi / m / 2)
    f = np.concatenate([[0.0], np.exp(-t * t) * (L * L + t * t)])
    return L, np.real(np.fft.fft(np.fft.fftshift(f)))[1:n + 1] / (2 * m)


_W = _faddeeva_coefficients(48)


def _faddeeva(z):
    L, a = _W
    d = L - 1j * z
    Z = (L + 1j * z) / d
    p = torch.zeros_like(z)
    for c in a[::-1]:
        p = p * Z + c
    return 2 * p / (d * d) + (1 / math.sqrt(math.pi)) / d


def _bassetti(sx, sy, x, y):
    """(Kx, Ky, Hxx, Hyy) of an upright Gaussian, sigma_x > sigma_y: Bassetti and Erskine's field of unit strength and
    the diagonal of its derivative's trace form.  sx, sy: numbers or tensors."""
    if float(torch.as_tensor(sx).mean()) < float(torch.as_tensor(sy).mean()):
        ky, kx, hy, hx = _bassetti(sy, sx, y, x)
        return kx, ky, hx, hy
    t2 = sx * sx - sy * sy
    den = (2 * t2) ** 0.5
    ax, ay = x.abs(), y.abs()
    g = torch.exp(-0.5 * (x * x / (sx * sx) + y * y / (sy * sy)))
    w = _faddeeva(torch.complex(ax / den, ay / den)) - g * _faddeeva(torch.complex(sy / sx * ax / den, sx / sy * ay / den))
    w = w * (2 * math.sqrt(math.pi) / den)
    kx, ky = torch.sign(x) * w.imag, torch.sign(y) * w.real
    t = x * kx + y * ky
    return kx, ky, (t - 2 * (1 - g * sy / sx)) / t2, (-t + 2 * (1 - g * sx / sy)) / t2


def _exact_soft(case, e, p):
    """Each slice kicked by the Gaussian with the other's moments, pair by pair."""
    S = (_Slices(e, case["s1"]), _Slices(p, case["s2"]))
    n1, n2 = e.shape[1], p.shape[1]
    k1, k2 = _scales(case)
    lum = 0.0

    def kick(c, own_center, mom, kbb):
        (mx, mpx, my, mpy), vx, vy = mom
        x, px, y, py, z, pz = c.unbind()
        s = 0.5 * (z - own_center)
        x, y, pz = x + s * px, y + s * py, pz - 0.25 * (px * px + py * py)
        a, d = (v[0] - 2 * s * v[1] + s * s * v[2] for v in (vx, vy))
        sx, sy = a.sqrt(), d.sqrt()
        u, v = x - mx + mpx * s, y - my + mpy * s
        kx, ky, hx, hy = _bassetti(sx, sy, u, v)
        dens = (torch.exp(-0.5 * (u * u / a + v * v / d)) / (sx * sy)).sum() / (2 * math.pi)
        pz = pz + 0.25 * kbb * (hx * 2 * (vx[1] - s * vx[2]) + hy * 2 * (vy[1] - s * vy[2]))
        pz = pz + 0.5 * kbb * (kx * mpx + ky * mpy)
        px, py = px + kbb * kx, py + kbb * ky
        return torch.stack([x - s * px, px, y - s * py, py, z, pz + 0.25 * (px * px + py * py)]), float(dens)

    for i, j in _pairs(*S):
        a, b = S[0].state[i], S[1].state[j]
        if not a.shape[1] or not b.shape[1]:
            continue
        w1, w2 = a.shape[1] / n1, b.shape[1] / n2
        S[0].state[i], dens = kick(a, S[1].center[j], _moments(b), w2 * k1)
        S[1].state[j], _ = kick(b, S[0].center[i], _moments(a), w1 * k2)
        lum += dens * w2 * RINGS["e"]["npart"] * RINGS["p"]["npart"] / n1
    S[0].back(e)
    S[1].back(p)
    return lum


# ---------------------------------------------------------------- the network
def _exact_net(case, seed):
    """The U-Net in 64 bits from the saved parameters; for training, its loss and gradients."""
    torch.backends.cudnn.enabled = False
    data = np.load(os.path.join(os.path.dirname(os.path.abspath(learned.__file__)), "data",
                                "field_correction_pic_48.npz"))
    flat = torch.from_numpy(data["params"]).to(DEVICE).double().requires_grad_(case["kind"] == "train")
    chans = [(8, 32), (32, 32), (32, 64), (64, 64), (64, 128), (128, 128), (128, 128), (256, 64), (128, 32), (64, 32),
             (32, 8)]
    layers, at = [], 0
    for ci, co in chans:
        w = flat[at:at + 9 * ci * co].view(co, 3, 3, ci).permute(0, 3, 1, 2)
        layers.append((w, flat[at + 9 * ci * co:at + 9 * ci * co + co]))
        at += 9 * ci * co + co
    x, target, mask = _net_input(case["batch"], seed)
    f = torch.nn.functional

    def conv(k, v):
        v = f.conv2d(v, layers[k][0], layers[k][1], padding=1)
        return torch.relu(v) if k < 10 else v

    def merge(v, skip):
        return torch.cat([f.interpolate(v, scale_factor=2, mode="nearest"), skip], dim=1)

    s1 = conv(1, conv(0, x.double().permute(0, 3, 1, 2)))
    s2 = conv(3, conv(2, f.avg_pool2d(s1, 2)))
    s3 = conv(5, conv(4, f.avg_pool2d(s2, 2)))
    v = conv(7, merge(conv(6, f.avg_pool2d(s3, 2)), s3))
    v = conv(9, merge(conv(8, merge(v, s2)), s1))
    out = conv(10, v)[:, :2].permute(0, 2, 3, 1)
    if case["kind"] == "forward":
        return out.detach()
    loss = (mask[..., None] * (out - target.double()) ** 2).sum() / (2.0 * mask.sum().double())
    loss.backward()
    return {"loss": float(loss), "grads": flat.grad.cpu().numpy()}
