"""The work that programs have this package do, as measurable cases.

``listed()`` gives twelve named cases, ``draw(rng)`` one more of the same
ranges; ``prepare`` makes what a program holds before the call, ``run`` is one
pass through the public entry points, ``work`` the bytes and flops that pass
cannot do without and ``exact`` its results in plain FP64 torch where they can
be had.

Kinds of cases, and the ranges that ``draw`` covers:

  rings      the PteraSoftware-signature Biot-Savart functions (collapsed and
             expanded; ring, chordwise and horseshoe legs) with NumPy or CUDA
             arrays: 60 to 10,000 points x 60 to 10,000 vortices
  sweep      all-pairs particle sweeps at given targets (velocity, gradient,
             stretching, vorticity; both cores; FP64): 100 to 8,000 targets x
             1,000 to 131,072 sources
  field      one VortexParticleField RK3 step with direct sweeps, FP64 (1,000
             to 6,000 particles) or FP32 (4,096 to 32,768)
  tree       one VortexParticleField RK3 step through the treecode with the
             analytic or learned far field: 2^14 to 2^18 particles
  hybrid     one panel-particle step of the heaving wing (FP64, a wake of 300
             to 3,000 particles) or of the flapping aircraft (learned far
             field, 2^14 to 2^20 particles)
  flutter    the batched Goland sweep: 8 to 64 airspeeds, 5 to 20 chords
  training   loss and gradients of the far-field network: 512 to 16,384 rows
"""
from __future__ import annotations

import math

import numpy as np
import torch

LEG_FLOP = 51            # one line segment at one point (add, multiply = 1, sqrt, div = 1)
LEGS = {"ring": 4, "chordwise": 2, "horseshoe": 3}
PAIR_FLOP = {"velocity": 30, "stretching": 57, "both": 62, "jacobian": 65, "vorticity": 45}
ERF_FLOP = 10            # more per pair with the Gaussian-erf core
RK3 = ((0.0, 1.0 / 3.0), (-5.0 / 9.0, 15.0 / 16.0), (-153.0 / 128.0, 8.0 / 15.0))
U_INF = (9.998, 0.0, 0.1745)     # 10 m/s at one degree
DT = 1.0 / 43.0                  # the flapping configuration's time step


def listed():
    return [
        # PteraSoftware calling the patched functions on a small wing: host
        # arrays in, a host array out, dominated by latency
        {"name": "rings_host_small", "kind": "rings", "legs": "ring", "expanded": False,
         "host": True, "points": 200, "vortices": 100},
        # the largest row of the reference's published benchmark: a long free
        # wake on itself
        {"name": "rings_collapsed_large", "kind": "rings", "legs": "ring", "expanded": False,
         "host": False, "points": 10000, "vortices": 10000},
        # influence-coefficient assembly of the horseshoe method, every pair
        # written out, sizes that are no multiple of any tile
        {"name": "horseshoe_expanded", "kind": "rings", "legs": "horseshoe", "expanded": True,
         "host": False, "points": 501, "vortices": 1003},
        # the wake's particles at a wing's collocation points and bound legs:
        # few targets, many sources
        {"name": "wake_on_panels_f64", "kind": "sweep", "quantity": "velocity",
         "core": "winckelmans", "targets": 384, "sources": 131071, "own": False},
        # the velocity gradient of a free wake at its own particles with the
        # function's default core (the reference quotes 7,000 particles)
        {"name": "jacobian_erf_f64", "kind": "sweep", "quantity": "jacobian",
         "core": "gaussianerf", "targets": 7001, "sources": 7001, "own": True},
        # a particle field with every default (FP64, Gaussian-erf core, direct
        # sweeps, relaxation), about the heaving wing's wake after 3 cycles
        {"name": "field_step_f64", "kind": "field", "core": "gaussianerf", "precision": "f64",
         "n": 3001, "relax": 0.3, "stretch": True},
        # a larger wake in single precision, still all pairs
        {"name": "field_step_f32c", "kind": "field", "core": "winckelmans",
         "precision": "f32c", "n": 32768, "relax": 0.0, "stretch": True},
        # a wake that needs the treecode, set up as the reference's solver
        # sets up its field (relaxation on)
        {"name": "field_step_learned", "kind": "tree", "far_field": "learned", "n": 131072,
         "leaf": 32, "relax": 0.3, "stretch": True},
        # the panel-particle step at the size of a reference run: many small
        # launches, FP64 throughout
        {"name": "hybrid_step_wing", "kind": "hybrid", "aircraft": False, "n": 2001},
        # the headline configuration: 192 panels and a million particles
        {"name": "hybrid_step_aircraft", "kind": "hybrid", "aircraft": True, "n": 1 << 20},
        # the aeroelastic sweep of 64 airspeeds, mixed precision
        {"name": "flutter_sweep", "kind": "flutter", "speeds": 64, "chords": 20.0,
         "precision": "f32c"},
        # one minibatch of the far-field network's training
        {"name": "training_gradients", "kind": "training", "rows": 8192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rings", "rings", "sweep", "sweep", "field", "field", "tree", "hybrid",
                       "hybrid", "flutter", "training"])
    if kind == "rings":
        expanded = rng.random() < 0.4
        legs = rng.choice(["ring", "horseshoe"] if expanded else
                          ["ring", "ring", "chordwise", "horseshoe"])
        top = 3000 if expanded else 10000
        return {"kind": kind, "legs": legs, "expanded": expanded, "host": rng.random() < 0.4,
                "points": _log(rng, 60, top), "vortices": _log(rng, 60, top)}
    if kind == "sweep":
        own = rng.random() < 0.5
        q = rng.choice(["velocity", "jacobian", "stretching", "both", "vorticity"] if own else
                       ["velocity", "velocity", "jacobian"])
        n = _log(rng, 1000, 8000 if own else 131072)
        return {"kind": kind, "quantity": q, "core": rng.choice(["winckelmans", "gaussianerf"]),
                "targets": n if own else _log(rng, 100, 1000), "sources": n, "own": own}
    if kind == "field":
        f64 = rng.random() < 0.5
        return {"kind": kind, "core": rng.choice(["winckelmans", "gaussianerf"]),
                "precision": "f64" if f64 else "f32c",
                "n": _log(rng, 1000, 6000) if f64 else _log(rng, 4096, 32768),
                "relax": rng.choice([0.0, 0.3]), "stretch": rng.random() < 0.7}
    if kind == "tree":
        return {"kind": kind, "far_field": rng.choice(["m2l", "learned"]),
                "n": _log(rng, 1 << 14, 1 << 18), "leaf": rng.choice([32, 48, 64]),
                "relax": rng.choice([0.0, 0.3]), "stretch": rng.random() < 0.7}
    if kind == "hybrid":
        aircraft = rng.random() < 0.5
        return {"kind": kind, "aircraft": aircraft,
                "n": _log(rng, 1 << 14, 1 << 20) if aircraft else _log(rng, 300, 3000)}
    if kind == "flutter":
        return {"kind": kind, "speeds": rng.randint(8, 64),
                "chords": round(rng.uniform(5.0, 20.0), 1),
                "precision": rng.choice(["f32c", "f32c", "f64"])}
    return {"kind": kind, "rows": _log(rng, 512, 16384)}


# ---- inputs ----------------------------------------------------------------------


def _slab(n, seed, x0=9.0):
    """A grown wake: n particles over a 20 x 10 x 2 slab, strengths
    N(0, (1e-3)^2), cores 1.3 x the mean spacing."""
    rng = np.random.default_rng(seed)
    pos = rng.uniform([x0, -5.0, -1.0], [x0 + 20.0, 5.0, 1.0], size=(n, 3))
    gamma = rng.normal(0.0, 1e-3, size=(n, 3))
    sigma = np.full(n, 1.3 * (400.0 / n) ** (1.0 / 3.0))
    return pos, gamma, sigma


def _wake(n, seed):
    """n vortex rings of a rolled-up wake sheet behind a wing of span 10:
    corners BR, FR, FL, BL (n, 3), strengths, core radii, ages."""
    rng = np.random.default_rng(seed)
    cols = max(4, int(math.sqrt(n / 2.0)))
    rows = -(-n // cols)
    x = 1.0 + 0.15 * np.arange(rows + 1)[:, None] + 0.02 * rng.standard_normal((rows + 1, cols + 1))
    y = (np.linspace(-5.0, 5.0, cols + 1)[None, :]
         + 0.02 * rng.standard_normal((rows + 1, cols + 1)))
    z = 0.2 * np.sin(0.8 * x + 0.3 * y) + 0.02 * rng.standard_normal((rows + 1, cols + 1))
    v = np.stack([x, y, z], axis=-1)
    pick = [v[1:, 1:], v[:-1, 1:], v[:-1, :-1], v[1:, :-1]]
    corners = [np.ascontiguousarray(c.reshape(-1, 3)[:n]) for c in pick]
    strengths = 0.3 * rng.standard_normal(n) + 0.5
    ages = np.repeat(DT * np.arange(rows), cols)[:n].copy()
    return corners, strengths, np.full(n, 0.03), ages


def _ring_inputs(case, seed):
    """Half of the points are vertices of the wake itself (a free wake
    convects them), the others lie over the wing and its near field."""
    n, m = case["points"], case["vortices"]
    corners, s, rc, ages = _wake(m, seed)
    rng = np.random.default_rng(seed + 1)
    near = rng.uniform([0.0, -5.0, -0.3], [3.0, 5.0, 0.3], size=(n, 3))
    k = min(n // 2, m)
    near[:k] = corners[1][rng.permutation(m)[:k]]
    return near, corners, s, rc, ages


def _cuda(a):
    return torch.as_tensor(a, device="cuda")


def _sweep_inputs(case, seed):
    pos, gam, sig = _slab(case["sources"], seed, x0=1.0)
    if case["own"]:
        return pos, gam, pos, gam, sig
    rng = np.random.default_rng(seed + 1)
    tgt = rng.uniform([0.0, -5.0, -0.2], [1.0, 5.0, 0.2], size=(case["targets"], 3))
    return tgt, None, pos, gam, sig


def _network_inputs(case, seed):
    """Packed weights (48-128-128-128-32), biases, features and targets of
    the magnitudes that training sees."""
    g = torch.Generator().manual_seed(seed)
    blocks = [torch.randn(o, i, generator=g) * math.sqrt(2.0 / i) * k
              for (o, i, k) in ((128, 48, 1.0), (128, 128, 1.0), (128, 128, 1.0), (32, 128, 0.1))]
    w = torch.cat([x.reshape(-1) for x in blocks]).numpy()
    b = (0.05 * torch.randn(416, generator=g)).numpy()
    X = (0.5 * torch.randn(case["rows"], 48, generator=g)).to(torch.bfloat16)
    X[:, 35:] = 0.0
    T = 0.3 * torch.randn(case["rows"], 32, generator=g)
    return w, b, X, T


# ---- cases -----------------------------------------------------------------------


def _prepare_rings(case, seed):
    from fluxvortex_gb300 import aerodynamics as A
    pts, corners, s, rc, ages = _ring_inputs(case, seed)
    name = {("ring", False): "collapsed_velocities_from_ring_vortices",
            ("chordwise", False): "collapsed_velocities_from_ring_vortices_chordwise_segments",
            ("horseshoe", False): "collapsed_velocities_from_horseshoe_vortices",
            ("ring", True): "expanded_velocities_from_ring_vortices",
            ("horseshoe", True): "expanded_velocities_from_horseshoe_vortices"}[
                (case["legs"], case["expanded"])]
    to = (lambda a: a) if case["host"] else _cuda
    args = [to(a) for a in (pts, *corners, s, rc)]
    tail = (15.06e-6,) if case["legs"] == "horseshoe" else (to(ages), 15.06e-6)
    counts = ((lambda: np.zeros(4, np.int64)) if case["host"] else
              (lambda: torch.zeros(4, dtype=torch.int64, device="cuda")))
    return {"fn": getattr(A, name), "args": args, "tail": tail, "counts": counts}


def _run_rings(st):
    counts = st["counts"]()
    v = st["fn"](*st["args"], counts, *st["tail"])
    return {"velocity": v, "counts": counts}


def _prepare_sweep(case, seed):
    t, tg, p, g, s = _sweep_inputs(case, seed)
    p, g, s = _cuda(p), _cuda(g), _cuda(s)
    return {"case": case, "src": (p, g, s), "tgt": p if case["own"] else _cuda(t),
            "tgt_gamma": g if case["own"] else None}


def _run_sweep(st):
    from fluxvortex_gb300 import kernel as K
    q, core = st["case"]["quantity"], st["case"]["core"]
    t, tg, src = st["tgt"], st["tgt_gamma"], st["src"]
    if q == "velocity":
        return K.velocity_from_particles(t, *src, core, "f64")
    if q == "jacobian":
        return K.jacobian_from_particles(t, tg, *src, core, "f64")
    if q == "vorticity":
        return K.vorticity_from_particles(t, *src, core, "f64")
    if q == "stretching":
        return K.stretching_from_particles(t, tg, *src, core, "f64")
    return list(K.velocity_and_stretching(t, tg, *src, core, "f64"))


def _prepare_field(case, seed):
    """A field and the state that every pass starts from."""
    from fluxvortex_gb300.particles import VortexParticleField
    far = case.get("far_field")
    kw = dict(far_field=far, leaf_target=case["leaf"]) if far else {}
    f = VortexParticleField(max_particles=case["n"] + 1024, rlxf=case["relax"],
                            kernel=case.get("core", "winckelmans"),
                            precision=case.get("precision", "f32c"), **kw)
    f.add_particles_batch(*_slab(case["n"], seed))
    return {"field": f, "start": f.snapshot(), "stretch": case["stretch"],
            "u_inf": np.array(U_INF)}


def _run_field(st):
    f = st["field"]
    f.restore(st["start"])
    f.advect_rk3(DT, st["u_inf"], stretch=st["stretch"])
    out = f.snapshot()
    return {k: out[k] for k in ("pos", "gamma", "sigma", "age")}


def _prepare_hybrid(case, seed):
    """Ten steps shed the ring rows that stay rings; then the grown wake is
    seeded, and every pass is the step that follows."""
    from fluxvortex_gb300.geometry import flapping_aircraft, heaving_wing
    from fluxvortex_gb300.hybrid import HybridStep
    n = case["n"]
    if case["aircraft"]:
        cfg = flapping_aircraft(n_keep=10, free_vpm=True, stretch=True, sigma_rule="edge",
                                max_particles=n + 2048, far_field="learned")
        hs = HybridStep(cfg, precision="f32c")
        hs.field.tree.leaf_target = 32
    else:
        cfg = heaving_wing(n_keep=10, free_vpm=True, stretch=True, sigma_rule="edge",
                           max_particles=n + 2048)
        hs = HybridStep(cfg, precision="f64")
    for _ in range(10):
        hs.step()
    hs.field.add_particles_batch(*_slab(n, seed, x0=9.0 if case["aircraft"] else 4.0))
    return {"step": hs, "start": hs.snapshot()}


def _run_hybrid(st):
    hs = st["step"]
    hs.restore(st["start"])
    hs.step()
    out = hs.snapshot()
    f = out["field"]
    return {"W": out["W"], "wg": out["wg"], "gamma": out["gamma"], "cl": out["cl"],
            "cdi": out["cdi"], "pos": f["pos"], "alpha": f["gamma"], "sigma": f["sigma"],
            "n": f["np"]}


def _prepare_flutter(case, seed):
    from fluxvortex_gb300.flutter import FlutterSweep, goland
    rng = np.random.default_rng(seed)
    cfg = goland(num_chords=case["chords"], tip_w=0.05 * rng.uniform(0.8, 1.2),
                 tip_theta_deg=2.0 * rng.uniform(0.8, 1.2))
    V = cfg.velocities(case["speeds"])
    return FlutterSweep(cfg, V, precision=case["precision"], threads=256)


def _run_flutter(sw):
    sw.reset()
    sw.run(graph=True)
    return {k: sw.st[k] for k in ("hist_w", "hist_th", "d", "v")}


def _prepare_training(case, seed):
    from fluxvortex_gb300.learned import FarFieldMLP
    w, b, X, T = _network_inputs(case, seed)
    return {"net": FarFieldMLP(w, b), "X": X.cuda(), "T": T.cuda()}


def _run_training(st):
    net = st["net"]
    loss, Y = net.gradients(st["X"], st["T"])
    return {"loss": loss, "Y": Y, "gw": net.gw, "gb": net.gb}


_PREPARE = {"rings": _prepare_rings, "sweep": _prepare_sweep, "field": _prepare_field,
            "tree": _prepare_field, "hybrid": _prepare_hybrid, "flutter": _prepare_flutter,
            "training": _prepare_training}
_RUN = {"rings": _run_rings, "sweep": _run_sweep, "field": _run_field, "tree": _run_field,
        "hybrid": _run_hybrid, "flutter": _run_flutter, "training": _run_training}


def prepare(case, seed):
    return case["kind"], _PREPARE[case["kind"]](case, seed)


def run(state):
    kind, st = state
    return _RUN[kind](st)


# ---- work ------------------------------------------------------------------------


def _near(n, leaf):
    """Particles that the opening angle 0.5 leaves to direct summation per
    target: the leaves within (r_T + r_S) / 0.5 of its own."""
    return min(n, 4.0 / 3.0 * math.pi * (2.0 * math.sqrt(3.0)) ** 3 * leaf)


def _field_flops(n, pairs, stretch, relax, erf):
    per = 3 * PAIR_FLOP["velocity"] + (3 * PAIR_FLOP["stretching"] if stretch else 0)
    per += ERF_FLOP * (3 + 3 * stretch) if erf else 0
    per += PAIR_FLOP["vorticity"] + ERF_FLOP if relax else 0
    return pairs * per + 300.0 * n


def work(case):
    kind = case["kind"]
    if kind == "rings":
        n, m = case["points"], case["vortices"]
        out = n * m * 24 if case["expanded"] else n * 24
        return {"bytes": n * 24 + m * 120 + out + 32,
                "flops": float(n) * m * LEGS[case["legs"]] * LEG_FLOP}
    if kind == "sweep":
        n, m, q = case["targets"], case["sources"], case["quantity"]
        per = PAIR_FLOP[q] + (ERF_FLOP if case["core"] == "gaussianerf" else 0)
        return {"bytes": m * 56 + n * (24 + {"both": 48, "jacobian": 72}.get(q, 24)),
                "flops": float(n) * m * per}
    if kind in ("field", "tree"):
        n = case["n"]
        pairs = n * (float(n) if kind == "field" else _near(n, case["leaf"]))
        return {"bytes": n * 64 * 2,
                "flops": _field_flops(n, pairs, case["stretch"], case["relax"] > 0,
                                      case.get("core") == "gaussianerf")}
    if kind == "hybrid":
        panels = 192 if case["aircraft"] else 120
        n = case["n"] + 4 * (panels // (6 if case["aircraft"] else 10))
        pairs = n * (_near(n, 32) if case["aircraft"] else float(n))
        rings = 2.0 * panels * 10 * (panels / (6.0 if case["aircraft"] else 10.0))
        flops = (_field_flops(n, pairs, True, False, False)
                 + 2.0 * panels * n * PAIR_FLOP["velocity"]
                 + (2.0 * panels * panels + rings) * 4 * LEG_FLOP + 2.0 / 3.0 * panels ** 3)
        return {"bytes": n * 64 * 2 + panels * 400, "flops": flops}
    if kind == "flutter":
        panels, dt, chord = 32, 0.003, 1.8288
        steps, pairs = 0.0, 0.0
        for v in np.linspace(80.0, 180.0, case["speeds"]):
            k = math.ceil(case["chords"] * chord / (v * dt))
            steps += k
            pairs += sum(min(2048, 32 * max(0, i - 10)) for i in range(k))
        flops = (steps * ((2 * panels * panels + 2 * panels * 80) * 4 * LEG_FLOP
                          + 2.0 / 3.0 * panels ** 3 + 2 * 27 * 27 * 3)
                 + 2.0 * panels * pairs * PAIR_FLOP["velocity"])
        return {"bytes": steps * 16 + case["speeds"] * 27 * 8 * 6, "flops": flops}
    rows = case["rows"]
    macs = 48 * 128 + 2 * 128 * 128 + 128 * 32
    return {"bytes": rows * (96 + 128 + 128) + 2 * macs * 4,
            "flops": rows * (2.0 * macs * 3 - 2.0 * 48 * 128)}


# ---- plain FP64 results ----------------------------------------------------------


def _exact_rings(case, seed):
    pts, corners, s, rc, ages = (np.asarray(a) if not isinstance(a, list) else a
                                 for a in _ring_inputs(case, seed))
    p = _cuda(pts)
    c = [_cuda(x) for x in corners]
    s, rc, ages = _cuda(s), _cuda(rc), _cuda(ages)
    if case["legs"] == "horseshoe":
        ages = torch.zeros_like(ages)
    legs = {"ring": ((0, 1), (1, 2), (2, 3), (3, 0)), "chordwise": ((0, 1), (2, 3)),
            "horseshoe": ((0, 1), (1, 2), (2, 3))}[case["legs"]]
    rc2 = rc * rc + 5.02572 * (15.06e-6 + 1e-4 * s.abs()) * ages
    n, m = p.shape[0], s.shape[0]
    out = torch.empty((n, m, 3) if case["expanded"] else (n, 3), dtype=torch.float64,
                      device="cuda")
    chunk = max(1, 4_000_000 // m)
    for i in range(0, n, chunk):
        d = [x[None] - p[i:i + chunk, None] for x in c]
        length = [x.norm(dim=2) for x in d]
        v = torch.zeros_like(d[0])
        for a, b in legs:
            r0sq = (c[b] - c[a]).pow(2).sum(1)
            tol = 1e-10 * r0sq.sqrt()
            r3 = torch.linalg.cross(d[a], d[b])
            r3sq = r3.pow(2).sum(2)
            r12 = length[a] * length[b]
            k = (s / (4.0 * math.pi) * (length[a] + length[b]) * (r12 - (d[a] * d[b]).sum(2))
                 / (r12 * (r3sq + r0sq * rc2)))
            skip = ((r0sq.sqrt() < 2.22e-16) | (length[a] < tol) | (length[b] < tol)
                    | (r3sq.sqrt() < 1e-10 * r12))
            v += torch.where(skip, torch.zeros_like(k), k)[..., None] * r3
        out[i:i + chunk] = v if case["expanded"] else v.sum(1)
    return {"velocity": out.cpu().numpy() if case["host"] else out, "counts": None}


def _core(r2, sig, core):
    """f = g(r / sigma) / r^3 and f'(r) / r of the two cores."""
    if core == "winckelmans":
        q = r2 + sig * sig
        t = q.rsqrt()
        return (r2 + 2.5 * sig * sig) * t ** 5, -(3.0 * r2 + 10.5 * sig * sig) * t ** 7
    c = math.sqrt(2.0 / math.pi)
    x = r2 / (sig * sig)
    h, dh = torch.zeros_like(x), torch.zeros_like(x)
    xs = x.clamp(max=1.0)
    for k in range(16, -1, -1):          # g / rho^3 = c sum (-1)^k x^k / (2^k k! (2k + 3))
        a = (-1.0) ** k / (2.0 ** k * math.factorial(k) * (2 * k + 3))
        h = h * xs + a
        if k:
            dh = dh * xs + 2 * k * a
    r = r2.clamp(min=1e-300).sqrt()
    rho = r / sig
    e = torch.exp(-0.5 * x)
    g = torch.erf(rho / math.sqrt(2.0)) - c * rho * e
    small = x < 0.5
    f = torch.where(small, c * h / sig ** 3, g / r ** 3)
    fp = torch.where(small, c * dh / sig ** 5, (c * x * e / sig - 3.0 * g / r) / r ** 4)
    return f, fp


def _pairs(q, core, t, tg, p, g, s):
    """One all-pairs sweep: the outputs of quantity q at targets t."""
    m = p.shape[0]
    n_out = {"jacobian": (9,), "both": (3, 3)}.get(q, (3,))
    out = [torch.empty((t.shape[0], k), dtype=torch.float64, device="cuda") for k in n_out]
    chunk = max(1, 4_000_000 // m)
    a = -g[None] / (4.0 * math.pi)
    for i in range(0, t.shape[0], chunk):
        d = t[i:i + chunk, None] - p[None]
        r2 = d.pow(2).sum(2)
        f, fp = _core(r2, s[None], core)
        aa = a.expand_as(d)
        dxa = torch.linalg.cross(d, aa)
        res = []
        if q in ("velocity", "both"):
            res.append((f[..., None] * dxa).sum(1))
        if q in ("stretching", "both"):
            G = tg[i:i + chunk, None].expand_as(d)
            w = fp * (d * G).sum(2)
            res.append((f[..., None] * torch.linalg.cross(G, aa) + w[..., None] * dxa).sum(1))
        if q == "vorticity":
            res.append(((fp * (d * aa).sum(2))[..., None] * d
                        - aa * (fp * r2 + 2.0 * f)[..., None]).sum(1))
        if q == "jacobian":
            J = torch.einsum("tsi,tsj->tij", fp[..., None] * dxa, d)
            fa = torch.einsum("ts,si->ti", f, a[0])
            for (r, c, k, sg) in ((0, 1, 2, 1), (0, 2, 1, -1), (1, 0, 2, -1), (1, 2, 0, 1),
                                  (2, 0, 1, 1), (2, 1, 0, -1)):
                J[:, r, c] += sg * fa[:, k]
            res.append(J.reshape(-1, 9))
        for o, x in zip(out, res):
            o[i:i + chunk] = x
    return out


def _exact_sweep(case, seed):
    t, tg, p, g, s = (None if a is None else _cuda(a) for a in _sweep_inputs(case, seed))
    out = _pairs(case["quantity"], case["core"], t, tg, p, g, s)
    if case["quantity"] == "jacobian":
        return out[0].reshape(-1, 3, 3)
    return out if case["quantity"] == "both" else out[0]


def _exact_field(case, seed):
    pos, gam, sig = (_cuda(a) for a in _slab(case["n"], seed))
    core = case.get("core", "winckelmans")
    u_inf = _cuda(np.array(U_INF))
    rX, rG, rs = torch.zeros_like(pos), torch.zeros_like(gam), torch.zeros_like(sig)
    for a, b in RK3:
        u = _pairs("velocity", core, pos, None, pos, gam, sig)[0] + u_inf
        sp = u.norm(dim=1, keepdim=True)
        u = torch.where(sp > 50.0, u * (50.0 / sp), u)
        rX = a * rX + DT * u
        pos = pos + b * rX
        if not case["stretch"]:
            continue
        S = _pairs("stretching", core, pos, gam, pos, gam, sig)[0]
        g2 = gam.pow(2).sum(1)
        Z = torch.where(g2 > 1e-20, 0.2 * (S * gam).sum(1) / g2, torch.zeros_like(g2))
        Z = Z.clamp(-10.0 / DT, 10.0 / DT)
        rG = a * rG + DT * (S - 3.0 * Z[:, None] * gam)
        rs = a * rs - DT * sig * Z
        gam, sig = gam + b * rG, sig + b * rs
        n2 = gam.pow(2).sum(1, keepdim=True)
        gam = torch.where(n2 > 1e4, gam * (1e4 / n2).sqrt(), gam)
        sig = sig.clamp(1e-6, 5.0)
    if case["relax"] > 0:
        k = case["relax"]
        w = _pairs("vorticity", "gaussianerf", pos, None, pos, gam, sig)[0]
        gn, wn = gam.norm(dim=1, keepdim=True), w.norm(dim=1, keepdim=True)
        h = w / wn
        new = (1.0 - k) * gam + k * gn * h
        b2 = 1.0 - 2.0 * (1.0 - k) * k * (1.0 - (new * h).sum(1, keepdim=True)
                                          / gn.clamp(min=1e-12))
        new = new / b2.clamp(min=0.01).sqrt()
        gam = torch.where((gn > 1e-15) & (wn > 1e-12), new, gam)
    return {"pos": pos, "gamma": gam, "sigma": sig, "age": torch.full_like(sig, DT)}


def _exact_training(case, seed):
    w, b, X, T = _network_inputs(case, seed)
    w = torch.as_tensor(w).to(torch.bfloat16).double().cuda().requires_grad_(True)
    b = torch.as_tensor(b).double().cuda().requires_grad_(True)
    h, T, at, bt = X.double().cuda(), T.double().cuda(), 0, 0
    for l, (o, i) in enumerate(((128, 48), (128, 128), (128, 128), (32, 128))):
        h = h @ w[at:at + o * i].reshape(o, i).T + b[bt:bt + o]
        if l < 3:
            h = torch.nn.functional.silu(h)
        at, bt = at + o * i, bt + o
    loss = (h[:, :30] - T[:, :30]).pow(2).sum()
    (loss / (case["rows"] * 30)).backward()
    return {"loss": loss.detach().reshape(1), "Y": h.detach(), "gw": w.grad, "gb": b.grad}


def exact(case, seed):
    kind = case["kind"]
    if kind == "rings":
        return _exact_rings(case, seed)
    if kind == "sweep":
        return _exact_sweep(case, seed)
    if kind == "field" or (kind == "tree" and case["n"] <= 1 << 16):
        return _exact_field(case, seed)
    if kind == "training":
        return _exact_training(case, seed)
    return None
