"""The solver's work as its users have it done, case by case, through the public entry points of
``lightweight-mb-color-gradient-lbm_gb300/mbcg.py``.

    listed()             the cases, with their names
    draw(rng)            one more case from the same ranges
    prepare(case, seed)  what a program holds before the call: the case handle (or the caller's own
                         arrays, or a running server) with a developed two-phase state on it
    run(state)           one pass through the entry points, and what it computes
    work(case)           bytes and operations that one pass cannot do without
    exact(case, seed)    what run() returns, by a plain torch restatement of the model in 64 bits

A developed state is a two-phase field (a drop, a perturbed heavy-over-light interface, a wavy
liquid column) in a moving ambient, all made from the seed.  run() returns the fluid nodes of the
state (and the inlet and outlet layers of a jet, which a step writes too), all 11 moments in one
tensor as ``Case.copy_out`` lays them out.  In the 16-bit storage forms it returns the stored
slots, with the colour slot read as the colour field phi (the slot itself jumps between -1 and +1
where phi passes through zero).
"""
import importlib
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "lightweight-mb-color-gradient-lbm_gb300"))
mbcg = importlib.import_module("mbcg")

PRECISION = {"fp32": mbcg.FP32, "fp16": mbcg.FP16, "bf16": mbcg.BF16}
TORCH_TYPE = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
DEV = "cuda"


def listed():
    return [
        # the smallest call: one step of a small drop, as a program that looks at the state after
        # every step makes it (latency of one launch)
        {"name": "drop32_step", "kind": "drop", "q": 27, "L": 32, "prec": "fp32", "steps": 1},
        # the Laplace-test drop in its 64^3 box, stepped in blocks between two pressure samples
        {"name": "drop64_q19", "kind": "drop", "q": 19, "L": 64, "prec": "fp32", "steps": 20},
        # the largest drop of the serving mix
        {"name": "drop192_q27", "kind": "drop", "q": 27, "L": 192, "prec": "fp32", "steps": 2},
        # Rayleigh-Taylor, walls, gravity and density ratio 3, at its full size
        {"name": "rti128", "kind": "rti", "q": 27, "L": 128, "H": 512, "prec": "fp32", "steps": 2},
        # Rayleigh-Taylor in a small box whose edges are no multiple of anything, D3Q19
        {"name": "rti61_q19", "kind": "rti", "q": 19, "L": 61, "H": 243, "prec": "fp32", "steps": 8},
        # the liquid jet at full size, FP32: the headline workload
        {"name": "jet256", "kind": "jet", "q": 27, "nx": 256, "ny": 256, "nz": 1024, "prec": "fp32", "steps": 1},
        # the same jet in the FP16 storage form
        {"name": "jet256_fp16", "kind": "jet", "q": 27, "nx": 256, "ny": 256, "nz": 1024, "prec": "fp16", "steps": 1},
        # a ragged D3Q19 jet in the BF16 storage form
        {"name": "jet_ragged_bf16", "kind": "jet", "q": 19, "nx": 187, "ny": 203, "nz": 611, "prec": "bf16", "steps": 1},
        # the reference's own jet (128^3 lattice, jet along y, convective outlet) in its main loop's
        # split form: collide-and-stream, boundary pass, swap
        {"name": "split128", "kind": "split", "q": 27, "nx": 126, "ny": 126, "nz": 126, "steps": 4},
        # the same loop on the caller's own dense arrays with an odd row length, as a program that
        # keeps the reference's memory layout calls it
        {"name": "raw_odd", "kind": "raw", "q": 27, "nx": 129, "ny": 118, "nz": 121, "steps": 2},
        # FP64 conservation sums and phase statistics with droplet labelling of a large jet
        {"name": "analysis", "kind": "analysis", "q": 27, "nx": 192, "ny": 192, "nz": 512},
        # a stream of requests through the batching server: submit, wait, fetch
        {"name": "serve_mix", "kind": "serve", "requests": 8, "L": 48, "H": 96, "steps": 48},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["drop", "drop", "rti", "rti", "jet", "jet", "split", "raw", "analysis", "serve"])
    q = rng.choice([19, 27])
    prec = rng.choice(["fp32", "fp32", "fp16", "bf16"])
    # the 16-bit forms round stochastically: runs are compared after one step
    steps = 1 if prec != "fp32" else rng.choice([1, 2, 5])
    if kind == "drop":
        return {"kind": kind, "q": q, "L": log(24, 200), "prec": prec, "steps": steps}
    if kind == "rti":
        L = log(24, 128)
        return {"kind": kind, "q": q, "L": L, "H": rng.randint(2 * L, 4 * L), "prec": prec, "steps": steps}
    if kind == "jet":
        return {"kind": kind, "q": q, "nx": log(40, 256), "ny": log(40, 256), "nz": log(80, 600), "prec": prec,
                "steps": 1}
    if kind in ("split", "raw"):
        return {"kind": kind, "q": q, "nx": log(40, 200), "ny": log(40, 200), "nz": log(40, 200),
                "steps": rng.choice([1, 2, 3])}
    if kind == "analysis":
        return {"kind": kind, "q": q, "nx": log(48, 200), "ny": log(48, 200), "nz": log(96, 500)}
    return {"kind": "serve", "requests": rng.randint(3, 10), "L": log(24, 64), "H": rng.randint(64, 128),
            "steps": rng.choice([16, 24, 40])}


# ------------------------------------------------------------------ parameters and initial states
def params_of(case, seed):
    kind, prec = case["kind"], PRECISION[case.get("prec", "fp32")]
    if kind == "drop":
        return mbcg.bubble_params(case["L"], q=case["q"], precision=prec)
    if kind == "rti":
        return mbcg.rti_params(case["L"], case["H"], q=case["q"], precision=prec)
    if kind in ("jet", "analysis"):
        return mbcg.jet_params(case["nx"], case["ny"], case["nz"], q=case["q"], precision=prec, seed=seed + 1,
                               diameter=min(32.0, 0.3 * min(case["nx"], case["ny"])))
    # the reference's jet: along y, blue, convective outlet
    return mbcg.reference_jet_params(case["nx"] + 2, case["ny"] + 2, case["nz"] + 2, q=case["q"], tau=0.8, sigma=0.05,
                                     beta=0.7, radius=min(12.0, 0.2 * min(case["nx"], case["nz"])))


def inout_axis(p):
    return next((a for a in range(3) if p.bc[a] == mbcg.BC_INOUT), -1)


def wrap(t, p):
    """Ghost layers of the periodic axes of t (..., nz, ny, nx): the opposite fluid layer."""
    for a in range(3):
        if p.bc[a] == mbcg.BC_PERIODIC:
            d, n = t.dim() - 1 - a, t.shape[t.dim() - 1 - a]
            t.select(d, 0).copy_(t.select(d, n - 2))
            t.select(d, n - 1).copy_(t.select(d, 1))
    return t


def dense_state(case, p, seed):
    """A developed state as (11, nz, ny, nx) FP32, ghost frame included."""
    r = random.Random(seed)
    n = (p.nx, p.ny, p.nz)
    ax = [torch.arange(k, dtype=torch.float32, device=DEV).reshape([-1 if d == 2 - a else 1 for d in range(3)])
          for a, k in enumerate(n)]
    s = torch.zeros((11, p.nz, p.ny, p.nx), dtype=torch.float32, device=DEV)
    ia = inout_axis(p)
    if ia >= 0:
        t = [a for a in range(3) if a != ia]
        rad = torch.sqrt((ax[t[0]] - p.jet_center[0]) ** 2 + (ax[t[1]] - p.jet_center[1]) ** 2)
        edge = p.jet_radius * (1 + 0.06 * torch.sin(2 * math.pi * ax[ia] / 40.0 + r.uniform(0, 6.28)))
        depth = 0.6 * n[ia] + r.uniform(-3, 3)
        phi = torch.tanh(torch.minimum(edge - rad, depth - ax[ia]) / 2.0)
        core = 0.5 * (1 + phi)
        if p.jet_phase < 0:
            phi = -phi
    elif p.ic == mbcg.IC_BUBBLE:
        c = [0.5 * (k - 1) + r.uniform(-2, 2) for k in n]
        rad = torch.sqrt(sum((ax[a] - c[a]) ** 2 for a in range(3)))
        phi = torch.tanh((p.bubble_radius + r.uniform(-1, 1) - rad) / 3.0)
    else:
        amp = p.rti_amplitude * r.uniform(0.7, 1.3)
        pos = p.rti_position + amp * torch.cos(2 * math.pi * (ax[0] / (n[0] - 2) + r.random())) * \
            torch.cos(2 * math.pi * (ax[1] / (n[1] - 2) + r.random()))
        phi = torch.tanh((ax[2] - pos) / 4.0)
    s[0] = 0.5 * (1 + phi) * p.rho_r0
    s[1] = 0.5 * (1 - phi) * p.rho_b0
    damp = 1.0
    for a in range(3):  # no flow through or along walls
        if p.bc[a] == mbcg.BC_WALL:
            damp = torch.sin(math.pi * (ax[a] - 0.5) / (n[a] - 2))
    for a in range(3):
        b = (a + 1) % 3
        s[2 + a] = damp * 0.01 * (r.uniform(0.2, 0.6) + torch.sin(2 * math.pi * (ax[b] / (n[b] - 2) + r.random())))
    if ia >= 0:
        s[2 + ia] += p.jet_velocity * core
        last, inner = s.select(3 - ia, n[ia] - 1), s.select(3 - ia, n[ia] - 2)
        last.copy_(inner)
        face = s.select(3 - ia, 0)
        face.zero_()
        disc = (rad.select(2 - ia, 0) <= p.jet_radius).float()
        face[0 if p.jet_phase > 0 else 1] = disc
        face[1 if p.jet_phase > 0 else 0] = 1 - disc
        face[2 + ia] = disc * p.jet_velocity
    for a in range(3):
        if p.bc[a] == mbcg.BC_WALL:
            for g, f in ((0, 1), (n[a] - 1, n[a] - 2)):
                s.select(3 - a, g).copy_(s.select(3 - a, f))
                s[2:5].select(3 - a, g).zero_()
    return wrap(s, p)


def to_slots(s, p):
    """The 16-bit forms' slots (include/mbcg.h) of a dense state, in the state's own precision."""
    rho = s[0] + s[1]
    c = torch.where(s[0] >= s[1], 2 * s[1] / rho, -(2 * s[0] / rho))
    phi = torch.copysign(1 - c.abs(), c)
    out = torch.empty_like(s)
    out[0] = (rho - (0.5 * (p.rho_r0 + p.rho_b0) + 0.5 * phi * (p.rho_r0 - p.rho_b0))) / p.rho_scale
    out[1] = c
    out[2:5] = s[2:5] / p.u_ref
    out[5:] = s[5:] / p.pi_scale
    return out


def from_slots(v, p):
    """The moments (64-bit) that 16-bit slots stand for."""
    v = v.double()
    c = v[1]
    phi = torch.copysign(1 - c.abs(), c)
    rho = 0.5 * (p.rho_r0 + p.rho_b0) + 0.5 * phi * (p.rho_r0 - p.rho_b0) + p.rho_scale * v[0]
    minor = 0.5 * rho * c.abs()
    red = ~torch.signbit(c)
    out = torch.empty_like(v)
    out[0] = torch.where(red, rho - minor, minor)
    out[1] = torch.where(red, minor, rho - minor)
    out[2:5] = v[2:5] * p.u_ref
    out[5:] = v[5:] * p.pi_scale
    return out


def stored(case, s, p):
    """The dense state in the case's storage type."""
    prec = case.get("prec", "fp32")
    return s if prec == "fp32" else to_slots(s, p).to(TORCH_TYPE[prec])


# ------------------------------------------------------------------ device views
class _Memory:
    """A case's device memory for torch.  Tensors made from it keep it, and so its case, alive."""

    def __init__(self, owner, ptr, count, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 3}


def view_of(case, m, p, prec):
    """(11, nz, ny, nx) torch view of one of a case's states (mbcg_fields)."""
    es = 4 if prec == "fp32" else 2
    step = (m.f[1] - m.f[0]) // es
    flat = torch.as_tensor(_Memory(case, m.f[0], 10 * step + m.pitch * p.ny * p.nz, "<f4" if es == 4 else "<i2"),
                           device=DEV)
    if es == 2:
        flat = flat.view(TORCH_TYPE[prec])
    return flat.as_strided((11, p.nz, p.ny, p.nx), (step, m.pitch * p.ny, m.pitch, 1))


def computed(t, p):
    """The nodes a step writes: the fluid, and a jet axis's inlet and outlet layers."""
    for a in range(3):
        if p.bc[a] != mbcg.BC_INOUT:
            d = t.dim() - 1 - a
            t = t.narrow(d, 1, t.shape[d] - 2)
    return t


def outputs(v, prec):
    if prec == "fp32":
        return v
    return [v[0], torch.copysign(1 - v[1].abs(), v[1]), v[2:]]


def requests_of(case, seed):
    """The requests of a serving case: drops and Rayleigh-Taylor boxes of several sizes by turns."""
    r = random.Random(seed)
    asked = []
    for k in range(case["requests"]):
        if k % 2 == 0:
            L = max(20, int(case["L"] * (1.0 - 0.07 * k)))
            asked.append(mbcg.bubble_params(L, q=27 if k % 4 else 19, radius=0.25 * L + r.uniform(-1, 1)))
        else:
            L = max(16, int(case["L"] * (0.6 - 0.04 * k)))
            asked.append(mbcg.rti_params(L, case["H"], q=27 if k % 4 == 1 else 19,
                                         amplitude=0.05 * L * r.uniform(0.7, 1.3)))
    return asked


# ------------------------------------------------------------------ the cases
def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return {"kind": kind, "steps": case["steps"], "asked": requests_of(case, seed),
                "server": mbcg.Server(arena_bytes=1 << 30, keep_results=1)}
    p = params_of(case, seed)
    s = dense_state(case, p, seed)
    if kind == "raw":
        a, b = s, s.clone()
        return {"kind": kind, "p": p, "lib": mbcg.Library.get(), "t": [a, b], "steps": case["steps"], "done": 0,
                "m": [mbcg.moments_from_tensors([x[f] for f in range(11)], p.nx) for x in (a, b)]}
    prec = case.get("prec", "fp32")
    c = mbcg.Case(p)
    views = [view_of(c, m, p, prec) for m in c.fields()]
    for v in views:
        v.copy_(stored(case, s, p))
    return {"kind": kind, "case": c, "prec": prec, "steps": case.get("steps", 0), "cur": 0,
            "views": [computed(v, p) for v in views]}


def run(state):
    kind = state["kind"]
    if kind in ("drop", "rti", "jet"):
        state["case"].step(state["steps"])
        state["cur"] ^= state["steps"] & 1
        return outputs(state["views"][state["cur"]], state["prec"])
    if kind == "split":
        c = state["case"]
        for _ in range(state["steps"]):
            c.rcs()
            c.bc()
            c.swap()
        state["cur"] ^= state["steps"] & 1
        return state["views"][state["cur"]]
    if kind == "raw":
        lib, p, m = state["lib"], state["p"], state["m"]
        for _ in range(state["steps"]):
            a, b = m[state["done"] & 1], m[1 - (state["done"] & 1)]
            state["done"] += 1
            lib.check(lib.mbcg_rcs_moments(p, a, b, state["done"], None), "rcs")
            lib.check(lib.mbcg_bc_moments(p, b, a, state["done"], None), "bc")
        return computed(state["t"][state["done"] & 1], p)
    if kind == "analysis":
        d = state["case"].diagnostics()
        st = state["case"].phase_statistics(components=True)
        return {"sums": np.array([d["mass_r"], d["mass_b"]] + d["momentum"]),
                "area": st["interface_area"], "centroid": np.array(st["centroid"]),
                "counts": np.array([d["nonfinite"], d["nodes"], int(st["volume_tracked"]), int(st["volume_other"]),
                                    st["interface_nodes"], int(st["penetration"]), st["components"],
                                    st["largest_component"], st["detached"], st["detached_volume"]])}
    srv = state["server"]
    ids = [srv.submit(p, state["steps"]) for p in state["asked"]]
    out = []
    for rid, p in zip(ids, state["asked"]):
        srv.wait(rid)
        out.append(srv.fetch(rid, p.shape)[:, 1:-1, 1:-1, 1:-1])
        srv.release(rid)
    return out


def work(case):
    """A time step reads and writes the 11 moments of every fluid node once (22 values a node and
    step) and needs some 14 operations a direction to rebuild, collide and project."""
    kind = case["kind"]
    if kind == "serve":
        nodes = sum(p.active_nodes() for p in requests_of(case, 0))
        return {"bytes": 88 * nodes * case["steps"], "flops": 320 * nodes * case["steps"]}
    if kind == "drop":
        nodes = case["L"] ** 3
    elif kind == "rti":
        nodes = case["L"] ** 2 * (case["H"] - 2)
    else:
        nodes = case["nx"] * case["ny"] * case["nz"]
    if kind == "analysis":
        return {"bytes": 44 * nodes, "flops": 30 * nodes}  # every moment read once, a few sums out
    each = 4 if case.get("prec", "fp32") == "fp32" else 2
    return {"bytes": 22 * each * nodes * case["steps"], "flops": 14 * case["q"] * nodes * case["steps"]}


# ------------------------------------------------------------------ the model in 64 bits
def directions(q):
    w27 = (8 / 27, 2 / 27, 1 / 54, 1 / 216)
    w19 = (1 / 3, 1 / 18, 1 / 36)
    out = []
    for z in (-1, 0, 1):
        for y in (-1, 0, 1):
            for x in (-1, 0, 1):
                n = x * x + y * y + z * z
                if q == 27 or n < 3:
                    out.append(((x, y, z), (w27 if q == 27 else w19)[n]))
    return out


def uniform_noise(seed, step, node, comp):
    """xi in [-1, 1) of the inlet noise: SplitMix64 finaliser on (seed, step), then (node, component)."""
    def mix(z):
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))
    with np.errstate(over="ignore"):
        h = mix(np.array([seed], dtype=np.uint64) + np.uint64(0x9E3779B97F4A7C15) * np.uint64(step + 1))
        h = mix(h ^ (node.astype(np.uint64) * np.uint64(4) + np.uint64(comp)))
    return (h >> np.uint64(40)).astype(np.float64) / 8388608.0 - 1.0


def inner(t, p, shift=(0, 0, 0)):
    """The fluid nodes of t displaced by -shift."""
    for a in range(3):
        d = t.dim() - 1 - a
        t = t.narrow(d, 1 - shift[a], t.shape[d] - 2)
    return t


def step64(p, S, step):
    """One time step of the dense 64-bit state S (ghost frame valid): the new state."""
    n, dirs, ia = (p.nx, p.ny, p.nz), directions(p.q), inout_axis(p)
    wall = next((a for a in range(3) if p.bc[a] == mbcg.BC_WALL), -1)
    rr, rb = S[0], S[1]
    rho = rr + rb
    neq = S[2:]
    if ia >= 0:  # a ghost source takes its non-equilibrium part from the fluid layer behind it
        neq = neq.clone()
        neq.select(3 - ia, 0).copy_(neq.select(3 - ia, 1))
        neq.select(3 - ia, n[ia] - 1).copy_(neq.select(3 - ia, n[ia] - 2))
    # colour gradient at the fluid nodes
    psi = (rr - rb) / rho
    if ia >= 0:
        psi.select(2 - ia, n[ia] - 1).copy_(psi.select(2 - ia, n[ia] - 2))
    if wall >= 0:
        psi.select(2 - wall, 0).copy_(psi.select(2 - wall, 1))
        psi.select(2 - wall, n[wall] - 1).copy_(psi.select(2 - wall, n[wall] - 2))
    F = torch.zeros((3,) + tuple(rho.shape), dtype=torch.float64, device=DEV)
    for c, w in dirs:
        if any(c):
            at = inner(psi, p, (-c[0], -c[1], -c[2]))
            for a in range(3):
                if c[a]:
                    inner(F[a], p).add_(at, alpha=3 * w * c[a])
    wrap(F, p)
    mixed = 4 * rr * rb / rho ** 2 > 1e-4
    if ia >= 0:
        mixed.select(2 - ia, 0).fill_(False)
        mixed.select(2 - ia, n[ia] - 1).fill_(False)
    absF = F.square().sum(0).sqrt()
    strong = mixed & (absF > 1e-4)
    oms = 1 - 1 / p.tau
    A = 0.5 * p.sigma / (4 * (1 / 9) * p.tau)
    hA = torch.where(mixed, A * absF, torch.zeros_like(absF))
    if p.omega2_conservative:
        hA = torch.where(strong, hA, torch.zeros_like(hA))
    qF = torch.where(strong, A / absF.clamp_min(1e-300), torch.zeros_like(absF))
    ratio = p.rho_r0 != p.rho_b0
    low = min(p.rho_r0, p.rho_b0)
    K = rr * (low / p.rho_r0 - 1) + rb * (low / p.rho_b0 - 1) if ratio else None
    dc = torch.where(strong, p.beta * rr * rb / rho ** 2 / absF.clamp_min(1e-300) * (rho + K if ratio else rho),
                     torch.zeros_like(absF))
    del strong, mixed, psi
    # a population is w times a polynomial in its velocity: coefficients by the powers of cx, cy, cz
    u, v = S[2:5], neq[0:3]
    P2 = {(0, 0): neq[3], (0, 1): neq[4], (1, 1): neq[5], (1, 2): neq[6], (2, 2): neq[7], (0, 2): neq[8]}
    g = [p.gravity[a] for a in range(3)]
    forced = any(g)
    co = {}

    def put(axes, t):
        k = tuple(axes.count(a) for a in range(3))
        co[k] = co[k] + t if k in co else t

    put([], rho - 1.5 * rho * u.square().sum(0) - 1.5 * oms * (P2[0, 0] + P2[1, 1] + P2[2, 2]) - hA)
    if ratio:
        put([], K)
    if forced:
        put([], -1.5 * rho * sum(g[a] * u[a] for a in range(3)))
    for a in range(3):
        put([a], 3 * rho * u[a] + (1.5 * rho * g[a] if forced else 0))
        for b in range(a, 3):
            f = 4.5 if a == b else 9.0
            put([a, b], f * (rho * u[a] * u[b] + oms * P2[a, b]) + (1 if a == b else 2) * qF * F[a] * F[b])
            if forced:
                put([a, b], 0.5 * f * rho * (g[a] * u[b] + g[b] * u[a]))
        for b in range(3):
            if b != a:  # the third-order moment aab against c_a c_a c_b - cs^2 c_b
                t = 13.5 * (rho * u[a] * u[a] * u[b] +
                            oms * (P2[a, a] * v[b] + 2 * P2[min(a, b), max(a, b)] * v[a]))
                if forced:
                    t = t + 13.5 * rho * (g[a] * u[a] * u[b] + 0.5 * g[b] * u[a] * u[a])
                put([a, a, b], t)
                put([b], t * (-1 / 3))
    t = 27.0 * (rho * u[0] * u[1] * u[2] + oms * (P2[0, 1] * v[2] + P2[0, 2] * v[1] + P2[1, 2] * v[0]))
    if forced:
        t = t + 13.5 * rho * (g[0] * u[1] * u[2] + g[1] * u[0] * u[2] + g[2] * u[0] * u[1])
    put([0, 1, 2], t)
    B0 = -10 / 27 if p.q == 27 else -1 / 3

    def population(c, w, cut):
        """(total, red) populations of velocity c at the nodes that cut selects."""
        gi = 0
        for k, t in co.items():
            s = 1
            for a in range(3):
                s *= c[a] ** k[a]
            if s:
                gi = gi + s * cut(t)
        gi = w * gi
        if not any(c):
            gi = gi + (w - B0) * cut(hA)
            if ratio:
                gi = gi - cut(K)
        ri = cut(rr) / cut(rho) * gi
        if any(c):
            fc = sum(c[a] * cut(F[a]) for a in range(3) if c[a])
            ri = ri + (w / math.sqrt(sum(k * k for k in c))) * cut(dc) * fc
        return gi, ri

    M = torch.zeros((11,) + tuple(inner(rho, p).shape), dtype=torch.float64, device=DEV)
    for c, w in dirs:
        gi, ri = population(c, w, lambda t: inner(t, p, c))
        if wall >= 0 and c[wall]:  # halfway bounce-back off the wall behind the node
            plane = 0 if c[wall] > 0 else n[wall] - 3
            own = population((-c[0], -c[1], -c[2]), w, lambda t: inner(t, p).select(2 - wall, plane))
            gi.select(2 - wall, plane).copy_(own[0])
            ri.select(2 - wall, plane).copy_(own[1])
        M[0] += ri
        M[1] += gi
        for a in range(3):
            if c[a]:
                M[2 + a].add_(gi, alpha=c[a])
        for k, (a, b) in enumerate(((0, 0), (0, 1), (1, 1), (1, 2), (2, 2), (0, 2))):
            h = c[a] * c[b] - (1 / 3 if a == b else 0)
            if h:
                M[5 + k].add_(gi, alpha=h)
        del gi, ri
    R = M[1].clone()
    M[1] -= M[0]
    G = [R * g[a] for a in range(3)] if forced else None
    for a in range(3):
        if forced:
            M[2 + a] += 0.5 * G[a]
        M[2 + a] /= R
    for k, (a, b) in enumerate(((0, 0), (0, 1), (1, 1), (1, 2), (2, 2), (0, 2))):
        M[5 + k] -= R * M[2 + a] * M[2 + b]
        if forced:
            M[5 + k] += 0.5 * (M[2 + a] * G[b] + M[2 + b] * G[a])
        if ratio and a == b:
            M[5 + k] -= (M[0] * (low / p.rho_r0 - 1) + M[1] * (low / p.rho_b0 - 1)) / 3
    out = S.clone()
    inner(out, p).copy_(M)
    del M
    if ia >= 0:
        d = 3 - ia
        face, first = out.select(d, 0), out.select(d, 1)
        t = [a for a in range(3) if a != ia]
        uu = torch.arange(n[t[0]], device=DEV, dtype=torch.float64).reshape(1, -1)
        vv = torch.arange(n[t[1]], device=DEV, dtype=torch.float64).reshape(-1, 1)
        disc = ((uu - p.jet_center[0]) ** 2 + (vv - p.jet_center[1]) ** 2 <= p.jet_radius ** 2).double()
        face[0 if p.jet_phase > 0 else 1] = disc
        face[1 if p.jet_phase > 0 else 0] = 1 - disc
        face[2:5] = 0
        face[2 + ia] = disc * p.jet_velocity
        if p.inlet_noise:
            stride = (1, p.nx, p.nx * p.ny)
            node = np.arange(n[t[0]])[None, :] * stride[t[0]] + np.arange(n[t[1]])[:, None] * stride[t[1]]
            for a in range(3):
                xi = uniform_noise(p.seed, step, node, a)
                face[2 + a] += disc * p.jet_velocity * p.inlet_noise * torch.from_numpy(xi).to(DEV)
        face[5:] = first[5:]
        last, old, end = out.select(d, n[ia] - 1), S.select(d, n[ia] - 1), out.select(d, n[ia] - 2)
        if p.outlet == mbcg.OUTLET_ZERO_GRADIENT:
            last.copy_(end)
        else:
            uc = end[2 + ia].clamp(0, 1)
            last[:5] = old[:5] - uc * (old[:5] - end[:5])
            last[5:] = end[5:]
    return wrap(out, p)


def initial64(p):
    """mbcg_init's drop and Rayleigh-Taylor states in 64 bits."""
    n = (p.nx, p.ny, p.nz)
    ax = [torch.arange(k, dtype=torch.float64, device=DEV).reshape([-1 if d == 2 - a else 1 for d in range(3)])
          for a, k in enumerate(n)]
    if p.ic == mbcg.IC_BUBBLE:
        rad = torch.sqrt(sum((ax[a] - p.bubble_center[a]) ** 2 for a in range(3)))
        phi = p.bubble_phase * torch.tanh((p.bubble_radius - rad) / p.bubble_width)
    else:
        pos = p.rti_position + p.rti_amplitude * torch.cos(2 * math.pi * p.rti_mode[0] * ax[0] / (n[0] - 2)) * \
            torch.cos(2 * math.pi * p.rti_mode[1] * ax[1] / (n[1] - 2))
        phi = p.rti_phase_above * torch.tanh((ax[2] - pos) / p.rti_width)
    s = torch.zeros((11, p.nz, p.ny, p.nx), dtype=torch.float64, device=DEV)
    s[0] = 0.5 * (1 + phi) * p.rho_r0
    s[1] = 0.5 * (1 - phi) * p.rho_b0
    return wrap(s, p)


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        out = []
        for p in requests_of(case, seed):
            s = initial64(p)
            for k in range(case["steps"]):
                s = step64(p, s, k + 1)
            out.append(inner(s, p).cpu().numpy())
        return out
    p = params_of(case, seed)
    s = dense_state(case, p, seed)
    if kind == "analysis":
        f = inner(s, p).double()
        rho = f[0] + f[1]
        sums = [f[0].sum(), f[1].sum()] + [(rho * f[2 + a]).sum() for a in range(3)]
        return {"sums": np.array([float(v) for v in sums]), "area": None, "centroid": None, "counts": None}
    prec = case.get("prec", "fp32")
    S = s.double() if prec == "fp32" else from_slots(stored(case, s, p), p)
    del s
    for k in range(case["steps"]):
        S = step64(p, S, k + 1)
    S = computed(S, p)
    if prec == "fp32":
        return S
    v = to_slots(S, p)
    return [v[0], torch.copysign(1 - v[1].abs(), v[1]), v[2:]]
