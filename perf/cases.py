"""The calls whose speed this repository answers for, and how each is set up, run and checked.

Every case goes through the package's public classes (``GpuSystem``, ``Mlp``, ``Analysis`` and the
``surrogate_*`` functions of ``souffle_gb300.gpu``), the way a user's program does.  Workloads are
those of the package: the 10-bead single-layer capsomere and the 42-bead two-layer capsomere, with
the shared options of ``souffle_gb300.workloads``.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "capsid-souffle_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from souffle_gb300 import analysis, geometry, gpu, state, workloads  # noqa: E402


# ---- the cases --------------------------------------------------------------------------------

def listed():
    return [
        # the smallest run there is: the test-suite's 200-bead system, where launches and latency count
        {"name": "md_patch_20", "kind": "md", "template": "patch_n3", "subunits": 20, "systems": 1, "steps": 100,
         "debye": 1.0, "conc": 800.0, "big_beads": 0},
        # the reference's default number of subunits (-S 64), an ordinary desktop run
        {"name": "md_bilayer_64", "kind": "md", "template": "bilayer_n5", "subunits": 64, "systems": 1, "steps": 100,
         "debye": 1.0, "conc": 800.0, "big_beads": 0},
        # the headline workload: 84,000 beads
        {"name": "md_bilayer_2000", "kind": "md", "template": "bilayer_n5", "subunits": 2000, "systems": 1,
         "steps": 100, "debye": 1.0, "conc": 800.0, "big_beads": 0},
        # the largest single system: 840,000 beads
        {"name": "md_bilayer_20000", "kind": "md", "template": "bilayer_n5", "subunits": 20000, "systems": 1,
         "steps": 40, "debye": 1.0, "conc": 800.0, "big_beads": 0},
        # a parameter sweep: 64 replicas of 20-500 subunits with their own attraction, screening
        # length and concentration, in one handle
        {"name": "md_replicas_64", "kind": "replicas", "systems": 64, "steps": 20, "surrogate": False},
        # Brownian dynamics (-D b) of a medium system, an odd number of subunits
        {"name": "bd_bilayer_333", "kind": "bd", "template": "bilayer_n5", "subunits": 333, "systems": 1, "steps": 50,
         "debye": 1.0, "conc": 800.0, "big_beads": 0},
        # the drop-in forceCalculation with its stretching and bending parts and a list rebuild:
        # positions in, forces out, every call
        {"name": "forces_bilayer_777", "kind": "forces", "template": "bilayer_n5", "subunits": 777, "rebuild": True,
         "parts": True, "debye": 1.0, "conc": 800.0, "big_beads": 0},
        # the energy block of an output step, with the per-bead energies that the movie writer prints
        {"name": "energies_bilayer_2000", "kind": "energies", "template": "bilayer_n5", "subunits": 2000,
         "per_bead": True, "debye": 1.0, "conc": 800.0, "big_beads": 0},
        # inference of the far-field network: the far pairs of the 256-replica sweep
        {"name": "mlp_forward_118016", "kind": "mlp_forward", "rows": 118016, "width": 128},
        # one minibatch of its training: loss and gradients of every parameter
        {"name": "mlp_gradients_4096", "kind": "mlp_gradients", "rows": 4096, "width": 128},
        # the parameter sweep with the trained far-field network in the force path
        {"name": "surrogate_replicas_64", "kind": "replicas", "systems": 64, "steps": 20, "surrogate": True},
        # post-run analysis: four trajectory frames of 86,000 beads from host arrays
        {"name": "analysis_2000", "kind": "analysis", "subunits": 2000, "frames": 4, "image": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: sizes over their logarithm, odd ones among them."""
    kind = rng.choice(["md", "md", "md", "bd", "forces", "energies", "mlp_forward", "mlp_gradients", "replicas",
                       "analysis"])
    if kind in ("md", "bd", "forces", "energies"):
        small = rng.random() < 0.25
        c = {"kind": kind, "template": "patch_n3" if small else "bilayer_n5",
             "subunits": _log_int(rng, 20, 400) if small else _log_int(rng, 20, 8000),
             "debye": round(rng.choice([1.0, 1.0, rng.uniform(0.7, 2.0)]), 3),
             "conc": round(rng.choice([800.0, rng.uniform(200.0, 1000.0)]), 1),
             "big_beads": rng.choice([0, 0, 0, 8]) if kind in ("md", "bd") else 0}
        if kind in ("md", "bd"):
            c["systems"] = 1
            c["steps"] = rng.choice([10, 17, 20, 33, 40])
        elif kind == "forces":
            c["rebuild"] = True
            c["parts"] = rng.random() < 0.5
        else:
            c["per_bead"] = rng.random() < 0.5
        return c
    if kind == "mlp_forward":
        return {"kind": kind, "rows": _log_int(rng, 100, 118016), "width": rng.choice([128, 256])}
    if kind == "mlp_gradients":
        return {"kind": kind, "rows": _log_int(rng, 500, 4096), "width": rng.choice([128, 256])}
    if kind == "replicas":
        return {"kind": kind, "systems": rng.randint(3, 48), "steps": 20, "surrogate": False}
    return {"kind": "analysis", "subunits": _log_int(rng, 50, 2000), "frames": rng.randint(1, 4),
            "image": rng.randint(0, 1)}


# ---- inputs -----------------------------------------------------------------------------------

def _template(name):
    return geometry.template_by_name(name)


def _warm(w, seed):
    """The workload as in a run under way: some subunits (a sixteenth, at most 200) moved into contact with another one
    (closest beads 1.05 to 1.6 sigma apart, so that the LJ and WCA terms act), and every subunit out
    of its rest shape by normal displacements of 0.015 sigma (a spring of 1000 kT moves by 0.03)."""
    rng = np.random.default_rng(40_000 + seed)
    L, n = w.state.box, w.template.n_beads
    wrap = lambda d: d - L * np.floor(d / L + 0.5)  # noqa: E731
    p = w.state.pos.reshape(-1, n, 3)
    local = wrap(p - p[:, :1])
    c = p[:, 0] + local.mean(axis=1)
    local -= local.mean(axis=1, keepdims=True)
    apart = 2 * float(np.sqrt(((w.template.pos - w.template.pos.mean(axis=0)) ** 2).sum(axis=1)).max()) + 1.0
    S = len(p)
    order = rng.permutation(S)
    for k in range(min(200, max(4, S // 16))):
        host, guest = order[2 * k], order[2 * k + 1]
        u = rng.normal(size=3)
        u /= np.linalg.norm(u)
        want = rng.uniform(1.05, 1.6)
        rel = local[host][:, None] - local[guest][None]
        lo, hi = 0.0, 9.5  # the largest centre distance whose closest beads are `want` apart
        for d in np.arange(9.0, 0.0, -0.5):
            if np.sqrt(((rel - d * u) ** 2).sum(-1)).min() < want:
                lo = d
                break
            hi = d
        for _ in range(6):
            mid = 0.5 * (lo + hi)
            if np.sqrt(((rel - mid * u) ** 2).sum(-1)).min() < want:
                lo = mid
            else:
                hi = mid
        at = c[host] + hi * u
        d = np.sqrt((wrap(c - at) ** 2).sum(-1))
        d[[host, guest]] = np.inf
        if d.min() > apart:
            c[guest] = at
    p = (local + c[:, None]).reshape(-1, 3)
    p = wrap(p + 0.015 * rng.standard_normal(p.shape))
    w.state.pos = np.where(p >= L / 2, p - L, p)
    return w


def _workload(case, seed):
    over = {"c": state.salt_for_debye_length(case["debye"]), "C": case["conc"]}
    if case["kind"] == "bd":
        over.update(D="b", d=100.0)
    return _warm(workloads.make(_template(case["template"]), case["subunits"], seed=1000 + seed, **over), seed)


BIG = dict(sigma=6.0, charge=-78.0, shc=3.5)  # the reference's -a 3 -G -78 -H 3.5


def _big_beads(case, w, seed):
    n = case.get("big_beads", 0)
    return workloads.place_big_beads(w, n, radius=BIG["sigma"] / 2, seed=50 + seed) if n else None


def _replica_workloads(case, seed):
    """The sweep of ``workloads.replicas``: the systems' sizes and parameters belong to the case,
    their initial states to the seed."""
    rng = np.random.default_rng(case["systems"])
    t = geometry.bilayer_n5()
    out = []
    for k in range(case["systems"]):
        S = int(rng.integers(20, 501))
        over = {"E": float(rng.uniform(1.5, 3.0)), "c": state.salt_for_debye_length(float(rng.uniform(0.5, 2.0))),
                "C": float(rng.uniform(200.0, 1600.0))}
        out.append(_warm(workloads.make(t, S, seed=1000 * seed + k, name=f"replica{k}", **over), 1000 * seed + k))
    return out


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    out = t.numpy()
    out[...] = a
    return out


def _handle(ws):
    return gpu.GpuSystem(ws[0].template, [gpu.system_params(w.opt, w.derived, int(w.opt.S), w.center_local) for w in ws])


N_IN, N_OUT = 64, 132  # the network's shape for the 42-bead capsomere: 64 -> w -> w -> w -> 6 + 3 * 42


def _mlp_shapes(width):
    dims = [N_IN, width, width, width, N_OUT]
    return [(dims[i + 1], dims[i]) for i in range(4)]


def _mlp_data(case, seed):
    """Parameters (flat, the layout of souffle_mlp_set_params), normalised inputs and targets."""
    rng = np.random.default_rng(7000 + seed)
    parts = []
    for o, i in _mlp_shapes(case["width"]):
        lim = math.sqrt(3.0 / i)
        parts.append(rng.uniform(-lim, lim, (o, i)).astype(np.float32).reshape(-1))
        parts.append(rng.uniform(-0.1, 0.1, o).astype(np.float32))
    x = rng.standard_normal((case["rows"], N_IN), dtype=np.float32)
    t = rng.standard_normal((case["rows"], N_OUT), dtype=np.float32)
    return np.concatenate(parts), x, t


def _trained_replicas(ws):
    """A handle over the replicas with the far-field network trained a little and switched on."""
    s = _handle(ws)
    far_cap = max(4096, 16 * sum(int(w.opt.S) for w in ws))
    net = gpu.Mlp(N_IN, N_OUT, max_batch=far_cap, seed=7, width=128)
    gpu.surrogate_attach(s, net, ws[0].template.pos, switch_radius=3.0, far_capacity=far_cap, judge_tolerance=1.0)
    s.set_state(np.concatenate([w.state.pos for w in ws]), np.concatenate([w.state.vel for w in ws]))
    x = torch.empty((far_cap, N_IN), dtype=torch.float32, device="cuda")
    t = torch.empty((far_cap, N_OUT), dtype=torch.float32, device="cuda")
    n = gpu.surrogate_collect(s, x.data_ptr(), t.data_ptr(), far_cap)
    gpu.surrogate_fit(s, x.data_ptr(), t.data_ptr(), n, 3, 4096, 1e-3, seed=11)
    gpu.surrogate_enable(s, True)
    return s


def prepare(case, seed):
    k = case["kind"]
    st = {"case": case}
    if k in ("md", "bd", "replicas", "forces", "energies"):
        if k == "replicas":
            ws = _replica_workloads(case, seed)
        else:
            ws = [_workload(case, seed)]
        if k == "replicas" and case["surrogate"]:
            st["sys"] = _trained_replicas(ws)
        else:
            st["sys"] = _handle(ws)
            big = _big_beads(case, ws[0], seed)
            if big is not None:
                st["sys"].set_big_beads(big, **BIG)
        pos = np.concatenate([w.state.pos for w in ws])
        vel = np.concatenate([w.state.vel for w in ws])
        if k in ("md", "bd", "replicas"):
            # what a driver program keeps: page-locked state buffers
            st["pos"], st["vel"] = _pinned(pos), _pinned(vel)
            st["pos_out"], st["vel_out"] = _pinned(np.zeros_like(pos)), _pinned(np.zeros_like(vel))
        elif k == "forces":
            st["pos"] = pos
        else:
            st["sys"].set_state(pos, vel)
            st["sys"].md_begin()
    elif k in ("mlp_forward", "mlp_gradients"):
        p, x, t = _mlp_data(case, seed)
        st["net"] = gpu.Mlp(N_IN, N_OUT, max_batch=case["rows"], seed=1, width=case["width"])
        st["net"].set_params(p)
        st["x"] = torch.from_numpy(x).cuda()
        if k == "mlp_forward":
            st["y"] = torch.empty((case["rows"], N_OUT), dtype=torch.float32, device="cuda")
        else:
            st["t"] = torch.from_numpy(t).cuda()
    else:
        types, frames, box, np_ = workloads.analysis_frames(case["subunits"], case["frames"], seed=900 + seed)
        st["an"] = analysis.Analysis(frames.shape[1], np_, box, image=case["image"])
        st["types"], st["frames"] = types, frames
    return st


# ---- one pass ---------------------------------------------------------------------------------

def run(st):
    case = st["case"]
    k = case["kind"]
    if k in ("md", "bd", "replicas"):
        # a simulation segment: state in, initial forces, steps, state out
        s = st["sys"]
        s.set_state(st["pos"], st["vel"])
        s.md_begin()
        s.md_enqueue(0, case["steps"])
        s.snapshot_enqueue(0, st["pos_out"], st["vel_out"])
        s.snapshot_wait(0)
        return {"pos": st["pos_out"], "vel": st["vel_out"], "scalars": [np.array(s.md_scalars(0))]}
    if k == "forces":
        s = st["sys"]
        s.set_state(st["pos"])
        f = s.forces(rebuild=case["rebuild"], parts=case["parts"])
        return list(f) if case["parts"] else [f]
    if k == "energies":
        if case["per_bead"]:
            tot, beads = st["sys"].energies(0, per_bead=True)
        else:
            tot, beads = st["sys"].energies(0), {}
        return {"totals": {n: tot[n] for n in ("kinetic", "stretching", "bending", "lj", "electrostatic")},
                "beads": beads}
    if k == "mlp_forward":
        st["net"].forward(st["x"].data_ptr(), case["rows"], st["y"].data_ptr())
        return st["y"]
    if k == "mlp_gradients":
        loss, g = st["net"].gradients(st["x"].data_ptr(), st["t"].data_ptr(), case["rows"])
        return {"loss": loss, "grad": g}
    return st["an"].frames(st["frames"], st["types"])


# ---- what a pass cannot do without ------------------------------------------------------------

PAIR_FLOPS = 30.0    # one directed screened-Coulomb pair on a bead's list
EDGE_FLOPS = 30.0
QUAD_FLOPS = 300.0


def _md_flops(t, n_sub, steps, debye):
    # partners of a bead inside its own subunit, once per unordered pair, plus the bonded terms
    intra = n_sub * t.n_beads * (t.n_beads - 1) / 2.0
    quads = float(np.count_nonzero(np.asarray(t.edge_type)))
    return steps * (intra * PAIR_FLOPS + n_sub * (len(t.edges) * EDGE_FLOPS + quads * QUAD_FLOPS))


def work(case):
    k = case["kind"]
    if k in ("md", "bd"):
        t = _template(case["template"])
        n = case["subunits"] * t.n_beads
        return {"bytes": 4.0 * 24 * n, "flops": _md_flops(t, case["subunits"], case["steps"] + 1, case["debye"])}
    if k == "replicas":
        t = _template("bilayer_n5")
        sub = 260 * case["systems"]
        return {"bytes": 4.0 * 24 * sub * t.n_beads, "flops": _md_flops(t, sub, case["steps"] + 1, 1.25)}
    if k == "forces":
        t = _template(case["template"])
        n = case["subunits"] * t.n_beads
        return {"bytes": 24.0 * n * (4 if case["parts"] else 2), "flops": _md_flops(t, case["subunits"], 1, case["debye"])}
    if k == "energies":
        t = _template(case["template"])
        n = case["subunits"] * t.n_beads
        return {"bytes": n * (48.0 + (40.0 if case["per_bead"] else 0.0)),
                "flops": _md_flops(t, case["subunits"], 1, case["debye"])}
    if k in ("mlp_forward", "mlp_gradients"):
        p = sum(o * i for o, i in _mlp_shapes(case["width"]))
        f = 2.0 * case["rows"] * p
        if k == "mlp_forward":
            return {"bytes": 4.0 * case["rows"] * (N_IN + N_OUT) + 4.0 * p, "flops": f}
        first = 2.0 * case["rows"] * N_IN * case["width"]
        return {"bytes": 4.0 * case["rows"] * (N_IN + N_OUT) + 8.0 * p, "flops": 3.0 * f - first}
    n = case["subunits"] * 43
    pcf = 4.0 * case["subunits"]
    return {"bytes": case["frames"] * (28.0 * n + 8.0 * 4 * case["subunits"]),
            "flops": case["frames"] * 10.0 * pcf * pcf / 2}


# ---- the same results in 64 bits --------------------------------------------------------------
# Plain torch on the GPU in float64: the reference's formulas (forces.cpp, energies.cpp, edge.cpp,
# functions.cpp, md.cpp) over arrays.

class _Exact:
    """One system's force field over float64 tensors."""

    def __init__(self, w, big=None):
        t, o, d = w.template, w.opt, w.derived
        dev = "cuda"
        self.np, self.S = t.n_beads, int(o.S)
        f64 = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=dev)  # noqa: E731
        i64 = lambda a: torch.as_tensor(np.asarray(a, dtype=np.int64), device=dev)    # noqa: E731
        self.L, self.o, self.d, self.cl = float(d.box), o, d, w.center_local
        self.q, self.sig, self.m, self.type = f64(t.charge), f64(t.diameter), f64(t.mass), i64(t.types)
        self.edges, self.len0 = i64(t.edges).reshape(-1, 2), f64(t.edge_len0)
        self.w = self.q * torch.exp(d.kappa * self.sig / 2) / (1 + d.kappa * self.sig / 2) * math.sqrt(d.lb)
        att = torch.zeros((self.np, self.np), dtype=torch.bool, device=dev)
        for a, b in t.lj_attract:
            att |= (self.type[:, None] == a) & (self.type[None, :] == b)
        self.att = att
        shc = (self.sig[:, None] + self.sig[None, :]) / 2
        self.shc = shc
        self.eps = torch.where(att, torch.where(self.type[None, :] == 7, 50.0, float(o.E)), 1.0).double()
        self.s6 = torch.where(att, self.sig[:, None] ** 6 + 0 * shc, shc ** 6)
        self.cut2 = torch.where(att, torch.full_like(shc, d.ecut ** 2), (1.12246205 * shc) ** 2)
        self.qq = self.q[:, None] * self.q[None, :]
        # bending quads of the edges with a bending type: both faces in face order
        faces, quads = [tuple(int(v) for v in f) for f in t.faces], []
        for e, (a, b) in enumerate(t.edges):
            if not t.edge_type[e]:
                continue
            fs = [f for f in faces if a in f and b in f]
            quads.append((int(a), int(b), fs[0], fs[1]))
        self.f0 = i64([x[2] for x in quads]).reshape(-1, 3)
        self.f1 = i64([x[3] for x in quads]).reshape(-1, 3)
        self.quad_beads = i64([[x[0], x[1], next(v for v in x[2] if v not in x[:2]),
                                next(v for v in x[3] if v not in x[:2])] for x in quads]).reshape(-1, 4)
        self.big = f64(big) if big is not None else None

    def wrap(self, x):
        return x - self.L * torch.round(x / self.L)

    def bonded(self, pos):
        """Stretching and bending forces [S, np, 3]."""
        p = pos.reshape(self.S, self.np, 3)
        a, b = self.edges[:, 0], self.edges[:, 1]
        lv = self.wrap(p[:, a] - p[:, b])
        ln = lv.norm(dim=-1)
        f = lv * ((self.len0 - ln) * self.o.s / ln)[..., None]
        sf = torch.zeros_like(p).index_add_(1, a, f).index_add_(1, b, -f)
        # -grad of kb (1 - |n0 . n1|) by autograd over per-quad vectors from the subunit's first bead
        x = self.wrap(p - p[:, :1]).detach().requires_grad_(True)
        with torch.enable_grad():
            self.bend_energy(x).sum().backward()
        return sf, -x.grad

    def bend_energy(self, x):
        def area(f):
            return torch.linalg.cross(x[:, f[:, 1]] - x[:, f[:, 0]], x[:, f[:, 2]] - x[:, f[:, 1]])
        A0, A1 = area(self.f0), area(self.f1)
        c = (A0 * A1).sum(-1) / (A0.norm(dim=-1) * A1.norm(dim=-1))
        return self.o.b * (1 - c.abs())

    def blocks(self, pos, r2max):
        """Subunit pairs (i, j), both directions and i == j, with centre distance^2 < r2max."""
        c = pos.reshape(self.S, self.np, 3)[:, self.cl]
        out = []
        step = max(1, 40_000_000 // self.S)
        for i0 in range(0, self.S, step):
            d = self.wrap(c[i0:i0 + step, None] - c[None])
            ij = ((d * d).sum(-1) < r2max).nonzero()
            out.append(ij + torch.tensor([i0, 0], device=ij.device))
        return torch.cat(out)

    def rebuild(self, pos):
        """Directed bead pairs on the reference's lists (its prefilter and stale-distance rule kept)."""
        nl2 = float(self.d.nlist_cutoff) ** 2
        p = pos.reshape(self.S, self.np, 3)
        blk = self.blocks(pos, 2.25 * nl2)
        gi, gj = [], []
        n, cl = self.np, self.cl
        eye = torch.eye(n, dtype=torch.bool, device=pos.device)
        charged = (self.qq != 0) & ~eye
        step = max(1, 8_000_000 // (n * n))
        for b0 in range(0, len(blk), step):
            b = blk[b0:b0 + step]
            i, j = b[:, 0], b[:, 1]
            d = self.wrap(p[i][:, :, None] - p[j][:, None])
            r2 = (d * d).sum(-1)
            same = (i == j)[:, None, None]
            seen = torch.where(same, charged, torch.ones_like(charged))
            zero = (i == 0) | (j == 0)
            if bool(zero.any()):
                for k in zero.nonzero().reshape(-1).tolist():
                    stale = torch.zeros_like(eye)
                    if int(i[k]) == 0:
                        stale[cl, :] = True
                    if int(j[k]) == 0:
                        stale[:, cl] = True
                    fresh = (seen[k] & ~stale).reshape(-1)
                    at = torch.arange(n * n, device=pos.device)
                    last = torch.cummax(torch.where(fresh, at, torch.full_like(at, -1)), 0).values
                    init = r2[k, cl, cl] if int(i[k]) != int(j[k]) else torch.zeros((), dtype=r2.dtype, device=r2.device)
                    flat = r2[k].reshape(-1)
                    r2[k] = torch.where(last >= 0, flat[last.clamp(min=0)], init).reshape(n, n)
            hit = (seen & (r2 < nl2)).nonzero()
            gi.append(i[hit[:, 0]] * n + hit[:, 1])
            gj.append(j[hit[:, 0]] * n + hit[:, 2])
        self.gi, self.gj = torch.cat(gi), torch.cat(gj)

    def pair_force(self, pos):
        out = torch.zeros_like(pos)
        kap, ecut_el = self.d.kappa, self.d.ecut_el
        for k0 in range(0, len(self.gi), 16_000_000):
            i, j = self.gi[k0:k0 + 16_000_000], self.gj[k0:k0 + 16_000_000]
            li, lj = i % self.np, j % self.np
            d = self.wrap(pos[i] - pos[j])
            r2 = (d * d).sum(-1)
            r = r2.sqrt()
            c = self.w[li] * self.w[lj] * torch.exp(-kap * r) / r2 * (kap + 1 / r)
            if ecut_el != 0:
                c = torch.where(r < ecut_el, c, torch.zeros_like(c))
            inter = (i // self.np) != (j // self.np)
            s6 = self.s6[li, lj] / (r2 * r2 * r2)
            lj_c = 48.0 * self.eps[li, lj] * s6 * (s6 - 0.5) / r2
            c = c + torch.where(inter & (r2 < self.cut2[li, lj]), lj_c, torch.zeros_like(c))
            out.index_add_(0, i, d * c[:, None])
        return out

    def big_force(self, pos):
        l = torch.arange(pos.shape[0], device=pos.device) % self.np
        sl, wl = self.sig[l], self.w[l]
        kap, sb, shc = self.d.kappa, BIG["sigma"], BIG["shc"]
        wb = BIG["charge"] * math.exp(kap * sb / 2) / (1 + kap * sb / 2) * math.sqrt(self.d.lb)
        out = torch.zeros_like(pos)
        for b in self.big:
            d = self.wrap(b - pos)
            r = d.norm(dim=-1)
            c = torch.where(r < self.d.ecut_el, wb * wl * torch.exp(-kap * r) / r ** 2 * (kap + 1 / r), 0 * r)
            delta = (sb + sl) / 2 - shc
            s6 = (shc / (r - delta)) ** 6
            c = c + torch.where(r < delta + 1.12246205 * shc, 48 * s6 * (s6 - 0.5) / r / (r - delta), 0 * r)
            out -= d * c[:, None]
        return out

    def forces(self, pos, rebuild):
        if rebuild:
            self.rebuild(pos)
        sf, bf = self.bonded(pos)
        sf, bf = sf.reshape(-1, 3), bf.reshape(-1, 3)
        f = sf + bf + self.pair_force(pos)
        if self.big is not None:
            f = f + self.big_force(pos)
        return f, sf, bf


class _Chain:
    """The Nose-Hoover chain in double (update_chain_xi, THERMOSTAT::update_eta)."""

    def __init__(self, o, T, n):
        m = int(o.q)
        self.q = [o.Q] + [1.0] * (m - 2) + [0.0] if m > 1 else [0.0]
        self.dof = [3.0 * n] + [1.0] * (m - 2) + [3.0 * n] if m > 1 else [3.0 * n]
        self.xi, self.dt, self.T = [0.0] * (m + 1), o.t, T

    def link(self, j, ke):
        if self.q[j] == 0:
            return
        x, dt = self.xi, self.dt
        g = 2 * ke - self.dof[0] * self.T if j == 0 else self.q[j - 1] * x[j - 1] ** 2 - self.dof[j] * self.T
        x[j] = x[j] * math.exp(-0.5 * dt * x[j + 1]) + 0.5 * dt / self.q[j] * g * math.exp(-0.25 * dt * x[j + 1])

    def backward(self, ke):
        for j in range(len(self.q) - 1, -1, -1):
            self.link(j, ke)
        return math.exp(-0.5 * self.dt * self.xi[0])

    def forward(self, ke):
        for j in range(len(self.q)):
            self.link(j, ke)


def _minstd_uniforms(x, count):
    """count values of uniform_real_distribution(-0.5, 0.5) from minstd_rand0 at state x, and the next state."""
    M, g = 2147483647, 2 * count
    draws = np.empty(g, dtype=np.int64)
    draws[0] = x * 16807 % M
    have, mult = 1, 16807
    while have < g:
        k = min(have, g - have)
        draws[have:have + k] = draws[:k] * mult % M
        have += k
        mult = mult * mult % M if have < g else mult
    r = 2147483646.0
    u = ((draws[0::2] - 1).astype(np.float64) + (draws[1::2] - 1).astype(np.float64) * r) / (r * r)
    return np.minimum(u, 0.99999999999999988898) - 0.5, int(draws[-1])


def _exact_md(w, steps, big, dt):
    e = _Exact(w, big)
    pos = torch.as_tensor(w.state.pos, dtype=torch.float64, device="cuda").clone()
    vel = torch.as_tensor(w.state.vel, dtype=torch.float64, device="cuda").clone()
    n = pos.shape[0]
    mass = e.m.repeat(e.S)[:, None]
    brownian = w.opt.D == "b"
    f, _, _ = e.forces(pos, True)
    ke = float((0.5 * mass * vel * vel).sum())
    ch = _Chain(w.opt, w.derived.T_reduced, n)
    lcg, vcom = 69521, 0.0
    for a in range(steps):
        ef = 1.0 if brownian else ch.backward(ke)
        kick = 0.5 * dt * math.sqrt(ef) / mass
        if brownian:
            drag = -mass * vel / float(w.opt.d)
        vel = vel * ef + f * kick
        pos = e.wrap(pos + vel * dt)
        f, _, _ = e.forces(pos, a % int(w.opt.B) == 0)
        if brownian:
            big_n = 0 if big is None else len(big)
            u, lcg = _minstd_uniforms(lcg, 3 * (n + big_n))
            noise = torch.as_tensor(u[:3 * n].reshape(n, 3), device="cuda") * torch.sqrt(24 * mass / (float(w.opt.d) * dt))
            f = f + noise - noise.mean(0) + drag
        vel = vel * ef + f * kick
        ke = float((0.5 * mass * vel * vel).sum())
        if not brownian:
            ch.forward(ke)
        mean = vel.mean(0)
        vel = vel - mean
        vcom = float(mean.norm())
    return pos.cpu().numpy(), vel.cpu().numpy(), np.array([ke, 0.0 if brownian else ch.xi[0], vcom])


def _exact_energies(w):
    e = _Exact(w)
    d, o = w.derived, w.opt
    pos = torch.as_tensor(w.state.pos, dtype=torch.float64, device="cuda")
    vel = torch.as_tensor(w.state.vel, dtype=torch.float64, device="cuda")
    n, np_ = pos.shape[0], e.np
    p = pos.reshape(e.S, np_, 3)
    a, b = e.edges[:, 0], e.edges[:, 1]
    half = 0.25 * o.s * (e.len0 - e.wrap(p[:, a] - p[:, b]).norm(dim=-1)) ** 2
    se = torch.zeros((e.S, np_), dtype=torch.float64, device="cuda").index_add_(1, a, half).index_add_(1, b, half)
    be_q = 0.25 * e.bend_energy(e.wrap(p - p[:, :1]))
    be = torch.zeros_like(se)
    for k in range(4):
        be.index_add_(1, e.quad_beads[:, k], be_q)
    ke = 0.5 * e.m.repeat(e.S) * (vel * vel).sum(-1)
    reach = max(d.ecut, d.ecut_el) + 2 * 1.2 * float((p - p[:, :1]).sub(e.L * torch.round((p - p[:, :1]) / e.L)).norm(dim=-1).max())
    blk = e.blocks(pos, reach * reach)
    blk = blk[blk[:, 1] >= blk[:, 0]]
    ne, ce = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2))
    ys = torch.exp(d.kappa * e.shc) / ((1 + d.kappa * e.sig[:, None] / 2) * (1 + d.kappa * e.sig[None, :] / 2))
    upper = torch.triu(torch.ones((np_, np_), dtype=torch.bool, device="cuda"), 1)
    s6t = e.shc ** 6
    ec6 = d.ecut ** 6
    for b0 in range(0, len(blk), 4000):
        i, j = blk[b0:b0 + 4000, 0], blk[b0:b0 + 4000, 1]
        r = e.wrap(p[i][:, :, None] - p[j][:, None]).norm(dim=-1)
        same = (i == j)[:, None, None]
        ok = torch.where(same, upper, torch.ones_like(upper))
        r = torch.where(ok, r, torch.full_like(r, 1e9))
        el = ys * e.qq * d.lb * (torch.exp(-d.kappa * r) / r - math.exp(-d.kappa * d.ecut_el) / d.ecut_el)
        el = torch.where(r < d.ecut_el, el, torch.zeros_like(el))
        q6 = s6t / r ** 6
        wca = torch.where(r < 1.12246205 * e.shc, 4 * q6 * (q6 - 1) + 1, torch.zeros_like(r))
        sh = 4 * o.E * ((s6t / ec6) * ((s6t / ec6) - 1))
        lj = torch.where(r < d.ecut, 4 * o.E * q6 * (q6 - 1) - sh, torch.zeros_like(r))
        lj = torch.where(same, torch.zeros_like(r), torch.where(e.att, lj, wca))
        at = (i[:, None] * np_ + torch.arange(np_, device="cuda")).reshape(-1)
        ce.index_add_(0, at, el.sum(2).reshape(-1))
        ne.index_add_(0, at, lj.sum(2).reshape(-1))
    return {"se": se.reshape(-1), "be": be.reshape(-1), "ne": ne, "ce": ce, "ke": ke}


def _exact_mlp(case, seed):
    p, x, t = _mlp_data(case, seed)
    par, k = [], 0
    for o, i in _mlp_shapes(case["width"]):
        for shape in ((o, i), (o,)):
            n = int(np.prod(shape))
            par.append(torch.as_tensor(p[k:k + n].reshape(shape).astype(np.float64), device="cuda").requires_grad_(True))
            k += n
    h = torch.as_tensor(x, device="cuda").double()
    with torch.enable_grad():
        for l in range(4):
            h = h @ par[2 * l].T + par[2 * l + 1]
            if l < 3:
                h = h * torch.sigmoid(h)
        if case["kind"] == "mlp_forward":
            return h.detach()
        loss = ((h - torch.as_tensor(t, device="cuda").double()) ** 2).mean()
        loss.backward()
    return {"loss": float(loss), "grad": torch.cat([q.grad.reshape(-1) for q in par])}


def exact(case, seed):
    k = case["kind"]
    if k in ("mlp_forward", "mlp_gradients"):
        return _exact_mlp(case, seed)
    if k == "analysis" or (k == "replicas" and case["surrogate"]):
        return None  # whole numbers; a learned approximation
    if k == "replicas":
        ws = _replica_workloads(case, seed)
        parts = [_exact_md(w, case["steps"], None, w.opt.t) for w in ws]
        return {"pos": np.concatenate([q[0] for q in parts]), "vel": np.concatenate([q[1] for q in parts]),
                "scalars": [parts[0][2]]}
    w = _workload(case, seed)
    if k in ("md", "bd"):
        pos, vel, sc = _exact_md(w, case["steps"], _big_beads(case, w, seed), w.opt.t)
        return {"pos": pos, "vel": vel, "scalars": [sc]}
    if k == "forces":
        e = _Exact(w)
        f, sf, bf = e.forces(torch.as_tensor(w.state.pos, dtype=torch.float64, device="cuda"), True)
        return [f, sf, bf] if case["parts"] else [f]
    en = _exact_energies(w)
    tot = {"kinetic": "ke", "stretching": "se", "bending": "be", "lj": "ne", "electrostatic": "ce"}
    return {"totals": {a: float(en[b].sum()) for a, b in tot.items()}, "beads": en if case["per_bead"] else {}}
