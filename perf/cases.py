"""Timed cases of the forward path, through the public entry points.

A head is a set of nested closed surfaces, each a geodesic sphere of some
frequency f (10 f^2 + 2 vertices, 20 f^2 triangles: f = 8 and 16 have the sizes of
the three- and four-times subdivided icosahedra), bent by a smooth radial field and
with conductivities around the nominal ones, both made from the seed.  Electrodes
lie on scalp triangles, magnetometers around the head, dipoles inside the brain.

Every case is one of the calls a forward-modelling program makes:

  gain      forward_gain: head matrix, factorization, sensor rows, sources, gains
  headmat   HeadMat
  dsm       DipSourceMat
  solver    Solver on a head matrix in hand, and the solve of the sensor rows
  solve     Solver.solve of new right-hand sides with a factorization kept
  direct    GainEEG and GainMEG from an explicit inverse (om_minverser + om_gain)
  gradient  adjoint.gain and its backward pass
  batch     a captured BatchForward, its models given new dipoles and replayed

`exact` restates the same quantities in plain torch, in 64 bits: the closed-form
triangle integrals, the 16-point rule, the adaptive rule of the sources, a dense
solve.
"""
from __future__ import annotations

import contextlib
import functools
import math

import numpy as np
import torch

from openmeeg_gb300 import adjoint, api

RADII = {3: (0.87, 0.92, 1.0), 4: (0.85, 0.88, 0.92, 1.0)}
SIGMA = {3: (1.0, 0.0125, 1.0), 4: (0.33, 1.79, 0.0042, 0.33)}
K = 1.0 / (4.0 * math.pi)
MAG = 1e-7


# ---- cases ------------------------------------------------------------------

def _case(kind, freqs, **more):
    c = {"kind": kind, "freqs": "-".join(str(f) for f in freqs), "precision": "fp64", "dipoles": 0, "eeg": 0, "meg": 0}
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: a coarse test head, where launches and latency count
        _case("gain", (4, 4, 4), name="gain_fp64_smallest", dipoles=8, eeg=16, meg=10),
        # the sample head's size in the default precision, EEG and a few magnetometers
        _case("gain", (8, 8, 8), name="gain_fp64_sample_head", dipoles=200, eeg=64, meg=32),
        # a finer head in the default precision, uneven surfaces, combined EEG and MEG
        _case("gain", (13, 12, 11), name="gain_fp64_fine_head", dipoles=500, eeg=64, meg=151),
        # the sample head's size in mixed precision
        _case("gain", (8, 8, 8), name="gain_mixed_sample_head", precision="mixed", dipoles=200, eeg=64),
        # the headline workload: 17926 unknowns, 2000 dipoles, EEG and MEG, mixed precision
        _case("gain", (16, 16, 16), name="gain_mixed_headline", precision="mixed", dipoles=2000, eeg=64, meg=151),
        # a head matrix to be written to a file or passed on, four ragged surfaces
        _case("headmat", (7, 9, 10, 11), name="headmat_fp64_4_layers"),
        # new sources on a fine head
        _case("dsm", (16, 14, 14), name="dipsourcemat_fp64", dipoles=500),
        # a head matrix from elsewhere, factored once for the electrodes
        _case("solver", (10, 9, 11), name="solver_fp64_from_headmat", eeg=64, meg=0),
        # new right-hand sides on a factorization that is kept
        _case("solve", (12, 11, 12), name="solve_mixed_kept_factor", precision="mixed", eeg=64, meg=151),
        # gains from an explicit inverse, the documented two-step pipeline
        _case("direct", (8, 8, 8), name="gain_from_inverse_fp64", dipoles=1000, eeg=64, meg=151),
        # conductivity and dipole gradients of a combined gain
        _case("gradient", (8, 8, 8), name="gain_gradient_fp64", dipoles=100, eeg=64, meg=32),
        # many heads of uneven size in one replayed graph
        _case("batch", (8, 8, 8), name="batch_mixed_4_heads", precision="mixed", dipoles=300, eeg=64, models=4),
    ]


def draw(rng):
    kind = rng.choice(["gain", "gain", "gain", "headmat", "dsm", "solver", "solve", "direct", "gradient", "batch"])
    layers = rng.choice([3, 3, 4])

    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def freqs(lo, hi):
        top = log(lo, hi)
        return [max(lo, top - rng.randrange(0, 3)) for _ in range(layers)]

    if kind == "gain":
        p = rng.choice(["fp64", "mixed"])
        return _case(kind, freqs(4, (12 if layers == 3 else 10) if p == "fp64" else (16 if layers == 3 else 13)),
                     precision=p, dipoles=log(8, 1500), eeg=log(16, 64), meg=rng.choice([0, log(10, 151)]))
    if kind == "headmat":
        return _case(kind, freqs(4, 11), precision=rng.choice(["fp64", "mixed"]))
    if kind == "dsm":
        return _case(kind, freqs(4, 16), dipoles=log(20, 500))
    if kind == "solver":
        return _case(kind, freqs(4, 10), precision=rng.choice(["fp64", "mixed"]), eeg=log(16, 64),
                     meg=rng.choice([0, log(10, 151)]))
    if kind == "solve":
        return _case(kind, freqs(4, 11), precision=rng.choice(["fp64", "mixed"]), eeg=log(16, 64),
                     meg=rng.choice([0, log(10, 151)]))
    if kind == "direct":
        return _case(kind, freqs(4, 9), precision=rng.choice(["fp64", "mixed"]), dipoles=log(20, 1500),
                     eeg=log(16, 64), meg=log(10, 151))
    if kind == "gradient":
        return _case(kind, freqs(4, 8), precision=rng.choice(["fp64", "mixed"]), dipoles=log(8, 100),
                     eeg=log(16, 64), meg=rng.choice([0, log(10, 32)]))
    return _case(kind, freqs(4, 9), precision="mixed", dipoles=log(50, 500), eeg=log(16, 64), models=rng.randrange(2, 6))


# ---- inputs -----------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _geodesic(f):
    """Unit geodesic sphere of frequency f: vertices, triangles (inward normals)."""
    t = (1.0 + math.sqrt(5.0)) / 2.0
    ico = np.array([(-1, t, 0), (1, t, 0), (-1, -t, 0), (1, -t, 0), (0, -1, t), (0, 1, t), (0, -1, -t), (0, 1, -t),
                    (t, 0, -1), (t, 0, 1), (-t, 0, -1), (-t, 0, 1)], np.float64)
    ico /= np.linalg.norm(ico[0])
    faces = [(0, 11, 5), (0, 5, 1), (0, 1, 7), (0, 7, 10), (0, 10, 11), (1, 5, 9), (5, 11, 4), (11, 10, 2), (10, 7, 6),
             (7, 1, 8), (3, 9, 4), (3, 4, 2), (3, 2, 6), (3, 6, 8), (3, 8, 9), (4, 9, 5), (2, 4, 11), (6, 2, 10),
             (8, 6, 7), (9, 8, 1)]
    grid = [(i, j) for i in range(f + 1) for j in range(f + 1 - i)]
    at = {ij: n for n, ij in enumerate(grid)}
    small = []
    for i in range(f):
        for j in range(f - i):
            small.append((at[i, j], at[i, j + 1], at[i + 1, j]))
            if i + j < f - 1:
                small.append((at[i + 1, j], at[i, j + 1], at[i + 1, j + 1]))
    small, ij = np.array(small), np.array(grid)
    keys, tris = [], []
    for n, (a, b, c) in enumerate(faces):
        w = np.zeros((len(grid), 12), np.int64)   # integer weights of the 12 corners: equal for a shared point
        w[:, a], w[:, b], w[:, c] = f - ij[:, 0] - ij[:, 1], ij[:, 0], ij[:, 1]
        keys.append(w)
        tris.append(small + n * len(grid))
    w, inverse = np.unique(np.concatenate(keys), axis=0, return_inverse=True)
    v = w @ ico
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    return v, inverse.reshape(-1)[np.concatenate(tris)]


def _unit(g, n):
    v = g.standard_normal((n, 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


class _Inputs:
    """Host arrays of one head: surfaces, domains, dipoles, sensors."""

    def __init__(self, freqs, case, seed):
        g = np.random.default_rng([seed, *freqs])
        layers = len(freqs)
        dirs, coef = _unit(g, 6), g.standard_normal(6)
        self.vertices, self.triangles = [], []
        for f, r in zip(freqs, RADII[layers]):
            v, t = _geodesic(f)
            p = v @ dirs.T
            bend = (np.hstack([p[:, :3], p[:, 3:] ** 2 - 1.0 / 3.0]) @ coef) / np.abs(coef).sum()
            self.vertices.append(v * (r * (1.0 + 0.02 * bend))[:, None])
            self.triangles.append(t)
        self.sigma = [s * float(np.exp(g.uniform(-0.2, 0.2))) for s in SIGMA[layers]] + [0.0]
        self.domains = []
        for k in range(layers + 1):
            bounds = ([k] if k else []) + ([-(k + 1)] if k < layers else [])
            self.domains.append(("dom%d" % k, bounds, self.sigma[k]))
        n = case["dipoles"]
        rmax = 0.8 * RADII[layers][0] / 0.87
        self.dipoles = np.hstack([_unit(g, n) * (rmax * g.random((n, 1)) ** (1 / 3)), _unit(g, n)])
        # electrodes: a point of a scalp triangle, a little outside; its weights are the triangle's
        v, t = self.vertices[-1], self.triangles[-1]
        self.el_tri = g.choice(len(t), case["eeg"], replace=case["eeg"] > len(t))
        w = 0.1 + g.random((case["eeg"], 3))
        self.el_w = w / w.sum(axis=1, keepdims=True)
        p = v[t[self.el_tri]]
        nrm = np.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])   # inward
        nrm /= np.maximum(np.linalg.norm(nrm, axis=1, keepdims=True), 1e-300)
        self.electrodes = np.einsum("ij,ijk->ik", self.el_w, p) - 1e-3 * nrm
        q = _unit(g, case["meg"])
        tilt = q + 0.2 * _unit(g, case["meg"])
        self.squids = np.hstack([1.2 * q, tilt / np.linalg.norm(tilt, axis=1, keepdims=True)])
        self.cotangent = g.standard_normal((case["eeg"] + case["meg"], n)) if case["kind"] == "gradient" else None

    def geometry(self):
        return api.Geometry.from_meshes(self.vertices, self.triangles, self.domains)


def _freqs(case):
    return [int(f) for f in case["freqs"].split("-")]


def _models(case):
    """The surfaces of each head of a batch: ragged sizes around the case's, three and four layers."""
    f = _freqs(case)
    out = []
    for k in range(case["models"]):
        m = [max(4, x + (k * 5 + 3 * i) % 7 - 2) for i, x in enumerate(f)]
        out.append(m + [m[0]] if k % 3 == 2 and len(m) == 3 else m)
    return out


@functools.lru_cache(maxsize=None)
def _stream():
    return torch.cuda.Stream()


@contextlib.contextmanager
def _on_stream():
    """The library's work and torch's own on one stream, so that each sees the other's results."""
    with torch.cuda.stream(_stream()):
        api.Context.default().bind_current_stream()
        yield


def _cuda(a):
    return torch.as_tensor(a, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    kind, prec = case["kind"], case["precision"]
    torch.cuda.synchronize()
    if kind == "batch":
        heads = [_Inputs(f, case, seed + 1000 * k) for k, f in enumerate(_models(case))]
        new = [np.hstack([0.95 * h.dipoles[::-1, :3], h.dipoles[:, 3:]]) for h in heads]
        with _on_stream():
            plan = api.BatchForward([(h.geometry(), h.dipoles, h.electrodes, None) for h in heads], precision=prec,
                                    n_branches=4)
            torch.cuda.synchronize()
        return {"kind": kind, "plan": plan, "dipoles": new}
    h = _Inputs(_freqs(case), case, seed)
    s = {"kind": kind, "precision": prec}
    with _on_stream():
        s["geo"] = h.geometry()
        s["dipoles"] = _cuda(h.dipoles)
        s["electrodes"] = _cuda(h.electrodes) if case["eeg"] else None
        s["squids"] = _cuda(h.squids) if case["meg"] else None
        if kind == "gradient":
            s["sigma"] = torch.tensor(h.sigma, dtype=torch.float64)
            s["domains"], s["cotangent"] = h.domains, _cuda(h.cotangent)
            s["electrodes"] = h.electrodes if case["eeg"] else None
            s["squids"] = h.squids if case["meg"] else None
        if kind in ("solver", "solve", "direct"):
            m = _Bem(h)
            hm = m.head_matrix()
            rows = m.sensor_rows()
            if kind == "direct":
                s["inverse"], s["dsm"] = torch.linalg.inv(hm), m.sources()
                s["h2em"] = (None, *m.eeg_triplets())
                s["h2mm"], s["ds2mm"] = rows[case["eeg"]:].contiguous(), m.primary_field()
            else:
                s["hm"], s["rhs"] = hm, rows.T.contiguous()
                if kind == "solve":
                    s["solver"] = api.Solver(s["geo"], precision=prec, hm=hm)
                    del s["hm"]
        torch.cuda.synchronize()
    return s


def run(state):
    kind = state["kind"]
    with _on_stream():
        if kind == "gain":
            return api.forward_gain(state["geo"], state["dipoles"], state["electrodes"], state["squids"],
                                    precision=state["precision"])[:2]
        if kind == "headmat":
            return api.HeadMat(state["geo"], precision=state["precision"])
        if kind == "dsm":
            return api.DipSourceMat(state["geo"], state["dipoles"])
        if kind == "solver":
            return api.Solver(state["geo"], precision=state["precision"], hm=state["hm"]).solve(state["rhs"])
        if kind == "solve":
            return state["solver"].solve(state["rhs"])
        if kind == "direct":
            return (api.GainEEG(state["inverse"], state["dsm"], state["h2em"], precision=state["precision"]),
                    api.GainMEG(state["inverse"], state["dsm"], state["h2mm"], state["ds2mm"],
                                precision=state["precision"]))
        if kind == "gradient":
            sigma = state["sigma"].clone().requires_grad_(True)
            dipoles = state["dipoles"].clone().requires_grad_(True)
            gain = adjoint.gain(sigma, dipoles, state["geo"], state["domains"], state["electrodes"], state["squids"],
                                precision=state["precision"])
            return (gain.detach(), *torch.autograd.grad(gain, [sigma, dipoles], state["cotangent"]))
        plan = state["plan"]
        for i, d in enumerate(state["dipoles"]):
            plan.set_dipoles(i, d)
        plan.run()
        return [plan.gains(i)[0] for i in range(len(plan))]


# ---- the work of one pass ---------------------------------------------------

def _head_work(freqs, case, kind):
    nt, nv = [20 * f * f for f in freqs], [10 * f * f + 2 for f in freqs]
    n = sum(nv) + sum(nt[:-1])
    k, nd = case["eeg"] + case["meg"], case["dipoles"]
    pairs = [(i, i) for i in range(len(nt))] + [(i + 1, i) for i in range(len(nt) - 1)]
    last = len(nt) - 1
    # about 70 operations for a single-layer value, 90 for the three double-layer ones, 16 points each
    s = sum(nt[a] * (nt[a] + 1) / 2 if a == b else nt[a] * nt[b] for a, b in pairs)
    d = sum(nt[a] * nt[b] * ((a != last) + (a != b and b != last)) for a, b in pairs)
    assembly = 16.0 * (70 * s + 90 * d)
    sources = 80.0 * 40 * nd * nt[0]
    rows = nv[0] + nt[0]
    geometry = 24.0 * (sum(nv) + sum(nt))
    if kind == "headmat":
        return geometry + 8.0 * n * n, assembly
    if kind == "dsm":
        return geometry + 8.0 * nd * n, sources
    if kind == "solver":
        return 8.0 * n * n + 16.0 * n * k, n ** 3 / 3 + 2.0 * n * n * k
    if kind == "solve":
        return 4.0 * n * n + 16.0 * n * k, 2.0 * n * n * k
    if kind == "direct":
        return 8.0 * n * (n + nd + k) + 8.0 * nd * k, 2.0 * n * n * case["meg"] + 2.0 * n * nd * k
    flops = assembly + n ** 3 / 3 + 2.0 * n * n * k + sources + 2.0 * rows * nd * k
    if kind == "gradient":   # the second solve and the block traces, the pulled-back sources
        flops += 4.0 * n * n * k + sources + 4.0 * n * nd * k
    return geometry + 8.0 * nd * (6 + k), flops


def work(case):
    heads = _models(case) if case["kind"] == "batch" else [_freqs(case)]
    done = [_head_work(f, case, case["kind"]) for f in heads]
    return {"bytes": sum(b for b, _ in done), "flops": sum(f for _, f in done)}


# ---- the same in plain torch, 64 bits ----------------------------------------

# the 16-point rule of the reference implementation, with its tabulated digits
_A, _B, _C, _D = 0.008394777409957, 0.728492392955404, 0.263112829634639, 0.027230314174434
_RULE = [(0.333333333333333, 0.333333333333333, 0.333333333333333, 0.144315607677786),
         (0.081414823414554, 0.459292588292722, 0.459292588292722, 0.095091634267284),
         (0.459292588292722, 0.081414823414554, 0.459292588292722, 0.095091634267284),
         (0.459292588292722, 0.459292588292722, 0.081414823414554, 0.095091634267284),
         (0.898905543365937, 0.050547228317031, 0.050547228317031, 0.032458497623198),
         (0.050547228317031, 0.898905543365937, 0.050547228317031, 0.032458497623198),
         (0.050547228317031, 0.050547228317031, 0.898905543365937, 0.032458497623198),
         (0.658861384496479, 0.170569307751760, 0.170569307751761, 0.103217370534718),
         (0.170569307751760, 0.658861384496479, 0.170569307751761, 0.103217370534718),
         (0.170569307751760, 0.170569307751761, 0.658861384496479, 0.103217370534718),
         (_A, _B, _C, _D), (_B, _A, _C, _D), (_B, _C, _A, _D), (_A, _C, _B, _D), (_C, _A, _B, _D), (_C, _B, _A, _D)]
_CHUNK = 1 << 22   # values of one temporary


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


class _Mesh:
    def __init__(self, vertices, triangles):
        self.v, self.t = _cuda(vertices), torch.as_tensor(triangles, device="cuda")
        self.nv, self.nt = len(vertices), len(triangles)
        self.p = self.v[self.t]                                            # nt x 3 corners x 3
        n = torch.linalg.cross(self.p[:, 1] - self.p[:, 0], self.p[:, 2] - self.p[:, 0])
        nrm = torch.linalg.norm(n, dim=1)
        self.area, self.n = 0.5 * nrm, n / nrm[:, None]
        self.edge = self.p[:, [1, 2, 0]] - self.p                          # corner i to corner i + 1
        self.len = torch.linalg.norm(self.edge, dim=2)
        self.unit = self.edge / self.len[:, :, None]
        self.en = torch.linalg.cross(self.n[:, None].expand_as(self.unit), -self.unit)
        r = _cuda(_RULE)
        self.w = r[:, 3]
        self.q = torch.einsum("qj,tjk->tqk", r[:, :3], self.p).reshape(-1, 3)
        # triangles around each vertex (padded with weight 0) and the corner it is there
        order = torch.argsort(self.t.reshape(-1), stable=True)
        vert = self.t.reshape(-1)[order]
        count = torch.bincount(vert, minlength=self.nv)
        slot = torch.arange(3 * self.nt, device="cuda") - (torch.cumsum(count, 0) - count)[vert]
        deg = int(count.max())
        self.around = torch.zeros((self.nv, deg), dtype=torch.int64, device="cuda")
        self.corner = torch.zeros_like(self.around)
        self.there = torch.zeros((self.nv, deg), dtype=torch.float64, device="cuda")
        self.around[vert, slot], self.corner[vert, slot], self.there[vert, slot] = order // 3, order % 3, 1.0
        opposite = self.p[:, [1, 2, 0]] - self.p[:, [2, 0, 1]]
        self.curl = (opposite / self.area[:, None, None])[self.around, self.corner] * self.there[:, :, None]

    def seen_from(self, x, a, b):
        """Corners of triangles a..b relative to the points x: vectors, distances, height, half solid angle."""
        r = [[self.p[a:b, i, c, None] - x[None, :, c] for c in range(3)] for i in range(3)]
        d = [torch.sqrt(_dot(v, v)) for v in r]
        n = [self.n[a:b, c, None] for c in range(3)]
        h = _dot(r[0], n)
        den = d[0] * d[1] * d[2] + d[0] * _dot(r[1], r[2]) + d[1] * _dot(r[2], r[0]) + d[2] * _dot(r[0], r[1])
        return r, d, n, h, torch.atan2(2 * h * self.area[a:b, None], den)

    def single(self, x, a, b):
        """Integral of 1/|y - x| over triangles a..b, at the points x."""
        r, d, _, h, half = self.seen_from(x, a, b)
        s = 0.0
        for i in range(3):
            en = [self.en[a:b, i, c, None] for c in range(3)]
            s = s + _dot(r[i], en) * torch.atanh(self.len[a:b, i, None] / (d[i] + d[(i + 1) % 3]))
        flat = (2 * h * self.area[a:b, None]).abs() < 1e-10
        return 2 * s - h * torch.where(flat, 0.0, 2 * half)

    def double(self, x, a, b):
        """Integrals of the double-layer kernel times the three P1 functions of triangles a..b, at x."""
        r, d, n, h, half = self.seen_from(x, a, b)
        s = [0.0, 0.0, 0.0]
        for i in range(3):
            j = (i + 1) % 3
            u = [self.unit[a:b, i, c, None] for c in range(3)]
            lg = torch.log((d[j] + _dot(r[j], u)) / (d[i] + _dot(r[i], u)))
            s = [s[c] + u[c] * lg for c in range(3)]
        out = []
        for i in range(3):
            p, q = r[(i + 1) % 3], r[(i + 2) % 3]
            z = (p[1] * q[2] - p[2] * q[1], p[2] * q[0] - p[0] * q[2], p[0] * q[1] - p[1] * q[0])
            e = [self.edge[a:b, (i + 1) % 3, c, None] for c in range(3)]
            v = (_dot(z, n) * half + 0.5 * h * _dot(e, s)) / self.area[a:b, None]
            out.append(torch.where(h.abs() < 1e-10, 0.0, v))
        return out

    def over(self, values):
        """Values at this mesh's rule points, rows x (nt * 16), integrated over its triangles."""
        return (values.view(values.shape[0], self.nt, 16) @ self.w) * self.area


def _single_block(a, b):
    out = torch.empty((a.nt, b.nt), dtype=torch.float64, device="cuda")
    step = max(1, _CHUNK // (16 * b.nt))
    for i in range(0, a.nt, step):
        out[i:i + step] = b.over(a.single(b.q, i, min(a.nt, i + step)))
    return torch.triu(out) + torch.triu(out, 1).T if a is b else out


def _double_block(a, b):
    """Rows: triangles of a; columns: vertices of b."""
    part = [torch.empty((b.nt, a.nt), dtype=torch.float64, device="cuda") for _ in range(3)]
    step = max(1, _CHUNK // (16 * a.nt))
    for i in range(0, b.nt, step):
        for j, v in enumerate(b.double(a.q, i, min(b.nt, i + step))):
            part[j][i:i + step] = a.over(v)
    out = torch.zeros((b.nv, a.nt), dtype=torch.float64, device="cuda")
    for k in range(b.around.shape[1]):
        for j in range(3):
            w = b.there[:, k] * (b.corner[:, k] == j)
            out += w[:, None] * part[j][b.around[:, k]]
    return out.T


def _hyper_block(a, b, s):
    """-1/4 sum over the components of curl^T S curl."""
    out = 0.0
    for c in range(3):
        u = 0.0
        for k in range(b.around.shape[1]):
            u = u + s[:, b.around[:, k]] * b.curl[:, k, c]
        for k in range(a.around.shape[1]):
            out = out + a.curl[:, k, c, None] * u[a.around[:, k]]
    return -0.25 * out


class _Bem:
    """The symmetric formulation for nested closed surfaces with inward normals."""

    def __init__(self, h, sigma=None, dipoles=None):
        self.h = h
        self.m = [_Mesh(v, t) for v, t in zip(h.vertices, h.triangles)]
        self.sigma = list(h.sigma) if sigma is None else sigma
        self.dipoles = _cuda(h.dipoles) if dipoles is None else dipoles
        self.vbeg = np.concatenate([[0], np.cumsum([m.nv for m in self.m])])
        self.tbeg = self.vbeg[-1] + np.concatenate([[0], np.cumsum([m.nt for m in self.m])])
        self.size = int(self.tbeg[len(self.m) - 1])
        self.vs = [slice(int(a), int(b)) for a, b in zip(self.vbeg, self.vbeg[1:])]
        self.ts = [slice(int(a), int(b)) for a, b in zip(self.tbeg, self.tbeg[1:])]

    def head_matrix(self):
        hm = torch.zeros((self.size, self.size), dtype=torch.float64, device="cuda")

        def put(r, c, block):
            hm[r, c] = block
            if r != c:
                hm[c, r] = block.T

        last = len(self.m) - 1
        for i, a in enumerate(self.m):
            for j in ([i] if i == 0 else [i - 1, i]):
                b = self.m[j]
                inner, outer = self.sigma[i], self.sigma[i + 1]
                s = _single_block(a, b)
                if i == j:
                    cn, cd = K * (inner + outer), -2 * K
                    if i != last:
                        put(self.ts[i], self.ts[i], s * (K * (1 / inner + 1 / outer)))
                else:
                    cn, cd = -K * inner, K
                    if i != last:
                        put(self.ts[i], self.ts[j], s * (-K / inner))
                put(self.vs[i], self.vs[j], _hyper_block(a, b, s) * cn)
                if i != last:
                    put(self.ts[i], self.vs[j], _double_block(a, b) * cd)
                if i != j:
                    put(self.ts[j], self.vs[i], _double_block(b, a) * cd)
        v = self.vs[last]   # the outermost surface's constant
        hm[v, v] = hm[v, v] + hm[v.start, v.start] / self.m[last].nv
        return hm

    def eeg_triplets(self):
        """(columns, weights) of the electrodes' rows, n x 3 each."""
        return (self.vs[-1].start + self.m[-1].t[torch.as_tensor(self.h.el_tri, device="cuda")], _cuda(self.h.el_w))

    def sensor_rows(self):
        ne = len(self.h.electrodes)
        rows = []
        if ne:
            cols, w = self.eeg_triplets()
            rows.append(torch.zeros((ne, self.size), dtype=torch.float64, device="cuda").scatter_(1, cols, w))
        if len(self.h.squids):
            x, o = _cuda(self.h.squids[:, :3]), _cuda(self.h.squids[:, 3:])
            o = o / torch.linalg.norm(o, dim=1, keepdim=True)
            parts = []
            for i, m in enumerate(self.m):
                s = m.single(x, 0, m.nt) / 2
                jump = self.sigma[i] - self.sigma[i + 1]
                f = 0.0   # the curl is (edge end - edge start) / area; the field's edge runs the other way
                for k in range(m.around.shape[1]):
                    f = f - (m.curl[:, k] @ o.T) * s[m.around[:, k]]
                parts.append(f.T * (MAG * jump))
            parts.append(torch.zeros((len(x), self.size - int(self.vbeg[-1])), dtype=torch.float64, device="cuda"))
            rows.append(torch.cat(parts, 1))
        return torch.cat(rows, 0)

    def primary_field(self):
        s = _cuda(self.h.squids)
        d = s[:, None, :3] - self.dipoles[None, :, :3]
        f = torch.linalg.cross(self.dipoles[None, :, 3:].expand_as(d), d) / torch.linalg.norm(d, dim=2, keepdim=True) ** 3
        return MAG * (f * (s[:, 3:] / torch.linalg.norm(s[:, 3:], dim=1, keepdim=True))[:, None]).sum(2)

    def sources(self):
        m = self.m[0]
        pot, der = [], []
        step = max(1, (1 << 20) // m.nt)
        for i in range(0, len(self.dipoles), step):
            d = self.dipoles[i:i + step]
            n = len(d)
            pair = (torch.arange(n, device="cuda").repeat_interleave(m.nt), torch.arange(m.nt, device="cuda").repeat(n))
            pot.append(_adaptive(_potential, m, d, pair, 1).view(n, m.nt))
            der.append(_adaptive(_derivative, m, d, pair, 3).view(n, m.nt, 3))
        pot, der = torch.cat(pot), torch.cat(der)
        vert = 0.0
        for k in range(m.around.shape[1]):
            vert = vert + der[:, m.around[:, k], m.corner[:, k]] * m.there[:, k]
        out = torch.zeros((self.size, len(pot)), dtype=torch.float64, device="cuda")
        out[self.vs[0]] = -K * vert.T
        out[self.ts[0]] = (-K / self.sigma[0]) * pot.T
        return out

    def gains(self):
        rows = self.sensor_rows()
        g = torch.linalg.solve(self.head_matrix(), rows.T).T @ self.sources()
        ne = len(self.h.electrodes)
        return g[:ne] if ne else None, g[ne:] + self.primary_field() if len(self.h.squids) else None


def _potential(m, d, tri, x):
    v = x - d[:, None, :3]
    n2 = (v * v).sum(2)
    return ((d[:, None, 3:] * v).sum(2) / (n2 * torch.sqrt(n2)))[:, :, None]


def _derivative(m, d, tri, x):
    """The dipole's normal derivative times the three barycentric coordinates."""
    e1, e2 = m.p[tri, 1] - m.p[tri, 0], m.p[tri, 2] - m.p[tri, 0]
    c11, c12, c22 = (e1 * e1).sum(1), (e1 * e2).sum(1), (e2 * e2).sum(1)
    det = c11 * c22 - c12 * c12
    v = x - m.p[tri, 0][:, None]
    d1, d2 = (v * e1[:, None]).sum(2), (v * e2[:, None]).sum(2)
    l1, l2 = (d1 * c22[:, None] - d2 * c12[:, None]) / det[:, None], (d2 * c11[:, None] - d1 * c12[:, None]) / det[:, None]
    y = x - d[:, None, :3]
    inv = 1.0 / (y * y).sum(2)
    q = d[:, None, 3:]
    grad = q - y * (3 * (q * y).sum(2) * inv)[:, :, None]
    g = (grad * m.n[tri][:, None]).sum(2) * (inv * torch.sqrt(inv))
    return g[:, :, None] * torch.stack([1 - l1 - l2, l1, l2], 2)


def _adaptive(f, m, dipoles, pair, dim, levels=10, tol=1e-3):
    """The reference's adaptive rule: a triangle's value is that of its four parts' once the two agree."""
    rule = _cuda(_RULE)
    which = torch.arange(len(pair[0]), device="cuda")
    corners, area = m.p[pair[1]], m.area[pair[1]]

    def integrate(which, corners, area):
        x = torch.einsum("qj,njk->nqk", rule[:, :3], corners)
        return torch.einsum("q,nqc->nc", rule[:, 3], f(m, dipoles[pair[0][which]], pair[1][which], x)) * area[:, None]

    total = torch.zeros((len(pair[0]), dim), dtype=torch.float64, device="cuda")
    with torch.no_grad():
        coarse = integrate(which, corners, area)
    for level in range(levels, -1, -1):
        mid = 0.5 * (corners[:, [1, 2, 0]] + corners[:, [2, 0, 1]])
        p, q = corners.unbind(1), mid.unbind(1)
        parts = [torch.stack(c, 1) for c in ((p[0], q[1], q[2]), (q[0], p[1], q[2]), (q[0], q[1], p[2]), q)]
        values = [integrate(which, c, 0.25 * area) for c in parts]
        fine = values[0] + values[1] + values[2] + values[3]
        done = torch.linalg.norm(coarse - fine, dim=1) <= tol * torch.linalg.norm(coarse, dim=1)
        if level == 0:
            done = torch.ones_like(done)
        total = total.index_add(0, which[done], fine[done])
        more = ~done
        if not bool(more.any()):
            break
        which, area = which[more].repeat(4), 0.25 * area[more].repeat(4)
        corners = torch.cat([c[more] for c in parts])
        coarse = torch.cat([v[more] for v in values]).detach()
    return total


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        heads = [_Inputs(f, case, seed + 1000 * k) for k, f in enumerate(_models(case))]
        for h in heads:
            h.dipoles = np.hstack([0.95 * h.dipoles[::-1, :3], h.dipoles[:, 3:]])
        return [_Bem(h).gains()[0] for h in heads]
    h = _Inputs(_freqs(case), case, seed)
    if kind == "gradient":
        s = [torch.tensor(x, dtype=torch.float64, device="cuda", requires_grad=x != 0.0) for x in h.sigma]
        d = _cuda(h.dipoles).requires_grad_(True)
        ge, gm = _Bem(h, s, d).gains()
        gain = torch.cat([g for g in (ge, gm) if g is not None])
        *gs, gd = torch.autograd.grad(gain, [x for x in s if x.requires_grad] + [d], _cuda(h.cotangent))
        return gain.detach(), torch.stack([*gs, torch.zeros_like(gs[0])]).cpu(), gd
    m = _Bem(h)
    if kind == "gain":
        return m.gains()
    if kind == "headmat":
        return m.head_matrix()
    if kind == "dsm":
        return m.sources()
    rows = m.sensor_rows()
    if kind in ("solver", "solve"):
        return torch.linalg.solve(m.head_matrix(), rows.T)
    g = (rows @ torch.linalg.inv(m.head_matrix())) @ m.sources()
    ne = case["eeg"]
    return g[:ne], g[ne:] + m.primary_field()
