"""The extraction workloads whose speed this framework is judged by.

A case is one of three calls that a user's program makes:

* ``file``: input files in, capacitance matrices out, through the extraction
  server (``count`` files submitted at once, then every result taken): mesh
  and link construction, coefficient fill and GMRES, all of it timed.
* ``solve``: coefficient fill and GMRES of a model that is resident on the
  GPU (``Problem.fill`` and ``Problem.solve``): every conductor's right-hand
  side, or every geometry's of a concatenated batch.
* ``product``: the hierarchical product with ``columns`` vectors in device
  memory (``Problem.matvec_device``), the operator of a caller's own solver.

Shapes are the k x k bus crossings (in vacuum, or in a dielectric slab with
its interface) and the spheres of ``fastercap_gb300.geometry``, at the mesh
switches of the benchmark (-m4e-4 -d2.5, -m5e-4 -d2) and of the reference's
coarse runs (-m0.01). The seed scales the whole geometry by up to 2 %, so that
another seed's panels, coefficients and matrices are others at nearly the same
panel and link counts; a product's seed makes its vectors. Launch-shape measurement is off, as in the server: the programs
meant here solve a model once, and it makes results the same from run to run.
"""

from __future__ import annotations

import atexit
import functools
import json
import math
import os
import random
import tempfile

import numpy as np
import torch

import fastercap_gb300 as fc
from fastercap_gb300 import geometry as geo

LISTED = [
    # the smallest call: a 2x2 crossing at a 1 % mesh (528 panels), file to
    # matrix; what a designer's script waits for per variation
    dict(name="file_small", kind="file", shape="crossing", k=2, length=10.0, pitch=3.0, gap=1.0, mesh=0.01, ratio=1.0,
         count=1, precision="mixed", tol=1e-4, steps=18),
    # one ordinary extraction request of the serving workload, alone: 14
    # conductors, about 90,000 panels, 11 million links
    dict(name="file_request", kind="file", shape="crossing", k=7, length=31.5, pitch=2.19, gap=1.7, mesh=4e-4, ratio=2.5,
         count=1, precision="mixed", tol=1e-4, steps=46),
    # one large request: 22 conductors, about 160,000 panels, 28 million links
    dict(name="file_large", kind="file", shape="crossing", k=11, length=23.5, pitch=2.08, gap=1.03, mesh=4e-4, ratio=2.5,
         count=1, precision="mixed", tol=1e-4, steps=53),
    # eight requests of uneven size (7,000 to 25,000 panels) in the server at once
    dict(name="file_burst", kind="file", shape="crossing", k=7, length=31.5, pitch=2.19, gap=1.7, mesh=1e-3, ratio=2.0,
         count=8, precision="mixed", tol=1e-4, steps=37),
    # resident model, few conductors: launches and latency count
    dict(name="solve_small", kind="solve", shape="crossing", k=2, length=53.6, pitch=2.49, gap=2.3, mesh=4e-4, ratio=2.5,
         count=1, precision="mixed", tol=1e-4, steps=35),
    # resident model, 22 right-hand sides in one batch
    dict(name="solve_bus", kind="solve", shape="crossing", k=11, length=23.5, pitch=2.08, gap=1.03, mesh=4e-4, ratio=2.5,
         count=1, precision="mixed", tol=1e-4, steps=53),
    # conductors in a dielectric slab: interface panels evaluate the normal field
    dict(name="solve_slab", kind="solve", shape="slab", k=8, length=40.0, pitch=2.0, gap=1.5, mesh=1e-5, ratio=1.0,
         count=1, precision="mixed", tol=1e-4, steps=42),
    # one right-hand side and a link list far larger than the L2 cache
    dict(name="solve_sphere", kind="solve", shape="sphere", k=4, length=1.0, pitch=0.0, gap=0.0, mesh=3e-4, ratio=1.0,
         count=1, precision="mixed", tol=1e-4, steps=8),
    # six uneven geometries concatenated into one problem
    dict(name="solve_batch", kind="solve", shape="crossing", k=9, length=36.9, pitch=2.73, gap=1.6, mesh=5e-4, ratio=2.0,
         count=6, precision="mixed", tol=1e-4, steps=36),
    # the reference's own arithmetic, for a user who checks against it
    dict(name="solve_fp64", kind="solve", shape="crossing", k=3, length=31.5, pitch=2.18, gap=2.19, mesh=4e-4, ratio=2.5,
         count=1, precision="fp64", tol=1e-4, steps=36),
    # the operator alone, one vector, for a caller's own iteration
    dict(name="product_one", kind="product", shape="sphere", k=4, length=1.0, pitch=0.0, gap=0.0, mesh=3e-4, ratio=1.0,
         count=1, precision="mixed", columns=1),
    # an odd number of vectors in FP64
    dict(name="product_fp64", kind="product", shape="crossing", k=6, length=27.2, pitch=2.74, gap=1.75, mesh=4e-4, ratio=2.5,
         count=1, precision="fp64", columns=7),
]


def listed():
    return [dict(c) for c in LISTED]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random) -> dict:
    """One more case: bus crossings of 2 to 11 bars a layer, 10 to 60 um long,
    pitch 2-4, gap 1-3 (the serving workload's ranges) in vacuum or a slab,
    or a sphere; coarse to fine meshes."""
    kind = rng.choice(["file", "file", "solve", "solve", "solve", "product"])
    shape = "crossing" if kind == "file" else rng.choice(["crossing", "crossing", "crossing", "slab", "sphere"])
    c = dict(kind=kind, shape=shape, k=rng.randint(2, 11), length=round(_log(rng, 10.0, 55.0), 3),
             pitch=round(rng.uniform(2.0, 4.0), 3), gap=round(rng.uniform(1.0, 3.0), 3), count=1)
    # at most about the panels of the largest listed case
    finest = 4e-4 if c["k"] * c["length"] < 300.0 else 6e-4
    c["mesh"], c["ratio"] = float("%.3g" % _log(rng, finest, 1e-2)), rng.choice([1.5, 2.0, 2.5])
    c["precision"] = rng.choice(["mixed", "mixed", "fp64"]) if kind != "file" else "mixed"
    if shape == "slab":
        c["mesh"], c["ratio"] = float("%.3g" % _log(rng, 1.2e-5, 1e-3)), 1.0
    if shape == "sphere":
        c.update(k=rng.choice([3, 4]), length=1.0, pitch=0.0, gap=0.0, mesh=float("%.3g" % _log(rng, 4e-4, 1e-2)), ratio=1.0)
    if kind == "product":
        c["columns"] = rng.randint(1, 32) if c["precision"] == "mixed" else rng.randint(1, 12)
        return c
    c["tol"] = rng.choice([1e-2, 1e-3, 1e-4])
    c["steps"] = 8 if shape == "sphere" else {1e-2: 15, 1e-3: 28, 1e-4: 42}[c["tol"]]
    if kind == "file":
        c["count"] = rng.choice([1, 1, 3])
    elif shape == "crossing" and rng.random() < 0.25:
        c["count"], c["mesh"] = rng.randint(2, 5), max(c["mesh"], 8e-4)
    if kind == "solve" and c["precision"] == "fp64":
        # an FP64 solve costs several times a mixed one
        c["k"], c["mesh"] = min(c["k"], 5), max(c["mesh"], 4e-4 if shape != "slab" else 2e-5)
    return c


# ----------------------------------------------------------------- inputs

_dir = tempfile.TemporaryDirectory(prefix="cases_")
atexit.register(_dir.cleanup)


@functools.lru_cache(maxsize=None)
def _context() -> fc.Context:
    return fc.Context(0)


@functools.lru_cache(maxsize=None)
def _server(slots: int) -> fc.Server:
    return _context().server(slots=slots)


@functools.lru_cache(maxsize=None)
def _sphere(depth: int):
    return geo.icosphere(depth)


def _key(case: dict) -> str:
    return json.dumps({k: case[k] for k in ("shape", "k", "length", "pitch", "gap", "count")}, sort_keys=True)


def _text(case: dict, index: int, scale: float) -> str:
    """Input file `index` of the case, every length times `scale`."""
    if case["shape"] == "sphere":
        vert, tri = _sphere(case["k"])
        p = (vert * (scale * case["length"]))[tri].reshape(len(tri), 9)
        lines = ["* sphere", "C sphere.txt  1.0  0.0 0.0 0.0", "End", "File sphere.txt", "* sphere"]
        lines += ["T sphere  " + " ".join("%.9e" % x for x in row) for row in p]
        return "\n".join(lines + ["End"]) + "\n"
    k, length, pitch, gap = case["k"], case["length"], case["pitch"], case["gap"]
    if index:  # the other geometries of a batch: sizes of their own, the same for every seed
        rng = random.Random("%s %d" % (_key(case), index))
        k, length = rng.randint(2, case["k"]), rng.uniform(10.0, max(10.0, case["length"]))
        pitch, gap = rng.uniform(2.0, 4.0), rng.uniform(1.0, 3.0)
    slab = None
    if case["shape"] == "slab":
        top = 2.0 + gap + 0.5
        slab = (top * scale, 1.0, 3.9, 1.5 * length * scale)
    return geo.Crossing(k=k, length=length * scale, pitch=pitch * scale, gap=gap * scale, width=scale, height=scale,
                        eps_r=3.9 if slab else 1.0, slab=slab).text()


def _files(case: dict, seed: int) -> list:
    # a product's vectors are as long as its panels: the same for every seed
    scale = 1.0 if case["kind"] == "product" else 1.0 + 0.02 * random.Random(seed).random()
    paths = []
    for i in range(case["count"]):
        fd, path = tempfile.mkstemp(suffix=".txt", dir=_dir.name)
        with os.fdopen(fd, "w") as f:
            f.write(_text(case, i, scale))
        paths.append(path)
    return paths


def _models(case: dict, seed: int) -> list:
    return [fc.Model.build(p, mesh_eps=case["mesh"], eps_ratio=case["ratio"], ctx=_context()) for p in _files(case, seed)]


def _precision(case: dict) -> int:
    return fc.PREC_MIXED if case["precision"] == "mixed" else fc.PREC_FP64


def _vectors(n: int, columns: int, seed: int):
    """Charge vectors as a Krylov iteration has them: normalised, signs mixed,
    smooth parts and noise."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.randn((columns, n), generator=gen, dtype=torch.float64, device="cuda")
    q += torch.linspace(0.5, 2.0, columns, dtype=torch.float64, device="cuda")[:, None]
    return q / q.norm(dim=1, keepdim=True)


def prepare(case: dict, seed: int) -> dict:
    if case["kind"] == "file":
        # as many slots as a burst has files: the server is there before the requests
        return {"case": case, "paths": _files(case, seed), "server": _server(case["count"])}
    models = _models(case, seed)
    model, geom = fc.Model.concat(models) if len(models) > 1 else (models[0], None)
    prob = _context().problem(model, _precision(case))
    prob.set_tuning(False)
    if geom is not None:
        prob.set_geometries(geom)
    state = {"case": case, "prob": prob}
    if case["kind"] == "product":
        prob.fill()
        state["q"] = _vectors(prob.n_panels, case["columns"], seed)
        state["v"] = torch.empty_like(state["q"])
        torch.cuda.synchronize()  # the problem works on a stream of its own
    return state


def run(state: dict):
    case = state["case"]
    if case["kind"] == "file":
        jobs = [state["server"].submit_file(p, precision=_precision(case), tol=case["tol"], mesh_eps=case["mesh"],
                                            eps_ratio=case["ratio"]) for p in state["paths"]]
        out = [j.result() for j in jobs]
        return {"cap": [c for c, _ in out], "iterations": [i for _, i in out]}
    prob = state["prob"]
    if case["kind"] == "product":
        prob.matvec_device(state["q"].data_ptr(), state["v"].data_ptr(), case["columns"])
        return {"v": state["v"]}
    prob.fill()
    cap, its = prob.solve(tol=case["tol"])
    return {"cap": cap, "iterations": its} if case["count"] == 1 else {"cap": list(cap), "iterations": list(its)}


# ------------------------------------------------------------------- work


@functools.lru_cache(maxsize=None)
def _counts(shape_json: str):
    case = json.loads(shape_json)
    ms = _models(case, 1)
    return [(m.n_panels, m.n_links, len(m.conductor_names)) for m in ms]


def work(case: dict) -> dict:
    """A product streams a coefficient and a source word per link and reads
    and writes its vectors. A solve has one product, and two passes over its
    vector and basis vectors, per step; a fill reads a source word and writes
    a coefficient per link. Making links writes a word per link."""
    counts = _counts(json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True))
    word = 8 if case["precision"] == "mixed" else 12
    bytes_, flops = 0.0, 0.0
    for panels, links, cond in counts:
        if case["kind"] == "product":
            k = case["columns"]
            bytes_ += links * word + 16.0 * k * panels
            flops += 2.0 * k * links
            continue
        s = case["steps"]
        bytes_ += links * word * (s + 1.0) + 8.0 * cond * panels * (0.5 * s * s + 2.0 * s)
        flops += 2.0 * cond * links * s + 2.0 * cond * panels * s * s
        bytes_ += links * word
        flops += 30.0 * links
        if case["kind"] == "file":
            bytes_ += 4.0 * links + 200.0 * panels
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------- the same outputs in 64 bits

FOUR_PI_E0 = 1.1126500559756e-10  # the reference's constants (Solver/Potential.h:41-45)
TWO_E0 = 1.7708375634e-11
EPS = 1e-6
DIEL, OUTSIDE, SUPER = 2, 4, 128  # element type bits


def _dot(a, b):
    return (a * b).sum(-1)


def _rule(points):
    t = torch.tensor(points, dtype=torch.float64, device="cuda")
    return t, torch.full((len(points),), 1.0 / len(points), dtype=torch.float64, device="cuda")


def _rules():
    """Quadrature points in triangle coordinates (their third is 1 - the other
    two), with equal weights: three interior points, the edge midpoints, six
    interior points."""
    a, b, c = 0.659027622374092, 0.231933368553031, 0.109039009072877
    third = _rule([(2 / 3, 1 / 6), (1 / 6, 2 / 3), (1 / 6, 1 / 6)])
    mid = _rule([(0.0, 0.5), (0.5, 0.0), (0.5, 0.5)])
    six = _rule([(a, b), (a, c), (b, a), (b, c), (c, a), (c, b)])
    return {1: six, 2: mid, 3: third}


def _sides(v):
    """The sides of single-precision triangles, each a difference of two
    stored vertices rounded as they are (part of the method: it moves a
    coefficient by up to 1e-7)."""
    return [(v[:, (i + 1) % 3] - v[:, i]).double() for i in range(3)]


def _quadrature(r, v, normal, rule):
    s1, s2, s3 = _sides(v)
    cross = torch.linalg.cross(s1, s2)
    double_area, length = _dot(cross, cross).sqrt(), _dot(s1, s1).sqrt()
    x = s1 / length[:, None]
    y = torch.linalg.cross(x, cross / double_area[:, None])
    down = -_dot(s3, y)
    edge = x * -_dot(s3, x)[:, None] + y * down[:, None]
    total = torch.zeros(len(r), dtype=torch.float64, device="cuda")
    for (px, py), w in zip(rule[0].tolist(), rule[1]):
        d = r - (v[:, 0].double() + px * s1 + (1.0 - px - py) * edge)
        m = _dot(d, d).sqrt()
        total += w * (1.0 / m if normal is None else _dot(d, normal) / m**3)
    return total * (-length * down / double_area)


def _analytic(r, v):
    """Potential at r of a unit charge spread evenly over the triangle v."""
    side = _sides(v)
    n = torch.linalg.cross(side[0], side[1])
    double_area = _dot(n, n).sqrt()
    n = n / double_area[:, None]
    rel = v.double() - r[:, None, :]
    dist = _dot(rel, rel).sqrt()
    d = -_dot(n, rel[:, 0])
    flat = rel - n[:, None, :] * (rel * n[:, None, :]).sum(-1, keepdim=True)
    total = torch.zeros(len(r), dtype=torch.float64, device="cuda")
    for i in range(3):
        j = (i + 1) % 3
        l = side[i] / _dot(side[i], side[i]).sqrt()[:, None]
        u = torch.linalg.cross(l, n)
        p0s, lp, lm = _dot(flat[:, j], u), _dot(flat[:, j], l), _dot(flat[:, i], l)
        p0 = p0s.abs()
        tol = EPS * torch.where(lp > lm, lp.abs(), lm.abs())
        ap, am = dist[:, j] + lp, dist[:, i] + lm
        keep = (p0 > tol) & (ap.abs() > tol) & (am.abs() > tol)
        r0 = p0 * p0 + d * d
        angle = torch.atan(p0 * lp / (r0 + d.abs() * dist[:, j])) - torch.atan(p0 * lm / (r0 + d.abs() * dist[:, i]))
        term = torch.sign(p0s) * (p0 * torch.log(ap / am) - d.abs() * angle)
        total += torch.where(keep, term, torch.zeros_like(term))
    return 2.0 * total / double_area


class _Operator:
    """A model's coefficients and its hierarchical product in 64 bits."""

    def __init__(self, a: dict):
        def put(name, dtype=None):
            t = torch.from_numpy(np.array(a[name])).cuda()
            return t if dtype is None else t.to(dtype)

        f64, i64 = torch.float64, torch.int64
        kind, left = put("node_type", i64), put("node_left", i64)
        vert = put("node_vertices").reshape(-1, 3, 3)
        cent, side = put("node_centroid"), put("node_maxside")
        normal = put("node_normal", f64)
        size = _dot(normal, normal).sqrt()[:, None]
        is_super = (kind & SUPER)[:, None] != 0
        normal = torch.where(is_super, torch.where(size < 1e-12, torch.zeros_like(normal), normal / size), normal)
        normal = torch.where((kind & OUTSIDE)[:, None] != 0, normal, -normal)
        ptr, src = put("link_ptr", i64), put("link_src", i64)
        self.n_nodes, self.n = len(kind), len(a["leaf_diel"])
        row = torch.repeat_interleave(torch.arange(self.n_nodes, device="cuda"), ptr[1:] - ptr[:-1])
        coef = torch.empty(len(src), dtype=f64, device="cuda")
        rules = _rules()
        for lo in range(0, len(src), 4_000_000):
            i, j = row[lo:lo + 4_000_000], src[lo:lo + 4_000_000]
            off = (cent[i] - cent[j]).to(f64)  # the difference of two stored (single) centroids, rounded as they are
            dist = _dot(off, off).sqrt()
            rho = dist / torch.maximum(side[i], side[j])
            band = (rho >= 1).to(i64) + (rho >= 2) + (rho >= 4) + (rho >= 10)
            diel = (kind[i] & DIEL) != 0
            out = torch.empty(len(i), dtype=f64, device="cuda")
            for b in range(5):
                for field in (False, True):
                    at = ((band == b) & (diel == field)).nonzero()[:, 0]
                    if not len(at):
                        continue
                    ii, jj = i[at], j[at]
                    r, v, nn = cent[ii].to(f64), vert[jj], normal[ii]
                    if b == 4:
                        val = _dot(off[at], nn) / dist[at]**3 if field else 1.0 / dist[at]
                    elif b > 0:
                        val = _quadrature(r, v, nn if field else None, rules[b])
                    elif field:
                        h = (dist[at] / 20.0)[:, None]
                        val = (_analytic(r - nn * h, v) - _analytic(r + nn * h, v)) / (2.0 * h[:, 0])
                    else:
                        val = _analytic(r, v)
                    out[at] = val
            coef[lo:lo + 4_000_000] = out / FOUR_PI_E0
        del row
        self.links = torch.sparse_csr_tensor(ptr, src, coef, (self.n_nodes, self.n_nodes), check_invariants=False)
        self.first, self.last = put("node_leaf_first", i64), put("node_leaf_first", i64) + put("node_leaf_count", i64)
        # leaves: the nodes without children, in leaf order
        leaf = (left < 0).nonzero()[:, 0]
        leaf = leaf[torch.argsort(self.first[leaf])]
        self.leaf = leaf
        self_coef = _analytic(cent[leaf].to(f64), vert[leaf]) / FOUR_PI_E0
        self.weight = torch.zeros(self.n, dtype=f64, device="cuda")
        area, sub = put("node_area"), a["leaf_diel"]
        self.cond = []
        for c in range(len(a["cond_is_diel"])):
            lo = int(a["cond_leaf_first"][c])
            hi = lo + int(a["cond_leaf_count"][c])
            if a["cond_is_diel"][c]:
                outer, inner = float(a["cond_outperm"][c]), float(a["cond_inperm"][c])
                self_coef[lo:hi] = (inner + outer) / (TWO_E0 * (outer - inner) * area[leaf[lo:hi]])
            else:
                w = a["cond_surf_outperm"][int(a["cond_surf_ptr"][c]) + np.asarray(sub[lo:hi], np.int64)]
                self.weight[lo:hi] = torch.from_numpy(np.array(w)).cuda()
                self.cond.append((lo, hi))
        self.self_coef = self_coef

    def product(self, q):
        """v = P q for q of shape [k][n]."""
        zero = torch.zeros((len(q), 1), dtype=torch.float64, device="cuda")
        total = torch.cat([zero, q.cumsum(1)], 1)
        charge = (total[:, self.last] - total[:, self.first]).T.contiguous()
        charge[self.leaf] = q.T
        pot = (self.links @ charge).T
        # every node's potential reaches the leaves below it
        step = torch.zeros((len(q), self.n + 1), dtype=torch.float64, device="cuda")
        inner = torch.ones(self.n_nodes, dtype=torch.bool, device="cuda")
        inner[self.leaf] = False
        step.index_add_(1, self.first[inner], pot[:, inner])
        step.index_add_(1, self.last[inner], -pot[:, inner])
        return self.self_coef * q + pot[:, self.leaf] + step.cumsum(1)[:, :-1]

    def solve(self, tol):
        """GMRES with the Jacobi preconditioner and the reference's start and
        stopping test (Solver/SolveCapacitance.cpp:2288-2574)."""
        cap = torch.zeros((len(self.cond), len(self.cond)), dtype=torch.float64)
        its = np.zeros(len(self.cond), np.int32)
        for c, (lo, hi) in enumerate(self.cond):
            b = torch.zeros(self.n, dtype=torch.float64, device="cuda")
            b[lo:hi] = 1.0
            x0 = b / self.self_coef
            r = b - self.product(x0[None])[0]
            norm_r, norm_b = float(r.norm()), float(b.norm())
            x = x0
            if norm_r / norm_b >= tol:
                basis, cols, g = [r / norm_r], [], [norm_r]
                rot = []
                for i in range(min(1000, self.n)):
                    w = self.product((basis[-1] / self.self_coef)[None])[0]
                    q = torch.stack(basis)
                    h = q @ w
                    w = w - h @ q
                    hn = float(w.norm())
                    col = h.tolist() + [hn]
                    basis.append(w / hn)
                    for j, (cs, sn) in enumerate(rot):
                        col[j], col[j + 1] = cs * col[j] - sn * col[j + 1], cs * col[j + 1] + sn * col[j]
                    length = math.hypot(col[i], col[i + 1])
                    cs, sn = col[i] / length, -col[i + 1] / length
                    rot.append((cs, sn))
                    col[i] = cs * col[i] - sn * col[i + 1]
                    cols.append(col[: i + 1])
                    g[i:] = [cs * g[i], sn * g[i]]
                    its[c] = i + 1
                    if abs(g[i + 1]) / norm_b < tol:
                        break
                m = len(cols)
                upper = np.zeros((m, m))
                for i, col in enumerate(cols):
                    upper[: i + 1, i] = col
                z = np.linalg.solve(upper, np.array(g[:m]))
                y = torch.from_numpy(z).cuda() @ torch.stack(basis[:m])
                x = x0 + y / self.self_coef
            for d, (a, e) in enumerate(self.cond):
                cap[c, d] = (self.weight[a:e] * x[a:e]).sum()
        return cap.numpy(), its


def exact(case: dict, seed: int):
    """The panels and links are the model's; everything computed from them is
    plain torch in 64 bits."""
    models = _models(case, seed)
    if sum(m.n_links for m in models) > 100_000_000:
        return None
    ops = (_Operator(m.arrays) for m in models)
    if case["kind"] == "product":
        op = next(ops)
        return {"v": op.product(_vectors(op.n, case["columns"], seed))}
    out = [op.solve(case["tol"]) for op in ops]
    if case["kind"] == "solve" and case["count"] == 1:
        return {"cap": out[0][0], "iterations": None}
    return {"cap": [c for c, _ in out], "iterations": [None] * len(out)}
