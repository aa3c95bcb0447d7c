"""The workloads that the speed of this framework is measured on, as calls of its public entry points.

Each case is a plain dict; ``listed()`` gives the fixed ones, ``draw(rng)`` another of the
same ranges, ``prepare(case, seed)`` what a program holds before the call, ``run(state)`` one
pass, ``work(case)`` the least bytes and operations of a pass and ``exact(case, seed)`` the
pass's results in 64-bit torch arithmetic written out here, where that is short enough to
evaluate.

Families (``what``):
  relax    upload positions, a few relaxation steps, download the new positions: the loop of
           every run (a run is 200 to 500 such steps).  "settled" positions follow the target
           spacing, as from the first tens of steps on; "seeded" ones are uniform in the body,
           as Initialize_case leaves them, with many more neighbours.
  batch    the same over many small bodies at once (BatchRelaxation).
  setup    a new handle from level-set grids, its fields, and phi / normals at points.
  volume   the cut-cell volume pass that gives a geometry's particle number.
  cvp      centroidal Voronoi partition of the particles.
  tris     triangle mesh of the particles and its quality (2D).
  tets     tetrahedral mesh of the particles and its quality (3D).

FP32-split positions are handed on as float32, FP64-plain results as float64.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "sph-mesh-generation_gb300"))

from mrsph import BatchRelaxation, SPHMeshGeneration, cases  # noqa: E402


# ------------------------------------------------------------------ cases
def listed():
    return [
        # A small 2D body: the unit square less a disc on a 256^2 grid.  Launches count.
        {"name": "relax_disc_2d", "what": "relax", "geom": "disc", "n": 8745, "start": "settled", "steps": 8,
         "kernel": "wendland", "precision": "fp32"},
        # A small 3D body with the reference's default smoothing kernel.
        {"name": "relax_star_3d", "what": "relax", "geom": "star3", "n": 20000, "start": "settled", "steps": 4,
         "kernel": "hyperbolic", "precision": "fp32"},
        # The accurate path: FP64 arithmetic throughout, whole particle state read back.
        {"name": "relax_torus_fp64", "what": "relax", "geom": "torus", "n": 37249, "start": "settled", "steps": 2,
         "kernel": "wendland", "precision": "fp64"},
        # The square with 64 elliptic holes, spacing graded 1:8.
        {"name": "relax_ellipses_2d", "what": "relax", "geom": "ellipses", "n": 77551, "start": "settled",
         "steps": 4, "kernel": "wendland", "precision": "fp32"},
        # A medium 3D body in its first steps: uniform positions, 300 and more neighbours.
        {"name": "relax_torus_seeded", "what": "relax", "geom": "torus", "n": 301270, "start": "seeded", "steps": 4,
         "kernel": "wendland", "precision": "fp32"},
        # The benchmark body, 2.4 M particles, relaxed: where a long run spends its time.
        {"name": "relax_torus_settled", "what": "relax", "geom": "torus", "n": 2410164, "start": "settled",
         "steps": 4, "kernel": "wendland", "precision": "fp32"},
        # 24 star bodies, half 2D half 3D, stepped together.
        {"name": "batch_stars", "what": "batch", "count": 24, "n_min": 2000, "n_max": 60000, "steps": 4},
        # A geometry's set-up: level sets of 64 and 128 cells, fields, 100,000 samples.
        {"name": "setup_torus", "what": "setup", "geom": "torus", "fine": 32, "points": 100003, "precision": "fp64"},
        # The particle number of the benchmark body (256 x 256 x 96 cells).
        {"name": "volume_torus", "what": "volume", "geom": "torus", "fine": 64},
        # Partition of 300,000 particles into 128 domains.
        {"name": "cvp_torus", "what": "cvp", "geom": "torus", "n": 301270, "vps": 128, "iters": 12},
        # Triangle mesh of the square with elliptic holes.
        {"name": "tris_ellipses", "what": "tris", "geom": "ellipses", "n": 77551},
        # Tetrahedral mesh of a medium body.
        {"name": "tets_torus", "what": "tets", "geom": "torus", "n": 150001},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["relax"] * 6 + ["batch", "setup", "volume", "cvp", "tris", "tets"])
    if what == "relax":
        precision = "fp64" if rng.random() < 0.15 else "fp32"
        geom = rng.choice(["disc", "star2", "star3", "torus", "torus", "ellipses", "spheres"])
        start = rng.choice(["settled", "settled", "seeded"])
        top = {"disc": 300000, "star2": 100000, "star3": 200000, "torus": 1800000, "ellipses": 300000,
               "spheres": 1000000}[geom]
        if precision == "fp64":
            top = 37000
        elif start == "seeded":
            top = min(top, 500000)
        return {"what": "relax", "geom": geom, "n": _log(rng, 5000 if geom in ("torus", "spheres") else 2000, top),
                "start": start, "steps": 1 if precision == "fp64" else rng.randint(1, 4),
                "kernel": rng.choice(["wendland"] * 4 + ["hyperbolic", "cubic"]), "precision": precision}
    if what == "batch":
        return {"what": "batch", "count": rng.randint(2, 24), "n_min": 2000, "n_max": _log(rng, 5000, 60000),
                "steps": rng.randint(1, 4)}
    if what == "setup":
        return {"what": "setup", "geom": rng.choice(["torus", "star2", "star3", "disc"]), "fine": 32,
                "points": _log(rng, 1, 100000), "precision": rng.choice(["fp64", "fp32"])}
    if what == "volume":
        return {"what": "volume", "geom": rng.choice(["torus", "star2", "star3", "disc", "spheres"]),
                "fine": rng.choice([32, 64]), "seed": rng.randint(0, 1 << 20)}
    if what == "cvp":
        return {"what": "cvp", "geom": rng.choice(["torus", "star2", "star3", "disc"]), "n": _log(rng, 3000, 300000),
                "vps": _log(rng, 2, 128), "iters": rng.randint(2, 12)}
    if what == "tris":
        return {"what": "tris", "geom": rng.choice(["disc", "star2", "ellipses"]), "n": _log(rng, 2000, 77000)}
    return {"what": "tets", "geom": rng.choice(["torus", "star3", "spheres"]), "n": _log(rng, 5000, 150000)}


# ------------------------------------------------------------------ geometries
@functools.lru_cache(maxsize=64)
def _geometry(geom, n, kernel, precision, fine=0, number=5):
    """The workloads of mrsph.cases, sized for about n particles."""
    kw = {"kernel": kernel, "precision": precision}
    if geom == "disc":
        return cases.disc_hole_2d(spacing=math.sqrt(0.87434 / n), grid=256, **kw)
    if geom in ("star2", "star3"):
        return cases.star_shape(2 if geom == "star2" else 3, number, n, **kw)
    if geom == "ellipses":
        dx = 0.001 * math.sqrt(77551.0 / n)
        return cases.ellipses_2d(dx_min=dx, dx_max=8 * dx, grid=512, **kw)
    make, size, grade, grid = (cases.torus_3d, 0.005 * 2410164.0 ** (1 / 3.0), 4.0, fine or 64) if geom == "torus" \
        else (cases.spheres_3d, 0.005 * 353003.0 ** (1 / 3.0), 4.8, fine or 32)
    dx = size / n ** (1 / 3.0)
    for _ in range(200):  # the spacing range has to give a consistent cell-list plan
        try:
            extra = {"middle_dl": 1.6 * dx} if geom == "spheres" else {}
            return make(dx_min=dx, dx_max=grade * dx, fine_pkg=grid, nlevels=3 if grid >= 64 else 2, **extra, **kw)
        except ValueError:
            dx *= 1.003
    raise ValueError("no consistent spacing near %g" % dx)


def _of(case):
    return _geometry(case["geom"], case.get("n", 20000), case.get("kernel", "wendland"),
                     case.get("precision", "fp32"), case.get("fine", 0), case.get("seed", 5))


def _shifted(g, delta):
    """The body grown by delta: phi + delta on every level."""
    levels = [cases.LevelGrid(lv.box_l, lv.dpkg, lv.num_pkg, lv.margin, lv.phi + delta, lv.active)
              for lv in g.levels]
    return cases.Case(g.name, g.params, levels, g.n_particles)


def _finest_cell(g):
    return g.levels[-1].dpkg[0] / 4.0


def _morton(idx, bits):
    """Interleaved index of integer coordinates (dim x m)."""
    out = torch.zeros_like(idx[0])
    for b in range(bits):
        for d in range(len(idx)):
            out |= ((idx[d] >> b) & 1) << (b * len(idx) + d)
    return out


def _positions(g, n, start, seed):
    """n positions inside the body of case g, a function of the seed alone: systematic sampling
    of the interior cells in Z-order with density 1 / spacing^dim ("settled") or uniform where
    phi exceeds the smoothing length ("seeded"), jittered inside (fractions of) a cell."""
    p, lv = g.params, g.levels[-1]
    dim, m = p["dim"], 4 * lv.margin
    dev = torch.device("cuda")
    phi = torch.from_numpy(lv.phi).to(dev)
    phi = phi[m:-m, m:-m, m:-m] if dim == 3 else phi[:, m:-m, m:-m]
    mp = cases.max_phi(g.levels, dim)
    lo = p["min_dl"] if not p.get("scale_law") else p["middle_dl"]
    scale = lo + torch.tanh(2.5 * phi.abs() / mp) / math.tanh(2.5) * (p["max_dl"] - lo)
    if start == "settled":
        keep, weight = phi > 0, scale ** -dim
    else:
        keep, weight = phi > scale * p["cell_ratio"] / p["cutoff"], torch.ones_like(scale)
    idx = torch.nonzero(keep).t().flip(0)[:dim]  # x, y(, z) by column
    weight = weight[keep]
    order = torch.argsort(_morton(idx, 11))
    idx, weight = idx[:, order], weight[order]
    peak = float(weight.max() / weight.sum()) * n
    sub = 1
    while sub < 4 and sub ** dim < peak:
        sub *= 2
    part = torch.arange(sub ** dim, device=dev)
    local = torch.stack([sum(((part >> (b * dim + d)) & 1) << b for b in range(2)) for d in range(dim)])
    # whole weights: their running sum does not depend on the order of the additions
    weight = (weight * (2.0 ** 20 / weight.max())).long() + 1
    cum = torch.cumsum(weight, 0).double()
    weight = weight.double()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    at = (torch.arange(n, device=dev, dtype=torch.float64) + torch.rand(1, generator=gen, device=dev,
                                                                        dtype=torch.float64)) * (cum[-1] / n)
    cell = torch.searchsorted(cum, at).clamp_(max=len(cum) - 1)
    inside = (at - (cum[cell] - weight[cell])) / weight[cell]
    piece = (inside * sub ** dim).long().clamp_(0, sub ** dim - 1)
    xyz = torch.zeros(n, 3, dtype=torch.float64, device=dev)
    for d in range(dim):
        u = torch.rand(n, generator=gen, device=dev, dtype=torch.float64)
        xyz[:, d] = lv.box_l[d] + (idx[d][cell] + (local[d][piece] + u) / sub) * (lv.dpkg[d] / 4.0)
    return xyz[torch.randperm(n, generator=gen, device=dev)]


# ------------------------------------------------------------------ states
def _pinned(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out


def _loaded(g, xyz):
    """A handle that holds the positions, mapped and binned (Pre_run)."""
    s = SPHMeshGeneration(g)
    s.set_state({"xyz": xyz.cpu().numpy()}, pre_run=True)
    return s


def _star_numbers(case, seed):
    rng = np.random.default_rng(case["count"])  # the bodies; the seed makes their particles
    n = np.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"]), case["count"]))
    return [("star2" if k % 2 == 0 else "star3", int(v), 100 + k, seed * 64 + k) for k, v in enumerate(n)]


def prepare(case, seed):
    what = case["what"]
    if what == "batch":
        bodies = _star_numbers(case, seed)
        geoms = [_geometry(kind, n, "wendland", "fp32", 0, number) for kind, n, number, _ in bodies]
        x0 = [_pinned(_positions(g, g.n_particles, "settled", b[3])) for g, b in zip(geoms, bodies)]
        solvers = [_loaded(g, x) for g, x in zip(geoms, x0)]
        batch = BatchRelaxation(solvers)
        total = sum(len(x) for x in x0)
        out = torch.empty(total, 3, dtype=torch.float64, pin_memory=True)
        return {"what": what, "steps": case["steps"], "solvers": solvers, "batch": batch,
                "x0": [x.numpy() for x in x0], "keep": x0, "out": out,
                "parts": [p.numpy() for p in torch.split(out, [len(x) for x in x0])],
                "pos": torch.empty(total, 3, dtype=torch.float32)}
    g = _of(case)
    if what in ("setup", "volume"):
        rng = np.random.default_rng(seed)
        g = _shifted(g, (rng.random() - 0.5) * _finest_cell(g))
        if what == "volume":
            return {"what": what, "solver": SPHMeshGeneration(g)}
        lo, hi = np.array(g.params["box_l"]), np.array(g.params["box_r"])
        xyz = lo + rng.random((case["points"], 3)) * (hi - lo)
        return {"what": what, "geometry": g, "xyz": xyz, "precision": case["precision"]}
    n = int(case["n"])
    xyz = _positions(g, n, case.get("start", "settled"), seed)
    s = _loaded(g, xyz)
    if what == "relax":
        x0 = _pinned(xyz)
        out = torch.empty(n, 3, dtype=torch.float64, pin_memory=True)
        return {"what": what, "solver": s, "steps": case["steps"], "precision": case["precision"], "keep": x0,
                "x0": x0.numpy(), "out": out, "host": out.numpy(), "pos": torch.empty(n, 3, dtype=torch.float32)}
    if what == "cvp":
        return {"what": what, "solver": s, "vp": xyz[: case["vps"]].cpu().numpy(), "iters": case["iters"]}
    s.SPH_run_mesh_generation(1)  # neighbour rows for the mesh
    return {"what": what, "solver": s,
            "mesh": torch.empty((2 * n, 3) if what == "tris" else (8 * n, 4), dtype=torch.int32)}


def run(state):
    what = state["what"]
    if what == "relax":
        s = state["solver"]
        s.upload_positions(state["x0"])
        s.SPH_run_mesh_generation(state["steps"])
        if state["precision"] == "fp64":
            return s.particles(("xyz", "v", "h", "type"))
        s.download_positions(state["host"])
        return state["pos"].copy_(state["out"])
    if what == "batch":
        for s, x in zip(state["solvers"], state["x0"]):
            s.upload_positions(x)
        state["batch"].SPH_run_mesh_generation(state["steps"])
        state["batch"].sync()
        for s, part in zip(state["solvers"], state["parts"]):
            s.download_positions(part)
        return state["pos"].copy_(state["out"])
    if what == "setup":
        s = SPHMeshGeneration(state["geometry"])
        f = s.levelset_fields(len(state["geometry"].levels) - 1)
        phi, nrm, curv, tag = s.sample_levelset(state["xyz"])
        s.close()
        t = np.float32 if state["precision"] == "fp32" else np.float64
        return {"fields": f, "at": {"phi": phi.astype(t), "normal": nrm.astype(t), "curvature": curv.astype(t),
                                    "tag": tag}}
    s = state["solver"]
    if what == "volume":
        out = s.volume_mass(-1, cells=True)
        out.pop("device_ms")  # a time, not a result
        return out
    if what == "cvp":
        return s.Partitioning(state["vp"], max_iter=state["iters"])
    mesh, quality = s.Reconstruct_tris() if what == "tris" else s.Reconstruct_tets()
    # the program's own mesh array, of one size for every mesh of n particles
    state["mesh"][: len(mesh)].copy_(torch.from_numpy(mesh))
    state["mesh"][len(mesh):] = -1
    return state["mesh"], quality


# ------------------------------------------------------------------ least work
def _pair_work(dim, n, steps, real):
    """A step reads positions, spacing and viscosity and writes positions, type and viscosity; a
    pair costs a distance, a kernel value, its gradient and two vector terms."""
    pairs = (21.2 if dim == 2 else 73.6) * n  # spheres of 2 h, h = 1.3 spacings
    return {"bytes": steps * n * real * (2 * dim + 5), "flops": steps * pairs * (8 + 8 + 20 + 14)}


def work(case):
    what = case["what"]
    if what == "batch":
        parts = [_pair_work(2 if b[0] == "star2" else 3, b[1], case["steps"], 4) for b in _star_numbers(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    g = _of(case)
    dim = g.params["dim"]
    n = case.get("n", 0)
    cells = sum(lv.phi.size for lv in g.levels)
    if what == "relax":
        w = _pair_work(dim, n, case["steps"], 4 if case["precision"] == "fp32" else 8)
        return {"bytes": w["bytes"] + 48.0 * n, "flops": w["flops"]}
    if what == "setup":  # phi in, fields out; samples in and out
        return {"bytes": 8.0 * cells + 33.0 * g.levels[-1].phi.size + 68.0 * case["points"],
                "flops": 40.0 * cells + 100.0 * case["points"]}
    if what == "volume":
        return {"bytes": 24.0 * g.levels[-1].phi.size, "flops": 20.0 * g.levels[-1].phi.size}
    if what == "cvp":  # a point is compared with the VPs around its own
        return {"bytes": 28.0 * n, "flops": (case["iters"] + 1) * n * 27 * 8.0}
    # a particle reads itself and its neighbours and writes its share of the mesh
    return {"bytes": n * (24.0 + (24.0 if dim == 2 else 100.0)), "flops": n * (21.0 * 30 if dim == 2 else 74.0 * 200)}


# ------------------------------------------------------------------ results in 64 bits
class _Fields:
    """The level sets of a case in float64: phi, unit normals, curvature, cut-cell tags."""

    def __init__(self, g):
        self.g, self.p, self.dim = g, g.params, g.params["dim"]
        self.dev = torch.device("cuda")
        self.lv = [self._level(lv) for lv in g.levels]
        self.max_phi = max(f["max_phi"] for f in self.lv)
        cut = torch.cat([f["curv"][f["tag"]] for f in self.lv])
        self.max_curv, self.min_curv = (float(cut.max()), float(cut.min())) if len(cut) else (0.0, 1e20)
        self.dl0 = min(g.levels[0].dpkg[d] / 4.0 for d in range(self.dim))

    def _level(self, lv):
        dim, m = self.dim, 4 * lv.margin
        ph = torch.from_numpy(lv.phi).to(self.dev)
        dc = [lv.dpkg[d] / 4.0 for d in range(dim)]
        inner = torch.zeros_like(ph, dtype=torch.bool)
        inner[(slice(m, -m) if dim == 3 else slice(None), slice(m, -m), slice(m, -m))] = True

        def sh(*off):  # phi at (x + off[0], y + off[1], ...)
            return torch.roll(ph, [-o for o in off], [2 - d for d in range(len(off))])

        def ax(d, k):
            return sh(*[k if q == d else 0 for q in range(dim)])

        grad = []
        for d in range(dim):
            loc = (torch.arange(ph.shape[2 - d], device=self.dev) % 4).view([-1 if a == 2 - d else 1 for a in range(3)])
            side = torch.where(loc == 0, (ax(d, 1) - ph) / dc[d],
                               torch.where(loc == 3, (ph - ax(d, -1)) / dc[d], 0.5 * (ax(d, 1) - ax(d, -1)) / dc[d]))
            grad.append(torch.where(inner, 0.5 * (ax(d, 1) - ax(d, -1)) / dc[d], side))
        size = torch.sqrt(sum(v * v for v in grad)) + 1e-12
        n = [v / size for v in grad] + [torch.zeros_like(ph)] * (3 - dim)
        # a cell is cut when its centre and its corners (means of the cells around them) differ in sign
        offs = [[(c >> d) & 1 for d in range(dim)] for c in range(1 << dim)]
        sign = torch.sign(sum(sh(*[-o for o in off]) for off in offs) / len(offs))  # the cell's lower corner
        corners = [torch.roll(sign, [-o for o in off], [2 - d for d in range(dim)]) for off in offs]
        cut = torch.sign(ph) != corners[0]
        for c in corners[1:]:
            cut |= c != corners[0]
        cut &= inner
        d1 = [(8.0 * (ax(d, 1) - ax(d, -1)) - (ax(d, 2) - ax(d, -2))) / dc[d] / 12.0 for d in range(dim)]
        d2 = [(ax(d, 1) - 2 * ph + ax(d, -1)) / dc[d] / dc[d] for d in range(dim)]
        num = torch.zeros_like(ph)
        for a in range(dim):
            for b in range(a + 1, dim):
                def at(i, j):
                    return sh(*[i if q == a else j if q == b else 0 for q in range(dim)])
                mix = 0.25 * (at(1, 1) - at(-1, 1) - at(1, -1) + at(-1, -1)) / dc[a] / dc[b]
                num += d1[a] ** 2 * d2[b] - 2 * d1[a] * d1[b] * mix + d1[b] ** 2 * d2[a]
        den = sum(v * v for v in d1) ** 1.5
        lim = 2.0 / math.sqrt(sum(v * v for v in dc))
        curv = torch.where(cut, (num / den).clamp(-lim, lim).abs(), torch.zeros_like(ph))
        pos = ph[inner & (ph > 0)]
        return {"phi": ph, "n": n, "curv": curv, "tag": cut, "dc": dc, "lv": lv,
                "max_phi": float(pos.max()) if len(pos) else 0.0}

    def _cells(self, x):
        """The level and position (in cells of it, from its box) of every point."""
        which = torch.zeros(len(x), dtype=torch.long, device=self.dev)
        for l in range(1, len(self.lv)):
            lv = self.lv[l]["lv"]
            pk = [torch.floor((x[:, d] - lv.box_l[d]) / lv.dpkg[d]).long() for d in range(self.dim)]
            ok = torch.ones(len(x), dtype=torch.bool, device=self.dev)
            for d in range(self.dim):
                ok &= (pk[d] >= 0) & (pk[d] < lv.num_pkg[d])
            if lv.active is not None:
                np_ = [lv.num_pkg[d] + 2 * lv.margin if d < self.dim else 1 for d in range(3)]
                act = torch.from_numpy(np.ascontiguousarray(lv.active)).to(self.dev).reshape(-1)
                flat = torch.zeros_like(which)
                for d in reversed(range(self.dim)):
                    flat = flat * np_[d] + (pk[d].clamp(0, lv.num_pkg[d] - 1) + lv.margin)
                ok &= act[flat] != 0
            which[ok] = l
        return which

    def sample(self, x):
        """phi, normal and curvature by linear interpolation of the cell centres around x, and the
        tag of the cell that holds it."""
        n = len(x)
        phi, curv = torch.zeros(n, dtype=torch.float64, device=self.dev), torch.zeros(n, dtype=torch.float64, device=self.dev)
        nrm = torch.zeros(n, 3, dtype=torch.float64, device=self.dev)
        tag = torch.zeros(n, dtype=torch.bool, device=self.dev)
        which = self._cells(x)
        for l, f in enumerate(self.lv):
            at = torch.nonzero(which == l)[:, 0]
            if not len(at):
                continue
            lv, m = f["lv"], 4 * f["lv"].margin
            lo, w, own = [], [], []
            for d in range(self.dim):
                cs = (x[at, d] - lv.box_l[d]).clamp(0.0, lv.dpkg[d] * lv.num_pkg[d] - 1e-8)
                pk = torch.floor(cs / lv.dpkg[d]).clamp(-lv.margin, lv.num_pkg[d] + lv.margin - 1)
                rest = (cs - lv.dpkg[d] * pk) / f["dc"][d]
                rr = (rest - 0.5).clamp(-0.5, 3.5)
                own.append((pk * 4 + torch.floor(rest).clamp(0, 3)).long() + m)
                lo.append((pk * 4 + torch.floor(rr)).long() + m)
                w.append(rr - torch.floor(rr))
            shape = f["phi"].shape

            def flat(c):
                z = c[2] if self.dim == 3 else torch.zeros_like(c[0])
                return (z * shape[1] + c[1]) * shape[2] + c[0]

            tag[at] = f["tag"].reshape(-1)[flat(own)]
            for c in range(1 << self.dim):
                off = [(c >> d) & 1 for d in range(self.dim)]
                coef = torch.ones(len(at), dtype=torch.float64, device=self.dev)
                for d in range(self.dim):
                    coef = coef * (w[d] if off[d] else 1.0 - w[d])
                k = flat([lo[d] + off[d] for d in range(self.dim)])
                phi[at] += f["phi"].reshape(-1)[k] * coef
                curv[at] += f["curv"].reshape(-1)[k] * coef
                for d in range(self.dim):
                    nrm[at, d] += f["n"][d].reshape(-1)[k] * coef
        return phi, nrm, curv, tag

    def spacing(self, phi, curv):
        p = self.p
        lo = torch.full_like(phi, p["min_dl"])
        if p.get("scale_law", 0) == 1:
            q = ((self.max_curv - curv.abs()) / (self.max_curv - self.min_curv + 1e-20)).clamp(0.0, 1.0)
            mid = p["middle_dl"] if p["middle_dl"] > 0 else 5.0 * self.dl0
            lo = lo + q * q * (mid - p["min_dl"])
        s = lo + torch.tanh(2.5 * phi.abs() / self.max_phi) / math.tanh(2.5) * (p["max_dl"] - lo)
        return torch.where((phi > 0) | (phi.abs() < self.dl0), s, torch.full_like(phi, p["min_dl"]))


def _philox(c, seed):
    """Philox4x32-10 (Salmon et al., 2011) of four uint32 counters held in int64 arrays."""
    c = [v.copy() if isinstance(v, np.ndarray) else np.int64(v) for v in c]
    c = list(np.broadcast_arrays(*c))
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    c = [v.astype(np.uint64) for v in c]
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        lo = np.uint64(0xFFFFFFFF)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & lo, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & lo]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


class _Relaxation:
    """Relaxation steps of REAL and SURFACE particles in float64."""

    PAIRS = 4_000_000_000  # candidate pairs of a step above which it would take too long

    def __init__(self, g, x):
        self.f, self.p, self.dim = _Fields(g), g.params, g.params["dim"]
        n = len(x)
        z = x.new_zeros
        self.x, self.v, self.a, self.nu, self.dt, self.k = x.clone(), z(n, 3), z(n, 3), z(n), 0.0, 0
        self.h = z(n)
        self._map(first=True)
        self.x = x.clone()  # the positions uploaded by the pass

    def _info(self, phi, curv):
        s = self.f.spacing(phi, curv)
        return s * self.p["cell_ratio"] / self.p["cutoff"], s ** -self.dim

    def _map(self, first=False):
        f, x = self.f, self.x
        phi, n, curv, cut = f.sample(x)
        if first:
            self.h, _ = self._info(phi, curv)
        size = n.norm(dim=1)
        out = torch.where(phi < 0, 1.0, -1.0)[:, None] * n / (size + 1e-15)[:, None]
        self.surf = cut
        x = torch.where(cut[:, None], x + out * phi.abs()[:, None] + 0.0, x)
        x = torch.where(cut[:, None], x + out * (1e-5 * self.h)[:, None], x)
        phi, n, curv, _ = f.sample(x)
        self.h_new, self.rho = self._info(phi, curv)
        start = again = torch.nonzero((phi < 0) & ~cut)[:, 0]
        for t in range(2000):  # a REAL particle that left the body starts again at random
            if not len(again):
                break
            ids = again.cpu().numpy()
            y = x.new_zeros(len(again), 3)
            for d in range(self.dim):
                r = _philox((ids, np.int64(self.k), np.int64(t), np.int64((2 << 8) | d)), int(self.p["seed"]))
                u = [((r[q] >> np.uint64(5)).astype(np.float64) * 67108864.0 + (r[q + 1] >> np.uint64(6)).astype(np.float64))
                     / 9007199254740992.0 for q in (0, 2)]
                bl, br = self.p["box_l"][d], self.p["box_r"][d]
                y[:, d] = torch.from_numpy(np.clip(u[0] * (br - bl) + u[1] * 1e-3 + bl, bl + 1e-10, br - 1e-10))
            sp, sn, sc, _ = f.sample(y)
            ok = sp > self.h[again]
            at = again[ok]
            x[at], n[at], phi[at], curv[at] = y[ok], sn[ok], sp[ok], sc[ok]
            self.h_new[at], self.rho[at] = self._info(sp[ok], sc[ok])
            again = again[~ok]
        self.x, self.n = x, n
        if first:  # Pre_run keeps the spacing of the unmapped position
            self.h[start] = self.h_new[start]
        else:
            self.h = self.h_new

    def _pairs(self):
        """(i, j) lists of the neighbour relation, in chunks of i."""
        dim, x, reach = self.dim, self.x, self.h * self.p["cutoff"] + 1e-10
        big = float(reach.max())
        lo = x.min(0).values - big
        c = torch.floor((x - lo) / big).long()
        size = [int(v) + 2 for v in c.max(0).values]
        if dim == 2:
            c[:, 2], size[2] = 0, 1
        key = (c[:, 2] * size[1] + c[:, 1]) * size[0] + c[:, 0]
        order = torch.argsort(key)
        count = torch.bincount(key, minlength=size[0] * size[1] * size[2])
        start = torch.cumsum(count, 0) - count
        offs = [(a, b, e) for a in (-1, 0, 1) for b in (-1, 0, 1) for e in ((-1, 0, 1) if dim == 3 else (0,))]
        cells = []
        for o in offs:
            q = [c[:, d] + o[d] for d in range(3)]
            ok = (q[0] >= 0) & (q[1] >= 0) & (q[2] >= 0) & (q[0] < size[0]) & (q[1] < size[1]) & (q[2] < size[2])
            cells.append(torch.where(ok, (q[2].clamp(min=0) * size[1] + q[1].clamp(min=0)) * size[0] + q[0].clamp(min=0), -1)
                         .clamp(max=len(count) - 1))
        total = sum(torch.where(q >= 0, count[q.clamp(min=0)], 0) for q in cells)
        if int(total.sum()) > self.PAIRS:
            raise OverflowError
        edge = torch.cumsum(total, 0)
        a = 0
        while a < len(x):
            b = int(torch.searchsorted(edge, (edge[a - 1] if a else 0) + 60_000_000)) + 1
            b = min(max(b, a + 1), len(x))
            keep = []
            for q in cells:
                q = q[a:b]
                m = torch.where(q >= 0, count[q.clamp(min=0)], 0)
                i = torch.repeat_interleave(torch.arange(a, b, device=x.device), m)
                k = torch.arange(len(i), device=x.device) - torch.repeat_interleave(torch.cumsum(m, 0) - m, m)
                j = order[start[q.clamp(min=0)].repeat_interleave(m) + k]
                ok = (x[i] - x[j]).norm(dim=1) <= torch.maximum(reach[i], reach[j])
                keep.append((i[ok], j[ok]))
            yield torch.cat([k[0] for k in keep]), torch.cat([k[1] for k in keep])
            a = b

    def _kernel(self, dim, r, h, slope):
        """W(r, h) or dW/dr / r of the smoothing kernel in dim dimensions."""
        s, kind, pi = r / h, self.p["kernel"], 3.1415926
        if kind == cases.KERNELS["wendland"]:
            if dim == 1:
                return torch.zeros_like(s)
            c = (1.75 / pi / h ** 2) if dim == 2 else (21.0 / 16.0 / pi / h ** 3)
            t = (1.0 - 0.5 * s).clamp(min=0.0)
            return -5.0 * c * t ** 3 * s / h / (r + 1e-15) if slope else c * t ** 4 * (1.0 + 2.0 * s)
        if kind == cases.KERNELS["hyperbolic"]:
            c = (1 / 7.0 / h, 1 / (3.0 * pi) / h ** 2, 15.0 / (62.0 * pi) / h ** 3)[dim - 1]
            t = (2.0 - s).clamp(min=0.0)
            if slope:
                return c / h * torch.where(s < 1, -6.0 + 3.0 * s * s, -3.0 * t * t) / (r + 1e-20)
            return c * torch.where(s < 1, 6.0 - 6.0 * s + s ** 3, t ** 3)
        c = (0.666666667 / h, 0.454728408 / h ** 2, 0.318309886 / h ** 3)[dim - 1]
        t = (2.0 - s).clamp(min=0.0)
        if slope:
            return c / h * torch.where(s < 1, 3.0 * (-s + 0.75 * s * s), -0.75 * t * t) / (r + 1e-20)
        return c * torch.where(s < 1, 1 - 1.5 * s * s + 0.75 * s ** 3, 0.25 * t ** 3)

    def step(self):
        p, dim = self.p, self.dim
        self.x = self.x + (self.v + self.a * (0.5 * self.dt)) * self.dt
        self.k += 1
        self._map()
        n, h, surf, nrm = len(self.x), self.h, self.surf, self.n
        pairs = list(self._pairs())
        cos = math.cos(p["angle_thres"])
        total, count = h.new_zeros(n), h.new_zeros(n)
        vol = self.rho ** -2
        terms = []
        for i, j in pairs:
            d = self.x[i] - self.x[j]
            si = surf[i]
            d = torch.where(si[:, None], d - nrm[i] * (d * nrm[i]).sum(1, keepdim=True), d)
            use = ~si | (surf[j] & ((nrm[i] * nrm[j]).sum(1).abs() > cos))
            i, j, d, si = i[use], j[use], d[use], si[use]
            r = d.norm(dim=1)
            w = torch.where(si, self._kernel(dim - 1, r, h[i], False), self._kernel(dim, r, h[i], False))
            total.index_add_(0, i, w)
            count.index_add_(0, i, torch.ones_like(w))
            far = i != j
            i, j, d, si, r = i[far], j[far], d[far], si[far], r[far]
            hij = 0.5 * (h[i] + h[j])
            aw = torch.where(si, self._kernel(dim - 1, r, hij, True), self._kernel(dim, r, hij, True))
            terms.append((i, j, d, aw * (vol[i] + vol[j])))
        total = torch.where(count > 1, 1.0 / (total + 1e-15), total)

        def flat(a):  # the force on a SURFACE particle stays in its tangent plane
            return torch.where(surf[:, None], a - nrm * (a * nrm).sum(1, keepdim=True), a)

        a1 = h.new_zeros(n, 3)
        for i, j, d, c in terms:
            a1.index_add_(0, i, d * (-total[i] * c)[:, None])
        a1 = flat(a1)
        dt1 = float((0.25 * torch.sqrt(h / (a1.norm(dim=1) + 1e-15))).min())
        v = a1 * (0.5 * dt1)
        eta = self.nu * self.rho
        a2 = h.new_zeros(n, 3)
        for i, j, d, c in terms:
            vj = torch.where((~surf[i] & surf[j])[:, None], -v[i], v[j])
            visc = 2.0 * eta[i] * eta[j] / (eta[i] + eta[j] + 1e-15)
            a2.index_add_(0, i, (v[i] - vj) * (c * visc)[:, None])
        a2 = flat(a2 + v * p["damp_coeff"])
        u = v.norm(dim=1)
        self.nu = p["nu_coeff"] * h * u
        dt = torch.minimum(0.25 * torch.sqrt(h / (a2.norm(dim=1) + 1e-15)), h / 40.0 / (u + 1e-15))
        self.dt = float(torch.minimum(dt, 0.125 * h * h / (self.nu + 1e-15)).min())
        self.v, self.a = v, a2


def exact(case, seed):
    what = case["what"]
    if what == "setup":
        state = prepare(case, seed)
        f = _Fields(state["geometry"])
        top = f.lv[-1]
        phi, nrm, curv, _ = f.sample(torch.from_numpy(state["xyz"]).cuda())
        return {"fields": {"nx": top["n"][0], "ny": top["n"][1], "nz": top["n"][2], "curv": top["curv"],
                           "tag": None, "max_phi": f.max_phi},
                "at": {"phi": phi, "normal": nrm, "curvature": curv, "tag": None}}
    if what not in ("relax", "batch"):
        return None  # adaptive bisection, iterated Voronoi cells, meshes: no short plain form
    if what == "batch":
        todo = [(_geometry(kind, n, "wendland", "fp32", 0, number), own)
                for kind, n, number, own in _star_numbers(case, seed)]
        todo = [(g, _positions(g, g.n_particles, "settled", own)) for g, own in todo]
    else:
        g = _of(case)
        todo = [(g, _positions(g, int(case["n"]), case["start"], seed))]
    done = []
    for g, x in todo:
        if len(x) * case["steps"] > 1_500_000:
            return None
        try:
            r = _Relaxation(g, x)
            for _ in range(case["steps"]):
                r.step()
        except OverflowError:
            return None
        done.append(r)
    if case.get("precision") == "fp64":
        r = done[0]
        return {"xyz": r.x, "v": r.v + r.a * (0.5 * r.dt), "h": r.h, "type": None}
    return torch.cat([r.x for r in done])
