"""The workloads this library is timed on: BIEF's SOLVE and MATVEC as a
TELEMAC-2D time step, a stand-alone solve, a batch of meshes and a gradient
call them, from a 1,000-node test mesh to the 4M-node configuration.

A case is a dict of plain values.  Its mesh is an nx x ny grid of jittered
nodes, each quad cut into two triangles:
  split      'uniform': every quad along the same diagonal (the benchmark's
             meshes, node degree 6); 'mixed': a random diagonal per quad
             (degrees 4 to 8, as unstructured meshes have)
  numbering  'rows': row by row; 'local': at random within runs of four rows
             (an unstructured mesh numbered for bandwidth); 'random': nodes
             and elements in random order (numbered with no care at all)
  depth      'smooth' (5 + 4 sin cos, random phase) or 'loguniform' (0.5 to
             500 m per quad, three passes of neighbour averaging)
The right-hand side is A x_true with x_true drawn at random, so the exact
solution of every system is known.
"""
import math

import numpy as np
import torch

from opentelemac_b200 import autograd, bief, meshgen
from opentelemac_b200.batch import BatchSolver

DEV = "cuda:0"
F64 = torch.float64


# --------------------------------------------------------------------------
# meshes and operators, in plain numpy and torch
# --------------------------------------------------------------------------
class Grid:
    """Mesh, element coefficients and exact operator of one case, from the
    case's sizes and the seed alone."""

    def __init__(self, nx, ny, seed, split="uniform", numbering="rows", depth="smooth"):
        rng = np.random.default_rng([seed, nx, ny])
        self.nx, self.ny, self.n = nx, ny, nx * ny
        hx = 1.0 / (max(nx, ny) - 1)
        i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="xy")
        inner = ((i > 0) & (i < nx - 1) & (j > 0) & (j < ny - 1))
        x = (i + inner * rng.uniform(-0.2, 0.2, i.shape)) * hx
        y = (j + inner * rng.uniform(-0.2, 0.2, i.shape)) * hx
        qi, qj = np.meshgrid(np.arange(nx - 1, dtype=np.int32),
                             np.arange(ny - 1, dtype=np.int32), indexing="xy")
        a = (qj * nx + qi).ravel()
        corner = [a, a + 1, a + nx + 1, a + nx]
        cut = rng.random(a.size) < 0.5 if split == "mixed" else np.zeros(a.size, bool)
        ik = np.empty((2 * a.size, 3), dtype=np.int32)
        for k, (c0, c1) in enumerate(((0, 0), (1, 1), (2, 3))):
            ik[0::2, k] = np.where(cut, corner[c1], corner[c0])
        for k, (c0, c1) in enumerate(((0, 1), (2, 2), (3, 3))):
            ik[1::2, k] = np.where(cut, corner[c1], corner[c0])
        self.cut = cut
        quad = np.repeat(np.arange(a.size, dtype=np.int32), 2)
        self.new_id = None
        if numbering != "rows":
            if numbering == "random":
                new_id = rng.permutation(self.n)
                order = rng.permutation(ik.shape[0])
            else:
                run = np.arange(self.n) // (4 * nx)
                perm = np.lexsort((rng.random(self.n), run))
                new_id = np.empty(self.n, np.int64)
                new_id[perm] = np.arange(self.n)
                order = np.argsort(new_id[ik].min(axis=1), kind="stable")
            self.new_id = new_id
            ik = new_id[ik[order]].astype(np.int32)
            quad = quad[order]
            xn, yn = np.empty(self.n), np.empty(self.n)
            xn[new_id], yn[new_id] = x.ravel(), y.ravel()
            x, y = xn, yn
        self.ik = np.ascontiguousarray(ik)
        self.nelem = ik.shape[0]
        self.rng = rng
        self.x = torch.tensor(np.ascontiguousarray(x).ravel(), device=DEV)
        self.y = torch.tensor(np.ascontiguousarray(y).ravel(), device=DEV)
        self.ikd = torch.tensor(self.ik, device=DEV).long()
        xe, ye = self.x[self.ikd], self.y[self.ikd]
        self.x2, self.x3 = xe[:, 1] - xe[:, 0], xe[:, 2] - xe[:, 0]
        self.y2, self.y3 = ye[:, 1] - ye[:, 0], ye[:, 2] - ye[:, 0]
        self.area = 0.5 * (self.x2 * self.y3 - self.x3 * self.y2)
        if depth == "loguniform":
            h = np.exp(rng.uniform(math.log(0.5), math.log(500.0), (ny - 1, nx - 1)))
            for _ in range(3):
                p = np.pad(h, 1, mode="edge")
                h = (p[1:-1, 1:-1] + p[:-2, 1:-1] + p[2:, 1:-1] + p[1:-1, :-2] + p[1:-1, 2:]) / 5.0
            self.h = torch.tensor(h.ravel()[quad], device=DEV)
        else:
            s, t = rng.uniform(0, 2 * math.pi, 2)
            self.h = 5.0 + 4.0 * torch.sin(2 * math.pi * xe.mean(1) + s) * torch.cos(
                2 * math.pi * ye.mean(1) + t)

    def wave(self, coef):
        """Element matrices of M + coef_e K_e: off-diagonal terms (12, 13,
        23) and the three diagonal ones."""
        c = 0.25 * coef / self.area
        bpe = c * (self.y3 * self.y3 + self.x3 * self.x3)
        cpf = c * (self.y2 * self.y3 + self.x2 * self.x3)
        apd = c * (self.y2 * self.y2 + self.x2 * self.x2)
        m = self.area / 12.0
        return ((m + cpf - bpe, m + cpf - apd, m - cpf),
                (2 * m + apd + bpe - 2 * cpf, 2 * m + bpe, 2 * m + apd))

    def nodes(self, *w):
        """Per-node sums of the values w[k] of the elements' k-th points."""
        out = np.zeros(self.n)
        for k, v in enumerate(w):
            out += np.bincount(self.ik[:, k], v.cpu().numpy(), self.n)
        return torch.tensor(out, device=DEV)

    def product(self, off, dia, v, transposed=False):
        """A v for element matrices off = (12, 13, 23[, 21, 31, 32]), dia."""
        o = list(off) + (list(off) if len(off) == 3 else [])
        if transposed:
            o = o[3:] + o[:3]
        v1, v2, v3 = (v[self.ikd[:, k]].double() for k in range(3))
        return self.nodes(dia[0] * v1 + o[0] * v2 + o[1] * v3,
                          o[3] * v1 + dia[1] * v2 + o[2] * v3,
                          o[4] * v1 + o[5] * v2 + dia[2] * v3)

    def vector(self, salt=0):
        return torch.tensor(np.random.default_rng([int(self.rng.bit_generator.state["state"][
            "state"] % (1 << 31)), salt]).uniform(-1, 1, self.n), device=DEV)

    def segments(self):
        """GLOSEG columns: boundary edges first, then the others."""
        nx, ny = self.nx, self.ny
        k = np.arange(self.n).reshape(ny, nx)
        a, b = k[:-1, :-1].ravel(), k[:-1, 1:].ravel()
        c, d = k[1:, 1:].ravel(), k[1:, :-1].ravel()
        rim = [(k[0, :-1], k[0, 1:]), (k[:-1, -1], k[1:, -1]), (k[-1, 1:], k[-1, :-1]),
               (k[1:, 0], k[:-1, 0])]
        rest = [(k[1:-1, :-1], k[1:-1, 1:]), (k[:-1, 1:-1], k[1:, 1:-1]),
                (np.where(self.cut, b, a), np.where(self.cut, d, c))]
        g1 = np.concatenate([p.ravel() for p, _ in rim + rest])
        g2 = np.concatenate([q.ravel() for _, q in rim + rest])
        nb = sum(p.size for p, _ in rim)
        if self.new_id is not None:
            g1, g2 = self.new_id[g1], self.new_id[g2]
        lo, hi = np.minimum(g1[nb:], g2[nb:]), np.maximum(g1[nb:], g2[nb:])
        order = np.lexsort((hi, lo))
        return np.concatenate([g1[:nb], lo[order]]), np.concatenate([g2[:nb], hi[order]])


def grid_of(c, seed):
    return Grid(c["nx"], c["ny"], seed, c.get("split", "uniform"), c.get("numbering", "rows"),
                c.get("depth", "smooth"))


def skewed(g, off):
    """Off-diagonal terms of a nonsymmetric matrix: the symmetric ones with
    the transport of a tracer added (unequal terms (k,l) and (l,k))."""
    s = 0.15 * torch.sin(2 * math.pi * g.h)
    return [o * (1 + s) for o in off] + [o * (1 - s) for o in off]


def system(c, seed):
    """The case's grid, element matrices and exact solution."""
    g = grid_of(c, seed)
    off, dia = g.wave(c.get("dt", 1.0) ** 2 * 9.81 * g.h)
    return g, off, dia, g.vector()


def step_operator(c, seed):
    """A time step's operator as PROPAG builds it: MATMAS / DT plus MATDIFUV
    with U = DM1 per node (negative) and V = the depth per node, XMUL = -1."""
    g = grid_of(c, seed)
    dt = c["dt"]
    depth = 5.0 + 3.0 * torch.sin(7 * g.x + seed % 7) * torch.cos(5 * g.y)
    dm1 = -0.36 * 9.81 * dt * torch.ones_like(depth)
    u, v = dm1[g.ikd], depth[g.ikd]
    k = (u * (v + v.sum(1, keepdim=True))).sum(1) * (-1.0 / 48.0) / g.area
    a12 = (g.y3 * (g.y2 - g.y3) + g.x3 * (g.x2 - g.x3)) * k
    a13 = -(g.y2 * (g.y2 - g.y3) + g.x2 * (g.x2 - g.x3)) * k
    a23 = -(g.y2 * g.y3 + g.x2 * g.x3) * k
    m = g.area / 12.0 / dt
    off = (m + a12, m + a13, m + a23)
    dia = (2 * m - a12 - a13, 2 * m - a12 - a23, 2 * m - a13 - a23)
    truth = 0.2 * torch.sin(9 * g.x) * torch.cos(4 * g.y) + 0.01 * g.vector()
    return g, off, dia, truth, dm1, depth


def batch_sizes(c):
    rng = np.random.default_rng(c["ninst"])
    n = np.exp(rng.uniform(math.log(c["lo"]), math.log(c["hi"]), c["ninst"]))
    return [(max(3, int(math.sqrt(v))), max(3, int(v / int(math.sqrt(v))))) for v in n]


def batch_grids(c, seed):
    return [Grid(nx, ny, seed + 1000 * k) for k, (nx, ny) in enumerate(batch_sizes(c))]


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one product on a 10,201-node mesh, where the
        # launch is all there is (the reference's own loops call MATVEC so)
        dict(name="matvec_101", kind="matvec", nx=101, ny=101, op="X=AY", typext="S"),
        # the product at the benchmark's 1M nodes
        dict(name="matvec_1001", kind="matvec", nx=1001, ny=1001, op="X=AY", typext="S"),
        # a small stand-alone solve: the size of the smoke test's mesh
        dict(name="solve_41", kind="solve", nx=41, ny=41, eps=1e-8),
        # one wave-equation time step of an ordinary study: assembly of AM1
        # and a solve at a model's accuracy, few iterations, ragged sizes
        dict(name="step_401x379", kind="step", nx=401, ny=379, dt=0.002, eps=1e-6,
             split="mixed", numbering="local"),
        # the benchmark's binary64 solve
        dict(name="solve_1001", kind="solve", nx=1001, ny=1001, eps=1e-8),
        # segment storage, the default of TELEMAC-2D's dictionary, on an
        # irregular mesh
        dict(name="solve_seg_601x417", kind="solve", nx=601, ny=417, eps=1e-8, storage="seg",
             split="mixed", numbering="local"),
        # a nonsymmetric system (tracer transport) with CGSTAB
        dict(name="cgstab_333x301", kind="solve", nx=333, ny=301, eps=1e-8, slv=6, typext="Q",
             dt=0.05, split="mixed"),
        # a mesh numbered at random, mixed precision
        dict(name="mixed_random_307x293", kind="mixed", nx=307, ny=293, inner_tol=0.1,
             outer_tol=1e-8, split="mixed", numbering="random"),
        # the headline: mixed precision at 1M nodes
        dict(name="mixed_1001", kind="mixed", nx=1001, ny=1001, inner_tol=0.1, outer_tol=1e-8),
        # the largest configuration: 4.0M nodes, log-uniform depth
        dict(name="mixed_2001", kind="mixed", nx=2001, ny=2001, inner_tol=1e-4,
             outer_tol=1e-10, depth="loguniform"),
        # many meshes in one launch
        dict(name="batch_48", kind="batch", ninst=48, lo=2000, hi=60000, npt=4, threads=1024),
        # forward and adjoint solve with the gradient of the depth field
        dict(name="grad_251", kind="grad", nx=251, ny=251, eps=1e-12),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "matvec32", "solve", "solve", "solve", "step",
                       "mixed", "mixed", "batch", "grad"])
    top = dict(matvec=1200, matvec32=1200, solve=700, step=900, mixed=900, batch=0, grad=260)[kind]
    if kind == "batch":
        lo = _log(rng, 300, 4000)
        return dict(kind=kind, ninst=_log(rng, 3, 64), lo=lo, hi=lo * rng.randint(2, 12),
                    npt=rng.choice([1, 2, 4, 8]), threads=rng.choice([256, 512, 1024]))
    side = _log(rng, 23, top)
    c = dict(kind=kind, nx=max(17, int(side * rng.uniform(0.6, 1.4))), ny=max(17, side))
    c["split"] = rng.choice(["uniform", "mixed"])
    c["numbering"] = rng.choice(["rows", "rows", "local", "local", "random"])
    if kind == "matvec":
        c.update(op=rng.choice(["X=AY", "X=-AY", "X=CAY", "X=TAY"]),
                 typext=rng.choice(["S", "S", "Q"]), storage=rng.choice(["ebe", "ebe", "seg"]))
    elif kind == "matvec32":
        c.update(storage=rng.choice(["ebe", "seg"]))
    elif kind == "solve":
        slv = rng.choice([1, 1, 1, 1, 2, 6, 7])
        c.update(slv=slv, storage=rng.choice(["ebe", "ebe", "seg"]), precon=rng.choice([2, 2, 2, 0]),
                 modass=rng.choice([1, 1, 3]), eps=rng.choice([1e-6, 1e-8]))
        c["dt"] = 1.0 if slv == 1 else 0.05
        if slv == 6 and rng.random() < 0.5:
            c["typext"] = "Q"
        if slv == 7:
            c["krylov"] = rng.choice([3, 6, 10])
        if c["precon"] == 0:
            c["eps"], c["dt"] = 1e-10, 0.02   # unscaled: ||B|| is small, tested absolutely
    elif kind == "step":
        c.update(dt=rng.choice([0.0005, 0.002, 0.01]), eps=rng.choice([1e-4, 1e-6]))
    elif kind == "mixed":
        c.update(inner_tol=rng.choice([0.1, 0.1, 1e-4]), outer_tol=rng.choice([1e-8, 1e-10]),
                 depth=rng.choice(["smooth", "loguniform"]),
                 storage=rng.choice(["ebe", "ebe", "seg"]))
    else:
        c.update(eps=rng.choice([1e-10, 1e-12]))
    return c


def _stored(c, g, off, dia):
    """The case's matrix on a mesh handle, as a program stores it."""
    mesh = bief.Mesh(g.ik, g.n)
    A = bief.Matrix(mesh)
    if c.get("typext", "S") == "Q":
        A.set(g.nodes(*dia), torch.stack(skewed(g, off)).contiguous(), "Q", "Q")
    else:
        A.assemble_wave(g.x, g.y, (c.get("dt", 1.0) ** 2 * 9.81 * g.h).contiguous())
    if c.get("storage", "ebe") == "seg":
        mesh.set_segments(*g.segments())
        A.to_segments()
    return A


def prepare(c, seed):
    kind = c["kind"]
    s = dict(kind=kind, case=c)
    if kind == "batch":
        gs = batch_grids(c, seed)
        coefs = [9.81 * g.h for g in gs]
        B = BatchSolver([(g.n, g.ik) for g in gs])
        B.assemble_wave([g.x for g in gs], [g.y for g in gs], coefs)
        s.update(B=B, b=B.gather([g.product(*g.wave(k), g.vector()) for g, k in zip(gs, coefs)]))
        s["x"] = torch.zeros_like(s["b"])
        return s
    if kind == "grad":
        g, off, dia, truth = system(c, seed)
        s["prob"] = autograd.WaveProblem(g.x.cpu().numpy(), g.y.cpu().numpy(), g.ik,
                                         device=DEV, eps=c["eps"])
        s["coef"] = (9.81 * g.h).requires_grad_(True)
        s["b"] = g.product(off, dia, truth).requires_grad_(True)
        s["gx"] = g.product(off, dia, g.vector(1))
        return s
    if kind == "step":
        g, off, dia, truth, dm1, depth = step_operator(c, seed)
        s.update(A=bief.Matrix(bief.Mesh(g.ik, g.n)), xc=g.x, yc=g.y, u=dm1, v=depth)
        s["b"] = g.product(off, dia, truth)
        s["x0"] = 0.98 * truth   # the previous step's field
        s["x"] = torch.empty_like(truth)
        return s
    g, off, dia, truth = system(c, seed)
    s["A"] = _stored(c, g, off, dia)
    if kind == "matvec":
        s.update(x=torch.zeros_like(truth), y=truth)
    elif kind == "matvec32":
        s.update(x=torch.zeros(g.n, dtype=torch.float32, device=DEV), y=truth.float())
    else:
        s["x"] = torch.zeros_like(truth)
        q = skewed(g, off) if c.get("typext", "S") == "Q" else off
        s["b"] = g.product(q, dia, truth)
    return s


def run(s):
    c, kind = s["case"], s["kind"]
    if kind == "matvec":
        return bief.matvec(c["op"], s["x"], s["A"], s["y"], 0.75)
    if kind == "matvec32":
        return bief.matvec32(s["x"], s["A"], s["y"])
    if kind == "batch":
        s["x"].zero_()
        r = s["B"].solve_mixed(s["x"], s["b"], inner_tol=1e-4, outer_tol=1e-8,
                               nodes_per_thread=c["npt"], threads_per_block=c["threads"])
        return [s["x"], r["status"], r["inner"], r["outer"]]
    if kind == "grad":
        s["coef"].grad = s["b"].grad = None
        x = autograd.wave_solve(s["coef"], s["b"], s["prob"])
        x.backward(s["gx"])
        return [x.detach(), s["coef"].grad, s["b"].grad]
    if kind == "mixed":
        s["x"].zero_()
        st, outer, inner, relres = bief.solve_mixed(s["x"], s["A"], s["b"], 2, c["inner_tol"],
                                                    c["outer_tol"])
        return [s["x"], st, outer, inner]
    if kind == "step":
        s["A"].assemble_mass_diff(s["xc"], s["yc"], s["u"], s["v"], kind=12,
                                  xmul_mass=1.0 / c["dt"], xmul_dif=-1.0)
        s["x"].copy_(s["x0"])
    else:
        s["x"].zero_()
    cfg = bief.SlvCfg(slv=c.get("slv", 1), nitmax=20000, precon=c.get("precon", 2),
                      krylov=c.get("krylov", 0), eps=c["eps"], zero=0.0)
    st, nit, relres = bief.solve(s["x"], s["A"], s["b"], cfg, modass=c.get("modass", 1))
    return [s["x"], st, nit]


def exact(c, seed):
    kind = c["kind"]
    if kind == "batch":
        out = []
        for g in batch_grids(c, seed):
            v = torch.zeros((g.n + 31) // 32 * 32, dtype=F64, device=DEV)
            v[:g.n] = g.vector()
            out.append(v)
        out = torch.cat(out)
        return [out, None, None, None]
    if kind == "step":
        return [step_operator(c, seed)[3], None, None]
    g, off, dia, truth = system(c, seed)
    if kind == "grad":
        lam = g.vector(1)
        one = g.wave(torch.ones_like(g.h))[0]
        mass = g.area / 12.0
        k12, k13, k23 = (o - mass for o in one)
        l, u = lam[g.ikd], truth[g.ikd]
        grad = (k12 * (l[:, 0] - l[:, 1]) * (u[:, 0] - u[:, 1])
                + k13 * (l[:, 0] - l[:, 2]) * (u[:, 0] - u[:, 2])
                + k23 * (l[:, 1] - l[:, 2]) * (u[:, 1] - u[:, 2]))
        return [truth, grad, lam]
    if kind in ("matvec", "matvec32"):
        q = skewed(g, off) if c.get("typext", "S") == "Q" else off
        r = g.product(q, dia, truth.float() if kind == "matvec32" else truth,
                      transposed=c.get("op") == "X=TAY")
        return {"X=-AY": -1.0, "X=CAY": 0.75}.get(c.get("op"), 1.0) * r
    return [truth] + [None] * (3 if kind == "mixed" else 2)


# Bytes a pass cannot do without: per product the off-diagonal terms and the
# three node numbers of every element (segment storage: one term and two node
# numbers per edge), the diagonal and the two vectors; per CG iteration that
# and the vector updates.  Iterations: fits to counts of these operators (255
# on the 41 x 41 mesh, 2216 on 1001 x 1001 at 1e-8; about 11 per node spacing
# that a wave crosses in a time step).
def _iterations(c):
    side = max(c["nx"], c["ny"])
    digits = math.log10(1 / c.get("outer_tol", c.get("eps", 1e-8)))
    full = 33.0 * side ** 0.6 * (digits / 8.0) ** 2
    if c["kind"] == "step":
        return max(3.0, min(11.0 * 7.0 * c["dt"] * side * digits / 6.0, full))
    if c.get("dt", 1.0) < 1.0:
        return full * (0.5 if c.get("slv", 1) == 7 else 0.21)
    return full * (1.35 if c.get("depth") == "loguniform" else 1.0)


def work(c):
    kind = c["kind"]
    if kind == "batch":
        by = sum(33.0 * max(nx, ny) ** 0.6 * (24 * 2 * nx * ny + 48 * nx * ny)
                 for nx, ny in batch_sizes(c))
        return {"bytes": by, "flops": by * 0.3}
    n = c["nx"] * c["ny"]
    ne, ns = 2 * (c["nx"] - 1) * (c["ny"] - 1), 3 * n
    cols = 6 if c.get("typext", "S") == "Q" else 3
    seg = c.get("storage", "ebe") == "seg"
    if kind == "matvec32":
        by = (12 * ns if seg else 24 * ne) + 12 * n
    else:
        by = ns * (8 * cols // 3 + 8) + 24 * n if seg else ne * (8 * cols + 12) + 24 * n
    if kind in ("matvec", "matvec32"):
        return {"bytes": by, "flops": 12.0 * ne + 2 * n}
    it = _iterations(c)
    if kind == "mixed":
        per = (12 * ns if seg else 24 * ne) + 48 * n
    else:
        per = by + 64 * n
        if c.get("slv", 1) == 6:
            per = 2 * by + 120 * n
        elif c.get("slv", 1) == 7:
            per = c["krylov"] * (by + 8 * n * (c["krylov"] + 2))
    if kind == "grad":
        it *= 2
    return {"bytes": it * per, "flops": it * (12.0 * ne + 12 * n)}
