"""Performance cases of the transport operator, through its public entry points.

A case is one call that a driver of the operator makes again and again: an Apply
of a Krylov iteration (`apply`), the same through host vectors in the reference's
cell numbering (`apply_host`), the right-hand side of a time step (`rhs`), the
diffusion preconditioner (`dsa`), the Apply of many uneven problems (`batch`), a
whole solve (`solve`).  `listed()` names the sizes that are followed over time,
`draw()` gives others of the same ranges, `exact()` the same results from plain
torch in 64 bits.

FP32 sweeps are the inner operator of mixed-precision solves and the diffusion
correction is computed in FP32: those results are handed on in single precision,
which is what they hold.  FP64 results stay FP64.
"""
import math
import os
import random

import numpy as np
import torch

import ouranos_gb300 as og
from ouranos_gb300 import learned

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _case(name, kind, cells, order, quad, sn, l_max=0, precision="fp64", **more):
    c = {"name": name, "kind": kind, "nx": cells[0], "ny": cells[1], "nz": cells[2] if len(cells) > 2 else 0,
         "order": order, "quad": quad, "sn": sn, "l_max": l_max, "precision": precision}
    c.update(more)
    return c


def listed():
    return [
        # the smallest Apply in use: the CPU-runnable homogeneous problem of the
        # test-suite, where launches and the wavefront's latency are all there is
        _case("apply-2d-q1-32-s8", "apply", (32, 32), 1, "LS", 8),
        # the benchmark workload: heterogeneous 2-D, P3 scattering
        _case("apply-2d-q2-256-s16-p3", "apply", (256, 256), 2, "LS", 16, 3),
        # an ordinary mesh whose sides are no multiple of any tile, third order
        _case("apply-2d-q3-135x93-s12-p1", "apply", (135, 93), 3, "LS", 12, 1),
        # the thick diffusive 3-D problem in FP64 (true residuals, plain GMRES)
        _case("apply-3d-q1-64-glc12", "apply", (64, 64, 64), 1, "GLC", 12),
        # the angular sweep of the time-dependent problem: the largest mesh
        _case("apply-3d-q1-128-s8-fp32", "apply", (128, 128, 128), 1, "LS", 8, 0, "fp32"),
        # ragged 3-D boxes: second order with linearly anisotropic scattering ...
        _case("apply-3d-q2-37x29x41-s6-p1", "apply", (37, 29, 41), 2, "LS", 6, 1),
        # ... and third order, whose cells no lane's registers hold
        _case("apply-3d-q3-20x17x23-s4", "apply", (20, 17, 23), 3, "LS", 4),
        # a reference driver's own call: pageable host vectors in z-order numbering
        _case("host-2d-q1-128-s8-p1", "apply_host", (128, 128), 1, "LS", 8, 1),
        # right-hand side of an implicit Euler step: fixed source, the other
        # group's scattering, inflow, and psi of the last step
        _case("rhs-3d-q1-40x36x33-s8-step", "rhs", (40, 36, 33), 1, "LS", 8, 0, groups=2, inv_vdt=0.5),
        # the diffusion preconditioner at the step count of the thick problem
        _case("dsa-3d-q1-64-20", "dsa", (64, 64, 64), 1, "GLC", 4, 0, cg=20),
        # uneven 2-D problems in one launch, FP32 sweeps
        _case("batch-16-fp32", "batch", (256, 256), 2, "LS", 16, 1, "fp32", count=16, shapes=3),
        # the thick problem solved to 1e-8: FP32 sweeps, diffusion correction
        # started from the trained network
        _case("solve-3d-q1-64-glc12-learned", "solve", (64, 64, 64), 1, "GLC", 12, 0, "fp32",
              method="fgmres_learned", cg=3),
    ]


# the largest drawn call stays below the largest listed one
_LARGEST = (128 ** 3) * 80 * 8


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        kind = rng.choice(["apply", "apply", "apply", "apply", "apply_host", "rhs", "dsa", "batch", "solve"])
        precision = rng.choice(["fp64", "fp64", "fp32"])
        more = {}
        if kind == "batch":
            c = _case("", kind, (256, 256), 2, "LS", 16, 1, rng.choice(["fp64", "fp32", "fp32"]),
                      count=rng.randint(3, 20), shapes=rng.randint(10, 10 ** 6))
        else:
            dim = rng.choice([2, 2, 3])
            cells = tuple(_log_int(rng, 24, 320) if dim == 2 else _log_int(rng, 12, 96) for _ in range(dim))
            order = rng.choice([1, 1, 2, 2, 3, 4]) if dim == 2 else rng.choice([1, 1, 1, 2, 3])
            quad = rng.choice(["LS", "GLC"])
            sn = rng.choice([4, 6, 8, 12, 16] if dim == 2 else [4, 6, 8, 12])
            l_max = rng.choice([0, 1, 1, 2, 3] if dim == 2 else [0, 0, 1, 3])
            if kind == "apply_host":
                side = 1 << rng.randint(5, 8)
                cells, dim, order = (side, side), 2, min(order, 3)
            if kind == "rhs":
                precision = "fp64"
                more = {"groups": rng.choice([1, 2, 3]), "inv_vdt": rng.choice([0.0, 0.5, 2.0])}
            if kind == "dsa":
                precision, order, sn, l_max = "fp64", min(order, 2), 4, min(l_max, 1)
                more = {"cg": rng.randint(3, 30)}
            if kind == "solve":
                precision, order, l_max = "fp32", min(order, 2), min(l_max, 1)
                more = {"method": "fgmres_mixed", "cg": rng.choice([5, 10, 20])}
            if dim == 3 and order > 2 and kind == "rhs":
                continue
            c = _case("", kind, cells, order, quad, sn, l_max, precision, **more)
            nd = _dirs(c)
            if _cells(c) * nd * _n(c) > _LARGEST // 2 or (_n(c) > 27 and _cells(c) * nd > 3_000_000):
                continue
            if _cells(c) * nd * _n(c) > {"rhs": 40_000_000, "solve": 5_000_000}.get(kind, _LARGEST):
                continue
        del c["name"]
        return c


# ------------------------------------------------------------------ the problem
def _dim(c):
    return 3 if c["nz"] else 2


def _n(c):
    return (c["order"] + 1) ** _dim(c)


def _cells(c):
    return c["nx"] * c["ny"] * max(1, c["nz"])


def _dirs(c):
    return c["sn"] * (c["sn"] + 2) // (2 if _dim(c) == 2 else 1)


def _moments(c):
    L = c["l_max"]
    return (L + 1) * (L + 2) // 2 if _dim(c) == 2 else (L + 1) ** 2


def _blocks(cells, side):
    """Block number of every cell, x fastest; `side` cells to a block."""
    idx, mul = np.zeros(cells[::-1], dtype=np.int64), 1
    for a, n in enumerate(cells):
        shape = [1] * len(cells)
        shape[len(cells) - 1 - a] = n
        idx = idx + (np.arange(n) // side).reshape(shape) * mul
        mul *= (n + side - 1) // side
    return idx.reshape(-1), mul


def _problem(c, seed):
    """Materials of the seeded workloads on any box: in 2-D 8 x 8 blocks of
    sigma_t ~ LogUniform[0.1, 100] and c ~ U[0.5, 0.9999] with Henyey-Greenstein
    moments (g = 0.7), in 3-D blocks of 4^3 cells of a thick scatterer or a thin
    one.  One homogeneous material on the smallest mesh."""
    rng = np.random.default_rng(seed)
    dim = _dim(c)
    cells = (c["nx"], c["ny"], c["nz"])[:dim]
    quad = og.build_quadrature(c["quad"], c["sn"], c["l_max"], dim=dim)
    G, L = c.get("groups", 1), c["l_max"]
    if dim == 2 and _cells(c) <= 1024:
        mat, nm = np.zeros(_cells(c), np.int32), 1
        st, ratio, g = np.ones((1, G)), np.full((1, G), 0.5), 0.0
    elif dim == 2:
        mat, nm = _blocks(cells, -(-max(cells) // 8))
        st = np.exp(rng.uniform(math.log(0.1), math.log(100.0), (nm, G)))
        ratio, g = rng.uniform(0.5, 0.9999, (nm, G)), 0.7
    else:
        blk, nb = _blocks(cells, 4)
        mat, nm = rng.integers(0, 2, nb)[blk], 2
        st = np.array([[1.0], [100.0]]) * (1.0 + 0.25 * np.arange(G))
        ratio, g = np.array([[0.9], [0.999]]) * np.ones((1, G)), 0.4
    ss = np.zeros((nm, G, G, L + 1))
    for gf in range(G):
        for gt in range(G):
            share = 0.8 if gf == gt else 0.2 / max(1, G - 1)
            for l in range(L + 1):
                ss[:, gf, gt, l] = (share if G > 1 else 1.0) * ratio[:, gf] * st[:, gf] * g ** l
    rhs = c["kind"] == "rhs"
    bc = (1, 0, 2, 1, 0, 0) if rhs else (0,) * 6
    inc = rng.uniform(0.2, 2.0, (2 * dim, G)) if rhs else None
    sid = rng.integers(0, 2, _cells(c)).astype(np.int32)
    src = np.vstack([np.zeros(G), rng.uniform(0.5, 1.5, G)])
    order = og.zorder_cells(*cells) if c["kind"] == "apply_host" else None
    return og.Problem(dim, c["order"], cells, (0.0,) * dim, (10.0,) * dim, quad, st, ss, mat.astype(np.int32),
                      sid, src, bc, inc, order)


def _batch(c, seed):
    """Uneven members: the shapes come from the case, the materials from the seed."""
    r = random.Random(c["shapes"])
    out = []
    for i in range(c["count"]):
        side, p, sn = r.choice([32, 64, 100, 128, 200, 256]), r.choice([1, 2]), r.choice([4, 8, 12, 16])
        m = _case("", "apply", (side, side), p, "LS", sn, 1)
        out.append((m, seed * 1000 + i))
    return out


def _vector(rng_seed, nm, nd):
    """Flux moments of a Krylov vector: signed, the higher moments smaller."""
    g = torch.Generator(device=DEV)
    g.manual_seed(rng_seed)
    x = torch.randn(nm, nd, dtype=torch.float64, device=DEV, generator=g)
    x[1:] *= 0.3
    return x.reshape(-1)


def _inputs(c, seed):
    """The vectors of a call, as device tensors in the caller's numbering."""
    if c["kind"] == "batch":
        return torch.cat([_vector(s, _moments(m), _cells(m) * _n(m)) for m, s in _batch(c, seed)])
    x = _vector(seed, _moments(c), _cells(c) * _n(c))
    if c["kind"] != "rhs":
        return x
    g = torch.Generator(device=DEV)
    g.manual_seed(seed + 1)
    gf = torch.rand(c["groups"] * x.numel(), dtype=torch.float64, device=DEV, generator=g)
    psi = torch.rand(_dirs(c) * _cells(c) * _n(c), dtype=torch.float32, device=DEV, generator=g)
    return gf, psi


def prepare(case, seed):
    c = case
    if c["kind"] == "batch":
        batch = og.Batch([_problem(m, s) for m, s in _batch(c, seed)])
        x = _inputs(c, seed)
        return {"case": c, "op": batch, "x": x, "y": torch.empty_like(x)}
    p = _problem(c, seed)
    rt = og.RadiativeTransfer(p, precision="fp64" if c["kind"] == "solve" else c["precision"])
    s = {"case": c, "op": rt}
    if c["kind"] == "solve":
        s["x"] = torch.zeros(rt.length, dtype=torch.float64, device=DEV)
        rt.set_dsa(c["cg"])
        if c["method"] == "fgmres_learned":
            s["net"] = learned.Network.load(os.path.join(learned.WEIGHTS, "dsa_guess_thick3d.npz"), p.n_cells)
            learned.install(rt, s["net"])
        return s
    if c["kind"] == "rhs":
        s["x"], psi = _inputs(c, seed)
        if c["inv_vdt"]:
            rt.set_time_step(c["inv_vdt"])
            rt.set_angular_flux(psi.double().cpu().numpy())
        return s
    s["x"] = _inputs(c, seed)
    s["y"] = torch.empty_like(s["x"])
    if c["kind"] == "apply_host":
        s["x"], s["y"] = s["x"].cpu().numpy(), s["y"].cpu().numpy()
    if c["kind"] == "dsa":
        rt.set_dsa(c["cg"])
    return s


def run(state):
    c, op = state["case"], state["op"]
    if c["kind"] == "batch":
        y = op.apply(state["x"], precision=c["precision"], out=state["y"])
    elif c["kind"] == "rhs":
        y = op.rhs(state["x"], out=torch.zeros(op.length, dtype=torch.float64, device=DEV))
    elif c["kind"] == "solve":
        return op.solve(c["method"], x=state["x"], dsa=True)[0].float()
    elif c["kind"] == "dsa":
        return op.dsa_apply(state["x"], out=state["y"]).float()
    else:
        op.Apply(state["x"], state["y"])
        y = state["y"]
    return y.astype(np.float32) if c["precision"] == "fp32" and isinstance(y, np.ndarray) else \
        y.float() if c["precision"] == "fp32" else y


def work(case):
    """Vectors in and out once, materials once; per (cell, direction) the dense
    cell solve, the inflow faces and the two moment contractions."""
    c = case
    if c["kind"] == "batch":
        parts = [work(dict(m, precision=c["precision"])) for m, _ in _batch(c, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    dim, n, cells, nd, nm = _dim(c), _n(c), _cells(c), _dirs(c), _moments(c)
    fd = (c["order"] + 1) ** (dim - 1)
    if c["kind"] == "dsa":
        stencil = 27 if dim == 3 else 9
        return {"bytes": 16.0 * cells * n * nm + 16 * cells, "flops": cells * (c["cg"] * (2 * stencil + 12) + 4 * n * n)}
    vectors = 16.0 * cells * n * nm
    if c["kind"] == "rhs":  # every group's flux in, the right-hand side out, psi of the last step
        vectors = 8.0 * cells * n * nm * (c["groups"] + 2) + (4.0 * cells * n * nd if c["inv_vdt"] else 0)
    if c["kind"] == "solve":  # an Apply for each of some thirty iterations
        a = work(dict(c, kind="apply"))
        return {k: 30 * v for k, v in a.items()}
    solve = 2 * n * n + 2 * dim * (fd * fd + fd) + 4 * n * nm
    return {"bytes": vectors + 4 * cells, "flops": float(cells) * nd * solve + 2.0 * cells * n * n * nm}


# --------------------------------------------------- the same results in 64 bits
def _lagrange(p, x):
    """Values and derivatives of the Lagrange basis on the nodes j/p at x."""
    nodes = np.arange(p + 1) / p
    v, d = np.ones((p + 1, len(x))), np.zeros((p + 1, len(x)))
    for k in range(p + 1):
        others = [j for j in range(p + 1) if j != k]
        for j in others:
            v[k] *= (x - nodes[j]) / (nodes[k] - nodes[j])
        for m in others:
            t = np.full(len(x), 1.0 / (nodes[k] - nodes[m]))
            for j in others:
                if j != m:
                    t *= (x - nodes[j]) / (nodes[k] - nodes[j])
            d[k] += t
    return v, d


def _tensor(mats):
    """Tensor product of per-axis matrices, axis 0 fastest."""
    out = np.ones((1, 1))
    for m in mats:
        out = np.kron(m, out)
    return out


def _line(p):
    x, w = np.polynomial.legendre.leggauss(p + 2)
    x, w = 0.5 * (x + 1), 0.5 * w
    v, d = _lagrange(p, x)
    return (v * w) @ v.T, (d * w) @ v.T, (v * w) @ np.vstack([1 - x, x]).T  # mass, int b_j b_i', mixed with hats


class _Exact:
    """The operator written out: DG upwind cells swept level by level."""

    def __init__(self, prob, inv_vdt=0.0):
        self.p, self.dim, self.cells = prob, prob.dim, prob.n_cells
        self.n1 = prob.fe_order + 1
        h = [(b - a) / n for a, b, n in zip(prob.lower, prob.upper, prob.n_cells)]
        m, g, _ = _line(prob.fe_order)
        ident = [m * hh for hh in h]
        self.mass = _tensor(ident)
        last = np.zeros_like(m)
        last[-1, -1] = 1.0
        self.grad = [_tensor([g if a == b else ident[b] for b in range(self.dim)]) for a in range(self.dim)]
        self.out = [_tensor([last if a == b else ident[b] for b in range(self.dim)]) for a in range(self.dim)]
        self.face = [_tensor([ident[b] for b in range(self.dim) if b != a]) for a in range(self.dim)]
        comp = [(np.arange(self.n1 ** self.dim) // self.n1 ** a) % self.n1 for a in range(self.dim)]
        self.low = [np.flatnonzero(k == 0) for k in comp]
        self.high = [np.flatnonzero(k == self.n1 - 1) for k in comp]
        self.inv_vdt = inv_vdt

    def t(self, a):
        return torch.as_tensor(np.ascontiguousarray(a), device=DEV)

    def source(self, x, group_from, group_to):
        """sigma_s M x of every moment: [moment][cell][n]."""
        q = self.p.quad
        sig = self.t(self.p.sigma_s[:, group_from, group_to, :][:, q.moment_l])[self.t(self.p.material_id).long()]
        x = x.reshape(q.n_mom, self.p.total_cells, -1)
        return (x @ self.t(self.mass).T) * sig.T[:, :, None]

    def sweep(self, S, iso=None, psi_prev=None, inflow=False):
        """D L^-1 (M2D S + iso + inv_vdt M psi_prev + inflow): [moment][dof]."""
        P, q, dim, n = self.p, self.p.quad, self.dim, self.n1 ** self.dim
        shape = tuple(self.cells[::-1])
        N = P.total_cells
        mat = P.material_id.reshape(shape)
        phi = torch.zeros(q.n_mom, N, n, dtype=torch.float64, device=DEV)
        sig = P.sigma_t[:, 0] + self.inv_vdt
        idx = np.arange(N).reshape(shape)
        loc = np.arange(n).reshape((self.n1,) * dim)
        for oct_ in range(1 << dim):
            ds = [d for d in range(q.n_dir) if all((q.omega[d, a] < 0) == bool(oct_ >> a & 1) for a in range(dim))]
            if not ds:
                continue
            axes = tuple(dim - 1 - a for a in range(dim) if oct_ >> a & 1)
            cmap, lmap = np.flip(idx, axes).reshape(-1), np.flip(loc, axes).reshape(-1)
            om = np.abs(q.omega[ds])
            A = sig[None, :, None, None] * self.mass
            for a in range(dim):
                A = A + om[:, a, None, None, None] * (self.out[a] - self.grad[a])
            inv = self.t(np.linalg.inv(A))  # [d][material][n][n]
            Q = torch.einsum("dm,mcn->dcn", self.t(q.m2d[ds]), S)
            if iso is not None:
                Q = Q + iso
            if psi_prev is not None:
                Q = Q + self.inv_vdt * (psi_prev.reshape(q.n_dir, N, n)[self.t(np.array(ds))] @ self.t(self.mass).T)
            Q = Q[:, self.t(cmap.copy())][:, :, self.t(lmap.copy())]
            cls = self.t(mat.reshape(-1)[cmap]).long()
            pos = np.indices(shape).reshape(dim, -1)[::-1]  # per axis
            level = pos.sum(0)
            order = np.argsort(level, kind="stable")
            cuts = np.searchsorted(level[order], np.arange(level.max() + 2))
            stride = [int(np.prod(self.cells[:a])) for a in range(dim)]
            faces, enter = [], []
            for a in range(dim):
                f = torch.zeros(len(ds), N + 1, len(self.low[a]), dtype=torch.float64, device=DEV)  # row N: the boundary
                if inflow:
                    side = 2 * a + (oct_ >> a & 1)
                    b = P.bc_type[side]
                    on = (q.most_normal[side][ds] != 0) if b == 2 else np.full(len(ds), b == 1)
                    f[:, N, :] = self.t(np.where(on, P.inc_flux[side, 0], 0.0) / q.weight_sum)[:, None]
                faces.append(f)
                enter.append(self.t(np.where(pos[a] == 0, N, np.arange(N) - stride[a])))
            F = [self.t(om[:, a])[:, None, None] * self.t(self.face[a]) for a in range(dim)]
            order_t = self.t(order)
            psi = torch.empty(len(ds), N, n, dtype=torch.float64, device=DEV)
            for k in range(len(cuts) - 1):
                c = order_t[cuts[k]:cuts[k + 1]]
                b = Q[:, c].clone()
                for a in range(dim):
                    b[:, :, self.low[a]] += faces[a][:, enter[a][c]] @ F[a].transpose(1, 2)
                x = torch.einsum("dcij,dcj->dci", inv[:, cls[c]], b)
                psi[:, c] = x
                for a in range(dim):
                    faces[a][:, c] = x[:, :, self.high[a]]
            part = torch.einsum("md,dcn->mcn", self.t(q.d2m[:, ds]), psi)
            back, lback = np.argsort(cmap), np.argsort(lmap)
            phi += part[:, self.t(back)][:, :, self.t(lback)]
        return phi.reshape(-1)

    def apply(self, x):
        return x - self.sweep(self.source(x, 0, 0))

    def rhs(self, gf, psi):
        P, q = self.p, self.p.quad
        S = torch.zeros(q.n_mom, P.total_cells, self.n1 ** self.dim, dtype=torch.float64, device=DEV)
        for g in range(1, P.n_groups):
            S += self.source(gf.reshape(P.n_groups, -1)[g], g, 0)
        iso = self.t(P.source[P.source_id, 0] / q.weight_sum)[:, None] * self.t(self.mass.sum(1))
        return self.sweep(S, iso, psi.double() if self.inv_vdt else None, True)

    def dsa(self, v, steps):
        """v + f: Jacobi-CG steps of the vertex diffusion system from zero."""
        P, dim = self.p, self.dim
        h = [(b - a) / n for a, b, n in zip(P.lower, P.upper, P.n_cells)]
        m1, s1 = np.array([[2.0, 1.0], [1.0, 2.0]]) / 6, np.array([[1.0, -1.0], [-1.0, 1.0]])
        vert = [n + 1 for n in self.cells]
        pos = np.indices(tuple(self.cells[::-1])).reshape(dim, -1)[::-1]
        corner = np.zeros((P.total_cells, 1 << dim), dtype=np.int64)
        for k in range(1 << dim):
            mul = 1
            for a in range(dim):
                corner[:, k] += (pos[a] + (k >> a & 1)) * mul
                mul *= vert[a]
        st, s0 = P.sigma_t[:, 0], P.sigma_s[:, 0, 0, 0]
        s1v = P.sigma_s[:, 0, 0, 1] if P.l_max >= 1 else 0.0 * s0
        D, sa = 1.0 / (3.0 * (st - s1v)), np.maximum(st - s0, 0.0)
        mass = _tensor([m1 * hh for hh in h])
        stiff = sum(_tensor([s1 / h[a] if a == b else m1 * h[b] for b in range(dim)]) for a in range(dim))
        K = self.t((D[:, None, None] * stiff + sa[:, None, None] * mass)[P.material_id])
        for a in range(dim):  # Marshak: half the face mass on every (vacuum) side
            for s in (0, 1):
                e = np.zeros((2, 2))
                e[s, s] = 0.5
                on = self.t((pos[a] == (self.cells[a] - 1 if s else 0)).astype(np.float64))
                K += on[:, None, None] * self.t(_tensor([e if a == b else m1 * h[b] for b in range(dim)]))
        corner = self.t(corner)
        nv = int(np.prod(vert))

        def add(local):
            return torch.zeros(nv, dtype=torch.float64, device=DEV).index_add_(0, corner.reshape(-1), local.reshape(-1))

        def mul(z):
            return add((K @ z[corner][:, :, None])[:, :, 0])

        mixed = _line(P.fe_order)[2]
        n = self.n1 ** dim
        v0 = v[:P.total_cells * n].reshape(-1, n)
        r = add((v0 @ self.t(_tensor([mixed * hh for hh in h]))) * self.t(s0[P.material_id])[:, None])
        dinv = 1.0 / add(torch.diagonal(K, dim1=1, dim2=2))
        x, z = torch.zeros_like(r), r * dinv
        p, rz = z.clone(), torch.dot(r, z)
        for _ in range(steps):
            w = mul(p)
            al = rz / torch.dot(p, w)
            x, r = x + al * p, r - al * w
            z = r * dinv
            new = torch.dot(r, z)
            p, rz = z + (new / rz) * p, new
        hats = np.vstack([1 - np.arange(self.n1) / P.fe_order, np.arange(self.n1) / P.fe_order]).T
        out = v.clone()
        out[:P.total_cells * n] += (x[corner] @ self.t(_tensor([hats] * dim)).T).reshape(-1)
        return out


def exact(case, seed):
    c = case
    if c["kind"] == "batch":
        x, out, at = _inputs(c, seed), [], 0
        for m, s in _batch(c, seed):
            p = _problem(m, s)
            out.append(_Exact(p).apply(x[at:at + p.vector_length]))
            at += p.vector_length
        return torch.cat(out)
    if c["kind"] == "solve":
        return None
    p = _problem(c, seed)
    if c["kind"] == "rhs":
        return _Exact(p, c["inv_vdt"]).rhs(*_inputs(c, seed))
    x = _inputs(c, seed)
    if c["kind"] == "dsa":
        return _Exact(p).dsa(x, c["cg"])
    if c["kind"] != "apply_host":
        return _Exact(p).apply(x)
    z = torch.as_tensor(p.cell_order, device=DEV)
    nm, n = _moments(c), _n(c)
    y = _Exact(p).apply(x.reshape(nm, -1, n)[:, z].reshape(-1))
    out = torch.empty_like(y).reshape(nm, -1, n)
    out[:, z] = y.reshape(nm, -1, n)
    return out.reshape(-1).cpu().numpy()
