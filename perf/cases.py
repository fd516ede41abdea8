"""What is timed: the work that a solver program has this library do.

Every case goes through the public entry points of ``bcm_cgli_gb300.api``:
a device-resident context (or batch of cases) that marches dual-time steps,
the drop-in functions on host arrays in the reference driver's call order,
and the immersed-boundary preprocessing.  Workloads, resolutions and options
are those of the repository's benchmark and tests (Taylor-Green box, sphere
with immersed boundary on two cube levels, uneven sphere batches, isentropic
vortex; both precisions; RK and LU-SGS sub-iterations), at sizes whose
inputs are made quickly.

``exact`` restates the scheme in 64-bit torch, cube-vectorised, from its
definition, without this repository's code.
"""
from __future__ import annotations

import ctypes
import functools

import numpy as np
import torch

from bcm_cgli_gb300 import _lib, api, cases

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # The smallest calls: 8 cubes of 8^3 cells, one dual-time step of 10
        # RK sub-iterations per call (a coarse grid of a convergence study;
        # launches and their gaps are what it costs).
        dict(name="tiny_split_rk", family="tgv", n=8, size=2, precision="split", method="rk",
             subiters=10),
        # Cube edge not a multiple of 8 (the ragged resolutions the reference
        # allows: any multiple of 4).
        dict(name="ragged_split_rk", family="tgv", n=12, size=6, precision="split", method="rk",
             subiters=10),
        # The Taylor-Green configuration: 512 cubes of 24^3, 7.1 M cells.
        dict(name="tgv_split_rk", family="tgv", n=24, size=8, precision="split", method="rk",
             subiters=10),
        # LU-SGS sub-iterations, the implicit option, at the same resolution.
        dict(name="tgv_split_lusgs", family="tgv", n=24, size=6, precision="split",
             method="lusgs", subiters=10),
        # One sphere flow: immersed boundary, two cube levels, open box.
        dict(name="sphere_split_rk", family="sphere", n=16, size=400, precision="split",
             method="rk", subiters=10),
        # Uneven independent sphere flows in one batched context.
        dict(name="batch_split_rk", family="batch", n=16, size=6, hi=480, precision="split",
             method="rk", subiters=5),
        # The largest resident case: 512 cubes of 32^3, 16.8 M cells, LU-SGS.
        dict(name="large_split_lusgs", family="tgv", n=32, size=8, precision="split",
             method="lusgs", subiters=5),
        # The plain 64-bit method (the drop-in precision): the inviscid
        # vortex configuration, norms read every step.
        dict(name="vortex_fp64_rk", family="vortex", n=16, size=4, precision="fp64", method="rk",
             subiters=10),
        # 64-bit sphere: viscous, immersed boundary, level jumps, norms read.
        dict(name="sphere_fp64_rk", family="sphere", n=16, size=96, precision="fp64",
             method="rk", subiters=5),
        # 64-bit LU-SGS.
        dict(name="tgv_fp64_lusgs", family="tgv", n=24, size=4, precision="fp64",
             method="lusgs", subiters=5),
        # The drop-in functions on host arrays: one RK sub-iteration in the
        # reference driver's call order.
        dict(name="dropin_fp64_rk", family="dropin", n=16, size=72, precision="fp64",
             method="rk", subiters=1),
        # Setup: immersed-boundary tables of a 20,480-triangle body.
        dict(name="ibm_tables", family="ibm", n=16, size=160, levels=5),
    ]


def _bounded(subiters, precision, cells):
    """Sub-iterations of a drawn case: no more work than the largest listed."""
    return max(1, min(subiters, int((6e7 if precision == "split" else 2.2e6) / cells)))


def draw(rng):
    """One more case of the same families; sizes over the whole range."""
    kind = rng.choice(["tgv", "tgv", "tgv", "sphere", "sphere", "batch", "vortex", "dropin",
                       "ibm"])
    precision = rng.choice(["split", "split", "fp64"])
    method = rng.choice(["rk", "rk", "lusgs"])
    subiters = rng.randint(2, 10)
    if kind == "tgv":
        n = rng.choice([4, 8, 12, 16, 20, 24, 28, 32])
        cap = (6e6 if n % 8 == 0 else 3e6) if precision == "split" else 2.5e5  # cells
        top = max(2, int((cap / n ** 3) ** (1.0 / 3.0)))
        size = min(int(round(2 * (top / 2.0) ** rng.random())), 12)
        return dict(family="tgv", n=n, size=size, precision=precision, method=method,
                    subiters=_bounded(subiters, precision, size ** 3 * n ** 3))
    if kind == "sphere":
        n = rng.choice([8, 12, 16, 20])
        size = int(64 * ((400 if precision == "split" else 96) / 64.0) ** rng.random())
        return dict(family="sphere", n=n, size=size, precision=precision, method=method,
                    subiters=_bounded(subiters, precision, size * n ** 3))
    if kind == "batch":
        return dict(family="batch", n=rng.choice([8, 16]), size=rng.randint(2, 6),
                    hi=rng.randint(72, 480), precision="split", method=method,
                    subiters=min(subiters, 5))
    if kind == "vortex":
        n, size = rng.choice([8, 12, 16, 20]), rng.randint(2, 4)
        return dict(family="vortex", n=n, size=size, precision="fp64", method="rk",
                    subiters=_bounded(subiters, "fp64", size ** 3 * n ** 3))
    if kind == "dropin":
        return dict(family="dropin", n=rng.choice([8, 12, 16]), size=rng.randint(64, 72),
                    precision="fp64", method="rk", subiters=1)
    return dict(family="ibm", n=rng.choice([8, 12, 16]), size=rng.randint(64, 160),
                levels=rng.randint(3, 5))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=3)
def _grid(family, n, size, hi):
    """Host-side cases (grid, flags, tables, base flow) of a configuration: a
    list, one entry per independent case."""
    if family == "tgv":
        return [cases.taylor_green(ncx=size, n=n)]
    if family == "vortex":
        return [cases.isentropic_vortex(ncx=size, n=n)]
    if family == "batch":
        return cases.sphere_batch(ncase=size, seed=2024, n=n, lo=64, hi=hi)
    return [cases.sphere_cubes(size, n=n)]  # sphere, dropin, ibm


def _grid_of(case):
    return _grid(case["family"], case["n"], case["size"], case.get("hi", 0))


def _perturbed(base, seed):
    """The base flow with a seeded 1e-4 density perturbation (velocity and
    pressure kept), as a device array."""
    U = torch.tensor(base, device=DEV)
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    f = 1 + 1e-4 * (torch.rand(U.shape[:-1], generator=g, device=DEV, dtype=torch.float64) - 0.5)
    ke = 0.5 * (U[..., 1] ** 2 + U[..., 2] ** 2 + U[..., 3] ** 2) / U[..., 0].clamp_min(1e-30)
    U[..., :4] *= f[..., None]
    U[..., 4] += ke * (f - 1)
    return U


def _flat_base(grids):
    return grids[0].U if len(grids) == 1 else cases.CaseBatch(grids).U


class _DeviceArray:
    """A context's device array for torch (kept alive with its context)."""

    def __init__(self, ctx, ptr, shape):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8",
                                         "data": (int(ptr), False), "version": 2}


def _device_state(ctx):
    p = [ctypes.c_void_p() for _ in range(3)]
    _lib.check(_lib.lib().bcmg_case_device_state(ctx.h, *(ctypes.byref(x) for x in p)))
    return [torch.as_tensor(_DeviceArray(ctx, x.value, ctx.shape), device="cuda") for x in p]


def _body(case):
    """Triangles of the seeded body: an icosphere a little off the origin."""
    return lambda seed: cases.icosphere(
        case["levels"], 0.5, center=np.random.RandomState(seed % (1 << 31)).uniform(-0.01, 0.01, 3))


def prepare(case, seed):
    grids = _grid_of(case)
    if case["family"] == "ibm":
        return dict(case=case, grid=grids[0], tris=_body(case)(seed),
                    rows=int((grids[0].fws == 0).sum()))
    U = _perturbed(_flat_base(grids), seed).cpu().numpy()
    if case["family"] == "dropin":
        g = grids[0]
        api.reference_config_for(g)
        return dict(case=case, grid=g, lists=[api._one_based(x) for x in g.bc_lists()],
                    U1_=U, U1=U.copy(), U1q=U.copy(),
                    scratch=[np.zeros_like(U) for _ in range(4)], er=np.zeros(8))
    precision = api.PRECISION_SPLIT if case["precision"] == "split" else api.PRECISION_FP64
    if len(grids) > 1:
        ctx = api.BatchContext(grids, precision=precision)
    else:
        ctx = api.CaseContext(grids[0], precision=precision)
    if case["method"] == "lusgs":
        ctx.set_method(api.METHOD_LUSGS)
    ctx.set_state(U, U, U)
    return dict(case=case, ctx=ctx, out=_device_state(ctx))


def run(state):
    case = state["case"]
    if case["family"] == "ibm":
        # the table builder updates the flags in place: each call gets its own
        fws = state["grid"].fws.copy()
        minus, plus = api.ibm_preprocess(state["grid"], state["tris"], fws)
        # into a solver's fixed-size tables (one row per flagged ghost cell)
        return dict(fws=fws, used=[len(minus[0]), len(plus[0])],
                    minus=[_padded(x, state["rows"]) for x in minus],
                    plus=[_padded(x, state["rows"]) for x in plus])
    if case["family"] == "dropin":
        return _dropin_subiteration(state)
    if case["precision"] == "split":
        # as in the benchmark's resident loop: the step is enqueued, its
        # result is the state on the device
        state["ctx"].advance_async(1, case["subiters"])
        return dict(U1_=state["out"][0], U1=state["out"][1], U1q=state["out"][2])
    er = state["ctx"].advance(1, case["subiters"])
    return dict(U1_=state["out"][0], U1=state["out"][1], U1q=state["out"][2], er=er)


def _padded(x, rows):
    out = np.zeros((rows,) + x.shape[1:], x.dtype)
    out[:len(x)] = x
    return out


def _dropin_subiteration(s):
    g, U = s["grid"], s["U1_"]
    xl, xu, yl, yu, zl, zu = s["lists"]
    p1, p2, rku, res = s["scratch"]
    for RK in (1, 2, 3):
        api.BCM_X_boundary_condition(0, len(xl) - 1, len(xu) - 1, xl, xu, U)
        api.BCM_Y_boundary_condition(len(yl) - 1, len(yu) - 1, yl, yu, U)
        api.BCM_Z_boundary_condition(len(zl) - 1, len(zu) - 1, zl, zu, U)
        for fill, table in ((api.BCM_Ghostcell_minus, g.ibm_minus),
                            (api.BCM_Ghostcell_plus, g.ibm_plus)):
            if table is not None:
                W, G, I = table
                fill(0, (len(G) - 1) // 4, W, G, I, g.fws, U)
        api.BCM_Interface_for_case(g, U)
        api.BCM_Flux_XYZ_Viscous_Runge_kutta(0, g.ncube, RK, g.dT, g.dTau, g.e, g.fws, g.csl,
                                             g.cube_size, U, s["U1"], s["U1q"], p1, p2, rku, res,
                                             s["er"])
        api.BCM_Interface_for_case(g, U)
    return dict(U1_=U, U1p1=p1, U1p2=p2, Rku1=rku, Residual1=res, er=s["er"])


def work(case):
    """Bytes and operations of one pass.  A flux stage reads the state and two
    earlier levels and the flag of a cell and writes the state (164 B) and
    does about 1,900 additions, multiplications, divisions and roots (three
    faces of five reconstructed pairs and an upwind flux each, six viscous
    faces, source, preconditioner); an LU-SGS sweep about 450 more and the
    residual once in and out; a step's time shift moves two levels."""
    grids = _grid_of(case)
    if case["family"] == "ibm":
        g = grids[0]
        cells = int((g.fws == 0).sum())
        tris = 20 * 4 ** case["levels"]
        # triangles, flags in and out, tables out; ray test per pair of a
        # ghost cell and a triangle near its cube
        return {"bytes": 72.0 * tris + 8.0 * g.fws.size + 96.0 * cells,
                "flops": 30.0 * cells * tris}
    cells = sum(g.n_cells for g in grids)
    if case["family"] == "dropin":
        S3 = _flat_base(grids).nbytes
        return {"bytes": 3.0 * (3 * S3 + S3), "flops": 3.0 * 1900 * cells}
    if case["method"] == "rk":
        per = {"bytes": 3 * 164.0, "flops": 3 * 1900.0}
    else:
        per = {"bytes": 164.0 + 80.0, "flops": 1900.0 + 450.0}
    return {"bytes": cells * (case["subiters"] * per["bytes"] + 160.0),
            "flops": cells * case["subiters"] * per["flops"]}


# ---------------------------------------------------------------------------
# The same in plain 64-bit torch
# ---------------------------------------------------------------------------
K, RGAS, CV, PR = 1.4, 287.0, 717.5, 0.72


class _World:
    """Cubes of one or several cases in one array, with per-cube constants."""

    def __init__(self, grids):
        dev = DEV
        self.n = n = grids[0].n
        self.S = n + 4
        f64 = dict(dtype=torch.float64, device=dev)
        off, const, dx, fws, self.bc, self.ibm, faces = 0, [], [], [], [[] for _ in range(6)], [], {}
        for g in grids:
            m = g.ncube - 1
            ph = g.phys
            const.append(np.tile([ph.mu_L, ph.rho0, ph.P0, ph.Uin, g.dT, g.dTau, g.e], (m, 1)))
            dx.append(g.cube_size[1:] / n)
            fws.append(g.fws[1:])
            for t, x in enumerate(g.bc_lists()):
                self.bc[t] += [int(c) - 1 + off for c in x]
            for table in (g.ibm_minus, g.ibm_plus):
                if table is None:
                    continue
                W, G, I = table
                for r in range((len(G) - 1) // 4):
                    gc, ip = G[4 * r + 1:4 * r + 5], I[4 * r + 1:4 * r + 5]
                    self.ibm.append(((int(gc[0]) - 1 + off, *map(int, gc[1:])),
                                     (int(ip[0]) - 1 + off, *map(int, ip[1:])),
                                     W[8 * r + 1:8 * r + 9]))
            for c in range(1, g.ncube):
                for d in range(1, 7):
                    for slot in range(1, 5):
                        a = int(g.adj[c, slot, d])
                        if a <= 0:
                            continue
                        ax, side = (d - 1) // 2, (d - 1) % 2  # side: c's low / high face
                        if g.csl[a] == g.csl[c]:
                            if slot == 1:
                                faces.setdefault((0, ax, side, 0), []).append((c - 1 + off, a - 1 + off))
                        elif g.csl[a] < g.csl[c]:  # a is smaller: slot names its quadrant
                            faces.setdefault((2, ax, side, slot), []).append((c - 1 + off, a - 1 + off))
                            faces.setdefault((1, ax, 1 - side, slot), []).append((a - 1 + off, c - 1 + off))
            off += m
        self.C = off
        c = torch.tensor(np.concatenate(const), **f64)
        self.mu, self.rho0, self.P0, self.Uin, self.dT, self.dTau, self.e = (
            c[:, t].reshape(-1, 1, 1, 1) for t in range(7))
        self.dx = torch.tensor(np.concatenate(dx), **f64).reshape(-1, 1, 1, 1)
        self.fluid = torch.from_numpy(np.concatenate(fws) == 1).to(dev)
        self.T0 = self.P0 / self.rho0 / RGAS
        self.viscous = bool((self.mu != 0).any())
        self.faces = [(k, torch.tensor(v, device=dev).T) for k, v in faces.items()]
        self.bc = [torch.tensor(x, device=dev, dtype=torch.long) for x in self.bc]
        self.grids = grids
        self._ibm_groups()

    def _ibm_groups(self):
        """Entries in the order a serial pass sees: groups whose members read
        no cell that an earlier member of the group writes."""
        wrote, read, level = {}, {}, []
        for gc, ip, _ in self.ibm:
            cells = [(ip[0], ip[1] + a, ip[2] + b, ip[3] + c)
                     for a in (0, 1) for b in (0, 1) for c in (0, 1)]
            lv = max([wrote.get(x, -1) + 1 for x in cells] + [wrote.get(gc, -1) + 1, read.get(gc, 0)])
            for x in cells:
                read[x] = max(read.get(x, 0), lv)
            wrote[gc] = lv
            level.append(lv)
        self.groups = []
        for lv in range(max(level) + 1 if level else 0):
            m = [e for e, x in zip(self.ibm, level) if x == lv]
            self.groups.append((torch.tensor([x[0] for x in m], device=DEV),
                                torch.tensor([x[1] for x in m], device=DEV),
                                torch.tensor(np.array([x[2] for x in m]), device=DEV,
                                             dtype=torch.float64)))


def _press(q):
    rho = q[..., 0]
    u, v, w = q[..., 1] / rho, q[..., 2] / rho, q[..., 3] / rho
    vv = u * u + v * v + w * w
    return rho, u, v, w, vv, (q[..., 4] - 0.5 * rho * vv) * (K - 1)


def _boundaries(w, U):
    n = w.n
    nx = n + 1
    xl, xu, yl, yu, zl, zu = w.bc
    s = slice(2, n + 2)
    if len(xl):
        rho, _, _, _, _, p = _press(U[xl, 2, s, s])
        uin = w.Uin[xl, 0]
        z = torch.zeros_like(rho)
        g = torch.stack([rho, rho * uin, z, z, p / (K - 1) + 0.5 * rho * uin * uin], -1)
        U[xl, 0, s, s] = g
        U[xl, 1, s, s] = g
    if len(xu):
        g = U[xu, nx, s, s]
        U[xu, nx + 1, s, s] = g
        U[xu, nx + 2, s, s] = g
    for lst, src, d in ((yl, 2, (0, 1)), (yu, nx, (nx + 1, nx + 2))):
        if len(lst):
            g = U[lst, :, src, s]
            for t in d:
                U[lst, :, t, s] = g
    if len(zl):
        g = U[zl, :, :, 2] * torch.tensor([1., 1, 1, -1, 1], dtype=U.dtype, device=U.device)
        U[zl, :, :, 0] = g
        U[zl, :, :, 1] = g
    if len(zu):
        g = U[zu, :, :, nx]
        U[zu, :, :, nx + 1] = g
        U[zu, :, :, nx + 2] = g


_STENCIL = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 1, 1)]


def _ghosts(w, U):
    for gc, ip, wt in w.groups:
        o = torch.tensor(_STENCIL, device=DEV)
        q = U[ip[:, :1], ip[:, 1:2] + o[:, 0], ip[:, 2:3] + o[:, 1], ip[:, 3:4] + o[:, 2]]
        rho, u, v, ww, _, p = _press(q)
        r0, p0 = w.rho0[ip[:, 0], 0, 0, 0], w.P0[ip[:, 0], 0, 0, 0]
        d = gc[:, 1:] - ip[:, 1:]
        own = ((d >= 0) & (d <= 1)).all(1)
        slot = (d[:, None, :] == o[None]).all(2) & own[:, None]
        ws = (wt * slot).sum(1)
        wr = torch.where(slot, torch.zeros_like(wt), wt)  # all but the ghost's own slot
        # the ghost outside its stencil: halfway velocity
        R = (wt * (rho - r0[:, None])).sum(1) + r0
        P = (wt * (p - p0[:, None])).sum(1) + p0
        a, b, c = ((wt * x).sum(1) for x in (u, v, ww))
        out = torch.stack([R, 0.5 * R * a, 0.5 * R * b, 0.5 * R * c,
                           P / (K - 1) + 0.5 * R * 0.25 * (a * a + b * b + c * c)], -1)
        big = ws > 0.9999
        R2 = torch.where(big, (rho * slot).sum(1), (wr * (rho - r0[:, None])).sum(1) / (1 - ws) + r0)
        P2 = torch.where(big, (p * slot).sum(1), (wr * (p - p0[:, None])).sum(1) / (1 - ws) + p0)
        a, b, c = ((wr * x).sum(1) / (2 - ws) for x in (u, v, ww))
        out2 = torch.stack([R2, R2 * a, R2 * b, R2 * c,
                            P2 / (K - 1) + 0.5 * R2 * (a * a + b * b + c * c)], -1)
        U[gc[:, 0], gc[:, 1], gc[:, 2], gc[:, 3]] = torch.where(own[:, None], out2, out)


def _interface(w, U):
    n = w.n
    h = n // 2
    for (kind, ax, side, slot), (dst, src) in w.faces:
        A = U.movedim(1 + ax, 1)  # [cube][along][t0][t1][v]
        lo = 0 if side == 0 else n + 2
        if kind == 0:
            so = n if side == 0 else 2
            for l in range(2):
                A[dst, lo + l, 2:n + 2, 2:n + 2] = A[src, so + l, 2:n + 2, 2:n + 2]
            continue
        o0 = h if slot in (2, 4) else 0
        o1 = h if slot in (3, 4) else 0
        if kind == 1:
            big = A[src, n + 1 if side == 0 else 2, 2 + o0:2 + o0 + h, 2 + o1:2 + o1 + h]
            g = big.repeat_interleave(2, 1).repeat_interleave(2, 2)
            for l in range(2):
                A[dst, lo + l, 2:n + 2, 2:n + 2] = g
        else:
            for l in range(2):
                a0 = (n - 2 + 2 * l) if side == 0 else 2 * (l + 1)
                b = A[src, a0:a0 + 2, 2:n + 2, 2:n + 2].mean(1)
                b = b.reshape(len(src), h, 2, h, 2, 5).mean((2, 4))
                A[dst, lo + l, 2 + o0:2 + o0 + h, 2 + o1:2 + o1 + h] = b
    # edges: averages of the two face ghosts beside them; corners: of the two
    # edge cells beside them (first and second axis)
    V = U.clone()
    s = slice(2, n + 2)
    gh = ((1, 2), (n + 2, n + 1))
    for a, ai in gh:
        for b, bi in gh:
            U[:, s, a, b] = 0.5 * (V[:, s, ai, b] + V[:, s, a, bi])
            U[:, a, s, b] = 0.5 * (V[:, ai, s, b] + V[:, a, s, bi])
            U[:, a, b, s] = 0.5 * (V[:, ai, b, s] + V[:, a, bi, s])
    for a, ai in gh:
        for b, bi in gh:
            for c, ci in gh:
                U[:, a, b, c] = 0.5 * (U[:, a, bi, c] + U[:, ai, b, c])


def _recon(q, order):
    a, b, c, d, f, g = q
    o = order[..., None]
    ML = torch.where(o == 5, (2 * a - 13 * b + 47 * c + 27 * d - 3 * f) / 60,
                     torch.where(o == 3, (-b + 5 * c + 2 * d) / 6, c))
    MR = torch.where(o == 5, (-3 * b + 27 * c + 47 * d - 13 * f + 2 * g) / 60,
                     torch.where(o == 3, (2 * c + 5 * d - f) / 6, d))
    return ML, MR


def _roe(ax, ML, MR, e):
    r1, u1, v1, w1, vv1, p1 = _press(ML)
    r2, u2, v2, w2, vv2, p2 = _press(MR)
    h1, h2 = 0.5 * vv1 + K * p1 / r1 / (K - 1), 0.5 * vv2 + K * p2 / r2 / (K - 1)
    s1, s2 = r1.sqrt(), r2.sqrt()
    t = s1 + s2
    rho = (r1 * r2).sqrt()
    u, v, w, H = ((s1 * x + s2 * y) / t for x, y in ((u1, u2), (v1, v2), (w1, w2), (h1, h2)))
    vv = u * u + v * v + w * w
    C = (H - 0.5 * vv) * (K - 1)
    beta = torch.maximum(vv / C, e)
    un, n1, n2 = (u, v, w)[ax], (u1, v1, w1)[ax], (u2, v2, w2)[ax]
    tmp = 0.5 * (1 + beta) * un
    sp = 0.5 * (4 * beta * C + un * un * (1 - beta) ** 2).sqrt()
    dp, dn, an = p2 - p1, n2 - n1, un.abs()
    t3 = 0.5 * (1 - beta) * un * tmp / sp
    du = (sp - t3 - beta * an) * dp / rho / beta / C + tmp / sp * dn
    dP = tmp / sp * dp + (sp - an + t3) * rho * dn
    dr = du * rho
    d = MR - ML
    F = []
    for m in range(5):
        avg = (ML[..., m] * n1 + MR[..., m] * n2)
        if m == 4:
            avg = n1 * (ML[..., 4] + p1) + n2 * (MR[..., 4] + p2)
        elif m == 1 + ax:
            avg = avg + p1 + p2
        dis = an * d[..., m] + dr * (1.0, u, v, w, H)[m]
        if m == 1 + ax:
            dis = dis + dP
        if m == 4:
            dis = dis + dP * un
        F.append(0.5 * (avg - dis))
    return torch.stack(F, -1), 0.5 * (p1 + p2)


def _residual(w, U, U1, U1q):
    """(residual of the interior cells, force integrands of the non-fluid)."""
    n, S = w.n, w.S
    s = slice(2, n + 2)
    dx = w.dx
    dx5 = dx[..., None]
    acc, dPd = None, {}
    for ax in range(3):
        t = [s, s, s]
        t[ax] = slice(0, S)
        A = U[(slice(None), *t)].movedim(1 + ax, 1)
        f = w.fluid[(slice(None), *t)].movedim(1 + ax, 1)
        pos = torch.arange(2, n + 3, device=U.device)
        at = lambda X, o: X[:, (pos + o).clamp(0, S - 1)]  # noqa: E731
        q = [at(A, o) for o in (-3, -2, -1, 0, 1, 2)]
        fm2, fm1, f0, fp1 = (at(f, o) for o in (-2, -1, 0, 1))
        g = pos.reshape(1, -1, 1, 1)
        one, three, five = (torch.tensor(x, device=U.device) for x in (1, 3, 5))
        ob = torch.where(fp1 & fm1, torch.where((g == 2) | ~fm2, three, five), one)
        of = torch.where(f0 & fm2, torch.where((g == n + 2) | ~fp1, three, five), one)
        Fb, Pb = _roe(ax, *_recon([x[:, :n] for x in q], ob[:, :n]), w.e)
        Ff, Pf = _roe(ax, *_recon([x[:, 1:] for x in q], of[:, 1:]), w.e)
        r = ((Ff - Fb) / dx5).movedim(1, 1 + ax)
        acc = r if acc is None else acc + r
        if ax != 1:
            dPd[ax] = (Pf - Pb).movedim(1, 1 + ax)
        del q, Fb, Ff, r
    rho, u, v, ww, _, p = _press(U)
    T = p / (rho * RGAS)
    prim = (u, v, ww, T)
    vis = [None] * 5
    if w.viscous:
        def at3(X, o):
            return X[:, 2 + o[0]:n + 2 + o[0], 2 + o[1]:n + 2 + o[1], 2 + o[2]:n + 2 + o[2]]

        def sh(ax, k):
            return tuple(k if a == ax else 0 for a in range(3))

        add = lambda a, b: tuple(x + y for x, y in zip(a, b))  # noqa: E731
        out = None
        for ax in range(3):
            face = []
            for sgn in (-1, 1):
                o = sh(ax, sgn)
                c0 = [at3(X, (0, 0, 0)) for X in prim]
                c1 = [at3(X, o) for X in prim]
                Tm = 0.5 * (c0[3] + c1[3])
                mu = w.mu * (Tm / w.T0) ** 1.5 * (w.T0 + 110.) / (Tm + 110.)
                grad = [None] * 3
                grad[ax] = [sgn * (b - a) / dx for a, b in zip(c0, c1)]
                for ta in range(3):
                    if ta != ax:
                        up, dn = sh(ta, 1), sh(ta, -1)
                        grad[ta] = [(at3(X, up) + at3(X, add(up, o)) - at3(X, dn) -
                                     at3(X, add(dn, o))) / 4 / dx for X in prim[:3]]
                div = grad[0][0] + grad[1][1] + grad[2][2]
                tau = [mu * (grad[m][ax] + grad[ax][m]) for m in range(3)]
                tau[ax] = mu * (2 * grad[ax][ax] - 2.0 / 3.0 * div)
                heat = sum(0.5 * (c0[m] + c1[m]) * tau[m] for m in range(3))
                face.append(tau + [heat + mu * CV * K * grad[ax][3] / PR])
            d = [(b - a) / dx for a, b in zip(*face)]
            out = d if out is None else [x + y for x, y in zip(out, d)]
        vis = [None] + out
    src = -(3 * U[:, s, s, s] - 4 * U1[:, s, s, s] + U1q[:, s, s, s]) / (2 * w.dT[..., None])
    R = src - acc
    for m in range(1, 5):
        if vis[m] is not None:
            R[..., m] += vis[m]
    zero = torch.zeros_like(dPd[0])
    f6 = -(-dPd[0] / dx + (vis[1] if vis[1] is not None else zero)) * dx ** 3
    f7 = -(-dPd[2] / dx + (vis[3] if vis[3] is not None else zero)) * dx ** 3
    return R, f6, f7


def _precondition(w, q, R):
    rho, u, v, ww, vv, p = _press(q)
    dT, dTau = w.dT, w.dTau
    T = p / rho
    C = K * T
    H = 0.5 * vv + C / (K - 1)
    b = torch.maximum(vv / C, w.e)
    t = C * (2 * dT + 3 * dTau) * (2 * dT + 3 * b * dTau)
    t2 = (K - 1) * (b - 1) * dT * dT
    t3 = H - H * K - vv + K * (T + vv)
    D = 3 * C * b * dTau
    vel = (u, v, ww)
    # rows 1..4 share the coupling (1, u, v, w, H) x (..., -u, -v, -w, 1)
    lin = R[..., 4] - (u * R[..., 1] + v * R[..., 2] + ww * R[..., 3])
    out = [2 * dT * (-2 * (-(K - 1) * (H - vv) - t3 * b) * dT + D) * R[..., 0] + 4 * t2 * lin]
    for m in range(3):
        um = vel[m]
        diag = 2 * dT * (2 * C * dT + D)  # the part without velocity products
        # d[m][m] = diag + 2 dT (-2K u^2 (b-1) dT + 2 u^2 (b-1) dT) = diag - 4 u^2 t2
        out.append(4 * um * t3 * (b - 1) * dT * dT * R[..., 0] + diag * R[..., 1 + m] +
                   4 * um * t2 * lin)
    d44 = 2 * dT * (2 * H * (K - 1) * (b - 1) * dT + C * (2 * dT + 3 * b * dTau))
    out.append(4 * H * t3 * (b - 1) * dT * dT * R[..., 0] + d44 * R[..., 4] +
               4 * H * t2 * (lin - R[..., 4]))
    return torch.stack([dTau * x / t for x in out], -1)


def _change(w, old, new, fluid, f6, f7):
    """Sums of squared changes of p, u, v, w, T over fluid cells and of the
    force integrands over the others, of one case."""
    a, b = _press(old), _press(new)
    z = torch.zeros((), dtype=old.dtype, device=old.device)
    d = [b[5] - a[5], b[1] - a[1], b[2] - a[2], b[3] - a[3], b[5] / b[0] - a[5] / a[0]]
    tot = [torch.where(fluid, x * x, z).sum() for x in d]
    tot += [torch.where(fluid, z, x).sum() for x in (f6, f7)]
    g = w.grids[0]
    er = [0.0] + [float(x.sqrt()) / (g.phys.mpi_ncube * w.n ** 3) for x in tot[:5]]
    q = 0.5 * g.phys.rho0 * g.phys.U0 ** 2 * 2.602
    return er + [float(tot[5]) / q, float(tot[6]) / q]


def _sweep(w, q, R, fluid, omega=1.5):
    """LU-SGS increment: forward and backward sweeps over planes i+j+k."""
    n, C = w.n, w.C
    rho, u, v, ww, vv, p = _press(q)
    c = (K * p / rho).sqrt()
    H = (q[..., 4] + p) / rho
    r = [x.abs() + c for x in (u, v, ww)]
    T = p / rho / RGAS
    nu = w.mu * (T / w.T0) ** 1.5 * (w.T0 + 110.) / (T + 110.) * (K / PR) / rho
    rs = r[0] + r[1] + r[2]
    dg = 1.5 / w.dT + omega * rs / w.dx + 6.0 * nu / (w.dx * w.dx)
    rows = lambda x: x.reshape(C, n ** 3).T.contiguous()  # noqa: E731
    vel, rr = [rows(x) for x in (u, v, ww)], [rows(x) for x in r]
    vv, H, nu, dg, fl = rows(vv), rows(H), rows(nu), rows(dg), rows(fluid)
    dq = R.reshape(C, n ** 3, 5).transpose(0, 1).contiguous()
    ih = (0.5 / w.dx).reshape(1, C)
    ih2 = (1.0 / (w.dx * w.dx)).reshape(1, C)
    ids = torch.arange(n ** 3, device=q.device)
    ijk = torch.stack([ids // (n * n), (ids // n) % n, ids % n])
    plane = ijk.sum(0)
    order = torch.argsort(plane, stable=True)
    cnt = torch.bincount(plane, minlength=3 * n - 2).tolist()
    start = np.concatenate([[0], np.cumsum(cnt)])
    stride = (n * n, n, 1)

    def offdiag(at, D, lower):
        x = dq[at]
        U, V, W = (y[at] for y in vel)
        un = (U, V, W)[D]
        dp = (K - 1) * (x[..., 4] - (U * x[..., 1] + V * x[..., 2] + W * x[..., 3]) +
                        0.5 * vv[at] * x[..., 0])
        t = x[..., 1 + D] - un * x[..., 0]
        a = [x[..., 1 + D], un * x[..., 1] + U * t, un * x[..., 2] + V * t,
             un * x[..., 3] + W * t, un * (x[..., 4] + dp) + H[at] * t]
        a[1 + D] = a[1 + D] + dp
        a = torch.stack(a, -1)
        wgt = (omega * rr[D][at])[..., None]
        vis = (nu[at] * ih2)[..., None]
        h = ih[..., None]
        out = h * (a + wgt * x) + vis * x if lower else h * (a - wgt * x) - vis * x
        return torch.where(fl[at][..., None], out, torch.zeros_like(out))

    for lower in (True, False):
        hs = range(3 * n - 2) if lower else range(3 * n - 3, -1, -1)
        for h in hs:
            at = order[start[h]:start[h + 1]]
            acc = torch.zeros((len(at), C, 5), dtype=q.dtype, device=q.device)
            for D in range(3):
                ok = ijk[D][at] > 0 if lower else ijk[D][at] < n - 1
                nb = at[ok] + (-stride[D] if lower else stride[D])
                if len(nb):
                    acc[ok] += offdiag(nb, D, lower)
            d = dg[at][..., None]
            x = (dq[at] + acc) / d if lower else dq[at] - acc / d
            dq[at] = torch.where(fl[at][..., None], x, torch.zeros_like(x))
    return dq.transpose(0, 1).reshape(C, n, n, n, 5)


def exact(case, seed):
    if case["family"] == "ibm":
        return None
    grids = _grid_of(case)
    w = _World(grids)
    full = _perturbed(_flat_base(grids), seed)
    U = full[1:].clone()
    U1, U1q = U.clone(), U.clone()
    n = w.n
    s = (slice(None),) + (slice(2, n + 2),) * 3
    fluid = w.fluid[s]
    f5 = fluid[..., None]
    emax, er = [0.0] * 6, [0.0] * 8
    for _ in range(case["subiters"]):
        if case["method"] == "rk":
            for RK in (1, 2, 3):
                _boundaries(w, U)
                _ghosts(w, U)
                _interface(w, U)
                R, f6, f7 = _residual(w, U, U1, U1q)
                old = U[s].clone()
                x = torch.where(f5, _precondition(w, old, R), torch.zeros_like(old))
                if RK == 1:
                    new = p1 = old + x
                elif RK == 2:
                    new = p2 = 0.75 * old + 0.25 * p1 + 0.25 * x
                else:
                    new = old / 3.0 + 2.0 / 3.0 * p2 + 2.0 / 3.0 * x
                new = torch.where(f5, new, old)
                U[s] = new
                if RK == 3 and len(grids) == 1:
                    er = _change(w, old, new, fluid, f6, f7)
                _interface(w, U)
        else:
            _boundaries(w, U)
            _ghosts(w, U)
            _interface(w, U)
            R, f6, f7 = _residual(w, U, U1, U1q)
            old = U[s].clone()
            new = old + _sweep(w, old, R, fluid)
            U[s] = new
            if len(grids) == 1:
                er = _change(w, old, new, fluid, f6, f7)
            _interface(w, U)
        if case["family"] != "dropin":
            for v in range(1, 6):
                emax[v] = max(emax[v], er[v])
                er[v] = er[v] / emax[v] if emax[v] else 0.0
    back = lambda x: torch.cat([full[:1], x])  # noqa: E731  (slot 0 is unused)
    if case["family"] == "dropin":
        return dict(U1_=back(U), U1p1=None, U1p2=None, Rku1=None, Residual1=None,
                    er=np.array(er))
    U1q[s] = U1[s]
    U1[s] = U[s]
    out = dict(U1_=back(U), U1=back(U1), U1q=back(U1q))
    if case["precision"] != "split":
        out["er"] = np.array(er)
    return out
