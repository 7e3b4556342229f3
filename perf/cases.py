"""Workloads of the multi-fluid Hall-MHD step, as programs on this framework run them.

A pass advances the solves that a program holds on the GPU by a few steps
(Context.step, or Batch.request / run / poll) and returns their conserved
state; the `request` cases serve a whole request on a grid that is already
loaded.  Sizes are those of the framework's tests, of its benchmark workloads
(cubes, the ensemble of uneven periodic boxes, the magnetosphere shells and the
implicit resistive cube) and odd ones in between.

A pass takes an even number of steps: the conserved states are double-buffered,
so after it they are in the arrays that they were in before, and the views of
the device arrays that prepare() makes stay those of the current state.
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

from mpcns_mercury_b200 import Context, capi, reference_constants
from mpcns_mercury_b200 import magnetosphere as M
from mpcns_mercury_b200 import setup as S
from mpcns_mercury_b200.capi import Batch, SolveDesc

NGHOST = 4
STATE = ("U_H", "U_Na", "B_xi", "B_eta", "B_zeta")
FIELD = {"U_H": "U_H", "U_Na": "U_NA", "B_xi": "B_XI", "B_eta": "B_ETA", "B_zeta": "B_ZETA"}

_topologies = M.TopologyCache()  # a program keeps a grid's tables for all its solves on that grid


def listed():
    return [
        # the smallest solve the tests and the smoke run take: nothing but latency and launches
        {"name": "box_8_fp64", "kind": "box", "nx": 8, "ny": 8, "nz": 8, "precision": 0, "steps": 20},
        # the single-block case of the reference's test setup
        {"name": "box_32_fp64", "kind": "box", "nx": 32, "ny": 32, "nz": 32, "precision": 0, "steps": 20},
        # an odd box with the artificial resistivity on
        {"name": "box_ragged_fp64", "kind": "box", "nx": 33, "ny": 47, "nz": 70, "precision": 0, "steps": 10,
         "artificial": True},
        # one mid-size block in mixed precision
        {"name": "box_64_mixed", "kind": "box", "nx": 64, "ny": 64, "nz": 64, "precision": 1, "steps": 10},
        # the largest block of the ensemble's range, in full precision
        {"name": "box_64x64x128_fp64", "kind": "box", "nx": 64, "ny": 64, "nz": 128, "precision": 0, "steps": 10},
        # the cube workload of the benchmark in mixed precision
        {"name": "box_96_mixed", "kind": "box", "nx": 96, "ny": 96, "nz": 96, "precision": 1, "steps": 10},
        # many uneven boxes advanced together
        {"name": "boxes_24_mixed", "kind": "boxes", "solves": 24, "sizes": 1, "precision": 1, "steps": 10},
        # the implicit resistive substep on a cube: long conjugate-gradient solves
        {"name": "implicit_64_fp64", "kind": "box", "nx": 64, "ny": 64, "nz": 64, "precision": 0, "steps": 2,
         "resistive": True},
        # the smallest magnetosphere shell of the tests
        {"name": "shell_8_fp64", "kind": "shells", "na": 8, "nr": 12, "grids": 1, "solves": 1, "precision": 0,
         "steps": 10, "resistive": False},
        # the magnetosphere configuration: dipole, Hall, electron pressure, implicit resistivity
        {"name": "shell_48_fp64", "kind": "shells", "na": 48, "nr": 96, "grids": 1, "solves": 1, "precision": 0,
         "steps": 10, "resistive": True},
        # the ensemble of resistive magnetosphere shells in mixed precision: several grids, several solves on each
        {"name": "shells_6_mixed", "kind": "shells", "na": 45, "nr": 72, "grids": 3, "solves": 6, "precision": 1,
         "steps": 4, "resistive": True},
        # a request of the serving loop on a grid that is loaded: new upstream, initial state, derived fields, steps
        {"name": "request_24_mixed", "kind": "request", "na": 24, "nr": 40, "precision": 1, "steps": 50,
         "resistive": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "box", "box", "boxes", "shells", "shells", "request"])
    precision = rng.randrange(2)
    if kind == "box":
        resistive = rng.random() < 0.25
        c = {"kind": kind, "nx": _log_int(rng, 8, 96), "ny": _log_int(rng, 8, 96), "nz": _log_int(rng, 8, 128),
             "precision": precision, "steps": 2 if resistive else rng.choice([4, 10])}
        if resistive:
            c.update(nx=_log_int(rng, 16, 64), ny=_log_int(rng, 16, 64), nz=_log_int(rng, 16, 64), resistive=True)
        elif rng.random() < 0.25:
            c["artificial"] = True
        return c
    if kind == "boxes":
        return {"kind": kind, "solves": rng.randint(2, 24), "sizes": rng.randrange(1, 1 << 20), "precision": precision,
                "steps": rng.choice([4, 10])}
    if kind == "request":
        return {"kind": kind, "na": _log_int(rng, 8, 32), "nr": _log_int(rng, 12, 48), "precision": precision,
                "steps": rng.choice([10, 50]), "resistive": rng.random() < 0.5}
    grids = rng.randint(1, 3)
    return {"kind": kind, "na": _log_int(rng, 8, 44), "nr": _log_int(rng, 12, 72), "grids": grids,
            "solves": grids * rng.randint(1, 2), "precision": precision, "steps": rng.choice([2, 4, 10]),
            "resistive": rng.random() < 0.5}


# ------------------------------------------------------------------ what a case holds
def _box_sizes(case):
    """Cells per axis of every box: 24 to 64 along x and y, 24 to 128 along z."""
    if case["kind"] == "box":
        return [(case["nx"], case["ny"], case["nz"])]
    r = random.Random(case["sizes"])
    return [(_log_int(r, 24, 64), _log_int(r, 24, 64), _log_int(r, 24, 128)) for _ in range(case["solves"])]


def _box_constants(case):
    kw = dict(cfl=0.4)
    if case.get("resistive"):
        kw.update(resistive=True, res_rtol=1e-10, res_max_it=2000)
    if case.get("artificial"):
        kw.update(arti_eta_max=1e-4, arti_J_start=1.0, arti_J_on=8.0)
    return reference_constants(**kw)


def _eta(geom):
    return S.resistivity_eta(geom, reference_constants())


def _shell_cases(case, seed):
    """The shells of a case: `grids` grids around (na, nr), the solves dealt
    over them, each with its own upstream conditions drawn from the seed."""
    r = random.Random(seed)
    out = []
    for s in range(case.get("solves", 1)):
        g = s % case.get("grids", 1)
        na, nr = case["na"] - 3 * g if case["na"] > 16 else case["na"] + g, case["nr"] + 5 * g
        up = (r.uniform(2.0, 6.0) * 4.031e5, M.UPSTREAM[1], r.uniform(0.5, 3.0) * 4e7, M.UPSTREAM[3], 0.0, 0.0, 0.0,
              0.0, r.uniform(-0.4, 0.4) * 1e-9)
        kw = dict(resistive=True, **M.ETA_CONFIG) if case["resistive"] else dict(resistive=False)
        out.append(M.ShellCase(na=na, nr=nr, upstream=up, na_fraction=r.uniform(1e-4, 1e-2), **kw))
    return out


class _Holder:
    """Device memory of a solve as an array, keeping the solve alive."""

    def __init__(self, owner, ptr, shape, strides, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": tuple(shape), "strides": tuple(strides),
                                         "typestr": typestr, "version": 2}


def _views(owner, cells, precision, view):
    """The blocks' conserved state on the cells (blocks, 10, i, j, k) and their
    face fluxes on the owned index box (blocks, 3, i, j, k); view(field, block,
    comp) gives an array's address, ghost width and strides."""
    es, typestr = (4, "<f4") if precision else (8, "<f8")
    out = []
    n = cells[0]
    for fields, ext in (((("U_H", 5), ("U_NA", 5)), n),
                        ((("B_XI", 1), ("B_ETA", 1), ("B_ZETA", 1)), tuple(v + 1 for v in n))):
        at = [[view(f, b, c) for f, nc in fields for c in range(nc)] for b in range(len(cells))]
        base, G, si, sj = at[0][0]
        first = base + es * (G * si + G * sj + G)
        cstep = at[0][1][0] - base
        bstep = at[1][0][0] - base if len(cells) > 1 else cstep * len(at[0])
        for b, row in enumerate(at):
            for q, (p, g, i, j) in enumerate(row):
                assert (p, g, i, j) == (base + b * bstep + q * cstep, G, si, sj)
        h = _Holder(owner, first, (len(cells), len(at[0])) + tuple(ext), (bstep, cstep, si * es, sj * es, es), typestr)
        out.append(torch.as_tensor(h, device="cuda"))
    return out


def _device_view(call):
    def view(field, block, comp):
        p, G, si, sj = ctypes.c_void_p(), ctypes.c_int32(), ctypes.c_int64(), ctypes.c_int64()
        ext = (ctypes.c_int32 * 3)()
        capi.check(call(capi.FIELD_ID[field], block, comp, ctypes.byref(p), ctypes.byref(G), ctypes.byref(si),
                        ctypes.byref(sj), ext), "device view")
        return p.value, G.value, si.value, sj.value

    return view


class _Solve:
    """One solve in a context of its own, advanced by Context.step."""

    def __init__(self, ctx, cells, precision, steps):
        self.ctx, self.steps = ctx, steps
        self.out = _views(ctx, cells, precision, _device_view(lambda *a: capi.lib().mhd_device_view(ctx.ctx, *a)))

    def run(self):
        dt = self.ctx.step(self.steps)
        return [dt] + self.out


class _Batch:
    """Solves advanced together: a request to each, the steps, a poll."""

    def __init__(self, batch, slots, cells, precision, steps):
        self.batch, self.slots, self.steps = batch, slots, steps
        self.out = []
        for slot, c in zip(slots, cells):
            self.out += _views(batch, c, precision,
                               _device_view(lambda *a, s=slot: capi.lib().mhd_batch_device_view(batch.b, s, *a)))

    def run(self):
        for slot in self.slots:
            self.batch.request(slot, self.steps)
        self.batch.run(self.steps)
        self.batch.poll()
        return self.out


class _Request(_Batch):
    """A request on a loaded grid: its upstream conditions and initial state
    set on the device, the ghost layers filled, the derived fields refreshed,
    its steps taken."""

    def __init__(self, batch, slot, case, k, precision, steps):
        super().__init__(batch, [slot], [case.cells], precision, steps)
        self.case, self.k = case, k
        self.uh, self.un = M.initial_state(case, k)

    def run(self):
        b, slot, n = self.batch, self.slots[0], self.case.cells[0]
        capi.check(capi.lib().mhd_batch_set_constants(b.b, slot, ctypes.byref(self.k)), "set constants")
        lo = (-NGHOST,) * 3
        hi = tuple(c + NGHOST for c in n)
        for blk in range(6):
            b.fill(slot, "U_H", self.uh, lo, hi, block=blk)
            b.fill(slot, "U_NA", self.un, lo, hi, block=blk)
            for ax, f in enumerate(("B_XI", "B_ETA", "B_ZETA")):
                b.fill(slot, f, [0.0], lo, tuple(h + (a == ax) for a, h in enumerate(hi)), block=blk)
        b.sync(slot, "UCELL")
        b.sync(slot, "BFACE")
        b.prepare(slot)
        return super().run()


def prepare(case, seed):
    precision, steps = case["precision"], case["steps"]
    if case["kind"] in ("box", "boxes"):
        k = _box_constants(case)
        sizes = _box_sizes(case)
        if case["kind"] == "box":
            target = Context([sizes[0]], NGHOST, k, precision=precision)
            slots, slot_args = [0], [()]
        else:
            target = Batch(len(sizes), precision)
            slots = [target.add_periodic(n, NGHOST, k) for n in sizes]
            slot_args = [(s,) for s in slots]
        for q, (n, sa) in enumerate(zip(sizes, slot_args)):
            nodes, state = S.cube_state(n, solve_id=1000 * (seed % (1 << 40)) + q)
            target.setup_geometry(*sa, nodes)
            if case.get("resistive"):
                for name, a in _eta(_geometry(n)).items():
                    target.upload(*sa, name.upper(), a.data, a.lo, a.hi)
            for name in STATE:
                a = state[name]
                target.upload(*sa, FIELD[name], a.data, a.lo, a.hi)
            target.sync(*sa, "UCELL")
            target.sync(*sa, "BFACE")
            target.prepare(*sa)
        if case["kind"] == "box":
            return _Solve(target, [sizes[0]], precision, steps)
        return _Batch(target, slots, [[n] for n in sizes], precision, steps)
    cases = _shell_cases(case, seed)
    ks = [M.constants(c) for c in cases]
    if case["kind"] == "shells" and len(cases) == 1:
        ctx = M.context(cases[0], precision=precision, k=ks[0], topologies=_topologies)
        return _Solve(ctx, cases[0].cells, precision, steps)
    batch = Batch(len(cases), precision)
    slots, first = [], {}
    for c, k in zip(cases, ks):
        grid = (c.na, c.nr)
        if grid in first:
            slot = batch.add_like(first[grid], k)
        else:
            d = SolveDesc(c.cells, NGHOST, k, precision=precision, topology=_topologies.get(c))
            slot = first[grid] = batch.add(d)
        M.set_up(batch, c, slot=slot, k=k)
        batch.prepare(slot)
        slots.append(slot)
    if case["kind"] == "request":
        return _Request(batch, slots[0], cases[0], ks[0], precision, steps)
    return _Batch(batch, slots, [c.cells for c in cases], precision, steps)


def run(state):
    return state.run()


def work(case):
    """Bytes and operations of a pass.  Per cell and step: 10 conserved values
    and 3 face fluxes read and written, and the static fields (metric 10 in
    double; 9 face areas and lengths' worth of Hall and Hodge data, 18 + 36
    reconstruction weights, 9 edge vectors, 3 tapers, 3 background fluxes,
    cell centres and photo rate 4) read once; with the implicit substep one
    application of its operator (21 values per cell)."""
    es = 4 if case["precision"] else 8
    if case["kind"] in ("box", "boxes"):
        cells = sum(a * b * c for a, b, c in _box_sizes(case))
    else:
        cells = sum(c.cell_count() for c in _shell_cases(case, 0))
    words = 2 * 13 + 12 + 18 + 36 + 9 + 3 + 3 + 4
    per_step = words * es + 10 * 8
    if case.get("resistive"):
        per_step += 21 * 8
    return {"bytes": float(cells) * per_step * case["steps"], "flops": 1500.0 * cells * case["steps"]}


# ------------------------------------------------------------------ the step in 64 bits
# One periodic block, whole-array torch: index 0 .. n - 1 of every location,
# neighbours by periodic shifts.
def _geometry(n):
    lo, x, y, z = S.cube_nodes(n, 0.05)
    return S.Geometry(n, lo, x, y, z)


def _m(a, ax):  # value one index lower
    return torch.roll(a, 1, ax)


def _p(a, ax):  # value one index higher
    return torch.roll(a, -1, ax)


class _Exact:
    def __init__(self, case, seed):
        self.n = n = _box_sizes(case)[0]
        self.c = c = _box_constants(case)
        self.dev = dev = "cuda" if torch.cuda.is_available() else "cpu"
        geom = _geometry(n)
        nodes = S.Nodes(n, *S.cube_nodes(n, 0.05))
        st = S.orszag_tang_state(nodes, solve_id=1000 * (seed % (1 << 40)))

        def own(a):
            return torch.from_numpy(np.ascontiguousarray(a.data[a.sl((0, 0, 0), n)])).to(dev).movedim(-1, 0)

        f = geom.fields
        self.U = [own(st["U_H"]), own(st["U_Na"])]
        self.B = [own(st[q])[0] for q in ("B_xi", "B_eta", "B_zeta")]
        self.JD = [own(f[q]) for q in ("JDxi", "JDet", "JDze")]
        self.Jac = own(f["Jac"])[0]
        self.area = [own(f[q])[0] for q in ("Area_xi", "Area_eta", "Area_zeta")]
        self.dl = [own(f[q])[0] for q in ("dl_xi", "dl_eta", "dl_zeta")]
        self.dr = [own(f[q]) for q in ("dr_xi", "dr_eta", "dr_zeta")]
        self.beta = [own(f[q])[0] for q in ("beta_xi", "beta_eta", "beta_zeta")]
        self.alpha = [own(f[q])[0] for q in ("alpha_xi", "alpha_eta", "alpha_zeta")]
        self.WB, self.WJ = own(f["Bcell_from_Bface_w"]), own(f["Jcell_from_Jedge_w"])
        self.photo = own(S.photo_rate(geom)[1])[0]
        self.xyz = [own(f[q])[0] for q in ("cell_x", "cell_y", "cell_z")]
        self.corner = [torch.from_numpy(q).to(dev) for q in S.uniform_state(gamma=c.gamma)]
        self.eta = [own(a)[0] for a in _eta(geom).values()] if case.get("resistive") else None
        self.An = [torch.sqrt((j * j).sum(0)) for j in self.JD]
        self.K = [0.5 * (j + _p(j, a + 1)) for a, j in enumerate(self.JD)]  # JD averaged to the cells
        self.derived()

    def density_number(self, rH, rN):
        c = self.c
        nH, nN = rH.clamp(min=0) / c.M_H * c.M_ref, rN.clamp(min=0) / c.M_Na * c.M_ref
        ne = nH + nN
        eff = torch.sqrt(ne * ne + c.ne_hall_floor ** 2)
        return nH, nN, ne, eff

    def curl_current(self, B):
        """alpha C^T (beta B) on the edges."""
        b = [x * y for x, y in zip(self.beta, B)]
        cc = [(_m(b[1], 2) - b[1]) + (b[2] - _m(b[2], 1)), (b[0] - _m(b[0], 2)) + (_m(b[2], 0) - b[2]),
              (_m(b[0], 1) - b[0]) + (b[1] - _m(b[1], 0))]
        return [x * a for x, a in zip(cc, self.alpha)]

    @staticmethod
    def curl(E):
        """Circulation of the edge values around the faces."""
        return [(E[1] - _p(E[1], 2)) + (_p(E[2], 1) - E[2]), (_p(E[0], 2) - E[0]) + (E[2] - _p(E[2], 0)),
                (E[0] - _p(E[0], 1)) + (_p(E[1], 0) - E[1])]

    def cells(self, U, Bc, Jc, K, Jac):
        """The derived cell fields from the conserved states, B and J at the cells."""
        c = self.c
        V, p, T = [], [], []
        for q, coeff in zip(U, (c.state_coeff_H, c.state_coeff_Na)):
            rho = q[0].clamp(min=1e-12)
            V.append(q[1:4] / rho)
            p.append(((c.gamma - 1) * (q[4] - 0.5 * rho * (V[-1] ** 2).sum(0)).clamp(min=0)).clamp(min=1e-12))
            T.append(p[-1] / (rho * coeff))
        nH, nN, ne, eff = self.density_number(U[0][0], U[1][0])
        up = (nH * V[0] + nN * V[1]) / ne
        ucon = [(k * up).sum(0) / (Jac.abs() + 1e-30) for k in K]
        JxB = torch.linalg.cross(Jc, Bc, dim=0)
        al = c.hall_coef / eff
        return dict(V=V, p=p, T=T, up=up, num=(nH, nN, eff), ucon=ucon, JxB=JxB, ehc=al * JxB,
                    hb=al.abs() * torch.sqrt((Bc * Bc).sum(0)))

    def derived(self):
        c, B = self.c, self.B
        s = [v for a in range(3) for v in (-B[a], _p(B[a], a))]
        self.Bc = torch.stack([sum(self.WB[6 * x + q] * s[q] for q in range(6)) for x in range(3)])
        self.J = J = self.curl_current(B)
        q = []
        for a, (u, v) in enumerate(((1, 2), (0, 2), (0, 1))):
            q += [J[a], _p(J[a], u), _p(J[a], v), _p(_p(J[a], u), v)]
        self.Jc = torch.stack([sum(self.WJ[12 * x + e] * q[e] for e in range(12)) for x in range(3)])
        self.cell = self.cells(self.U, self.Bc, self.Jc, self.K, self.Jac)
        B2, best = (self.Bc * self.Bc).sum(0), math.inf
        for U in self.U:
            rho = U[0].clamp(min=1e-2)
            V = U[1:4] / rho
            cs2 = c.gamma * (c.gamma - 1) * (U[4] - 0.5 * rho * (V * V).sum(0)) / rho
            den = 0
            for a in range(3):
                for nn, An in ((self.JD[a] / self.An[a], self.An[a]),
                               (_p(self.JD[a] / self.An[a], a + 1), _p(self.An[a], a))):
                    bn, un = (self.Bc * nn).sum(0), (V * nn).sum(0)
                    t = cs2 + c.inver_MA2 * B2 / rho
                    cf = torch.sqrt(0.5 * (t + torch.sqrt((t * t - 4 * cs2 * c.inver_MA2 * bn * bn / rho).clamp(min=0))))
                    den = den + (un.abs() + cf) * An
            best = min(best, float((c.CFL * self.Jac.abs() / den).min()))
        self.dt = best

    def pad(self, t):
        """Two ghost layers of periodic images around the last three axes."""
        for ax in (-3, -2, -1):
            t = torch.cat([t.narrow(ax, t.shape[ax] - 2, 2), t, t.narrow(ax, 0, 2)], ax)
        return t

    def emf(self):
        """The total EMF on the edges.  The conserved state's ghost cells that
        lie beyond two or three faces at once are never filled: they keep the
        uniform upstream state, so the edges along the box's own edges are
        evaluated with ghost layers, and an edge's images then averaged (the
        Hall EMF takes the image at index 0)."""
        c, pad, n = self.c, self.pad, self.n
        out = []
        for ax in range(3):
            i = torch.arange(-2, n[ax] + 2, device=self.dev)
            out.append(((i < 0) | (i >= n[ax])).view([-1 if q == ax else 1 for q in range(3)]).int())
        stale = out[0] + out[1] + out[2] > 1
        U = [torch.where(stale, q.view(5, 1, 1, 1), pad(u)) for u, q in zip(self.U, self.corner)]
        cell = self.cells(U, pad(self.Bc), pad(self.Jc), [pad(k) for k in self.K], pad(self.Jac))
        B, ucon = [pad(b) for b in self.B], cell["ucon"]
        area, dl, dr, J = ([pad(x) for x in v] for v in (self.area, self.dl, self.dr, self.J))
        bt = [0.5 * (B[a] + _p(B[a], a)) for a in range(3)]

        def flux(ba, fa):  # of the component ba of B through the face family fa
            uL, uR = _m(ucon[fa], fa), ucon[fa]
            bL, bR = _m(bt[ba], fa), bt[ba]
            GL, GR = uL * bL - _m(ucon[ba], fa) * B[fa], uR * bR - ucon[ba] * B[fa]
            return 0.5 * (GL + GR) - 0.5 * torch.maximum(uL.abs(), uR.abs()) * (bR - bL)

        pen = cell["p"][0] + cell["p"][1]
        for a in range(3):
            pen = 0.5 * (pen + _m(pen, a))
        pc = (c.rho_ref * c.U_ref) / (c.q_e * c.L_ref * c.B_ref * c.n_ref)
        E = []
        for a in range(3):
            u, v = (a + 1) % 3, (a + 2) % 3  # E_a from the faces of families u (flux of B_v) and v (flux of B_u)

            def around(f, x):  # over the four cells at the edge
                y = f(x, _m(x, u))
                return f(y, _m(y, v))

            def add(x, y):
                return x + y

            eu, ev = -flux(v, u), flux(u, v)
            e = 0.25 * (eu + _m(eu, v) + ev + _m(ev, u))
            mu, mv = around(torch.maximum, ucon[u].abs()), around(torch.maximum, ucon[v].abs())
            du, dv = B[v] - _m(B[v], u), B[u] - _m(B[u], v)
            e = e + 0.5 * (0.5 * mu * du - 0.5 * mv * dv)
            if c.ambipolar:
                eff = self.density_number(0.25 * around(add, U[0][0]), 0.25 * around(add, U[1][0]))[3]
                e = e - pc * (_p(pen, a) - pen) / eff
            if c.arti_eta_max > 0:
                mag = J[a].abs() / torch.sqrt((dr[a] ** 2).sum(0)).clamp(min=1e-30)
                q = ((mag - c.arti_J_start) / (c.arti_J_on - c.arti_J_start)).clamp(0, 1)
                e = e + c.arti_eta_max * q * q * (3 - 2 * q) * J[a]
            h = sum(0.25 * around(add, cell["ehc"][x]) * dr[a][x] for x in range(3))
            hb = around(torch.maximum, cell["hb"])
            L = dl[a].clamp(min=1e-14)
            iu = L / (0.5 * (area[v] + _m(area[v], u))).clamp(min=1e-14)
            iv = L / (0.5 * (area[u] + _m(area[u], v))).clamp(min=1e-14)
            h = h + 0.05 * hb * (iu * iu * du - iv * iv * dv)
            for ax in (0, 1, 2):  # index 0 .. n - 1, an image at n averaged in
                first = e.narrow(ax, 2, n[ax]).clone()
                if ax != a:
                    first.narrow(ax, 0, 1).copy_(0.5 * (e.narrow(ax, 2, 1) + e.narrow(ax, 2 + n[ax], 1)))
                e, h = first, h.narrow(ax, 2, n[ax])
            E.append(e + h)
        return E

    def fluid(self):
        c, g = self.c, self.c.gamma
        cell, out = self.cell, []
        dpe = 0
        if c.ambipolar:
            pe = cell["p"][0] + cell["p"][1]
            for a in range(3):  # the kernel's coefficients: the face below and the face of the cell
                dpe = dpe + 0.5 * (_m(self.JD[a], a + 1) + self.JD[a]) / self.Jac.abs() * (0.5 * (_p(pe, a) - _m(pe, a)))
        x, y, z = self.xyz
        vst = torch.where((x < 0) & (torch.sqrt(y * y + z * z) < 1), 1e-5, 5e-5)
        for s in range(2):
            U, V, p = self.U[s], cell["V"][s], cell["p"][s]
            rho = U[0]
            re = p / (g - 1) + 0.5 * rho * (V * V).sum(0)
            cs = torch.sqrt((g * p / rho.clamp(min=1e-30)).clamp(min=0))
            Q = torch.cat([rho[None], rho * V, re[None]])
            r = torch.zeros_like(U)
            for a in range(3):
                k, sk = self.JD[a], self.An[a]
                L = lambda t: torch.roll(t, 1, t.dim() - 3 + a)  # noqa: E731
                un, unL = (k * V).sum(0), (k * L(V)).sum(0)

                def phys(q, vel, pr):
                    return torch.cat([(q[0] * vel)[None], q[1:4] * vel + k * pr, ((q[4] + pr) * vel)[None]])

                rad = torch.maximum(unL.abs() + L(cs) * sk, un.abs() + cs * sk)
                F = 0.5 * (phys(L(Q), unL, L(p)) + phys(Q, un, p)) - 0.5 * rad * (Q - L(Q))
                r = r - (_p(F, a + 1) - F) / self.Jac
            nH, nN, eff = cell["num"]
            nS = nN if s else nH
            chi = nS / eff
            sub = torch.linalg.cross(V - cell["up"], self.Bc, dim=0)
            mom = c.momentum_induce_coeff * nS * sub + c.momentum_hall_coeff * chi * cell["JxB"] - chi * dpe
            M0 = c.M_Na if s else c.M_H
            a4 = c.L_ref / c.U_ref
            a5 = 3 * c.L_ref * c.k_Boltz * c.n_ref / (c.rho_ref * c.U_ref ** 3)
            u2 = (V * V).sum(0)
            e = (mom * V).sum(0) - a4 * rho * u2 * vst + a4 * rho * u2 * (c.M_Na / (M0 + c.M_Na)) * vst
            e = e + a5 * nS * vst * (1000.0 - cell["T"][s] * c.T_ref) * (M0 / (M0 + c.M_Na))
            r[1:4] += mom - a4 * rho * V * vst
            if s:
                r[0] += (c.L_ref / c.U_ref) * (c.m_Na / c.rho_ref) * 1e6 * self.photo
                e = e + 1e6 * c.L_ref * c.k_Boltz / (c.rho_ref * c.U_ref ** 3 * (g - 1)) * self.photo * 1000.0
            r[4] += e
            out.append(U + self.dt * r)
        return out

    def substep(self, dt):
        """(I + dt eta alpha C^T beta C) E = eta J(B*), B = B* - dt curl E, by
        conjugate gradients in the inner product weighted by 1 / (eta alpha)."""
        eta, al = torch.stack(self.eta), torch.stack(self.alpha)
        on = (eta > 0) & (al > 0)
        W = torch.where(on, 1 / (eta * al).clamp(min=1e-300), 0.0)

        def A(e):
            dB = [-dt * t for t in self.curl(list(e))]
            return torch.where(on, e - eta * torch.stack(self.curl_current(dB)), 0.0)

        r = torch.where(on, eta * torch.stack(self.curl_current(self.B)), 0.0)
        x, p = torch.zeros_like(r), r.clone()
        rho, r0 = (W * r * r).sum(), float(r.norm())
        for it in range(5000):
            if float(r.norm()) <= 1e-14 * r0:
                break
            q = A(p)
            a = rho / (W * p * q).sum()
            x, r = x + a * p, r - a * q
            new = (W * r * r).sum()
            p, rho = r + (new / rho) * p, new
        self.B = [b - dt * t for b, t in zip(self.B, self.curl(list(x)))]

    def step(self):
        E, dt = self.emf(), self.dt
        U = self.fluid()
        self.B = [b - dt * t for b, t in zip(self.B, self.curl(E))]
        self.U = U
        if self.eta is not None:
            self.substep(dt)
        self.derived()
        return dt


def exact(case, seed):
    if case["kind"] != "box" or case["nx"] * case["ny"] * case["nz"] > 300000:
        return None
    x = _Exact(case, seed)
    for _ in range(case["steps"]):
        dt = x.step()
    B = torch.nn.functional.pad(torch.stack(x.B)[None], (0, 1, 0, 1, 0, 1), mode="circular")
    return [dt, torch.cat(x.U)[None], B]
