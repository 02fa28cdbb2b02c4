"""Timed cases of the PIC-MCC path: what a program using scdat_b200 has it do, each through the
library's public entry points on a seeded synthetic plasma.

Every case is a box of hex cells split into 6 tets with a conducting or dielectric body in its
middle, electrons and H+, and periodic outer faces (at the wall potential), so that the plasma
stays in the box however often a case is run.  The body is at -10 V against Te = 1 eV (or floats
near -15 V against 5 eV), so it collects almost nothing from one run to the next.

Kinds: "step" one or more whole steps and what a driver reads back after them; "push" the
particle stage alone; "solve" the field stage alone for a new nodal charge; "batch" a sweep of
scenarios stepped together; "adjoint" a differentiated window; "pcg" the solver on a caller's own
matrix.  Results of the FP64 form are kept as FP64.  The precision form stores its particles in
FP32, and its fields are good to that, so its results are kept as FP32.  The particles themselves stay
on the GPU, as a driver leaves them there: where they went shows in the nodal charge, the ledger
and the energy of this pass and the next.

`exact` restates a case's first pass in plain FP64 torch: the tets are found from a point's cell
and the order of its local coordinates, the Laplacian from the edge weights per direction."""
import ctypes as C
import math

import numpy as np
import torch

from scdat_b200 import capi

QE, ME, MP, EPS0 = 1.602176634e-19, 9.1093837015e-31, 1.67262192369e-27, 8.8541878128e-12
PERMS = ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0))  # the 6 tets of a cell
HOST_PARTICLES = 3_000_000  # up to here the particles come from host arrays, above from the box seeder


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def _case(kind, nx, ny, nz, ppc, form, **kw):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, ppc=ppc, form=form, steps=1, precond="jacobi", rtol=1e-8, mcc=0, sort=0,
             ion_sort=0, deposit="linear", surface=False)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: the 8^3 probe box of the CPU baseline, one FP64 step at a time
        dict(_case("step", 8, 8, 8, 20, "fp64", mcc=2, sort=8), name="step fp64 8^3"),
        # a small scenario of a sweep in the precision form, one step at a time
        dict(_case("step", 16, 16, 16, 8, "mixed", rtol=1e-10, mcc=2, sort=4), name="step mixed 16^3"),
        # the plain FP64 benchmark configuration: 32^3 cells, 20 particles per cell and species
        dict(_case("step", 32, 32, 32, 20, "fp64", mcc=2, sort=8), name="step fp64 32^3"),
        # the precision benchmark's density, solver and re-sort settings on a 64^3 box (33 M particles)
        dict(_case("step", 64, 64, 64, 64, "mixed", precond="multigrid", rtol=1e-10, mcc=2, sort=1, ion_sort=16),
             name="step mixed 64^3"),
        # surface charging: a dielectric body that floats, secondaries, no collisions, an uneven box
        dict(_case("step", 47, 31, 38, 16, "mixed", rtol=1e-10, sort=4, ion_sort=16, surface=True),
             name="surface mixed 47x31x38"),
        # the particle stage alone at the differentiation workload's size and density, FP64 (7 M particles)
        dict(_case("push", 48, 48, 48, 32, "fp64"), name="push fp64 48^3"),
        # the same stage in the precision form on a ragged box, with the quadrature deposit
        dict(_case("push", 37, 53, 29, 13, "mixed", deposit="gauss3"), name="push mixed 37x53x29"),
        # the field stage alone, as a driver with its own particles calls it: multigrid, precision form
        dict(_case("solve", 64, 64, 64, 0, "mixed", precond="multigrid", rtol=1e-10), name="solve mixed 64^3"),
        # and Jacobi-CG in FP64, the default solver, on a ragged box
        dict(_case("solve", 33, 27, 41, 0, "fp64"), name="solve fp64 33x27x41"),
        # a sweep: 8 scenarios of uneven size, density and temperature in one batch, 4 steps a call
        dict(_case("batch", 16, 32, 0, 16, "mixed", steps=4, rtol=1e-10, mcc=2, sort=4), count=8,
             name="batch of 8, 16-32 cells"),
        # reverse mode: a window over a floating body with secondaries, checkpointed
        dict(_case("adjoint", 16, 16, 16, 8, "fp64", steps=4, rtol=1e-12, surface=True), checkpoint=2,
             name="adjoint fp64 16^3, 4 steps"),
        # the solver on a system the caller assembled and holds on the GPU
        dict(_case("pcg", 48, 48, 48, 0, "fp64"), name="pcg fp64 48^3"),
    ]


def _loguniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "push", "push", "solve", "solve", "batch", "adjoint", "pcg"])
    form = rng.choice(["fp64", "mixed"])
    e = _loguniform(rng, 8, 56)
    n = [max(6, int(round(e * rng.uniform(0.75, 1.25)))) for _ in range(3)]
    if kind == "batch":
        lo = rng.randint(8, 20)
        return dict(_case(kind, lo, lo + rng.randint(2, 12), 0, rng.randint(8, 24), "mixed", steps=rng.randint(1, 6),
                          rtol=1e-10, mcc=rng.choice([1, 2]), sort=4), count=rng.randint(2, 10))
    if kind == "adjoint":
        steps = rng.randint(2, 6)
        return dict(_case(kind, *(min(20, v) for v in n), rng.randint(2, 10), "fp64", steps=steps, rtol=1e-12,
                          surface=True), checkpoint=rng.randint(1, steps))
    if kind == "pcg":
        return _case(kind, *n, 0, "fp64")
    mg = form == "mixed" and min(n) >= 16 and rng.random() < 0.5
    precond, rtol = ("multigrid" if mg else "jacobi"), (1e-10 if form == "mixed" else 1e-8)
    if kind == "solve":
        return _case(kind, *n, 0, form, precond=precond, rtol=rtol)
    ppc = min(_loguniform(rng, 4, 64), max(2, 12_000_000 // (2 * n[0] * n[1] * n[2])))
    deposit = rng.choice(["linear", "linear", "linear", "nearest", "gauss3"])
    if kind == "push":
        return _case(kind, *n, ppc, form, deposit=deposit)
    sort = rng.choice([0, 1, 4, 8])
    return _case(kind, *n, ppc, form, precond=precond, rtol=rtol, deposit=deposit, sort=sort, ion_sort=4 * sort,
                 mcc=rng.choice([0, 1, 2]), surface=rng.random() < 0.25)


# ---------------------------------------------------------------------------------------------
# what a program has in hand before the call
# ---------------------------------------------------------------------------------------------
class _Species:
    def __init__(self, q, m, w):
        self.q, self.m, self.w = q, m, w


def _plasma(case):
    """Cell edge, time step, density, Te = Ti, bias of a case."""
    if case["surface"] and case["kind"] != "adjoint":  # the large surface-charging run's plasma
        n, te, bias = 1e9, 5.0, -15.0
        return math.sqrt(EPS0 * te / (n * QE)), 0.1 / math.sqrt(n * QE * QE / (EPS0 * ME)), n, te, bias
    h = 1.6 / case["nx"] if case["nx"] > 32 else 0.05
    return h, 2e-8, 1e10, 1.0, (-8.0 if case["surface"] else -10.0)


def _body(n):
    return tuple(((a - max(1, a // 4)) // 2, (a - max(1, a // 4)) // 2 + max(1, a // 4)) for a in n)


def _cells(n, body):
    """(cells, 3) index triples of the meshed cells, x fastest."""
    k, j, i = np.meshgrid(*(np.arange(a) for a in n[::-1]), indexing="ij")
    ijk = np.stack([i.ravel(), j.ravel(), k.ravel()], 1)
    inside = np.ones(len(ijk), bool)
    for a in range(3):
        inside &= (ijk[:, a] >= body[a][0]) & (ijk[:, a] < body[a][1])
    return ijk[~inside]


def _particles(n, body, h, ppc, te, m, seed, species):
    """Uniform positions in every meshed cell, a Maxwellian, and each particle's tet."""
    rng = np.random.default_rng([seed, species])
    cells = _cells(n, body)
    c = np.repeat(np.arange(len(cells)), ppc)
    u = rng.random((len(c), 3))
    x = (cells[c] + u) * h
    v = rng.standard_normal((len(c), 3)) * math.sqrt(te * QE / m)
    o = np.argsort(-u, axis=1, kind="stable")
    tet = 6 * c + 2 * o[:, 0] + (o[:, 1] > o[:, 2])
    return x, v, tet.astype(np.int32)


def _context(case, seed, n=None, plasma=None):
    n = n or (case["nx"], case["ny"], case["nz"])
    h, dt, density, te, bias = plasma or _plasma(case)
    body = _body(n)
    mesh = capi.kuhn_box_mesh(n, h, body=body, bias=bias)
    dep = {"nearest": capi.DEP_NEAREST, "linear": capi.DEP_LINEAR, "gauss3": capi.DEP_GAUSS3}[case["deposit"]]
    dom = capi.Domain(mesh["xyz"], mesh["tet"], mesh["dirichlet"], dt,
                      precision=capi.PREC_MIXED if case["form"] == "mixed" else capi.PREC_FP64, face_bc=(2,) * 6,
                      deposit_kernel=dep, pcg_rtol=case["rtol"], pcg_max_iter=20000, sort_interval=case["sort"])
    ppc = case["ppc"]
    if ppc:
        sp = [_Species(-QE, ME, density * h ** 3 / ppc), _Species(QE, MP, density * h ** 3 / ppc)]
        dom.set_species(sp)
        for s in range(2):
            if 2 * ppc * n[0] * n[1] * n[2] <= HOST_PARTICLES:
                dom.set_particles(s, *_particles(n, body, h, ppc, te, sp[s].m, seed, s))
            else:
                dom.seed_box(s, n, h, body, ppc, te, 1000 * seed + 17)
        if case["ion_sort"]:
            dom.set_species_sort_interval(1, case["ion_sort"])
        if case["mcc"]:
            for s in range(2):
                dom.set_elastic(s, 1e14, 1e-19, mode=case["mcc"])
    if case["precond"] == "multigrid":
        dom.set_preconditioner(capi.PRECOND_MULTIGRID)
    if case["surface"]:
        dom.set_surface_circuit(tuple(b[0] * h for b in body), tuple(b[1] * h for b in body), eps_r=3.0,
                                thickness=1e-3, v0=bias)
        dom.set_secondary_emission(1, 2.0, 300.0)
    dom.set_potential(mesh["phi"])
    dom.solve_field()
    return dom, mesh


class _Host:
    """Pinned buffers a driver keeps to read one context's fields into."""

    def __init__(self, dom, form):
        self.dom = dom
        self.raw = [torch.empty(k * dom.N, dtype=torch.float64, pin_memory=True) for k in (1, 1, 3)]
        self.kept = [torch.empty(r.numel(), dtype=torch.float32) for r in self.raw] if form == "mixed" else self.raw

    def read(self, want=(True, True, True)):
        ptr = [C.c_void_p(r.data_ptr()) if w else None for r, w in zip(self.raw, want)]
        self.dom._ck(self.dom.L.scdat_get_fields(self.dom.h, *ptr))
        if self.kept is not self.raw:
            for k, r, w in zip(self.kept, self.raw, want):
                if w:
                    k.copy_(r)
        return [k if w else None for k, w in zip(self.kept, want)]


def _charge(n, h, seed, dom):
    """A nodal charge (C) whose potential is of the order of volts, noise on a smooth part."""
    rng = np.random.default_rng([seed, 7])
    amp = EPS0 * h * 4.0 / h ** 3
    t = dom.xyz / (np.array(n) * h)
    return amp * (np.prod(np.sin(np.pi * t), axis=1) / max(n) ** 2 * 8 + 0.1 * rng.standard_normal(len(t)))


def _scenarios(case, seed):
    """Sizes even over the range, the rest drawn: one Debye length a cell, dt = 0.1 / omega_pe."""
    rng = np.random.default_rng([seed, 3])
    for k in range(case["count"]):
        e = case["nx"] + round((case["ny"] - case["nx"]) * k / max(1, case["count"] - 1))
        dens, te = 10 ** rng.uniform(8, 12), 10 ** rng.uniform(-1, 1)
        yield (e, e, e), (math.sqrt(EPS0 * te / (dens * QE)), 0.1 / math.sqrt(dens * QE * QE / (EPS0 * ME)), dens, te,
                          -10.0 * te)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "pcg":
        n, body, dev = (case["nx"], case["ny"], case["nz"]), None, "cuda"
        box = _Box(n, _body(n), _plasma(case)[0], "cpu")
        rp, col, val, diag = box.csr()
        b = np.random.default_rng([seed, 5]).standard_normal(len(diag)) * EPS0 * box.h
        t = [torch.from_numpy(a).to(dev) for a in (rp, col, val, diag, b)]
        return dict(case=case, sys=t, x=torch.zeros_like(t[4]), R=len(diag), it=C.c_int32(), rel=C.c_double())
    if kind == "batch":
        doms = [_context(case, seed + 100 * k, n, pl)[0] for k, (n, pl) in enumerate(_scenarios(case, seed))]
        return dict(case=case, doms=doms, batch=capi.Batch(doms), host=[_Host(d, "mixed") for d in doms])
    dom, mesh = _context(case, seed)
    s = dict(case=case, dom=dom, host=_Host(dom, case["form"]))
    if kind == "solve":
        s["rho"] = _charge((case["nx"], case["ny"], case["nz"]), _plasma(case)[0], seed, dom)
        s["phi0"] = mesh["phi"]
    return s


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def _read(dom, host, surface=False, want=(True, True, True)):
    st = dom.stats()
    out = dict(zip(("rho", "phi", "E"), host.read(want)), ledger=dom.ledger(), energy=st["total_energy"],
               active=st["active_particles"], substeps=st["substeps"], lost=st["lost_events"],
               collisions=st["mcc_collisions"])
    if surface:
        out["V"] = dom.surface_state()["V"]
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "pcg":
        state["x"].zero_()
        ptr = [C.c_void_p(t.data_ptr()) for t in state["sys"]]
        rc = capi.load().scdat_pcg_csr(state["R"], *ptr, C.c_void_p(state["x"].data_ptr()), case["rtol"], 20000, None,
                                       C.byref(state["it"]), C.byref(state["rel"]))
        if rc:
            raise capi.ScdatError(rc, "scdat_pcg_csr")
        return state["x"]
    if kind == "batch":
        state["batch"].step(case["steps"])
        return [dict(zip(("rho", "phi", "E"), h.read()), ledger=d.ledger()) for d, h in zip(state["doms"], state["host"])]
    dom = state["dom"]
    if kind == "step":
        dom.step(case["steps"])
        return _read(dom, state["host"], case["surface"])
    if kind == "push":
        dom.push()
        return _read(dom, state["host"], want=(True, False, False))
    if kind == "solve":
        dom.set_potential(state["phi0"])
        dom.set_charge_density(state["rho"])
        dom.solve_field()
        return state["host"].read((False, True, True))
    r = dom.adjoint_window(case["steps"], case["checkpoint"], g_V=(1.0 / 6.0,) * 6, te_ev=1.0)
    return dict({k: np.float64(r[k]) for k in ("J", "dbias", "dte", "ddelta")}, flags=int(r["flags"]),
                fields=state["host"].read())


def work(case):
    """Bytes: particle state and id read and written once a step, tet connectivity and geometry once,
    node fields and charge once, the matrix once a solve."""
    def one(n, steps, solves):
        b = _body(n)
        cells = n[0] * n[1] * n[2] - (b[0][1] - b[0][0]) * (b[1][1] - b[1][0]) * (b[2][1] - b[2][0])
        nodes = (n[0] + 1) * (n[1] + 1) * (n[2] + 1)
        v = 4 if case["form"] == "mixed" else 8
        parts = 2 * case["ppc"] * cells
        byte = steps * (parts * (12 * v + 8 + 4) + (6 * cells * 112 + nodes * 8 if parts else 0))
        byte += solves * nodes * (14 * (v + 4) + 6 * 8)
        return byte, steps * parts * 150 + solves * nodes * 100

    n, k = (case["nx"], case["ny"], case["nz"]), case["kind"]
    if k == "batch":
        got = [one(m, case["steps"], case["steps"]) for m, _ in _scenarios(case, 0)]
    else:
        got = [one(n, {"solve": 0, "pcg": 0, "adjoint": 2 * case["steps"]}.get(k, case["steps"]),
                   {"push": 0, "adjoint": 2 * case["steps"]}.get(k, case["steps"]))]
    return {"bytes": sum(a for a, _ in got), "flops": sum(f for _, f in got)}


# ---------------------------------------------------------------------------------------------
# the same in plain FP64 torch
# ---------------------------------------------------------------------------------------------
class _Box:
    """The box of 6-tet cells: Dirichlet nodes, edge weights per direction, control volumes."""

    DIRS = ((1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 1, 1))

    def __init__(self, n, body, h, dev):
        self.n, self.body, self.h, self.dev = n, body, h, dev
        sx, sy = n[0] + 1, (n[0] + 1) * (n[1] + 1)
        self.stride = (1, sx, sy)
        self.N = sy * (n[2] + 1)
        cells = torch.as_tensor(_cells(n, body), device=dev)
        base = cells[:, 0] + sx * cells[:, 1] + sy * cells[:, 2]
        self.W = torch.zeros(7, self.N, dtype=torch.float64, device=dev)
        self.cv = torch.zeros(self.N, dtype=torch.float64, device=dev)
        vol = max(h ** 3 / 6.0, 1e-12)
        for p in PERMS:
            v = [(0, 0, 0)]
            for a in p:
                v.append(tuple(v[-1][q] + (q == a) for q in range(3)))
            for i in range(4):
                at = base + sum(v[i][a] * self.stride[a] for a in range(3))
                self.cv.index_add_(0, at, torch.full((len(at),), vol / 4.0, dtype=torch.float64, device=dev))
                for j in range(i + 1, 4):
                    d = tuple(v[j][a] - v[i][a] for a in range(3))
                    w = EPS0 * vol / 6.0 / max(math.sqrt(sum(d)) * h, 1e-12) ** 2
                    self.W[self.DIRS.index(d)].index_add_(
                        0, at, torch.full((len(at),), w, dtype=torch.float64, device=dev))
        idx = torch.arange(self.N, device=dev)
        ijk = (idx % sx, idx // sx % (n[1] + 1), idx // sy)
        wall = torch.zeros(self.N, dtype=torch.bool, device=dev)
        hole = torch.ones(self.N, dtype=torch.bool, device=dev)
        for a in range(3):
            wall |= (ijk[a] == 0) | (ijk[a] == n[a])
            hole &= (ijk[a] >= body[a][0]) & (ijk[a] <= body[a][1])
        self.hole, self.inner = hole, ~(wall | hole)
        self.off = [sum(d[a] * self.stride[a] for a in range(3)) for d in self.DIRS]
        self.diag = torch.zeros(self.N, dtype=torch.float64, device=dev)
        for w, o in zip(self.W, self.off):
            self.diag += w
            self.diag[o:] += w[: self.N - o]

    def csr(self):
        """Off-diagonal CSR rows and the diagonal of the interior nodes' system."""
        inner = self.inner.numpy()
        row_of = np.cumsum(inner) - 1
        rows, cols, vals = [], [], []
        for w, o in zip(self.W.numpy(), self.off):
            i = np.nonzero((w[: self.N - o] != 0) & inner[: self.N - o] & inner[o:])[0]
            rows += [row_of[i], row_of[i + o]]
            cols += [row_of[i + o], row_of[i]]
            vals += [-w[i], -w[i]]
        rows, cols, vals = (np.concatenate(a) for a in (rows, cols, vals))
        order = np.lexsort((cols, rows))
        rp = np.zeros(int(inner.sum()) + 1, np.int64)
        np.add.at(rp, rows + 1, 1)
        return (np.cumsum(rp).astype(np.int32), cols[order].astype(np.int32), vals[order],
                np.ascontiguousarray(self.diag.numpy()[inner]))

    def apply(self, x):
        y = self.diag * x
        for w, o in zip(self.W, self.off):
            y[: self.N - o] -= w[: self.N - o] * x[o:]
            y[o:] -= w[: self.N - o] * x[: self.N - o]
        return y

    def solve(self, b, x):
        """A x = b on the interior nodes, x given on the others."""
        m = self.inner.to(torch.float64)
        x, dinv = x.clone(), m / torch.where(self.diag > 0, self.diag, torch.ones_like(self.diag))
        r = m * (b - self.apply(x))
        bb = float((m * (b - self.apply(x * (1 - m)))).square().sum()) or 1.0
        z = dinv * r
        p, rz = z.clone(), torch.dot(r, z)
        for k in range(5000):
            q = m * self.apply(p)
            a = rz / torch.dot(p, q)
            x += a * p
            r -= a * q
            if k % 8 == 0 and float(r.square().sum()) <= 1e-30 * bb:
                break
            z = dinv * r
            rz, old = torch.dot(r, z), rz
            p = z + (rz / old) * p
        return x

    def field(self, phi):
        """E = -the least-squares gradient over each node's edges."""
        M = torch.zeros(self.N, 3, 3, dtype=torch.float64, device=self.dev)
        g = torch.zeros(self.N, 3, dtype=torch.float64, device=self.dev)
        for w, o, d in zip(self.W, self.off, self.DIRS):
            e = torch.tensor(d, dtype=torch.float64, device=self.dev) * self.h
            on = (w[: self.N - o] != 0).to(torch.float64)[:, None]
            df = (phi[o:] - phi[: self.N - o])[:, None]
            M[: self.N - o] += on[:, :, None] * torch.outer(e, e)
            M[o:] += on[:, :, None] * torch.outer(e, e)
            g[: self.N - o] += on * e * df
            g[o:] += on * e * df
        ok = M.diagonal(dim1=1, dim2=2).sum(1) > 0
        E = torch.zeros_like(g)
        E[ok] = -torch.linalg.solve(M[ok], g[ok])
        return E

    def locate(self, x):
        """Cell, order of the local coordinates, and whether the point is in the mesh."""
        c = torch.floor(x / self.h).to(torch.int64)
        ok = torch.ones(len(x), dtype=torch.bool, device=self.dev)
        hole = ok.clone()
        for a in range(3):
            ok &= (c[:, a] >= 0) & (c[:, a] < self.n[a])
            hole &= (c[:, a] >= self.body[a][0]) & (c[:, a] < self.body[a][1])
        return c, torch.argsort(-(x / self.h - c), dim=1, stable=True), ok & ~hole

    def bary(self, x, c, p):
        u = torch.gather(x / self.h - c, 1, p)
        return torch.stack([1 - u[:, 0], u[:, 0] - u[:, 1], u[:, 1] - u[:, 2], u[:, 2]], 1)

    def nodes(self, c, p):
        s = torch.tensor(self.stride, device=self.dev)
        v = [(c * s).sum(1)]
        for a in range(3):
            v.append(v[-1] + s[p[:, a]])
        return torch.stack(v, 1)


def _inside(lam):
    return ((lam >= -1e-8) & (lam <= 1 + 1e-8)).all(1)


def _push(box, E, x, v, q, m, w, dt, deposit, rho, nseg=10):
    """One species through one step: positions, velocities, sub-steps, which were lost; adds to rho."""
    n = len(x)
    qm, qw = q / m, q * w
    c, p, _ = box.locate(x)
    vs = v.square().sum(1).sqrt()
    rem = torch.full((n,), dt, dtype=torch.float64, device=box.dev)
    lost = torch.zeros(n, dtype=torch.bool, device=box.dev)
    live, substeps = torch.arange(n, device=box.dev), 0

    def add(c, p, lam):
        rho.index_add_(0, box.nodes(c, p).reshape(-1), lam.reshape(-1))

    while len(live):
        xi, ci, pi, ri = x[live], c[live], p[live], rem[live]
        lam = box.bary(xi, ci, pi)
        Ei = (E[box.nodes(ci, pi)] * lam[:, :, None]).sum(1)
        Em = Ei.square().sum(1).sqrt()
        acc = Em * abs(qm)
        cap = (Em > 1e-10) & (acc > 1e-10) & (vs[live] > 1.0)
        adt = torch.where(cap, torch.minimum(ri, 0.1 * vs[live] / torch.where(cap, acc, torch.ones_like(acc))), ri)
        adt = torch.minimum(torch.maximum(adt, ri * 1e-3), ri)
        vi = v[live] + Ei * (qm * adt)[:, None]
        xn = xi + vi * adt[:, None]
        v[live], x[live] = vi, xn
        le = box.bary(xn, ci, pi)
        stay = _inside(le)
        if deposit == "nearest":
            add(ci[stay], pi[stay], qw * le[stay])
        else:
            add(ci[stay], pi[stay], qw * 0.5 * (lam[stay] + le[stay]))
        gone = ~stay
        cn, pn, ok = box.locate(xn[gone])
        c[live[gone]], p[live[gone]] = torch.where(ok[:, None], cn, ci[gone]), torch.where(ok[:, None], pn, pi[gone])
        a, b, cc, pp = xi[gone][ok], xn[gone][ok], cn[ok], pn[ok]
        if deposit == "nearest":
            pts = [(1.0, qw)]
        elif deposit == "linear":
            pts = [((k + 0.5) / nseg, qw / nseg) for k in range(nseg)]
        else:
            pts = [((k + 0.5 + 0.5 * g) / nseg, qw * f / nseg) for k in range(nseg)
                   for g, f in ((-math.sqrt(0.6), 5 / 18), (0.0, 8 / 18), (math.sqrt(0.6), 5 / 18))]
        for tau, wt in pts:
            lq = box.bary(a + tau * (b - a), cc, pp)
            on = _inside(lq)
            add(cc[on], pp[on], wt * lq[on])
        lost[live[gone][~ok]] = True
        rem[live] = ri - adt
        substeps += int(stay.sum() + ok.sum())
        live = live[(rem[live] > 1e-20) & ~lost[live]]
    return x, v, lost, substeps


def _exact_step(case, seed, n, plasma, field=True):
    """A step's outputs from the seeded particles: nodal charge, potential, field, ledger, energy, counts."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    h, dt, density, te, bias = plasma
    box = _Box(n, _body(n), h, dev)
    phi = torch.where(box.hole, bias, 0.0).to(torch.float64)
    zero = torch.zeros_like(phi)
    phi = box.solve(zero, phi)
    E = box.field(phi)
    rho, ledger, energy, active, substeps, lost_n = zero.clone(), np.zeros((7, 8)), 0.0, 0, 0, 0
    L = torch.tensor([a * h for a in n], dtype=torch.float64, device=dev)
    w = density * h ** 3 / case["ppc"]
    for s, (q, m) in enumerate(((-QE, ME), (QE, MP))):
        x, v, _ = _particles(n, box.body, h, case["ppc"], te, m, seed, s)
        x, v, lost, sub = _push(box, E, torch.as_tensor(x, device=dev), torch.as_tensor(v, device=dev), q, m, w, dt,
                                case["deposit"], rho)
        ke = 0.5 * m * v.square().sum(1)
        out = ((x < 0) | (x > L)).any(1)
        _, _, ok = box.locate(torch.where(out[:, None], torch.remainder(x, L), x))
        hit = lost & ~ok  # in no tet: collected by the body
        ledger[6, 0 if q < 0 else 1] += float(hit.sum()) * q * w
        ledger[6, 3] += float(ke[hit].sum()) * max(1.0, w)
        ledger[6, 4 if q < 0 else 5] += float(hit.sum())
        energy += float(ke.sum())
        active += len(x) - int(hit.sum())
        substeps += sub
        lost_n += int(lost.sum())
    got = dict(rho=rho.cpu(), ledger=ledger, energy=energy, active=active, substeps=substeps, lost=lost_n)
    if field:
        phi = box.solve(-rho * box.cv, phi)
        got.update(phi=phi.cpu(), E=box.field(phi).reshape(-1).cpu())
    return got


def exact(case, seed):
    kind, n = case["kind"], (case["nx"], case["ny"], case["nz"])
    if kind == "adjoint" or case["steps"] > 1 or case["surface"]:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "pcg":
        box = _Box(n, _body(n), _plasma(case)[0], dev)
        b = torch.zeros(box.N, dtype=torch.float64, device=dev)
        inner = torch.nonzero(box.inner)[:, 0]
        b[inner] = torch.from_numpy(np.random.default_rng([seed, 5]).standard_normal(len(inner)) * EPS0 * box.h).to(dev)
        return box.solve(b, torch.zeros_like(b))[inner]
    if kind == "solve":
        h, _, _, _, bias = _plasma(case)
        box = _Box(n, _body(n), h, dev)
        grid = np.stack([g.ravel() for g in np.meshgrid(*(np.arange(a + 1) * h for a in n[::-1]), indexing="ij")][::-1], 1)
        rho = torch.from_numpy(_charge(n, h, seed, type("", (), {"xyz": grid}))).to(dev)
        phi = box.solve(-rho * box.cv, torch.where(box.hole, bias, 0.0).to(torch.float64))
        return [None, phi.cpu(), box.field(phi).reshape(-1).cpu()]
    if 2 * case["ppc"] * n[0] * n[1] * n[2] > HOST_PARTICLES or kind == "batch":
        return None
    return _exact_step(case, seed, n, _plasma(case), field=kind == "step")
