"""Performance cases: time steps of the generated-style programs, called
through the Python mirror of the runtime.

A case is one call pattern of a user's program on one grid.  `prepare` makes
what the program has before its time loop (runtime, uploaded fields,
transmissibilities, index sets), `run` makes one pass of the loop from the
same start state and returns the fields that the program outputs:

  heat       implicit heat equation: one newtonSolve
  heat_run   the same program as a whole: runtime, set-up and 20 time steps,
             fields after every step (a small request of a serving loop)
  two_phase  fully implicit oil-water flow, two unknowns per cell: one
             newtonSolveSystem, 2D (nz = 0) or 3D, FP64 or `mixed`
  impes      the same flow with implicit pressure (newtonSolve, one unknown
             per cell) and explicit upwind transport substeps, one runtime
             call per operation
  swe        explicit shallow water: Heun steps with the CFL time step,
             output after `steps` of them

Inputs are made from the seed on the GPU in plain torch; `exact` computes the
same pass in plain torch FP64 (block tridiagonal elimination for the implicit
systems).
"""
import math

import numpy as np
import torch

import equelle_b200
from equelle_b200 import capi

DAY = 86400.0
MD = 9.869233e-16          # one millidarcy in m^2
VISC_W, VISC_O = 1e-3, 5e-3
GRAVITY, DRY, DUMMY, CFL = 9.81, 0.05, 1000.0, 0.45
SOLVER = dict(abs_res_tol=1e-10, linsolver_residual_tolerance=1e-12, linsolver_max_iterations=5000)


def listed():
    return [
        # the implicit heat configuration, one step: launches and round trips
        dict(name="heat 64x64", kind="heat", nx=64, ny=64),
        # the same program whole, as a request of the serving loop runs it
        dict(name="heat run 64x64", kind="heat_run", nx=64, ny=64, steps=20),
        # a large, ragged request of the serving mix (sides 64 to 1024)
        dict(name="heat 1000x701", kind="heat", nx=1000, ny=701),
        # a small instance of the batched mix (sides 32 to 512)
        dict(name="two-phase 48x40", kind="two_phase", nx=48, ny=40, nz=0, precision="double"),
        # a middle one, odd sides, with the FP32-stored preconditioner
        dict(name="two-phase 255x257 mixed", kind="two_phase", nx=255, ny=257, nz=0, precision="mixed"),
        # the largest of the batched mix
        dict(name="two-phase 512x512", kind="two_phase", nx=512, ny=512, nz=0, precision="double"),
        # a small odd reservoir in 3D
        dict(name="two-phase 33x31x17", kind="two_phase", nx=33, ny=31, nz=17, precision="double"),
        # the headline configuration
        dict(name="two-phase 128x128x64", kind="two_phase", nx=128, ny=128, nz=64, precision="double"),
        # sequential form: scalar pressure system in 3D, per-operation transport
        dict(name="impes 97x83x41", kind="impes", nx=97, ny=83, nz=41, steps=8),
        # shallow water on a test-size grid: launches and the CFL round trip
        dict(name="swe 64x48", kind="swe", nx=64, ny=48, steps=20),
        # a ragged middle size
        dict(name="swe 1023x777", kind="swe", nx=1023, ny=777, steps=20),
        # the shallow-water configuration
        dict(name="swe 4096x4096", kind="swe", nx=4096, ny=4096, steps=100),
    ]


def draw(rng):
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["heat", "heat_run", "two_phase", "two_phase", "two_phase", "impes", "swe", "swe"])
    if kind == "heat":
        return dict(kind=kind, nx=log_int(24, 1024), ny=log_int(24, 1024))
    if kind == "heat_run":
        return dict(kind=kind, nx=log_int(24, 128), ny=log_int(24, 128), steps=rng.randint(10, 30))
    if kind == "two_phase":
        precision = rng.choice(["double", "double", "mixed"])
        if rng.random() < 0.5:
            return dict(kind=kind, nx=log_int(32, 512), ny=log_int(32, 512), nz=0, precision=precision)
        return dict(kind=kind, nx=log_int(12, 128), ny=log_int(12, 128), nz=log_int(6, 64), precision=precision)
    if kind == "impes":
        return dict(kind=kind, nx=log_int(12, 96), ny=log_int(12, 96), nz=log_int(6, 48), steps=rng.randint(4, 12))
    return dict(kind=kind, nx=log_int(32, 4096), ny=log_int(32, 4096), steps=rng.randint(10, 40))


def work(case):
    """Each field of the pass read once and written once (8 bytes per value;
    shallow water: the state in and out and one bottom array in both stages
    of every step), and the arithmetic of one evaluation of the equations per
    Newton iteration the program needs at least."""
    n = case["nx"] * case["ny"] * max(case.get("nz", 0), 1)
    kind = case["kind"]
    if kind == "heat":
        return dict(bytes=8.0 * 5 * n, flops=20.0 * n)
    if kind == "heat_run":
        return dict(bytes=8.0 * 2 * n * case["steps"], flops=20.0 * n * case["steps"])
    if kind == "two_phase":
        return dict(bytes=8.0 * 10 * n, flops=3 * 150.0 * n)
    if kind == "impes":
        return dict(bytes=8.0 * (8 + 8 * case["steps"]) * n, flops=(40.0 + 50.0 * case["steps"]) * n)
    return dict(bytes=112.0 * n * case["steps"], flops=300.0 * n * case["steps"])


# ---- inputs (plain torch) --------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _smooth_field(shape, corr_len, gen):
    """Gaussian random field, mean 0 and deviation 1, covariance
    exp(-r / corr_len), by circulant embedding; shape slowest first."""
    ext = [2 * s for s in shape]
    r2 = torch.zeros(ext, dtype=torch.float64, device="cuda")
    for d, e in enumerate(ext):
        i = torch.arange(e, dtype=torch.float64, device="cuda")
        view = [1] * len(ext)
        view[d] = e
        r2 = r2 + (torch.minimum(i, e - i) ** 2).view(view)
    lam = torch.fft.fftn(torch.exp(-r2.sqrt() / corr_len)).real.clamp_min(0.0)
    noise = torch.complex(torch.randn(ext, generator=gen, device="cuda", dtype=torch.float64),
                          torch.randn(ext, generator=gen, device="cuda", dtype=torch.float64))
    f = torch.fft.ifftn(lam.sqrt() * noise).real[tuple(slice(0, s) for s in shape)]
    return (f - f.mean()) / f.std()


def _heat_inputs(case, seed):
    nx, ny = case["nx"], case["ny"]
    u0 = 0.5 + torch.rand(nx * ny, generator=_generator(seed), device="cuda", dtype=torch.float64)
    return dict(u0=u0, k=0.3, cv=1.0, dt=0.5, dir_faces=[(nx + 1) * j for j in range(ny)], dir_val=0.5)


def _flow_inputs(case, seed):
    """Log-normal permeability (100 mD, log deviation 1), an injector column
    in one corner and a producer column in the opposite one, and a water
    front that has left the injector."""
    nx, ny, nz = case["nx"], case["ny"], max(case["nz"], 1)
    gen = _generator(seed)
    shape = (nz, ny, nx) if case["nz"] else (ny, nx)
    perm = torch.exp(_smooth_field(shape, 8.0, gen) + math.log(100 * MD)).reshape(-1)
    ijk = torch.arange(nx * ny * nz, device="cuda")
    i, j = (ijk % nx).double(), ((ijk // nx) % ny).double()
    front = 0.25 * math.hypot(nx, ny) * (1.0 + 0.2 * _smooth_field(shape, 8.0, gen).reshape(-1))
    r = torch.hypot(i, j) / front
    sw0 = 0.2 + 0.5 * torch.exp(-r * r)
    dz = 2.0 if case["nz"] else 1.0
    inj = [nx * ny * k for k in range(nz)]
    prod = [(nx - 1) + nx * ((ny - 1) + ny * k) for k in range(nz)]
    rate = 0.2 * 100.0 * dz / DAY  # a well cell's pore volume a day
    cells = sorted(inj + prod)
    inj_set = set(inj)
    return dict(perm=perm, poro=0.2, sw0=sw0, dt=DAY, dz=dz, cells=cells, anchor=prod[0],
                rates=[rate if c in inj_set else -rate for c in cells])


def _swe_inputs(case, seed):
    """Depth 1 with eight Gaussian bumps over a smooth bottom, at rest."""
    nx, ny = case["nx"], case["ny"]
    rng = np.random.default_rng(seed)
    x = torch.arange(nx, device="cuda", dtype=torch.float64) + 0.5
    y = (torch.arange(ny, device="cuda", dtype=torch.float64) + 0.5).view(-1, 1)
    sigma = min(40.0, 0.1 * min(nx, ny))
    h = torch.ones(ny, nx, device="cuda", dtype=torch.float64)
    for _ in range(8):
        cx, cy = rng.uniform(0, nx), rng.uniform(0, ny)
        h += 0.1 * torch.exp(-((x - cx) ** 2 + (y - cy) ** 2) / (2 * sigma * sigma))
    kx, ky = (int(v) for v in rng.integers(1, 5, 2))
    px, py = rng.uniform(0, 2 * math.pi, 2)

    def bottom(xx, yy):
        return (0.05 * torch.sin(2 * math.pi * kx * xx / nx + px) * torch.sin(2 * math.pi * ky * yy / ny + py)).reshape(-1)

    zero = torch.zeros(nx * ny, device="cuda", dtype=torch.float64)
    return dict(h=h.reshape(-1), u=zero, v=zero, bn=bottom(x, y + 0.5), bs=bottom(x, y - 0.5), be=bottom(x + 0.5, y),
                bw=bottom(x - 0.5, y))


# ---- the programs, over the runtime ---------------------------------------
def _host(t):
    return t.cpu().numpy()


def _heat_program(er, c):
    """Set-up of the heat program; returns its initial field and its step."""
    ifaces, bf = er.interiorFaces(), er.boundaryFaces()
    first, second = er.firstCell(ifaces), er.secondCell(ifaces)
    itrans = c["k"] * (er.norm(ifaces) / er.norm(er.centroid(first) - er.centroid(second)))
    dir_boundary = er.entity_set(capi.FACES, c["dir_faces"])
    dir_value = er.collection(np.full(len(c["dir_faces"]), c["dir_val"]))
    bf_cells = er.trinaryIf(er.isEmpty(er.firstCell(bf)), er.secondCell(bf), er.firstCell(bf))
    bf_sign = er.trinaryIf(er.isEmpty(er.firstCell(bf)), er.operatorExtend(-1.0, bf), er.operatorExtend(1.0, bf))
    btrans = c["k"] * (er.norm(bf) / er.norm(er.centroid(bf) - er.centroid(bf_cells)))
    dir_cells = er.operatorOn(bf_cells, bf, dir_boundary)
    dir_sign = er.operatorOn(bf_sign, bf, dir_boundary)
    dir_trans = er.operatorOn(btrans, bf, dir_boundary)
    vol = er.norm(er.allCells())

    def residual(u, u0):
        ifluxes = -itrans * er.gradient(u)
        u_dir = er.operatorOn(u, er.allCells(), dir_cells)
        bfluxes = er.operatorExtend((dir_trans * dir_sign) * (u_dir - dir_value), dir_boundary, bf)
        fluxes = er.operatorExtend(ifluxes, ifaces, er.allFaces()) + er.operatorExtend(bfluxes, bf, er.allFaces())
        return (u - u0) + ((c["dt"] / (c["cv"] * vol)) * er.divergence(fluxes))

    return er.collection(_host(c["u0"])), lambda u0: er.newtonSolve(lambda u: residual(u, u0), u0)


class _Flow:
    """Set-up and functions of the two-phase programs."""

    def __init__(self, er, c):
        self.er, self.dt = er, c["dt"]
        self.cells, self.ifaces = er.allCells(), er.interiorFaces()
        self.first, self.second = er.firstCell(self.ifaces), er.secondCell(self.ifaces)
        vol = er.norm(self.cells)
        self.pv = er.collection(np.full(len(vol), c["poro"])) * vol
        perm = er.collection(_host(c["perm"]))
        fc, area, normal = er.centroid(self.ifaces), er.norm(self.ifaces), er.normal(self.ifaces)
        d1, d2 = er.centroid(self.first) - fc, er.centroid(self.second) - fc
        h1 = (-area * er.operatorOn(perm, self.cells, self.first)) * (er.dot(normal, d1) / er.dot(d1, d1))
        h2 = (area * er.operatorOn(perm, self.cells, self.second)) * (er.dot(normal, d2) / er.dot(d2, d2))
        self.trans = 1.0 / ((1.0 / h1) + (1.0 / h2))
        wells = er.entity_set(capi.CELLS, c["cells"])
        self.source = er.operatorExtend(er.collection(c["rates"]), wells, self.cells)
        anchor = er.entity_set(capi.CELLS, [c["anchor"]])
        self.is_anchor = er.operatorExtend(er.operatorExtend(1.0, anchor), anchor, self.cells) > 0.5
        self.insource_sw = er.operatorExtend(1.0, self.cells)
        self.sw0 = er.collection(_host(c["sw0"]))
        self.p0 = er.operatorExtend(0.0, self.cells)

    def upwind(self, flux, x):
        er = self.er
        return er.trinaryIf(flux >= 0.0, er.operatorOn(x, self.cells, self.first),
                            er.operatorOn(x, self.cells, self.second))

    def water_mob(self, sw):
        return (sw * sw) / VISC_W

    def oil_mob(self, sw):
        so = self.er.operatorExtend(1.0, self.cells) - sw
        return (so * so) / VISC_O

    def total_flux(self, p, mob):
        ngradp = -self.er.gradient(p)
        return (self.trans * self.upwind(ngradp, mob)) * ngradp

    def pressure(self, p, mob):
        er = self.er
        balance = (self.dt / self.pv) * (er.divergence(self.total_flux(p, mob)) - self.source)
        return er.trinaryIf(self.is_anchor, p, balance)

    def transported(self, sw, flux, dt):
        er = self.er
        zero = er.operatorExtend(0.0, self.cells)
        insource = er.trinaryIf(self.source > 0.0, self.source, zero)
        outsource = er.trinaryIf(self.source < 0.0, self.source, zero)
        mw, mo = self.water_mob(sw), self.oil_mob(sw)
        fracflow = mw / (mw + mo)
        q = (insource * self.insource_sw) + (outsource * fracflow)
        return (dt / self.pv) * (er.divergence(self.upwind(flux, fracflow) * flux) - q)

    def implicit_step(self):
        def pres(p, sw):
            return self.pressure(p, self.water_mob(sw) + self.oil_mob(sw))

        def trans(p, sw):
            flux = self.total_flux(p, self.water_mob(sw) + self.oil_mob(sw))
            return (sw - self.sw0) + self.transported(sw, flux, self.dt)

        p, sw = self.er.newtonSolveSystem([pres, trans], [self.p0, self.sw0])
        return p.value(), sw.value()

    def impes_step(self, substeps):
        mob = self.water_mob(self.sw0) + self.oil_mob(self.sw0)
        p = self.er.newtonSolve(lambda q: self.pressure(q, mob), self.p0)
        flux = self.total_flux(p, mob)
        sw = self.sw0
        for _ in range(substeps):
            sw = sw - self.transported(sw, flux, self.dt / substeps)
        return p.value(), sw.value()


class _ShallowWater:
    """Set-up and time step of the shallow-water program (Rusanov fluxes, wall
    fluxes, bathymetry source)."""

    def __init__(self, er, c):
        self.er = er
        self.bn, self.bs, self.be, self.bw = (er.collection(_host(c[k])) for k in ("bn", "bs", "be", "bw"))
        h, u, v = (er.collection(_host(c[k])) for k in ("h", "u", "v"))
        self.b_mid = (((self.bn + self.bs) + self.be) + self.bw) / 4.0
        self.ifaces, self.bound, self.cells = er.interiorFaces(), er.boundaryFaces(), er.allCells()
        self.vol, self.area = er.norm(self.cells), er.norm(er.allFaces())
        self.nrm, self.bnrm = er.normal(self.ifaces), er.normal(self.bound)
        self.first, self.second = er.firstCell(self.ifaces), er.secondCell(self.ifaces)
        bf = er.firstCell(self.bound)
        self.bcells = er.trinaryIf(er.isEmpty(bf), er.secondCell(self.bound), bf)
        self.b1, self.b2, self.bb = (er.operatorOn(self.b_mid, self.cells, s)
                                     for s in (self.first, self.second, self.bcells))
        self.sign = [er.trinaryIf(self.bnrm.col(d) > 0.0, er.operatorExtend(1.0, self.bound),
                                  er.operatorExtend(-1.0, self.bound)) for d in (0, 1)]
        self.bx, self.by = (self.be - self.bw) / 1.0, (self.bn - self.bs) / 1.0
        self.start = (h + self.b_mid, h * u, h * v)

    def side(self, w, hu, hv, b):
        er = self.er
        nx, ny = self.nrm.col(0), self.nrm.col(1)
        raw = w - b
        wet = raw > DRY
        height = er.trinaryIf(wet, raw, er.operatorExtend(DUMMY, self.ifaces))
        qn = (hu * nx) + (hv * ny)
        un = qn / height
        pressure = (0.5 * GRAVITY) * (height * height)
        zero = er.operatorExtend(0.0, self.ifaces)
        return (er.trinaryIf(wet, qn, zero), er.trinaryIf(wet, (hu * un) + (pressure * nx), zero),
                er.trinaryIf(wet, (hv * un) + (pressure * ny), zero),
                er.trinaryIf(wet, er.sqrt(un * un) + er.sqrt(GRAVITY * height), zero))

    def fluxes(self, q):
        er = self.er
        left = [er.operatorOn(x, self.cells, self.first) for x in q]
        right = [er.operatorOn(x, self.cells, self.second) for x in q]
        fl, fr = self.side(*left, self.b1), self.side(*right, self.b2)
        a = er.trinaryIf(fl[3] > fr[3], fl[3], fr[3])
        inner = [(0.5 * (fl[m] + fr[m])) - ((0.5 * a) * (right[m] - left[m])) for m in range(3)]
        height = er.operatorOn(q[0], self.cells, self.bcells) - self.bb
        wall = er.trinaryIf(height > DRY, (0.5 * GRAVITY) * (height * height), er.operatorExtend(0.0, self.bound))
        faces = er.allFaces()
        out = [er.operatorExtend(inner[0], self.ifaces, faces) * self.area]
        for d in (0, 1):
            w = (er.sqrt(self.bnrm.col(d) * self.bnrm.col(d)) * wall) * self.sign[d]
            out.append((er.operatorExtend(inner[d + 1], self.ifaces, faces)
                        + er.operatorExtend(w, self.bound, faces)) * self.area)
        return out

    def euler(self, q, dt):
        er = self.er
        w, hu, hv = q
        flux = self.fluxes(q)
        mx, my = ((w - self.be) + (w - self.bw)) / 2.0, ((w - self.bn) + (w - self.bs)) / 2.0
        wet = er.trinaryIf((w - self.b_mid) > DRY, er.operatorExtend(1.0, self.cells),
                           er.operatorExtend(0.0, self.cells))
        s0, s1 = (((-GRAVITY) * self.bx) * mx) * wet, (((-GRAVITY) * self.by) * my) * wet
        return (w + ((dt / self.vol) * (-er.divergence(flux[0]))),
                hu + ((dt / self.vol) * ((-er.divergence(flux[1])) + (self.vol * s0))),
                hv + ((dt / self.vol) * ((-er.divergence(flux[2])) + (self.vol * s1))))

    def max_speed(self, q):
        er = self.er
        raw = q[0] - self.b_mid
        wet = raw > DRY
        height = er.trinaryIf(wet, raw, er.operatorExtend(DUMMY, self.cells))
        u, v = q[1] / height, q[2] / height
        return er.maxReduce(er.trinaryIf(wet, er.sqrt((u * u) + (v * v)) + er.sqrt(GRAVITY * height),
                                         er.operatorExtend(0.0, self.cells)))

    def run(self, steps):
        q = self.start
        for _ in range(steps):
            dt = (CFL * 1.0) / self.max_speed(q)
            q2 = self.euler(self.euler(q, dt), dt)
            q = tuple((0.5 * a) + (0.5 * b) for a, b in zip(q, q2))
        return tuple(x.value() for x in q)


# ---- the cases ---------------------------------------------------------------
def _params(case):
    p = dict(grid_dim=3 if case.get("nz", 0) else 2, nx=case["nx"], ny=case["ny"], dx=1.0, dy=1.0)
    if case["kind"] == "swe":
        return p
    p.update(SOLVER)
    if case["kind"] in ("two_phase", "impes"):
        p.update(dx=10.0, dy=10.0, linsolver_precision=case.get("precision", "double"))
        if case["nz"]:
            p.update(nz=case["nz"], dz=2.0)
    return p


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("heat", "heat_run"):
        c = _heat_inputs(case, seed)
        if kind == "heat_run":
            return dict(kind=kind, params=_params(case), inputs=c, steps=case["steps"])
        er = equelle_b200.Runtime(_params(case))
        u0, step = _heat_program(er, c)
        return dict(kind=kind, u0=u0, step=step)
    er = equelle_b200.Runtime(_params(case))
    if kind == "swe":
        return dict(kind=kind, program=_ShallowWater(er, _swe_inputs(case, seed)), steps=case["steps"])
    return dict(kind=kind, flow=_Flow(er, _flow_inputs(case, seed)), steps=case.get("steps", 1))


def run(state):
    kind = state["kind"]
    if kind == "heat":
        return state["step"](state["u0"]).value()
    if kind == "heat_run":
        u, step = _heat_program(equelle_b200.Runtime(state["params"]), state["inputs"])
        fields = []
        for _ in range(state["steps"]):
            u = step(u)
            fields.append(u.value())
        return fields
    if kind == "swe":
        return state["program"].run(state["steps"])
    if kind == "impes":
        return state["flow"].impes_step(state["steps"])
    return state["flow"].implicit_step()


# ---- the same passes in plain torch FP64 -----------------------------------
class _SlabSystem:
    """Direct solver for a system on a Cartesian grid with `b` unknowns per
    cell and couplings between face neighbours: block elimination over slabs
    of cells across the longest axis.  Entries are given per cell (diag) and
    per interior face and direction."""

    def __init__(self, dims, b):
        # dims slowest first, as cell arrays reshape
        self.dims, self.b = dims, b
        self.axis = max(range(len(dims)), key=lambda d: dims[d])
        self.ns = dims[self.axis]
        self.m = int(np.prod(dims)) // self.ns

    @staticmethod
    def cost(dims, b):
        ns = max(dims)
        m = int(np.prod(dims)) // ns * b
        return ns * (2.0 * m ** 3 + 1e10)

    def slabs(self, x):
        """A per-cell array [cells, ...] as [slab, cell of the slab, ...]."""
        d = len(self.dims)
        y = x.reshape(*self.dims, *x.shape[1:]).movedim(self.axis, 0)
        return y.reshape(self.ns, self.m, *y.shape[d:])

    def cells(self, y):
        rest = [s for d, s in enumerate(self.dims) if d != self.axis]
        return y.reshape(self.ns, *rest, *y.shape[2:]).movedim(0, self.axis).reshape(-1, *y.shape[2:])

    def factor(self, diag, faces):
        """diag [cells, b, b]; faces: per axis (c1, c2, A12, A21), the cells of
        its faces and their couplings [faces, b, b]."""
        ns, m, b = self.ns, self.m, self.b
        n = diag.shape[0]
        number = self.slabs(torch.arange(n, device=diag.device))       # cell of (slab, place)
        place = torch.empty(n, dtype=torch.long, device=diag.device)
        slab = torch.empty(n, dtype=torch.long, device=diag.device)
        place[number.reshape(-1)] = torch.arange(m, device=diag.device).repeat(ns)
        slab[number.reshape(-1)] = torch.arange(ns, device=diag.device).repeat_interleave(m)
        inside = [f for d, f in enumerate(faces) if d != self.axis]
        c1, c2, a12, a21 = faces[self.axis]
        up = torch.zeros(ns, m, b, b, dtype=diag.dtype, device=diag.device)    # slab s to s + 1
        low = torch.zeros_like(up)                                             # slab s + 1 to s
        up[slab[c1], place[c1]] = a12
        low[slab[c1], place[c1]] = a21
        self.up, self.low, self.inv = up, low, []
        every = torch.arange(m, device=diag.device)
        ds = self.slabs(diag)
        for s in range(ns):
            D = torch.zeros(m, b, m, b, dtype=diag.dtype, device=diag.device)
            D[every, :, every, :] = ds[s]
            for f1, f2, g12, g21 in inside:
                k = slab[f1] == s
                D[place[f1[k]], :, place[f2[k]], :] = g12[k]
                D[place[f2[k]], :, place[f1[k]], :] = g21[k]
            if s:
                left = torch.einsum("iab,ibjc->iajc", low[s - 1], self.inv[-1].view(m, b, m, b))
                D -= torch.einsum("iajc,jcd->iajd", left, up[s - 1])
            self.inv.append(torch.linalg.inv(D.view(m * b, m * b)))
        return self

    def solve(self, rhs):
        ns, m, b = self.ns, self.m, self.b
        r = self.slabs(rhs).clone()
        for s in range(1, ns):
            y = (self.inv[s - 1] @ r[s - 1].reshape(-1)).view(m, b)
            r[s] -= torch.einsum("iab,ib->ia", self.low[s - 1], y)
        x = torch.empty_like(r)
        for s in range(ns - 1, -1, -1):
            if s < ns - 1:
                r[s] -= torch.einsum("iab,ib->ia", self.up[s], x[s + 1])
            x[s] = (self.inv[s] @ r[s].reshape(-1)).view(m, b)
        return self.cells(x)


def _face_cells(dims):
    """First and second cell of the interior faces, per axis (slowest first)."""
    n = torch.arange(int(np.prod(dims)), device="cuda").reshape(dims)
    return [(n.narrow(d, 0, dims[d] - 1).reshape(-1), n.narrow(d, 1, dims[d] - 1).reshape(-1))
            for d in range(len(dims))]


def _exact_heat(case, seed, steps):
    c = _heat_inputs(case, seed)
    dims = (case["ny"], case["nx"])
    n = case["nx"] * case["ny"]
    a = c["dt"] * c["k"] / c["cv"]
    diag = torch.ones(n, dtype=torch.float64, device="cuda")
    left = torch.arange(case["ny"], device="cuda") * case["nx"]
    diag[left] += 2.0 * a                      # half a cell to the boundary
    faces = []
    for c1, c2 in _face_cells(dims):
        g = torch.full((len(c1), 1, 1), -a, dtype=torch.float64, device="cuda")
        diag.index_add_(0, c1, torch.full_like(c1, a, dtype=torch.float64))
        diag.index_add_(0, c2, torch.full_like(c2, a, dtype=torch.float64))
        faces.append((c1, c2, g, g))
    system = _SlabSystem(dims, 1).factor(diag.view(-1, 1, 1), faces)

    def residual(u, u0):
        r = diag * u - u0
        r[left] -= 2.0 * a * c["dir_val"]
        for c1, c2 in _face_cells(dims):
            r.index_add_(0, c1, -a * u[c2])
            r.index_add_(0, c2, -a * u[c1])
        return r

    u, out = c["u0"], []
    for _ in range(steps):
        u0 = u
        for _ in range(3):
            u = u - system.solve(residual(u, u0).view(-1, 1)).view(-1)
        out.append(u)
    return out


class _ExactFlow:
    def __init__(self, case, seed):
        self.c = c = _flow_inputs(case, seed)
        self.dims = (case["nz"], case["ny"], case["nx"]) if case["nz"] else (case["ny"], case["nx"])
        h = [c["dz"], 10.0, 10.0] if case["nz"] else [10.0, 10.0]
        self.n = int(np.prod(self.dims))
        volume = 10.0 * 10.0 * c["dz"]
        self.pv = c["poro"] * volume
        self.faces = []
        for d, (c1, c2) in enumerate(_face_cells(self.dims)):
            area = volume / h[d]
            h1, h2 = area * c["perm"][c1] / (0.5 * h[d]), area * c["perm"][c2] / (0.5 * h[d])
            self.faces.append((c1, c2, 1.0 / (1.0 / h1 + 1.0 / h2)))
        self.q = torch.zeros(self.n, dtype=torch.float64, device="cuda")
        self.q[torch.tensor(c["cells"], device="cuda")] = torch.tensor(c["rates"], dtype=torch.float64, device="cuda")

    @staticmethod
    def mobilities(s):
        """Total mobility and fractional flow with their derivatives."""
        w, o = s * s / VISC_W, (1 - s) ** 2 / VISC_O
        dw, do = 2 * s / VISC_W, -2 * (1 - s) / VISC_O
        t = w + o
        return t, dw + do, w / t, (dw * o - w * do) / (t * t)

    def newton(self, coupled, sweeps):
        """p (and s when `coupled`) of one implicit step."""
        c, n, b = self.c, self.n, 2 if coupled else 1
        k = c["dt"] / self.pv
        p = torch.zeros(n, dtype=torch.float64, device="cuda")
        s = c["sw0"].clone()
        qin, qout = self.q.clamp_min(0.0), self.q.clamp_max(0.0)
        best = None
        for sweep in range(sweeps):
            mob, dmob, f, df = self.mobilities(s)
            r = torch.zeros(n, b, dtype=torch.float64, device="cuda")
            diag = torch.zeros(n, b, b, dtype=torch.float64, device="cuda")
            r[:, 0] = -k * self.q
            if coupled:
                r[:, 1] = (s - c["sw0"]) - k * (qin + qout * f)
                diag[:, 1, 1] = 1.0 - k * qout * df
            faces = []
            for c1, c2, T in self.faces:
                up1 = p[c1] - p[c2] >= 0
                up = torch.where(up1, c1, c2)
                ft = T * mob[up] * (p[c1] - p[c2])
                g = torch.zeros(len(c1), 2, b, b, dtype=torch.float64, device="cuda")  # d(flux) / d(cell 1, cell 2)
                g[:, 0, 0, 0] = T * mob[up]
                g[:, 1, 0, 0] = -T * mob[up]
                flux = ft.view(-1, 1)
                if coupled:
                    side = torch.where(up1, 0, 1)
                    every = torch.arange(len(c1), device="cuda")
                    dft = T * dmob[up] * (p[c1] - p[c2])
                    g[every, side, 0, 1] = dft
                    g[:, :, 1, :] = f[up].view(-1, 1, 1) * g[:, :, 0, :]
                    g[every, side, 1, 1] += df[up] * ft
                    flux = torch.stack([ft, f[up] * ft], 1)
                g = k * g
                r.index_add_(0, c1, k * flux)
                r.index_add_(0, c2, -k * flux)
                diag.index_add_(0, c1, g[:, 0])
                diag.index_add_(0, c2, -g[:, 1])
                faces.append([c1, c2, g[:, 1], -g[:, 0]])
            a = c["anchor"]
            r[a, 0] = p[a]
            diag[a, 0] = 0.0
            diag[a, 0, 0] = 1.0
            for face in faces:
                face[2][face[0] == a, 0] = 0.0
                face[3][face[1] == a, 0] = 0.0
            norm = float(r.norm())
            if best is not None and norm >= best[0] and sweep > 4:
                break
            if best is None or norm < best[0]:
                best = (norm, p, s)
            if sweep < 5:
                system = _SlabSystem(self.dims, b).factor(diag, faces)
            u = system.solve(r)
            p = p - u[:, 0]
            if coupled:
                s = s - u[:, 1]
        return best[1], best[2]

    def transport(self, p, substeps):
        c, s = self.c, self.c["sw0"]
        mob = self.mobilities(s)[0]
        qin, qout = self.q.clamp_min(0.0), self.q.clamp_max(0.0)
        for _ in range(substeps):
            f = self.mobilities(s)[2]
            div = torch.zeros_like(s)
            for c1, c2, T in self.faces:
                up = torch.where(p[c1] - p[c2] >= 0, c1, c2)
                ft = T * mob[up] * (p[c1] - p[c2]) * f[up]
                div.index_add_(0, c1, ft)
                div.index_add_(0, c2, -ft)
            s = s - (c["dt"] / substeps / self.pv) * (div - (qin + qout * f))
        return s


def _exact_swe(case, seed):
    c = {k: v.view(case["ny"], case["nx"]) for k, v in _swe_inputs(case, seed).items()}
    bm = (c["bn"] + c["bs"] + c["be"] + c["bw"]) / 4.0
    bx, by = c["be"] - c["bw"], c["bn"] - c["bs"]

    def side(q, normal):
        w, hu, hv, b = q
        wet = w - b > DRY
        h = torch.where(wet, w - b, DUMMY)
        qn = hu if normal == 0 else hv
        un, pr = qn / h, 0.5 * GRAVITY * h * h
        f = [qn, hu * un, hv * un]
        f[normal + 1] = f[normal + 1] + pr
        return [torch.where(wet, x, 0.0) for x in f] + [torch.where(wet, un.abs() + (GRAVITY * h).sqrt(), 0.0)]

    def divergence(q):
        total = [torch.zeros_like(bm) for _ in range(3)]
        h = q[0] - bm
        wall = torch.where(h > DRY, 0.5 * GRAVITY * h * h, 0.0)
        for normal, d in ((0, 1), (1, 0)):
            size = bm.shape[d]
            qb = [*q, bm]
            left = [x.narrow(d, 0, size - 1) for x in qb]
            right = [x.narrow(d, 1, size - 1) for x in qb]
            fl, fr = side(left, normal), side(right, normal)
            a = torch.maximum(fl[3], fr[3])
            for m in range(3):
                f = 0.5 * (fl[m] + fr[m]) - 0.5 * a * (right[m] - left[m])
                total[m].narrow(d, 0, size - 1).add_(f)
                total[m].narrow(d, 1, size - 1).sub_(f)
            total[normal + 1].narrow(d, size - 1, 1).add_(wall.narrow(d, size - 1, 1))
            total[normal + 1].narrow(d, 0, 1).sub_(wall.narrow(d, 0, 1))
        return total

    def euler(q, dt):
        w, hu, hv = q
        f = divergence(q)
        wet = torch.where(w - bm > DRY, 1.0, 0.0)
        s0 = -GRAVITY * bx * (w - 0.5 * (c["be"] + c["bw"])) * wet
        s1 = -GRAVITY * by * (w - 0.5 * (c["bn"] + c["bs"])) * wet
        return w - dt * f[0], hu + dt * (s0 - f[1]), hv + dt * (s1 - f[2])

    q = (c["h"] + bm, c["h"] * c["u"], c["h"] * c["v"])
    for _ in range(case["steps"]):
        h = q[0] - bm
        h = torch.where(h > DRY, h, DUMMY)
        speed = torch.where(q[0] - bm > DRY, ((q[1] / h) ** 2 + (q[2] / h) ** 2).sqrt() + (GRAVITY * h).sqrt(), 0.0)
        dt = CFL / speed.max()
        q2 = euler(euler(q, dt), dt)
        q = tuple(0.5 * a + 0.5 * b for a, b in zip(q, q2))
    return tuple(x.reshape(-1) for x in q)


def exact(case, seed):
    """The fields `run` returns, from the formulas; None where the direct
    solve would take too long."""
    kind = case["kind"]
    if kind == "swe":
        return _exact_swe(case, seed)
    if kind == "heat":
        return _exact_heat(case, seed, 1)[0]
    if kind == "heat_run":
        return _exact_heat(case, seed, case["steps"])
    dims = (case["nz"], case["ny"], case["nx"]) if case["nz"] else (case["ny"], case["nx"])
    coupled = kind == "two_phase"
    if _SlabSystem.cost(dims, 2 if coupled else 1) > 2e13 / (4 if coupled else 1):
        return None
    flow = _ExactFlow(case, seed)
    p, s = flow.newton(coupled, 12)
    return p, (s if coupled else flow.transport(p, case["steps"]))
