"""What a user of this package has it do, as cases that can be timed.

A case is a dict of plain values: the job (march, stages, linearise, autograd,
unrolled), the mesh (kind and size), the numerics (flux, reconstruction,
order) and the precision mode.  `prepare` makes what a program holds before
the call (the region with its grid products, the flow state, host and device
buffers), `run` is one pass through the public entry points, `exact` the same
results from plain torch in 64 bits.

The jobs:
  march      the solver's main loop between two outputs: the state goes up, a
             number of CFL-limited Runge-Kutta steps runs on the device, the
             state comes down
  stages     a host that keeps the loop to itself (coupled sources): every
             stage through the reference's own subroutines, gradients,
             fluxes, a source added to the residual, the update, with the
             gradients and residuals handed over on the device
  linearise  the tangent and the adjoint of the residual at one state, as a
             Newton-Krylov or sensitivity code asks for them
  autograd   the residual inside a torch program, forward and backward
  unrolled   the gradient of a time-integrated wall pressure with respect to
             the initial state, through checkpointed time steps

The mixed mode forms its residuals, gradients, increments and Jacobians in
FP32; its results are handed on in FP32, as a post-processor or a torch model
takes them.  The FP64 modes hand on FP64.
"""
import functools
import math

import numpy as np
import torch

from rocflu_gb300 import autograd, cases, gpu

ROE, HLLC, AUSM = cases.DISCR_ROE, cases.DISCR_HLLC, cases.DISCR_AUSM
BJ, BJ_COMP, VENKAT = cases.RECONST_BJ, cases.RECONST_BJ_COMP, cases.RECONST_VENKAT
WENO = cases.RECONST_WENO_XYZ
T0 = 0.01  # the clock of a run under way (the first step of a new run takes an imposed step instead)


def listed():
    return [
        # the one-dimensional verification run of every Euler code: few cells, many steps
        dict(name="march_sod_400x4x4_fp64", job="march", mesh="sod", n=400, flux=ROE, reconst=0, order=1,
             precision="fp64", steps=40),
        # the smallest call: the 8^3 gas-jump box, run bit for bit against the CPU code
        dict(name="march_gasjump_8_exact", job="march", mesh="closed", n=8, flux=HLLC, reconst=WENO, order=2,
             precision="fp64_exact", steps=20),
        # the production run: a planar shock over a dense sphere, 2.1 M cells
        dict(name="march_shocksphere_128_mixed", job="march", mesh="sphere", n=128, flux=HLLC, reconst=BJ, order=2,
             precision="mixed", steps=10),
        # the same flow as its all-FP64 verification run, on a coarser, odd-sized mesh
        dict(name="march_shocksphere_75_fp64", job="march", mesh="sphere", n=75, flux=HLLC, reconst=BJ, order=2,
             precision="fp64", steps=2),
        # a blast in a closed box on jittered tetrahedra, FP64, with the smooth limiter
        dict(name="march_blast_tets28_fp64", job="march", mesh="blast_tets", n=28, flux=HLLC, reconst=VENKAT, order=2,
             precision="fp64", steps=2),
        # the same at production size in the mixed mode
        dict(name="march_blast_tets48_mixed", job="march", mesh="blast_tets", n=48, flux=AUSM, reconst=BJ, order=2,
             precision="mixed", steps=6),
        # the solver's default reconstruction (WENO smoothing), mixed mode, a ragged size
        dict(name="march_shocksphere_77_weno_mixed", job="march", mesh="sphere", n=77, flux=HLLC, reconst=WENO,
             order=2, precision="mixed", steps=6),
        # the same reconstruction in FP64 on a fully periodic box
        dict(name="march_periodic_40_weno_fp64", job="march", mesh="periodic", n=40, flux=HLLC, reconst=WENO, order=2,
             precision="fp64", steps=2),
        # a particle or chemistry code that adds its sources stage by stage
        dict(name="stages_shocksphere_64_mixed", job="stages", mesh="sphere", n=64, flux=AUSM, reconst=BJ_COMP,
             order=2, precision="mixed", steps=2),
        # tangent and adjoint of the 196,608-cell sensitivity mesh in FP64
        dict(name="linearise_tets32_fp64", job="linearise", mesh="adjoint_tets", n=32, flux=ROE, reconst=BJ_COMP,
             order=2, precision="fp64", steps=1),
        # the residual as a layer of a torch program, mixed mode
        dict(name="autograd_tets32_mixed", job="autograd", mesh="adjoint_tets", n=32, flux=ROE, reconst=BJ_COMP,
             order=2, precision="mixed", steps=1),
        # a small data-assimilation or design gradient through time
        dict(name="unrolled_blast_32_mixed", job="unrolled", mesh="blast", n=32, flux=HLLC, reconst=BJ_COMP, order=2,
             precision="mixed", steps=4),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    job = rng.choice(["march"] * 6 + ["stages", "linearise", "autograd", "unrolled"])
    precision = rng.choice(["mixed", "mixed", "fp64", "fp64", "fp64_exact"])
    c = dict(job=job, flux=rng.choice([ROE, HLLC, AUSM]), order=2, precision=precision, steps=1)
    if job == "march":
        mesh = rng.choice(["sod", "closed", "sphere", "sphere", "blast_tets", "periodic", "blast"])
        c.update(mesh=mesh, reconst=rng.choice([BJ, BJ_COMP, WENO, VENKAT] if mesh == "sphere" else [BJ, BJ_COMP, WENO]))
        fp32 = precision == "mixed"
        if mesh == "sod":
            c.update(n=size(100, 1600), order=1, reconst=0, steps=rng.randint(10, 40), precision="fp64")
        elif mesh == "closed":
            c.update(n=size(6, 24), steps=rng.randint(5, 20))
        elif mesh == "blast_tets":
            c.update(n=size(6, 48 if fp32 else 26), steps=rng.randint(1, 3))
        else:
            c.update(n=size(12, 112 if fp32 else 60), steps=rng.randint(1, 6 if fp32 else 2))
    elif job == "stages":
        c.update(mesh="sphere", n=size(10, 72), reconst=rng.choice([BJ, BJ_COMP, WENO]))
    elif job == "unrolled":
        c.update(mesh="blast", n=size(8, 36), reconst=rng.choice([BJ, BJ_COMP]), flux=HLLC, precision="mixed",
                 steps=rng.randint(1, 4))
    else:
        c.update(mesh="adjoint_tets", n=size(5, 32), reconst=rng.choice([BJ_COMP, WENO]),
                 precision=rng.choice(["mixed", "fp64"]))
    return c


# --- inputs ------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _grid(mesh, n):
    """The case's mesh, patches and boundary types with the grid products that
    the solver's host hands over (faces, geometry, stencils): they belong to
    the mesh, whatever flow runs on it."""
    make = {"sod": lambda: cases.sod(nx=n), "closed": lambda: cases.gas_jump_closed(n),
            "sphere": lambda: cases.shock_sphere(n), "blast_tets": lambda: cases.blast_tets(n),
            "periodic": lambda: cases.gas_jump_periodic(n), "blast": lambda: cases.blast_hex(n),
            "adjoint_tets": lambda: cases.adjoint_tets(n)}[mesh]
    c = make()
    order = c.num.space_order
    c.num.space_order = 2
    setup = gpu.Setup(c)
    c.num.space_order = order
    return c, setup


def _case(case, seed):
    """The package's Case with the numerics of this case and a state of this
    seed: the mesh's own flow (shock tube, gas jump, shock and sphere, blast,
    uniform stream) with its strengths, and a smooth disturbance on all of it,
    both from the seed."""
    base, grid = _grid(case["mesh"], case["n"])
    num = cases.Numerics(space_order=case["order"], space_discr=case["flux"], reconst=case["reconst"], cfl=0.4,
                         cp=base.num.cp, gamma=base.num.gamma, dt_imposed=base.num.dt_imposed,
                         dt_min_limit=base.num.dt_min_limit)
    rng = np.random.default_rng([seed, case["n"]])
    patches = [cases.Patch(**{**p.__dict__, "order": min(p.order, case["order"])}) for p in base.patches]
    g = num.gamma
    if case["mesh"] == "adjoint_tets":
        cv = cases.conserved(np.ones(base.n_cells), 0.5 * np.ones(base.n_cells), 0.0, 0.0, 1.0 / g, g)
        cv = cv * (1.0 + 0.05 * rng.standard_normal(cv.shape))
        cv[:, 2:4] = 0.025 * rng.standard_normal((base.n_cells, 2))
    else:
        x = grid.cofg
        ext = x.max(axis=0) - x.min(axis=0)
        y = (x - x.min(axis=0)) / np.where(ext > 0, ext, 1.0)
        cv = base.cv0.copy()
        rho, vel = cv[:, 0].copy(), cv[:, 1:4] / cv[:, :1]
        p = (g - 1.0) * (cv[:, 4] - 0.5 * rho * (vel * vel).sum(axis=1))
        if case["mesh"] == "blast_tets":
            p = np.where(p > 1.5, 4.0, 1.0)
        amp = 1.0 + 0.1 * rng.uniform(-1, 1, 2)
        rho, p = rho ** amp[0], p ** (amp[1] if p.max() < 1e3 else 1.0)
        c0 = math.sqrt(g * float(p.min()) / float(rho.max()))

        def wave():
            k = rng.integers(1, 4, 3) * 2.0 * np.pi
            return np.cos(y @ k + rng.uniform(0, 2 * np.pi))

        rho = rho * (1.0 + 0.02 * wave())
        p = p * (1.0 + 0.02 * wave())
        vel = vel + 0.03 * c0 * np.stack([wave(), wave(), wave()], axis=1)
        cv = cases.conserved(rho, vel[:, 0], vel[:, 1], vel[:, 2], p, g)
    out = cases.Case(case["mesh"], base.xyz, base.c2v, patches, num, np.ascontiguousarray(cv))
    return out, grid, rng


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.copy_(torch.from_numpy(a))
    return t


def _fixed_dt(c, grid):
    """A step below the CFL limit of the state (the largest wave speed over the smallest cell width)."""
    rho, m, e = c.cv0[:, 0], c.cv0[:, 1:4], c.cv0[:, 4]
    u2 = (m * m).sum(axis=1) / rho ** 2
    p = (c.num.gamma - 1) * (e - 0.5 * rho * u2)
    speed = float((np.sqrt(u2) + np.sqrt(c.num.gamma * p / rho)).max())
    return 0.1 * float(grid.vol.min()) ** (1 / 3) / speed


def _directions(c, rng):
    """A direction in state space and one in residual space, of the sizes of the state's entries."""
    s = np.abs(c.cv0).mean(axis=0)
    return rng.standard_normal(c.cv0.shape) * s, rng.standard_normal(c.cv0.shape)


def _source(c, rng, dt):
    """A stage's source terms: a few per mille of the state over a step."""
    return 0.003 * np.abs(c.cv0).mean(axis=0) / dt * rng.standard_normal(c.cv0.shape)


def prepare(case, seed):
    c, grid, rng = _case(case, seed)
    r = gpu.Region(c, case["precision"], grid=grid)
    st = {"case": case, "region": r, "narrow": case["precision"] == "mixed"}
    nc = c.n_cells
    if case["job"] == "march":
        st["cv"], st["out"] = _pinned(c.cv0).numpy(), _pinned(np.zeros((nc, 5))).numpy()
    elif case["job"] == "stages":
        st["cv"], st["out"] = _pinned(c.cv0).numpy(), _pinned(np.zeros((nc, 5))).numpy()
        st["dt"] = _fixed_dt(c, grid)
        st["src"] = torch.from_numpy(_source(c, rng, st["dt"]) * grid.vol[:, None]).cuda()
        st["grad"] = torch.zeros((nc, 5, 3), dtype=torch.float64, device="cuda")
        st["rhs"] = torch.zeros((nc, 5), dtype=torch.float64, device="cuda")
    elif case["job"] == "linearise":
        st["cv"] = c.cv0
        st["dot"], st["bar"] = _directions(c, rng)
    elif case["job"] == "autograd":
        st["x"] = torch.from_numpy(c.cv0).requires_grad_(True)
        st["bar"] = torch.from_numpy(_directions(c, rng)[1])
    else:
        st["cv"], st["dt"] = c.cv0, _fixed_dt(c, grid)
    return st


# --- one pass ----------------------------------------------------------------
def _hand_on(st, a):
    t = torch.from_numpy(a) if isinstance(a, np.ndarray) else a
    return t.float() if st["narrow"] else t


def run(st):
    r, case = st["region"], st["case"]
    if case["job"] == "march":
        r.upload(st["cv"])
        done, time, _ = r.step(case["steps"], T0)
        r.download(st["out"], with_dv=False)
        return {"cv": _hand_on(st, st["out"]), "time": time - T0, "steps": done}
    if case["job"] == "stages":
        r.upload(st["cv"])
        dt = r.timestep(T0)
        for _ in range(case["steps"]):
            for istage in range(1, r.n_stages + 1):
                gpu.CellGradientsMP(r)
                r.get_grad(st["grad"].data_ptr())
                gpu.ConvectiveFluxesMP(r)
                r.add_rhs(st["src"].data_ptr())
                r.get_rhs(st["rhs"].data_ptr())
                gpu.RKUpdateMP(r, 1, istage, st["dt"])
        r.download(st["out"], with_dv=False)
        return {"dt": dt, "grad": _hand_on(st, st["grad"]), "rhs": _hand_on(st, st["rhs"]),
                "cv": _hand_on(st, st["out"])}
    if case["job"] == "linearise":
        return {"rhs_dot": _hand_on(st, r.jvp(st["cv"], st["dot"])), "cv_bar": _hand_on(st, r.vjp(st["cv"], st["bar"]))}
    if case["job"] == "autograd":
        st["x"].grad = None
        rhs = autograd.residual(st["x"], r)
        rhs.backward(st["bar"])
        return {"rhs": _hand_on(st, rhs.detach()), "cv_bar": _hand_on(st, st["x"].grad)}
    j, bar, _ = r.unrolled_adjoint(st["cv"], case["steps"], st["dt"], max(1, case["steps"] // 2), 1)
    return {"J": j, "cv_bar": _hand_on(st, bar)}


# --- what a pass cannot do without -------------------------------------------
def _sizes(case):
    """Cells, interior faces per cell and stencil members per cell (near enough for a bound)."""
    n = case["n"]
    if case["mesh"] == "sod":
        return 16 * n, 3 - 1 / n - 2 / 4, 0
    if case["mesh"] in ("blast_tets", "adjoint_tets"):
        return 6 * n ** 3, 2 - 1 / n, 40
    per = case["mesh"] == "periodic"
    return n ** 3, 3 if per else 3 - 3 / n, 26 if per else (3 - 2 / n) ** 3 - 1


def work(case):
    """Per stage: the state read and written, the mesh (faces, stencil ids) read once; arithmetic of the fit,
    the limiter, one flux per face and the update.  The tangent counts as two residuals, the adjoint as three."""
    nc, nf, s = _sizes(case)
    w = 4 if case["precision"] == "mixed" else 8
    stage_bytes = nc * (2 * 40 + 2 * s + nf * (10 * w + 8) + 3 * w)
    stage_flops = nc * (40 * s + (150 if case["reconst"] else 0) + (90 * s if case["reconst"] == WENO else 0)
                        + 250 * nf + 60)
    io = 40 * nc
    if case["job"] == "march":
        k, b = 3 * case["steps"], 2 * io
    elif case["job"] == "stages":
        k, b = 3 * case["steps"], 2 * io + 3 * case["steps"] * 5 * io
    elif case["job"] == "linearise":
        k, b = 5, 6 * io
    elif case["job"] == "autograd":
        k, b = 4, 4 * io
    else:
        k, b = 3 * case["steps"] * 5, 2 * io
    return {"bytes": float(k * stage_bytes + b), "flops": float(k * stage_flops)}


# --- the same in 64 bits -----------------------------------------------------
class _Plain:
    """The scheme in plain torch, FP64, on the grid products."""

    def __init__(self, c, grid):
        self.num, self.patches = c.num, c.patches
        dev = self.dev = "cuda" if torch.cuda.is_available() else "cpu"

        def put(a, t=torch.float64):
            return torch.as_tensor(np.ascontiguousarray(a)).to(dev, t)

        nc = self.nc = len(grid.vol)
        f2c = np.asarray(grid.f2c) - 1
        fc2 = grid.fc if grid.fc2 is None else grid.fc2
        self.c1, self.c2 = put(f2c[:, 0], torch.int64), put(f2c[:, 1], torch.int64)
        self.fn, self.area = put(grid.fn[:, :3]), put(grid.fn[:, 3])
        self.dl, self.dr = put(grid.fc - grid.cofg[f2c[:, 0]]), put(fc2 - grid.cofg[f2c[:, 1]])
        self.vol = put(grid.vol)
        self.bc = put(np.asarray(grid.bf2c) - 1, torch.int64)
        self.bfn, self.barea = put(grid.bfn[:, :3]), put(grid.bfn[:, 3])
        self.bd = put(grid.bfc - grid.cofg[np.asarray(grid.bf2c) - 1])
        self.boff = [int(o) for o in grid.patch_off]
        # a cell's faces as a table: neighbour (itself where there is none), offset, face, sign
        nf, nb = len(f2c), len(grid.bf2c)
        cell = np.concatenate([f2c[:, 0], f2c[:, 1], np.asarray(grid.bf2c) - 1])
        face = np.concatenate([np.arange(nf), np.arange(nf), nf + np.arange(nb)])
        sign = np.concatenate([np.ones(nf), -np.ones(nf), np.ones(nb)])
        nbr = np.concatenate([f2c[:, 1], f2c[:, 0], np.asarray(grid.bf2c) - 1])
        order = np.argsort(cell, kind="stable")
        first = np.concatenate([[0], np.cumsum(np.bincount(cell, minlength=nc))])
        col = np.arange(len(cell)) - first[cell[order]]
        width = int(col.max()) + 1

        def table(v, fill):
            a = np.full((nc, width), fill, v.dtype)
            a[cell[order], col] = v[order]
            return a

        self.cf, self.csgn = put(table(face, nf + nb), torch.int64), put(table(sign, 0.0))
        t = table(nbr, -1)
        t = np.where(t < 0, np.arange(nc)[:, None], t)
        self.cn, self.inner = put(t, torch.int64), put(table(face, nf + nb) < nf, torch.bool)
        d = torch.cat([self.dl, self.dr, self.bd])[torch.as_tensor(order).to(dev)]
        self.cd = torch.zeros((nc, width, 3), dtype=torch.float64, device=dev)
        self.cd[put(cell[order], torch.int64), put(col, torch.int64)] = d
        self.any_face = put(table(face, nf + nb) < nf + nb, torch.bool)
        if c.num.space_order == 2:
            off = np.asarray(grid.c2cs_off)
            rows = np.repeat(np.arange(nc), np.diff(off))
            col = np.arange(len(rows)) - off[:-1][rows]
            width = int(np.diff(off).max())
            ids = np.repeat(np.arange(nc)[:, None], width, 1)
            ids[rows, col] = np.asarray(grid.c2cs) - 1
            x, ids = put(grid.cofg), put(ids, torch.int64)
            d = x[ids] - x[:, None]
            if grid.c2cs_shift is not None:
                d[put(rows, torch.int64), put(col, torch.int64)] += put(grid.c2cs_shift)
            on = torch.zeros((nc, width), dtype=torch.bool, device=dev)
            on[put(rows, torch.int64), put(col, torch.int64)] = True
            r2 = torch.where(on, (d * d).sum(-1), torch.ones_like(d[..., 0]))
            s = d / r2[..., None] * on[..., None]
            # the inverse-distance weighted least-squares fit
            m = s.transpose(1, 2) @ d
            self.w = s @ torch.linalg.inv(m).transpose(1, 2)
            self.st, self.on = ids, on

    def primitive(self, cv):
        rho, u = cv[:, 0], cv[:, 1:4] / cv[:, :1]
        p = (self.num.gamma - 1) * (cv[:, 4] - 0.5 * rho * (u * u).sum(1))
        return torch.cat([rho[:, None], u, p[:, None]], 1)

    def fit(self, q):
        return torch.stack([((q[:, k][self.st] - q[:, k:k + 1])[..., None] * self.w).sum(1) for k in range(5)], 1)

    def gradients(self, q):
        """Limited gradients (cells, 5, 3)."""
        g, rc = self.fit(q), self.num.reconst
        if rc == WENO:
            own = 1.0 / (g * g + 1e-15)
            out = []
            for k in range(15):
                t = g.reshape(-1, 15)[:, k]
                tm = t[self.st]
                wm = self.on / (tm * tm + 1e-15)
                wo = own.reshape(-1, 15)[:, k]
                out.append((wo * t + (wm * tm).sum(1)) / (wo + wm.sum(1)))
            g = torch.stack(out, 1).reshape(-1, 5, 3)
            cols = []
            for k in range(5):
                if k in (0, 4):
                    low = ((q[:, k:k + 1] + (g[:, None, k] * self.cd).sum(-1) <= 0) & self.any_face).any(1)
                    cols.append(torch.where(low[:, None], torch.zeros_like(g[:, k]), g[:, k]))
                else:
                    cols.append(g[:, k])
            return torch.stack(cols, 1)
        if rc == 0:
            return g
        one = torch.ones_like(q[:, 0])
        cols = []
        for k in range(5):
            if rc == BJ and 1 <= k <= 3:
                cols.append(None)
                continue
            hi, lo = q[:, k], q[:, k]
            for f in range(self.cn.shape[1]):
                x = q[:, k][self.cn[:, f]]
                hi, lo = torch.where(x > hi, x, hi), torch.where(x < lo, x, lo)
            lim = one
            for f in range(self.cn.shape[1]):
                d2 = -(g[:, k] * self.cd[:, f]).sum(-1)
                live = self.inner[:, f] & (d2 != 0)
                ext = torch.where(d2 > 0, hi - q[:, k], lo - q[:, k])
                safe = torch.where(live, d2, one)
                if rc == VENKAT:
                    num = (ext * ext + self.vol) * safe + 2 * safe * safe * ext
                    den = safe * (ext * ext + 2 * safe * safe + ext * safe + self.vol)
                    phi = num / (den + 1e-12)
                else:
                    phi = ext / safe
                lim = torch.where(live & (phi < lim), phi, lim)
            cols.append(lim[:, None] * g[:, k])
        if rc == BJ:
            vel = self.frame_limited(q[:, 1:4], g[:, 1:4])
            cols[1:4] = [vel[:, 0], vel[:, 1], vel[:, 2]]
        return torch.stack(cols, 1)

    def frame_limited(self, u, g):
        """The velocity gradient limited along the strain rate's axes."""
        val, vec = _jacobi(0.5 * (g + g.transpose(1, 2)))
        rows = vec.transpose(1, 2) @ g                      # one row per axis
        al = []
        for j in range(3):
            a = vec[:, :, j]
            hi = lo = torch.zeros_like(u[:, 0])
            for f in range(self.cn.shape[1]):
                pr = (a * (u[self.cn[:, f]] - u)).sum(1)
                hi, lo = torch.maximum(hi, pr), torch.minimum(lo, pr)
            lim = torch.ones_like(hi)
            for f in range(self.cn.shape[1]):
                d2 = -(rows[:, j] * self.cd[:, f]).sum(1)
                live = self.inner[:, f] & (d2 != 0)
                phi = torch.where(d2 > 0, hi, lo) / torch.where(live, d2, torch.ones_like(d2))
                lim = torch.where(live & (phi < lim), phi, lim)
            al.append(lim)
        near = 1e-3 * val.abs().amax(1)
        e12, e23 = val[:, 1] - val[:, 0] <= near, val[:, 2] - val[:, 1] <= near
        a0, a1, a2 = al
        m01, m12 = torch.minimum(a0, a1), torch.minimum(a1, a2)
        m = torch.minimum(m01, a2)
        both = e12 & e23
        f0 = torch.where(both, m, torch.where(e12, m01, a0))
        f1 = torch.where(both, m, torch.where(e12, m01, torch.where(e23, m12, a1)))
        f2 = torch.where(both, m, torch.where(e12, a2, torch.where(e23, m12, a2)))
        return vec @ (torch.stack([f0, f1, f2], 1)[..., None] * rows)

    def flux(self, n, left, right, irl, irr):
        """Numerical flux per unit area of two states (rho, u, v, w, p)."""
        g, discr = self.num.gamma, self.num.space_discr
        rl, ul, pl = left[:, 0], left[:, 1:4], left[:, 4]
        rr, ur, pr = right[:, 0], right[:, 1:4], right[:, 4]
        ql, qr = (ul * n).sum(1), (ur * n).sum(1)
        al, ar = torch.sqrt(g * pl / rl), torch.sqrt(g * pr / rr)
        el, er = pl / (rl * (g - 1)) + 0.5 * (ul * ul).sum(1), pr / (rr * (g - 1)) + 0.5 * (ur * ur).sum(1)
        col = lambda a: a[:, None]  # noqa: E731
        if discr == AUSM:
            hl, hr = el + pl / rl, er + pr / rr
            af = 0.5 * (al + ar)
            ml, mr = ql / af, qr / af
            plus = torch.where(ml.abs() <= 1, 0.25 * (ml + 1) ** 2 + 0.125 * (ml * ml - 1) ** 2, 0.5 * (ml + ml.abs()))
            minus = torch.where(mr.abs() <= 1, -0.25 * (mr - 1) ** 2 - 0.125 * (mr * mr - 1) ** 2,
                                0.5 * (mr - mr.abs()))
            wl = torch.where(ml.abs() <= 1, 0.25 * (ml + 1) ** 2 * (2 - ml) + 0.1875 * ml * (ml * ml - 1) ** 2,
                             0.5 * (1 + torch.sign(ml)))
            wr = torch.where(mr.abs() <= 1, 0.25 * (mr - 1) ** 2 * (2 + mr) - 0.1875 * mr * (mr * mr - 1) ** 2,
                             0.5 * (1 - torch.sign(mr)))
            mf = plus + minus
            p, fl, fr = wl * pl + wr * pr, af * 0.5 * (mf + mf.abs()) * rl, af * 0.5 * (mf - mf.abs()) * rr
            return torch.cat([col(fl + fr), col(fl) * ul + col(fr) * ur + col(p) * n, col(fl * hl + fr * hr)], 1)
        if discr == HLLC:
            hl, hr = el + irl * pl, er + irr * pr
            s = torch.sqrt(rr / rl)
            us = (ul + col(s) * ur) / col(1 + s)
            qs, hs = (ql + s * qr) / (1 + s), (hl + s * hr) / (1 + s)
            a = torch.sqrt((g - 1) * (hs - 0.5 * (us * us).sum(1)))
            sl, sr = torch.minimum(ql - al, qs - a), torch.maximum(qr + ar, qs + a)
            sm = (rr * qr * (sr - qr) - rl * ql * (sl - ql) - pr + pl) / (rr * (sr - qr) - rl * (sl - ql))
            ps = pl + rl * (ql - sl) * (ql - sm)

            def side(r, u, p, e, q, sk):
                t = 1 / (sk - sm)
                rs, k = t * (sk - q) * r, (sk - q) * r
                mom = col(t) * (col(k) * u + col(ps - p) * n)
                en = t * (k * e + ps * sm - p * q)
                star = torch.cat([col(sm * rs), col(sm) * mom + col(ps) * n, col(sm * (en + ps))], 1)
                return star, torch.cat([col(q * r), col(q * r) * u + col(p) * n, col(q * (r * e + p))], 1)

            stl, fl = side(rl, ul, pl, el, ql, sl)
            stri, fr = side(rr, ur, pr, er, qr, sr)
            star = torch.where(col(sm > 0), stl, stri)
            return torch.where(col(sl > 0), fl, torch.where(col(sr < 0), fr, star))
        hl, hr = el + pl / rl, er + pr / rr
        rh = torch.sqrt(rl * rr)
        wt = rl / (rl + rh)
        uh, hh = col(wt) * ul + col(1 - wt) * ur, wt * hl + (1 - wt) * hr
        qh, sh = (uh * n).sum(1), 0.5 * (uh * uh).sum(1)
        ah = torch.sqrt((g - 1) * (hh - sh))
        l1, l2, l5 = (qh - ah).abs(), qh.abs(), (qh + ah).abs()
        fix = self.num.eps_entr * l5
        l1, l2, l5 = (torch.where(v > fix, v, (v * v + fix * fix) / (2 * fix)) for v in (l1, l2, l5))
        dr, du, dp = rr - rl, ur - ul, pr - pl
        dq = (du * n).sum(1)
        t1 = l1 * (dp - rh * ah * dq) / (2 * ah * ah)
        t5 = l5 * (dp + rh * ah * dq) / (2 * ah * ah)
        t2, t3 = l2 * (dr - dp / (ah * ah)), l2 * rh
        mom = (col(t1) * (uh - n * col(ah)) + col(t2) * uh + col(t3) * (du - n * col(dq))
               + col(t5) * (uh + n * col(ah)))
        en = t1 * (hh - qh * ah) + t2 * sh + t3 * ((uh * du).sum(1) - qh * dq) + t5 * (hh + qh * ah)
        dis = self.num.diss_fact * torch.cat([col(t1 + t2 + t5), mom, col(en)], 1)
        con = torch.cat([col(ql * rl + qr * rr), col(ql * rl) * ul + col(qr * rr) * ur + col(pl + pr) * n,
                         col(ql * rl * hl + qr * rr * hr)], 1)
        return 0.5 * (con - dis)

    def wall_and_outflow(self, ip, q, face):
        """Flux per unit area on patch ip from the cell's state q and the face state."""
        p, a, b = self.patches[ip], self.boff[ip], self.boff[ip + 1]
        n, g = self.bfn[a:b], self.num.gamma
        s = face if p.order == 2 else q
        rho, u, pr = s[:, 0], s[:, 1:4], s[:, 4]
        zero = torch.zeros_like(rho)
        if p.bc_type == cases.BC_SLIPWALL:
            return torch.cat([zero[:, None], pr[:, None] * n, zero[:, None]], 1)
        e = rho * (pr / (rho * (g - 1)) + 0.5 * (u * u).sum(1))

        def half(r, v, en, pk):
            qn = (v * n).sum(1)[:, None]
            return 0.5 * torch.cat([qn * r[:, None], qn * r[:, None] * v + pk[:, None] * n, qn * (en + pk)[:, None]], 1)

        inner = half(rho, u, e, pr)
        if p.outflow_type == cases.BCOPT_SUPERSONIC:
            return 2 * inner
        c = torch.sqrt(g * pr / rho)
        dp = pr - p.p_out
        ub = u + n * (dp / (rho * c))[:, None]
        back = (ub * n).sum(1) < 0
        ub = torch.where(back[:, None], torch.copysign(torch.ones_like(u), u) * torch.maximum(ub.abs(), u.abs()), ub)
        rb = rho - dp / (c * c)
        po = torch.full_like(rb, p.p_out)
        sub = (u * u).sum(1) < c * c
        ub, rb = torch.where(sub[:, None], ub, u), torch.where(sub, rb, rho)
        eb = torch.where(sub, rb * (po / (rb * (g - 1)) + 0.5 * (ub * ub).sum(1)), e)
        return inner + half(rb, ub, eb, po)

    def residual(self, cv):
        q = self.primitive(cv)
        ir = 1 / q[:, 0]
        left, right, grad = q[self.c1], q[self.c2], None
        if self.num.space_order == 2:
            grad = self.gradients(q)
            left = left + (grad[self.c1] * self.dl[:, None]).sum(-1)
            right = right + (grad[self.c2] * self.dr[:, None]).sum(-1)
        f = [self.flux(self.fn, left, right, ir[self.c1], ir[self.c2]) * self.area[:, None]]
        for ip in range(len(self.patches)):
            a, b = self.boff[ip], self.boff[ip + 1]
            if b > a:
                c = self.bc[a:b]
                face = q[c] + (grad[c] * self.bd[a:b, None]).sum(-1) if grad is not None else q[c]
                f.append(self.wall_and_outflow(ip, q[c], face) * self.barea[a:b, None])
        f = torch.cat(f + [torch.zeros((1, 5), dtype=torch.float64, device=self.dev)])
        rhs = 0
        for k in range(self.cf.shape[1]):
            rhs = rhs + self.csgn[:, k:k + 1] * f[self.cf[:, k]]
        return rhs, grad

    def dt(self, cv):
        q = self.primitive(cv)
        a = torch.sqrt(self.num.gamma * q[:, 4] / q[:, 0])
        vn = 0.5 * ((q[self.c1, 1:4] + q[self.c2, 1:4]) * self.fn).sum(1)
        s = (vn.abs() + 0.5 * (a[self.c1] + a[self.c2])) * self.area
        b = ((q[self.bc, 1:4] * self.bfn).sum(1).abs() + a[self.bc]) * self.barea
        s = torch.cat([s, b, torch.zeros(1, dtype=torch.float64, device=self.dev)])
        return float(min(self.num.cfl, 2.0) * (self.vol / s[self.cf].sum(1)).min())

    A, G = (8 / 15, 5 / 12, 0.75), (0.0, 17 / 25, 5 / 9)

    def stage(self, k, cv, old, dt, src=0.0):
        """Stage k of Wray's scheme: the new state, the residual kept for the next stage, the gradients."""
        rhs, grad = self.residual(cv)
        rhs = rhs + src
        inc = rhs if k == 0 else rhs - self.G[k] * old
        return cv - self.A[k] * dt / self.vol[:, None] * inc, rhs, grad

    def step(self, cv, dt):
        old = None
        for k in range(3):
            cv, old, _ = self.stage(k, cv, old, dt)
        return cv

    def patch_pressure(self, cv, ip):
        a, b = self.boff[ip], self.boff[ip + 1]
        q = self.primitive(cv)
        c = self.bc[a:b]
        p = q[c, 4]
        if self.patches[ip].order == 2:
            p = p + (self.gradients(q)[c, 4] * self.bd[a:b]).sum(1)
        return (p * self.barea[a:b]).sum()


def _jacobi(s):
    """Eigenvalues (ascending) and eigenvectors (columns) of symmetric 3x3 matrices by cyclic rotations."""
    r, v = s.clone(), torch.eye(3, dtype=s.dtype, device=s.device).expand_as(s).clone()
    total = (s * s).sum((1, 2))
    for _ in range(12):
        off = r[:, 0, 1] ** 2 + r[:, 0, 2] ** 2 + r[:, 1, 2] ** 2
        live = off > 1e-24 * total
        if not bool(live.any()):
            break
        for p, q in ((0, 1), (0, 2), (1, 2)):
            on = live & (r[:, p, q] != 0)
            theta = (r[:, q, q] - r[:, p, p]) / torch.where(on, 2 * r[:, p, q], torch.ones_like(r[:, p, q]))
            sg = torch.where(theta < 0, -torch.ones_like(theta), torch.ones_like(theta))
            t = torch.where(on, sg / (theta.abs() + torch.sqrt(theta * theta + 1)), torch.zeros_like(theta))
            c = 1 / torch.sqrt(t * t + 1)
            rot = torch.eye(3, dtype=s.dtype, device=s.device).expand_as(s).clone()
            rot[:, p, p] = rot[:, q, q] = c
            rot[:, p, q], rot[:, q, p] = t * c, -t * c
            r, v = rot.transpose(1, 2) @ r @ rot, v @ rot
    val = torch.diagonal(r, dim1=1, dim2=2)
    order = torch.argsort(val, dim=1, stable=True)
    return torch.gather(val, 1, order), torch.gather(v, 2, order[:, None].expand_as(v))




def exact(case, seed):
    c, grid, rng = _case(case, seed)
    s = _Plain(c, grid)
    cv = torch.as_tensor(c.cv0).to(s.dev)
    if case["job"] == "march":
        t = 0.0
        for _ in range(case["steps"]):
            dt = s.dt(cv)
            cv, t = s.step(cv, dt), t + dt
        return {"cv": cv, "time": t, "steps": None}
    if case["job"] == "stages":
        dt0, dt = s.dt(cv), _fixed_dt(c, grid)
        src = torch.as_tensor(_source(c, rng, dt) * grid.vol[:, None]).to(s.dev)
        for _ in range(case["steps"]):
            old = None
            for k in range(3):
                cv, old, grad = s.stage(k, cv, old, dt, src)
        return {"dt": dt0, "grad": grad, "rhs": old, "cv": cv}
    if case["job"] in ("linearise", "autograd"):
        cv.requires_grad_(True)
        dot, bar = _directions(c, rng)
        rhs, _ = s.residual(cv)
        # the adjoint is linear in its seed: its own derivative along dot is the tangent
        seed_ = torch.as_tensor(bar).to(s.dev).requires_grad_(True)
        (cv_bar,) = torch.autograd.grad(rhs, cv, seed_, create_graph=case["job"] == "linearise")
        if case["job"] == "autograd":
            return {"rhs": rhs.detach(), "cv_bar": cv_bar.detach()}
        (rhs_dot,) = torch.autograd.grad(cv_bar, seed_, torch.as_tensor(dot).to(s.dev))
        return {"rhs_dot": rhs_dot, "cv_bar": cv_bar.detach()}
    if case["reconst"] == BJ:
        return None  # its derivative is defined through perturbed eigenvectors, which plain autograd does not give
    cv.requires_grad_(True)
    x, dt, j = cv, _fixed_dt(c, grid), 0.0
    for _ in range(case["steps"]):
        x = s.step(x, dt)
        j = j + dt * s.patch_pressure(x, 1)
    (bar,) = torch.autograd.grad(j, cv)
    return {"J": float(j.detach()), "cv_bar": bar}
