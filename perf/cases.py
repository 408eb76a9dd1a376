"""The measured cases: what a user of this framework has it do, through the
Python call surface (``topopt3d_b200.TopOpt`` and the classes beside it).

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare`` makes what a user's program holds before the call, ``run`` is one
pass through the public entry points, ``work`` the bytes and operations a
pass cannot do without, and ``exact`` the result in 64-bit torch arithmetic
without this repository's code.

The kinds of work:

* ``step``     one design iteration: MatIntFnc, FEAssemble, FESolve from a
               zero guess, compliance and its design gradient
* ``optimize`` the optimisation loop itself: OC updates of a compliance
               problem with a volume constraint, warm-started solves, host
               arrays
* ``loads``    several load cases on an assembled hierarchy
* ``apply32``  the FP32 matrix-free operator on device buffers
* ``filter``   the density filter, forward and transpose
* ``buckling`` stress stiffness, the largest buckling factors and the design
               gradient of their aggregate
* ``mma``      one MMA update with several constraints
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import topopt3d_b200 as T
from topopt3d_b200 import problems as P

EPS = 1e-10          # the SIMP floor of MatIntFnc
PENAL = 3.0


# --------------------------------------------------------------------- cases

def listed():
    return [
        # the smallest meshes of the tests: launches and host work only
        dict(name="step_tiny_fp64", kind="step", nx=12, ny=6, nz=6, levels=2, rmin=1.5,
             precision="fp64", host=True),
        # the FP64 cantilever configuration, host arrays as a script passes them
        dict(name="step_small_fp64", kind="step", nx=48, ny=24, nz=24, levels=3, rmin=1.5,
             precision="fp64", host=True),
        # a medium mesh with odd element counts in every direction
        dict(name="step_odd_mixed", kind="step", nx=91, ny=47, nz=53, levels=4, rmin=1.5,
             precision="mixed", host=False),
        # the large cantilever (5.4M dof), mixed precision: the headline workload
        dict(name="step_large_mixed", kind="step", nx=192, ny=96, nz=96, levels=5, rmin=1.5,
             precision="mixed", host=False),
        # the same in plain FP64
        dict(name="step_large_fp64", kind="step", nx=192, ny=96, nz=96, levels=5, rmin=1.5,
             precision="fp64", host=False),
        # the optimisation loop of the OC configuration: 3 evaluations, 2 updates
        dict(name="optimize_mixed", kind="optimize", nx=64, ny=32, nz=32, levels=4, rmin=2.0,
             updates=2),
        # 8 load cases at once (the multi-load configuration)
        dict(name="loads8_mixed", kind="loads", nx=128, ny=64, nz=64, levels=5, rmin=1.5,
             precision="mixed", nrhs=8),
        # an uneven number of load cases on a ragged mesh, FP64
        dict(name="loads5_ragged_fp64", kind="loads", nx=75, ny=41, nz=34, levels=4, rmin=1.5,
             precision="fp64", nrhs=5),
        # the matrix-free operator alone, as a caller's own iteration uses it
        dict(name="apply32_large", kind="apply32", nx=192, ny=96, nz=96, levels=5, rmin=1.5),
        # a wide density filter, both directions
        dict(name="filter_wide", kind="filter", nx=128, ny=64, nz=64, levels=4, rmin=3.0),
        # the buckling column: 6 factors and their design gradient
        dict(name="buckling_column", kind="buckling", nx=96, ny=48, nz=48, levels=4, rmin=1.5,
             nev=6, block=12),
        # one MMA update with two constraints on the OC configuration's mesh
        dict(name="mma_two", kind="mma", nx=64, ny=32, nz=32, levels=4, rmin=2.0, m=2),
    ]


def _levels(nel):
    """GMG levels that leave a coarsest level of some six elements across."""
    n = max(1, int(math.floor(math.log2(max(1.0, min(nel) / 6.0)))) + 1)
    while True:
        d = [t + 1 for t in nel]
        for _ in range(n - 1):
            d = [(t + 1) // 2 for t in d]
        if 3 * d[0] * d[1] * d[2] <= 2500:
            return n
        n += 1


def _mesh(rng, lo, hi):
    """A box of up to 2 : 1 : 1, lo..hi elements across (log-uniform), even
    and odd sizes alike."""
    a = lo * (hi / lo) ** rng.random()
    ny = max(lo, min(hi, int(a * rng.uniform(0.9, 1.3))))
    nz = max(lo, min(hi, int(a * rng.uniform(0.9, 1.3))))
    nx = max(lo, min(2 * hi, int(a * rng.uniform(1.2, 2.0))))
    if rng.random() < 0.5:               # half of the meshes coarsen evenly
        nx, ny, nz = nx - nx % 2, ny - ny % 2, nz - nz % 2
    return nx, ny, nz


def draw(rng):
    kind = rng.choice(("step", "step", "step", "optimize", "loads", "loads", "apply32", "filter",
                       "buckling", "mma"))
    hi = {"step": 96, "optimize": 48, "loads": 64, "apply32": 96, "filter": 64, "buckling": 40,
          "mma": 48}[kind]
    lo = {"buckling": 12, "apply32": 16, "filter": 12, "optimize": 10, "mma": 10}.get(kind, 6)
    nel = _mesh(rng, lo, hi)
    if kind == "buckling":
        nel = (nel[0] // 2 + 1, nel[1], nel[2])
    c = dict(kind=kind, nx=nel[0], ny=nel[1], nz=nel[2], levels=_levels(nel), rmin=1.5)
    if kind == "step":
        c.update(precision=rng.choice(("fp64", "mixed")), host=max(nel) <= 64,
                 rmin=rng.choice((1.5, 1.5, 2.0)))
    elif kind == "optimize":
        c.update(updates=rng.randint(1, 2), rmin=2.0)
    elif kind == "loads":
        c.update(precision=rng.choice(("fp64", "mixed")), nrhs=rng.randint(2, 8))
    elif kind == "filter":
        c.update(rmin=rng.choice((1.5, 2.0, 2.5, 3.0)))
    elif kind == "buckling":
        c.update(nev=rng.randint(2, 6), block=12)
    elif kind == "mma":
        c.update(m=rng.randint(2, 4), rmin=2.0)
    return c


# -------------------------------------------------------------------- inputs

def _nel(c):
    return c["nx"], c["ny"], c["nz"]


def _sizes(c):
    nx, ny, nz = _nel(c)
    return nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)


def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed):
    g = torch.Generator(device=_dev())
    g.manual_seed(int(seed))
    return g


def _uniform(seed, n, lo, hi):
    return torch.rand(n, generator=_gen(seed), device=_dev(), dtype=torch.float64) * (hi - lo) + lo


def _design(c, seed):
    """A design in the middle of an optimisation: a smooth field of
    intermediate densities (random values on a grid 8 times coarser,
    interpolated) with a little scatter."""
    nx, ny, nz = _nel(c)
    grid = [1 + -(-n // 8) for n in (nz, ny, nx)]
    v = _uniform(seed, grid[0] * grid[1] * grid[2], 0.0, 1.0).reshape(1, 1, *grid)
    v = torch.nn.functional.interpolate(v, size=(nz, ny, nx), mode="trilinear",
                                        align_corners=True).reshape(-1)
    return 0.3 + 0.5 * v + _uniform(seed + 1000003, nx * ny * nz, 0.0, 0.05)


def _point_loads(c, seed):
    """Unit point loads on random nodes of the x = max face."""
    nx, ny, nz = _nel(c)
    r = np.random.default_rng(int(seed) + 77)
    F = np.zeros((c["nrhs"], 3 * _sizes(c)[1]))
    for j in range(c["nrhs"]):
        d = r.standard_normal(3)
        n = nx + (nx + 1) * (int(r.integers(0, ny + 1)) + (ny + 1) * int(r.integers(0, nz + 1)))
        F[j, 3 * n:3 * n + 3] = d / np.linalg.norm(d)
    return torch.from_numpy(F).to(_dev())


_streams = {}


def _stream():
    """The one stream a user's program issues this library's work on."""
    d = torch.cuda.current_device()
    if d not in _streams:
        _streams[d] = torch.cuda.Stream()
    return _streams[d]


def _problem(c):
    nel = _nel(c)
    t = T.TopOpt(nel, rmin=c["rmin"], mg_levels=c["levels"])
    P.apply_bcs(t, P.column_bcs(nel) if c["kind"] == "buckling" else P.cantilever_bcs(nel))
    t.penal = PENAL
    t.FEInitialize()
    t.set_stream(_stream().cuda_stream)
    return t


def _opts(c):
    # load cases are superposed afterwards, so they are solved a digit further
    return T.default_opts(precision=T.PREC_MIXED if c["precision"] == "mixed" else T.PREC_FP64,
                          rtol=1e-9 if c["kind"] == "loads" else 1e-8)


# ------------------------------------------------------------ prepare and run

class State:
    pass


def prepare(case, seed):
    s = State()
    s.kind = k = case["kind"]
    ne, nn = _sizes(case)
    if k == "mma":
        _prepare_mma(s, case, seed)
        return s
    s.t = t = _problem(case)
    x = _design(case, seed)
    torch.cuda.synchronize()
    if k == "step":
        s.opts = _opts(case)
        s.host = case["host"]
        if s.host:
            s.x, s.zero, s.dC, s.U = x.cpu().numpy(), np.zeros(3 * nn), None, np.zeros(3 * nn)
        else:
            s.x, s.zero = x, torch.zeros(3 * nn, device=x.device, dtype=torch.float64)
            s.dC, s.U = torch.empty_like(x), torch.empty_like(s.zero)
    elif k == "optimize":
        s.opts = T.default_opts(precision=T.PREC_MIXED)
        s.x, s.zero, s.updates = x.cpu().numpy(), np.zeros(3 * nn), case["updates"]
        t.function_list = [T.Compliance([1.0], 0.0, 1.0, True), T.Volume([0.4], 0.0, 1.0, False)]
    elif k == "loads":
        s.opts, s.nrhs = _opts(case), case["nrhs"]
        s.b = _point_loads(case, seed).reshape(-1)
        s.U = torch.zeros_like(s.b)
        t.MatIntFnc(x)
        t.FEAssemble(s.opts)
        s.t.solve(s.b, s.U, nrhs=s.nrhs, opts=s.opts)   # the block size is chosen here
    elif k == "apply32":
        t.MatIntFnc(x)
        s.u = (_uniform(seed + 1, 3 * nn, -1.0, 1.0)).to(torch.float32)
        s.y = torch.empty_like(s.u)
    elif k == "filter":
        s.x, s.g = x, _uniform(seed + 1, ne, -1.0, 0.0)
        s.rho, s.dx = torch.empty_like(x), torch.empty_like(x)
    elif k == "buckling":
        t.MatIntFnc(x)
        t.FEAssemble()
        t.FESolve()
        s.f = T.Stability([1.0], 0.0, 1.0, True, calc_gradient=True, nev=case["nev"],
                          block=case["block"])
    torch.cuda.synchronize()
    return s


def _prepare_mma(s, c, seed):
    """The state of an MMA run after two updates, and the functions' values
    at its design."""
    s.t = _problem(c)
    n, m = _sizes(c)[0], c["m"]
    r = np.random.default_rng(int(seed))
    s.xval = r.uniform(0.3, 0.6, n)
    s.xold1 = np.clip(s.xval + r.uniform(-0.05, 0.05, n), 0.0, 1.0)
    s.xold2 = np.clip(s.xold1 + r.uniform(-0.05, 0.05, n), 0.0, 1.0)
    s.low, s.upp = s.xval - 0.4, s.xval + 0.4
    s.dfdx = -r.uniform(0.1, 2.0, n) / n
    s.dgdx = np.zeros((n, m))
    for j in range(m):                    # volume shares, each of a part of the mesh
        part = slice(0, n) if j == 0 else slice((j - 1) * n // m, (j + 1) * n // m)
        s.dgdx[part, j] = r.uniform(0.8, 1.2, part.stop - part.start) / n
    s.g = np.array([0.02 / (j + 1) for j in range(m)])
    s.n = n


def run(s):
    t = s.t
    if s.kind == "step":
        t.set("U", s.zero)
        t.MatIntFnc(s.x)
        t.FEAssemble(s.opts)
        t.FESolve(s.opts)
        C, dC, _ = t.compliance(out=s.dC)
        return {"C": C, "dC": dC, "U": t.get("U", s.U)}
    if s.kind == "optimize":
        t.set("U", s.zero)
        oc = T.OC(n=t.nElem, maxiter=s.updates)
        oc.xval = s.x.copy()
        h = T.optimize(t, oc, opts=s.opts)
        return {"C": [r["values"][0] for r in h], "V": [r["values"][1] for r in h],
                "x": oc.xval, "U": t.U}
    if s.kind == "loads":
        with torch.cuda.stream(_stream()):
            s.U.zero_()
        t.solve(s.b, s.U, nrhs=s.nrhs, opts=s.opts)
        return s.U
    if s.kind == "apply32":
        rc = t._lib.tpo_apply_f32(t._h, ctypes.c_void_p(s.u.data_ptr()),
                                  ctypes.c_void_p(s.y.data_ptr()))
        if rc != 0:
            raise RuntimeError("tpo_apply_f32: %d" % rc)
        return s.y
    if s.kind == "filter":
        t.filter(s.x, s.rho)
        t.filter(s.g, s.dx, transpose=True)
        return {"rho": s.rho, "dx": s.dx}
    if s.kind == "buckling":
        s.f.Function(t)
        return {"lambda": s.f.lam, "value": s.f.values[0], "grad": s.f.gradients}
    mma = T.MMA(n=s.n, iter=3, fresh_start=False, xold1=s.xold1.copy(), xold2=s.xold2.copy(),
                low=s.low.copy(), upp=s.upp.copy())
    mma.xval = s.xval
    mma.Update(t, s.dfdx, s.g, s.dgdx)
    return {"x": mma.xval, "xold1": mma.xold1, "xold2": mma.xold2, "low": mma.low,
            "upp": mma.upp, "change": mma.Change}


# ---------------------------------------------------------------------- work

# fine-operator applications a solve to 1e-8 takes: some 14 PCG iterations,
# each the product K p and a V-cycle with four more on the finest level
_APPLIES = 14 * 5
_OPS = 153           # operations of one element in the matrix-free form


def work(case):
    ne, nn = _sizes(case)
    k = case["kind"]
    if k == "apply32":
        return {"bytes": 24 * nn + nn + 4 * ne, "flops": _OPS * ne}
    if k == "filter":
        taps = (4.0 / 3.0) * math.pi * case["rmin"] ** 3
        return {"bytes": 32 * ne, "flops": 4 * taps * ne}
    if k == "mma":
        return {"bytes": 8 * ne * (12 + case["m"]), "flops": 400.0 * ne}

    def applies(n, p):
        return n * (6 * p * nn + nn + p * ne), n * _OPS * ne

    if k == "buckling":
        b, f = applies(20 * 5 * case["block"] + _APPLIES * case["nev"], 8)
        return {"bytes": b, "flops": f}
    cols, p = 1, 8
    if k == "optimize":
        cols, p = case["updates"] + 1, 4
    elif case["precision"] == "mixed":
        p = 4
    if k == "loads":
        cols = case["nrhs"]
    b, f = applies(_APPLIES * cols, p)
    return {"bytes": b, "flops": f}


# ------------------------------------------------- the same in 64-bit torch

def _gauss_k0(nu=0.3, e0=1.0):
    """Stiffness of the unit hexahedron, 2x2x2 Gauss points, corners in
    lexicographic order (x fastest)."""
    lam = e0 / ((1 + nu) * (1 - 2 * nu))
    D = np.zeros((6, 6))
    D[:3, :3] = nu * lam
    D[range(3), range(3)] = (1 - nu) * lam
    D[range(3, 6), range(3, 6)] = e0 / (2 * (1 + nu))
    sg = np.array([[1.0 if (l >> d) & 1 else -1.0 for d in range(3)] for l in range(8)])
    K = np.zeros((24, 24))
    for q in range(8):
        xi = sg[q] / math.sqrt(3.0)
        B = np.zeros((6, 24))
        for l in range(8):
            h = [1 + sg[l, d] * xi[d] for d in range(3)]
            gx, gy, gz = (sg[l, 0] * h[1] * h[2] / 4, sg[l, 1] * h[0] * h[2] / 4,
                          sg[l, 2] * h[0] * h[1] / 4)
            B[0, 3 * l], B[1, 3 * l + 1], B[2, 3 * l + 2] = gx, gy, gz
            B[3, 3 * l], B[3, 3 * l + 1] = gy, gx
            B[4, 3 * l + 1], B[4, 3 * l + 2] = gz, gy
            B[5, 3 * l], B[5, 3 * l + 2] = gz, gx
        K += B.T @ D @ B / 8.0
    return K


class _Exact:
    def __init__(self, c):
        self.c, self.nel = c, _nel(c)
        nx, ny, nz = self.nel
        self.K0 = torch.from_numpy(_gauss_k0()).to(_dev())
        self.free = torch.ones(nz + 1, ny + 1, nx + 1, 1, device=_dev(), dtype=torch.float64)
        self.free[:, :, 0] = 0.0            # the cantilever's clamped face

    def _corners(self):
        nx, ny, nz = self.nel
        for l in range(8):
            i, j, k = l & 1, (l >> 1) & 1, l >> 2
            yield l, (slice(k, k + nz), slice(j, j + ny), slice(i, i + nx))

    def gather(self, u):
        return torch.cat([u[s] for _, s in self._corners()], dim=-1)

    def scatter(self, ye):
        nx, ny, nz = self.nel
        y = ye.new_zeros(nz + 1, ny + 1, nx + 1, 3)
        for l, s in self._corners():
            y[s] += ye[..., 3 * l:3 * l + 3]
        return y

    def mult(self, E, u):
        y = self.scatter((self.gather(u * self.free) @ self.K0) * E[..., None])
        return y * self.free + u * (1 - self.free)

    def solve(self, E, b, seconds=15.0):
        """Jacobi-preconditioned CG to a relative residual of 1e-13."""
        import time
        diag = self.scatter(E[..., None] * torch.diagonal(self.K0))
        dinv = self.free / diag + (1 - self.free)
        x = torch.zeros_like(b)
        r = b.clone()
        z = dinv * r
        p = z.clone()
        rz = (r * z).sum()
        stop = 1e-13 * float(b.norm())
        t0 = time.monotonic()
        for it in range(200000):
            q = self.mult(E, p)
            a = rz / (p * q).sum()
            x += a * p
            r -= a * q
            z = dinv * r
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
            if it % 50 == 49:
                if float(r.norm()) <= stop:
                    return x
                if time.monotonic() - t0 > seconds:
                    return None
        return None

    def taps(self):
        R = self.c["rmin"]
        n = int(R)
        for k in range(-n, n + 1):
            for j in range(-n, n + 1):
                for i in range(-n, n + 1):
                    d = math.sqrt(i * i + j * j + k * k)
                    if d < R:
                        yield i, j, k, 1.0 - d / R

    def cone(self, v):
        """sum_j W_ij v_j with the unscaled cone weights W (symmetric)."""
        nx, ny, nz = self.nel
        out = torch.zeros_like(v)

        def cut(n, d):   # rows and columns of a shift by d
            return slice(max(0, -d), n - max(0, d)), slice(max(0, d), n - max(0, -d))
        for i, j, k, w in self.taps():
            if abs(i) >= nx or abs(j) >= ny or abs(k) >= nz:
                continue
            (ri, ci), (rj, cj), (rk, ck) = cut(nx, i), cut(ny, j), cut(nz, k)
            out[rk, rj, ri] += w * v[ck, cj, ci]
        return out

    def box(self, v):
        nx, ny, nz = self.nel
        return v.reshape(nz, ny, nx)

    def moduli(self, x):
        """rho = P x, E and dE/drho, and the filter's row sums."""
        x = self.box(x)
        rows = self.cone(torch.ones_like(x))
        rho = self.cone(x) / rows
        return rho, EPS + (1 - EPS) * rho ** PENAL, (1 - EPS) * PENAL * rho ** (PENAL - 1), rows


def exact(case, seed):
    k = case["kind"]
    if k not in ("step", "loads", "apply32", "filter"):
        return None
    nx, ny, nz = _nel(case)
    e = _Exact(case)
    x = _design(case, seed)
    rho, E, dE, rows = e.moduli(x)
    if k == "filter":
        g = e.box(_uniform(seed + 1, _sizes(case)[0], -1.0, 0.0))
        return {"rho": rho.reshape(-1), "dx": e.cone(g / rows).reshape(-1)}
    if k == "apply32":
        u = _uniform(seed + 1, 3 * _sizes(case)[1], -1.0, 1.0).to(torch.float32).double()
        return e.mult(E, u.reshape(nz + 1, ny + 1, nx + 1, 3)).reshape(-1)
    if k == "loads":
        b = _point_loads(case, seed)
        out = []
        for j in range(case["nrhs"]):
            v = e.solve(E, b[j].reshape(nz + 1, ny + 1, nx + 1, 3), 18.0 / case["nrhs"])
            if v is None:
                return None
            out.append(v.reshape(-1))
        return torch.cat(out)
    F = x.new_zeros(nz + 1, ny + 1, nx + 1, 3)
    F[0, :, nx, 2] = -1.0 / (ny + 1)
    U = e.solve(E, F)
    if U is None:
        return None
    ue = e.gather(U)
    g = -dE * ((ue @ e.K0) * ue).sum(-1)
    return {"C": float((U * F).sum()), "dC": e.cone(g / rows).reshape(-1), "U": U.reshape(-1)}
