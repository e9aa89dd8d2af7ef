"""Performance cases of the pressure-equation library, through its public entry points.

A furnace run calls, once per SIMPLE outer iteration, the transport solves of
its momentum, energy and species equations (compute_residual_3d_mpi, then
line-by-line TDMA sweeps) and the pressure step: assembly, a capped Jacobi-PCG
(50 iterations, the reference's max_inner_pres) and the velocity and pressure
corrections. The cases are those calls on the meshes a user runs, from the
smoke mesh to the fine one, odd sizes among the drawn ones:

  cg         the pressure CG on device-resident arrays, pp starting from zero
  cg_host    the drop-in ``cg_3d`` on page-locked host arrays
  transport  residual and TDMA sweeps of one transport equation
  assemble   the assembly of the pressure-correction equation
  pcorr      the post-CG corrections
  pstep      assembly, CG and corrections chained (one pressure step)
  batch      many independent furnaces' pressure equations in one launch

Device arrays that a pass starts from are restored on the library's own
stream, which is what orders them before the call.
"""
import importlib
import math

import numpy as np
import torch

eaf = importlib.import_module("hornofusion-full3d_b200")
gen = importlib.import_module("hornofusion-full3d_b200.eafgen")

DEV = "cuda"
F64 = torch.float64
SMALL = 1e-30
TOL = eaf.SOR_TOL_PRESSURE
CAP = eaf.MAX_INNER_PRES
NAMES = ("aW", "aE", "aS", "aN", "aB", "aT", "aP", "Su")


def _case(kind, dims, **more):
    nr, nth, nz = dims
    return {"kind": kind, "nr": nr, "nth": nth, "nz": nz, **more}


def _batch_case(n0, n1, n2, n3, iters):
    """Systems of the four meshes of the repository's batch mix."""
    return {"kind": "batch", "n0": n0, "n1": n1, "n2": n2, "n3": n3, "iters": iters}


def listed():
    return [
        # the smallest call: the smoke mesh, where launches and latency count
        dict(_case("cg", (12, 24, 16), iters=CAP), name="cg-12x24x16"),
        # a mid-size serving mesh through the Fortran-style drop-in, host arrays
        dict(_case("cg_host", (35, 70, 50), iters=CAP), name="cg-host-35x70x50"),
        # an odd mesh that no tuning table knows
        dict(_case("cg", (41, 83, 57), iters=CAP), name="cg-41x83x57"),
        # the production mesh
        dict(_case("cg", (60, 120, 84), iters=CAP), name="cg-60x120x84"),
        # the fine mesh, whose working set is beyond L2
        dict(_case("cg", (120, 240, 168), iters=CAP), name="cg-120x240x168"),
        # one transport equation of the smoke, production and fine meshes
        dict(_case("transport", (12, 24, 16), sweeps=2), name="transport-12x24x16"),
        dict(_case("transport", (60, 120, 84), sweeps=3), name="transport-60x120x84"),
        dict(_case("transport", (120, 240, 168), sweeps=1), name="transport-120x240x168"),
        # assembly and corrections by themselves (a caller with its own solver)
        dict(_case("assemble", (60, 120, 84), flags=7), name="assemble-60x120x84"),
        dict(_case("pcorr", (60, 120, 84), gas=True), name="pcorr-60x120x84"),
        # the whole pressure step, device-resident
        dict(_case("pstep", (60, 120, 84), flags=7, iters=CAP), name="pstep-60x120x84"),
        # a campaign of uneven furnaces (the batch mix in its proportions)
        dict(_batch_case(13, 10, 7, 2, 200), name="batch-mix"),
    ]


def _draw_dims(rng, lo, hi):
    """A mesh of lo..hi cells (log-uniform): r shortest, theta about twice r."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    nr = max(3, round((n / 2.8) ** (1.0 / 3.0) * rng.uniform(0.75, 1.3)))
    nth = max(4, round(nr * rng.uniform(1.5, 2.6)))
    nz = max(3, int(n / (nr * nth)))
    return nr, nth, nz


def draw(rng):
    kind = rng.choice(["cg"] * 6 + ["cg_host"] * 2 + ["transport"] * 4 + ["assemble"] * 2
                      + ["pcorr"] * 2 + ["pstep"] * 3 + ["batch"])
    if kind == "cg":
        return _case(kind, _draw_dims(rng, 2e3, 3e6), iters=rng.randint(20, CAP))
    if kind == "cg_host":
        return _case(kind, _draw_dims(rng, 2e3, 3e5), iters=rng.randint(20, CAP))
    if kind == "transport":
        return _case(kind, _draw_dims(rng, 2e3, 8e5), sweeps=rng.randint(1, 3))
    if kind == "assemble":
        return _case(kind, _draw_dims(rng, 2e3, 1e6), flags=rng.choice([7, 7, 3, 1, 5, 0]))
    if kind == "pcorr":
        return _case(kind, _draw_dims(rng, 2e3, 1e6), gas=rng.random() < 0.7)
    if kind == "pstep":
        return _case(kind, _draw_dims(rng, 2e3, 8e5), flags=rng.choice([7, 7, 3, 1]),
                     iters=rng.randint(20, CAP))
    return _batch_case(rng.randint(2, 16), rng.randint(1, 12), rng.randint(0, 8),
                       rng.randint(0, 2), rng.randint(50, 200))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _halo(a):
    nz, nth, nr = a.shape
    h = torch.zeros((nz + 4, nth + 4, nr + 4), dtype=F64, device=a.device)
    h[2:-2, 2:-2, 2:-2] = a
    return h


def _wrap(h):
    """Periodic theta halo columns."""
    nth = h.shape[1] - 4
    lo, hi = h[:, nth:nth + 2].clone(), h[:, 2:4].clone()
    h[:, 0:2] = lo
    h[:, nth + 2:nth + 4] = hi
    return h


def _hmean(a, b):
    return 2.0 * a * b / (a + b)


def _pressure_system(nr, nth, nz, seed):
    """The pressure-correction operator of a steel bath under gas with scrap
    spheres on a uniform cylindrical mesh (the repository's generator's
    recipe), drawn on the GPU; halo-layout arrays in NAMES order."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    dr, dth, dz = gen.R_FURNACE / nr, 2.0 * math.pi / nth, gen.H_FURNACE / nz
    ar = lambda n: torch.arange(n, dtype=F64, device=DEV)  # noqa: E731
    rc = ((ar(nr) + 0.5) * dr)[None, None, :]
    th = ((ar(nth) + 0.5) * dth)[None, :, None]
    z = ((ar(nz) + 0.5) * dz)[:, None, None]
    x, y = rc * torch.cos(th), rc * torch.sin(th)
    bath = (z < gen.BATH_DEPTH) & (rc < gen.BATH_RADIUS) & (th > -1.0)
    rho = torch.where(bath, gen.RHO_STEEL, gen.RHO_GAS).to(F64)
    u = np.random.default_rng(seed).random((8 + min(56, nr // 3), 4))
    for a, b, c, d in u:
        rs, ts, zs, rad = gen.R_FURNACE * math.sqrt(a), 2 * math.pi * b, gen.H_FURNACE * c, 0.2 + 0.3 * d
        inside = (x - rs * math.cos(ts)) ** 2 + (y - rs * math.sin(ts)) ** 2 + (z - zs) ** 2 <= rad * rad
        rho = torch.where(inside, gen.RHO_SCRAP, rho)
    abar = torch.exp(math.log(1e2) + math.log(1e2) * torch.rand((nz, nth, nr), dtype=F64, device=DEV, generator=g))
    aE, aT = torch.zeros_like(rho), torch.zeros_like(rho)
    Ar = (ar(nr - 1) + 1.0) * dr * dth * dz
    aE[:, :, :-1] = _hmean(rho[:, :, :-1], rho[:, :, 1:]) * Ar * Ar / _hmean(abar[:, :, :-1], abar[:, :, 1:])
    aN = _hmean(rho, rho.roll(-1, 1)) * (dr * dz) ** 2 / _hmean(abar, abar.roll(-1, 1))
    Az = rc * dr * dth
    aT[:-1] = _hmean(rho[:-1], rho[1:]) * Az * Az / _hmean(abar[:-1], abar[1:])
    aW, aS, aB = torch.zeros_like(rho), aN.roll(1, 1), torch.zeros_like(rho)
    aW[:, :, 1:] = aE[:, :, :-1]
    aB[1:] = aT[:-1]
    aP = ((((aW + aE) + aS) + aN) + aB) + aT
    b = torch.randn((nz, nth, nr), dtype=F64, device=DEV, generator=g) * 1e-3
    b = b - b.mean()
    # the pinned cell (nr, 1, 1), its links folded
    for a in (aW, aE, aS, aN, aB, aT, b):
        a[0, 0, nr - 1] = 0.0
    aP[0, 0, nr - 1] = 1.0
    aE[0, 0, nr - 2] = 0.0
    aN[0, nth - 1, nr - 1] = 0.0
    aS[0, 1, nr - 1] = 0.0
    aB[1, 0, nr - 1] = 0.0
    return [_halo(a) for a in (aW, aE, aS, aN, aB, aT, aP, b)]


def _transport_system(nr, nth, nz, seed):
    """An upwind transport operator (asymmetric links, diagonally dominant,
    5 % identity rows) and a starting field, drawn on the GPU."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    rand = lambda *s: torch.rand(s, dtype=F64, device=DEV, generator=g)   # noqa: E731
    randn = lambda *s: torch.randn(s, dtype=F64, device=DEV, generator=g)  # noqa: E731

    def faces(*s):
        D, F = 0.5 + rand(*s), randn(*s)
        return D + F.clamp(min=0.0), D + (-F).clamp(min=0.0)  # seen from the + side, from the - side

    rp, rm = faces(nz, nth, nr + 1)
    tp, tm = faces(nz, nth, nr)
    zp, zm = faces(nz + 1, nth, nr)
    aW, aE = rp[:, :, :-1].clone(), rm[:, :, 1:].clone()
    aS, aN = tp.roll(1, 1).clone(), tm.clone()
    aB, aT = zp[:-1].clone(), zm[1:].clone()
    aW[:, :, 0] = 0.0
    aE[:, :, -1] = 0.0
    aB[0] = 0.0
    aT[-1] = 0.0
    aP = (aW + aE + aS + aN + aB + aT) * (1.0 + 0.1 * rand(nz, nth, nr))
    Su = randn(nz, nth, nr)
    trivial = rand(nz, nth, nr) < 0.05
    for a in (aW, aE, aS, aN, aB, aT, Su):
        a[trivial] = 0.0
    aP[trivial] = 1.0
    return [_halo(a) for a in (aW, aE, aS, aN, aB, aT, aP, Su)], _wrap(_halo(randn(nz, nth, nr)))


def _fields_on(f):
    """A generator's numpy fields as device tensors on an object of its kind."""
    c = f.copy()
    for k, v in c.__dict__.items():
        if isinstance(v, np.ndarray):
            setattr(c, k, torch.from_numpy(v).to(DEV))
    return c


STEP_STATE = ("p", "liq_ur", "liq_uth", "liq_uz", "gas_ur", "gas_uth", "gas_uz")


def _dims(case):
    return case["nr"], case["nth"], case["nz"]


def _batch_dims(case):
    out = []
    for k, ((nr, nth, nz, _), _) in enumerate(gen.BATCH_MIX):
        out += [(nr, nth, nz)] * case["n%d" % k]
    return out


def _batch_systems(case, seed):
    return [_pressure_system(*d, seed * 1000 + k) for k, d in enumerate(_batch_dims(case))]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "batch":
        dims = _batch_dims(case)
        s["arrays"] = _batch_systems(case, seed)
        s["phi"] = [torch.zeros(gen.halo_shape(*d), dtype=F64, device=DEV) for d in dims]
        b = s["solver"] = eaf.Batch(dims)
        for k, (a, phi) in enumerate(zip(s["arrays"], s["phi"])):
            b.set_system(k, a, phi, device_ptrs=True)
        s["stream"] = torch.cuda.ExternalStream(eaf.load().eaf_batch_stream(b._h))
        torch.cuda.synchronize()
        return s
    nr, nth, nz = _dims(case)
    if kind == "cg_host":
        s["arrays"] = []
        for a in _pressure_system(nr, nth, nz, seed):
            h = eaf.host_empty(tuple(a.shape))
            h[...] = a.cpu().numpy()
            s["arrays"].append(h)
        s["phi"] = eaf.host_empty(gen.halo_shape(nr, nth, nz))
        return s
    s["solver"] = eaf.CGSolver(nr, nth, nz)
    s["stream"] = torch.cuda.ExternalStream(s["solver"].stream)
    if kind == "cg":
        s["arrays"] = _pressure_system(nr, nth, nz, seed)
        s["phi"] = torch.zeros(gen.halo_shape(nr, nth, nz), dtype=F64, device=DEV)
    elif kind == "transport":
        s["arrays"], s["phi0"] = _transport_system(nr, nth, nz, seed)
        s["phi"] = s["phi0"].clone()
    elif kind == "pcorr":
        s["fields"] = _fields_on(gen.make_pcorr_fields(nr, nth, nz, seed, has_gas=case["gas"]))
    else:
        f = s["fields"] = _fields_on(gen.make_pressure_state(nr, nth, nz, seed, flags=case["flags"]))
        if kind == "pstep":
            s["state"] = [getattr(f, n) for n in STEP_STATE]
            s["state0"] = [a.clone() for a in s["state"]]
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "cg_host":
        s["phi"][...] = 0.0
        res, it = eaf.cg_3d(*s["arrays"], s["phi"], max_iter=case["iters"], tol=TOL)
        return {"phi": s["phi"], "residual": res, "n_iter": it}
    if kind == "cg":
        with torch.cuda.stream(s["stream"]):
            s["phi"].zero_()
        res, it, _ = s["solver"].solve(s["arrays"], s["phi"], case["iters"], TOL, device_ptrs=True)
        return {"phi": s["phi"], "residual": res, "n_iter": it}
    if kind == "transport":
        with torch.cuda.stream(s["stream"]):
            s["phi"].copy_(s["phi0"])
        res = s["solver"].residual(s["arrays"], s["phi"], device_ptrs=True)
        s["solver"].tdma(s["arrays"], s["phi"], case["sweeps"], device_ptrs=True)
        return {"phi": s["phi"], "residual": res}
    if kind == "pcorr":
        s["solver"].pressure_correct(s["fields"], device_ptrs=True)
        return s["fields"].outputs()
    if kind == "assemble":
        res = s["solver"].pressure_assemble(s["fields"], device_ptrs=True)
        return {**s["fields"].outputs(), "residual": res}
    if kind == "pstep":
        with torch.cuda.stream(s["stream"]):
            torch._foreach_copy_(s["state"], s["state0"])
        res, cg_res, it, _ = s["solver"].pressure_step(s["fields"], 0.7, case["iters"], TOL, device_ptrs=True)
        return {**s["fields"].outputs(), **dict(zip(STEP_STATE, s["state"])),
                "residual": res, "cg_residual": cg_res, "n_iter": it}
    with torch.cuda.stream(s["stream"]):
        torch._foreach_zero_(s["phi"])
    s["solver"].solve(max_iter=case["iters"], tol=TOL)
    got = [s["solver"].result(k) for k in range(len(s["phi"]))]
    return {"phi": s["phi"], "residual": np.array([r[0] for r in got]), "n_iter": np.array([r[1] for r in got])}


# ---------------------------------------------------------------------------
# Work: bytes at one read of each input and one write of each output, Krylov
# vectors and coefficients once per CG iteration (15 words a cell)
# ---------------------------------------------------------------------------
def _cg_work(n, nh, iters):
    return {"bytes": 120.0 * n * iters + 80.0 * nh, "flops": 26.0 * n * iters}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        w = [_cg_work(a * b * c, (a + 4) * (b + 4) * (c + 4), case["iters"]) for a, b, c in _batch_dims(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    nr, nth, nz = _dims(case)
    n, nh = nr * nth * nz, (nr + 4) * (nth + 4) * (nz + 4)
    if kind in ("cg", "cg_host"):
        return _cg_work(n, nh, case["iters"])
    if kind == "transport":  # residual, then per sweep and direction: right-hand side, Thomas
        return {"bytes": 80.0 * nh, "flops": n * (20.0 + 12.0 + 48.0 * case["sweeps"])}
    asm = {"bytes": (8.0 * (24 + 18) + 4.0 * (4 + 3)) * nh, "flops": 400.0 * n}
    cor = {"bytes": 300.0 * n, "flops": 60.0 * n}
    if kind == "assemble":
        return asm
    if kind == "pcorr":
        return cor
    cg = _cg_work(n, nh, case["iters"])
    return {k: asm[k] + cor[k] + cg[k] for k in asm}


# ---------------------------------------------------------------------------
# The same results in plain 64-bit torch and numpy
# ---------------------------------------------------------------------------
I2 = slice(2, -2)


def _in(a):
    return a[I2, I2, I2]


def _shift(a, axis, d):
    """The interior cells' neighbours along axis (0 z, 1 theta, 2 r)."""
    s = [I2] * 3
    s[axis] = slice(2 + d, a.shape[axis] - 2 + d)
    return a[tuple(s)]


def _cg_exact(arrays, max_iter, tol):
    """Jacobi-PCG from zero: (phi in the halo layout, residual, iterations)."""
    aW, aE, aS, aN, aB, aT, aP, b = [_in(a) for a in arrays]

    def mul(x):
        h = _wrap(_halo(x))
        return (aP * x - aW * _shift(h, 2, -1) - aE * _shift(h, 2, 1) - aS * _shift(h, 1, -1)
                - aN * _shift(h, 1, 1) - aB * _shift(h, 0, -1) - aT * _shift(h, 0, 1))

    d = aP.abs().clamp(min=SMALL)
    x, r = torch.zeros_like(b), b.clone()
    bnorm = float(b.square().sum().sqrt())
    if bnorm < SMALL:
        return _halo(x), 0.0, 0
    z = r / d
    p, rz = z, float((r * z).sum())
    res, it = float(r.square().sum().sqrt()) / bnorm, 0
    for it in range(1, max_iter + 1):
        q = mul(p)
        pq = float((p * q).sum())
        if abs(pq) < SMALL:
            it -= 1
            break
        alpha = rz / pq
        x = x + alpha * p
        r = r - alpha * q
        res = float(r.square().sum().sqrt()) / bnorm
        if res < tol:
            break
        z = r / d
        new = float((r * z).sum())
        p = z + (new / max(rz, SMALL)) * p
        rz = new
    return _wrap(_halo(x)), res, it


def _transport_exact(arrays, phi0, sweeps):
    A = {n: a.cpu().numpy() for n, a in zip(NAMES, arrays)}
    phi = phi0.cpu().numpy().copy()
    I = _in
    pc = I(phi)
    r = (I(A["Su"]) - I(A["aP"]) * pc
         + I(A["aW"]) * phi[I2, I2, 1:-3] + I(A["aE"]) * phi[I2, I2, 3:-1]
         + I(A["aS"]) * phi[I2, 1:-3, I2] + I(A["aN"]) * phi[I2, 3:-1, I2]
         + I(A["aB"]) * phi[1:-3, I2, I2] + I(A["aT"]) * phi[3:-1, I2, I2])
    links = sum(np.abs(I(A[n])) for n in NAMES[:6])
    live = ~((I(A["aP"]) == 1.0) & (links == 0.0))
    t = np.abs(I(A["Su"])) + np.abs(I(A["aP"]) * pc) + SMALL
    res = math.sqrt((r[live] ** 2).sum()) / (math.sqrt((t[live] ** 2).sum()) + SMALL)

    def tiny(v):
        return np.where(np.abs(v) < SMALL, np.copysign(SMALL, v), v)

    # (owner axis, chain axis, line axis), the first and second neighbour pairs, the line's own links
    plans = [((0, 1, 2), "aS", "aN", "aB", "aT", "aW", "aE"),
             ((0, 2, 1), "aW", "aE", "aB", "aT", "aS", "aN"),
             ((2, 1, 0), "aS", "aN", "aW", "aE", "aB", "aT")]
    nth = phi.shape[1] - 4
    factors = []
    for axes, *names in plans:
        lo, up = -A[names[4]].transpose(axes), -A[names[5]].transpose(axes)
        diag = A["aP"].transpose(axes)
        L = diag.shape[2] - 4
        M, CP = np.empty((L,) + diag.shape[:2]), np.empty((L,) + diag.shape[:2])
        cp = 0.0
        for e in range(L):
            m = tiny(diag[:, :, e + 2] - (lo[:, :, e + 2] * cp if e else 0.0))
            M[e] = m
            cp = up[:, :, e + 2] / m
            CP[e] = cp
        factors.append((np.nan_to_num(M), np.nan_to_num(CP)))
    for _ in range(sweeps):
        for (axes, *names), (M, CP) in zip(plans, factors):
            phi[:, 0:2] = phi[:, nth:nth + 2].copy()
            phi[:, nth + 2:nth + 4] = phi[:, 2:4].copy()
            V, S = phi.transpose(axes), A["Su"].transpose(axes)
            c1m, c1p, c2m, c2p, lm, lp = [A[n].transpose(axes) for n in names]
            B, C, L = [n - 4 for n in V.shape]
            for d in range(B + C - 1):  # lines (a, b) with a + b = d are independent
                a = np.arange(max(0, d - B + 1), min(C - 1, d) + 1) + 2
                b = d - (a - 2) + 2
                f = (S[b, a, I2] + c1m[b, a, I2] * V[b, a - 1, I2] + c1p[b, a, I2] * V[b, a + 1, I2]
                     + c2m[b, a, I2] * V[b - 1, a, I2] + c2p[b, a, I2] * V[b + 1, a, I2])
                f[:, 0] += lm[b, a, 2] * V[b, a, 1]
                f[:, -1] += lp[b, a, L + 1] * V[b, a, L + 2]
                f = np.ascontiguousarray(f.T)
                m, cp, lo = M[:, b, a], CP[:, b, a], np.ascontiguousarray(-lm[b, a, I2].T)
                f[0] /= m[0]
                for e in range(1, L):
                    f[e] = (f[e] - lo[e] * f[e - 1]) / m[e]
                for e in range(L - 2, -1, -1):
                    f[e] -= cp[e] * f[e + 1]
                V[b, a, I2] = f.T
    return {"phi": phi, "residual": res}


def _assemble_exact(f):
    """solve_pressure_correction up to its CG, on device tensors."""
    nr, nth, nz, fl = f.nr, f.nth, f.nz, f.flags
    room_on, gas_in, gas_comp = fl & 1, fl & 2, fl & 4
    dt, rho_gas, T_amb, beta = f.scalars
    one = torch.ones((), dtype=F64, device=DEV)
    zero = torch.zeros((nz, nth, nr), dtype=F64, device=DEV)
    live = f.cell_type != 0
    al, ag = f.act_l != 0, f.act_g != 0
    ok = live & (al | ag)
    coord = {2: f.r[None, None, :], 1: f.theta[None, :, None], 0: f.z[:, None, None]}
    full = {ax: coord[ax].expand(f.p.shape) for ax in coord}
    full[1] = full[1] * full[2]  # arc length r theta
    rng = {2: torch.arange(-1, nr + 3, device=DEV)[None, None, :], 1: torch.arange(-1, nth + 3, device=DEV)[None, :, None],
           0: torch.arange(-1, nz + 3, device=DEV)[:, None, None]}
    n_of = {2: nr, 1: nth, 0: nz}

    def grad(ax, periodic):
        p0, pm, pp = _in(f.p), _shift(f.p, ax, -1), _shift(f.p, ax, 1)
        if ax == 1:
            rc = _in(full[2])
            t = coord[1].expand(f.p.shape)
            x0, xm, xp = rc * _in(t), rc * _shift(t, 1, -1), rc * _shift(t, 1, 1)
        else:
            x0, xm, xp = _in(full[ax]), _shift(full[ax], ax, -1), _shift(full[ax], ax, 1)
        idx = _in(rng[ax].expand(f.p.shape))
        okm = _shift(ok, ax, -1) & (periodic | (idx > 1))
        okp = _shift(ok, ax, 1) & (periodic | (idx < n_of[ax]))
        return okm, okp, (p0 - pm) / (x0 - xm), (pp - p0) / (xp - x0), (pp - pm) / (xp - xm)

    def pick(okm, okp, lo, hi, both):
        v = torch.where(okm & okp, both, torch.where(okp, hi, torch.where(okm, lo, zero)))
        return _wrap(_halo(torch.where(_in(live), v, zero)))

    g = {ax: pick(*grad(ax, ax == 1)) for ax in (0, 1, 2)}
    w1 = al.to(F64) * f.liq_alpha * f.liq_rho * (1.0 - beta * (f.liq_T - T_amb))
    gz_gas = g[0]
    if gas_in:
        okm, okp, lo, hi, _ = grad(0, False)
        lo = lo + 0.5 * 9.81 * (_shift(w1, 0, -1) + _in(w1))
        hi = hi + 0.5 * 9.81 * (_in(w1) + _shift(w1, 0, 1))
        gz_gas = pick(okm, okp, lo, hi, 0.5 * (lo + hi))

    def faces(ax, A):
        """(lower, upper) cells of the n+1 faces normal to ax."""
        lo, hi = [I2] * 3, [I2] * 3
        lo[ax], hi[ax] = slice(1, -2), slice(2, -1)
        return A[tuple(lo)], A[tuple(hi)]

    out = {n: zero.clone() for n in ("aW", "aE", "aS", "aN", "aB", "aT", "Su", "Fs_r", "Fs_th", "Fs_z", "ac_r", "ac_th", "ac_z")}
    lk = {n: torch.zeros_like(zero, dtype=torch.int32) for n in ("lk_r", "lk_th", "lk_z")}
    flux = zero.clone()
    sides = {2: ("aW", "aE", "r", "ur"), 1: ("aS", "aN", "th", "uth"), 0: ("aB", "aT", "z", "uz")}
    for ph, act in (("liq", al), ("gas", ag)):
        if ph == "gas" and not gas_in:
            continue
        alpha = getattr(f, ph + "_alpha")
        for ax in (2, 1, 0):
            m_name, p_name, d_name, u_name = sides[ax]
            ap, u = getattr(f, ph + "_aP_" + u_name), getattr(f, ph + "_" + u_name)
            gr = gz_gas if (ph == "gas" and ax == 0) else g[ax]
            cond = alpha * f.vol / ap.clamp(min=SMALL)
            (cx, cq), (ax_, aq), (ux, uq), (gx, gq) = (faces(ax, v) for v in (cond, alpha, u, gr))
            d_f, a_f = 0.5 * (cq + cx), 0.5 * (aq + ax_)
            if ax == 1:
                t = coord[1].expand(f.p.shape)
                tx, tq = faces(1, t)
                delta = faces(1, full[2])[1] * (tq - tx)
            else:
                xx, xq = faces(ax, full[ax])
                delta = xq - xx
            px, pq = faces(ax, f.p)
            drive = 0.5 * (gq + gx) - (pq - px) / delta
            if ph == "gas" and ax == 0:
                wx, wq = faces(0, w1)
                drive = drive - 0.5 * 9.81 * (wx + wq)
            u_f = 0.5 * (uq + ux) + d_f * drive
            lx, lq = faces(ax, live & act)
            is_open = lx & lq
            if ph == "liq" and room_on:
                rx, rq = faces(ax, f.liq_room)
                is_open = is_open & ~((u_f > 0) & (rq <= 1e-4)) & ~((u_f < 0) & (rx <= 1e-4))
            m_side, p_side = [slice(None)] * 3, [slice(None)] * 3
            m_side[ax], p_side[ax] = slice(0, -1), slice(1, None)
            m_side, p_side = tuple(m_side), tuple(p_side)
            if ax == 1:
                area_m = area_p = _in(f.Ath)
            else:
                a = faces(ax, f.Ar if ax == 2 else f.Az)[0]
                area_m, area_p = a[m_side], a[p_side]
            for side, name, area, sign in ((m_side, m_name, area_m, 1.0), (p_side, p_name, area_p, -1.0)):
                c = torch.where(is_open[side], (a_f * d_f)[side] * area / delta[side], zero)
                F = torch.where(is_open[side], (a_f * u_f)[side] * area, zero)
                out[name] = out[name] + c
                out["Su"] = out["Su"] + sign * F
                flux = flux + F.abs()
                if sign < 0 and ph == "liq":
                    out["Fs_" + d_name] = F
                    out["ac_" + d_name] = c
                    lk["lk_" + d_name] = is_open[side].to(torch.int32)
    l_on, g_on, here, vol = _in(al), _in(ag), _in(live), _in(f.vol)
    if gas_comp:
        ga, gr = _in(f.gas_alpha), _in(f.gas_rho)
        src = ga * vol / dt * (gr - rho_gas * T_amb / _in(f.gas_T_old).clamp(min=100.0)) / gr.clamp(min=SMALL)
        cap = 0.2 * ga * vol / dt
        out["Su"] = out["Su"] - torch.where(g_on, torch.maximum(-cap, torch.minimum(cap, src)), zero)
    links = ("aW", "aE", "aS", "aN", "aB", "aT")
    aP = sum(out[n] for n in links) * (1.0 + 1e-6)
    if gas_comp:
        aP = aP + torch.where(g_on, ga / 101325.0 * vol / dt, zero)
    aP = aP + torch.where(l_on, _in(f.liq_alpha) * vol / (_in(f.liq_rho) * 4000.0 ** 2 * dt), zero)
    top = rng[0] == nz
    hole = (f.outlet != 0) & top
    dead = ~here | ~(l_on | g_on) | _in(hole)
    idx = {ax: _in(rng[ax].expand(f.p.shape)) for ax in rng}
    for name, ax, d in (("aW", 2, -1), ("aE", 2, 1), ("aS", 1, -1), ("aN", 1, 1), ("aB", 0, -1), ("aT", 0, 1)):
        cut = dead | _shift(hole, ax, d)
        if ax != 1:
            edge = idx[ax] == (1 if d < 0 else n_of[ax])
            cut = cut | edge | ~_shift(live, ax, d)
        out[name] = torch.where(cut, zero, out[name])
    out["Su"] = torch.where(dead, zero, out["Su"])
    out["aP"] = torch.where(dead, one, aP)
    total = float(torch.where(here & (l_on | g_on), out["Su"].abs(), zero).sum())
    res = total / max(float(torch.where(here, flux, zero).sum()), SMALL)
    made = {n: _halo(v) for n, v in out.items()}
    for n in ("Fs_r", "Fs_th", "Fs_z", "ac_r", "ac_th", "ac_z"):
        made[n] = _halo(torch.where(here, out[n], zero))
    for n, v in lk.items():
        made[n] = _halo(v.to(F64)).to(torch.int32)
    for n in ("pp", "Fc_r", "Fc_th", "Fc_z"):
        made[n] = torch.zeros_like(f.p)
    made["residual"] = res
    return made


def _correct_exact(f):
    """The post-CG corrections in place on the device tensors of f."""
    nr, nz = f.nr, f.nz
    here = _in(f.cell_type) != 0
    pp = f.pp
    for d, ax in (("r", 2), ("th", 1), ("z", 0)):
        link = (_in(getattr(f, "lk_" + d)) == 1) & here
        F = _in(getattr(f, "Fs_" + d)) + _in(getattr(f, "ac_" + d)) * (_in(pp) - _shift(pp, ax, 1))
        c = _in(getattr(f, "Fc_" + d))
        c.copy_(torch.where(link, F, c))
    rc = f.r[None, None, 2:-2]
    step = {2: (f.r[3:-1] - f.r[1:-3])[None, None, :], 1: rc * (f.theta[3:-1] - f.theta[1:-3])[None, :, None],
            0: (f.z[3:-1] - f.z[1:-3])[:, None, None]}
    wall = {2: torch.zeros(nr, dtype=torch.bool, device=DEV), 0: torch.zeros(nz, dtype=torch.bool, device=DEV)}
    for w in wall.values():
        w[0] = w[-1] = True
    wall = {2: wall[2][None, None, :], 1: torch.zeros((1, 1, 1), dtype=torch.bool, device=DEV), 0: wall[0][:, None, None]}
    for ph, act in (("liq", f.act_l), ("gas", f.act_g)):
        if ph == "gas" and not f.has_gas:
            continue
        for d, ax in (("ur", 2), ("uth", 1), ("uz", 0)):
            ap = _in(getattr(f, ph + "_aP_" + d))
            u = _in(getattr(f, ph + "_" + d))
            new = u - _in(getattr(f, ph + "_alpha")) * _in(f.vol) / ap * (_shift(pp, ax, 1) - _shift(pp, ax, -1)) / step[ax]
            u.copy_(torch.where(here & (_in(act) != 0) & ~wall[ax] & (ap.abs() > SMALL), new, u))
    f.p.copy_((f.p + f.alpha_p * pp).clamp(-gen.P_HYDRO_CAP, gen.P_HYDRO_CAP))
    active = (f.cell_type != 0) & ((f.act_l != 0) | (f.act_g != 0))
    w = active.to(F64)
    pw = torch.where(active, f.p, torch.zeros_like(f.p))
    near = [(ax, d) for ax in (2, 1, 0) for d in (-1, 1)]
    count = sum(_shift(w, *k) for k in near)
    mean = sum(_shift(pw, *k) for k in near) / count.clamp(min=1.0)
    p = _in(f.p)
    p.copy_(torch.where(here & ~_in(active), mean, p))
    for n in ("Fc_r", "Fc_th", "Fc_z", "p", "lk_r", "lk_th", "lk_z"):
        _wrap(getattr(f, n))


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        got = [_cg_exact(a, case["iters"], TOL) for a in _batch_systems(case, seed)]
        return {"phi": [x[0] for x in got], "residual": np.array([x[1] for x in got]), "n_iter": np.array([x[2] for x in got])}
    nr, nth, nz = _dims(case)
    if kind in ("cg", "cg_host"):
        phi, res, it = _cg_exact(_pressure_system(nr, nth, nz, seed), case["iters"], TOL)
        return {"phi": phi, "residual": res, "n_iter": it}
    if kind == "transport":
        return _transport_exact(*_transport_system(nr, nth, nz, seed), case["sweeps"])
    if kind == "pcorr":
        f = _fields_on(gen.make_pcorr_fields(nr, nth, nz, seed, has_gas=case["gas"]))
        _correct_exact(f)
        return f.outputs()
    f = _fields_on(gen.make_pressure_state(nr, nth, nz, seed, flags=case["flags"]))
    made = _assemble_exact(f)
    if kind == "assemble":
        return made
    res = made.pop("residual")
    for n, v in made.items():
        setattr(f, n, v)
    f.pp, cg_res, it = _cg_exact([getattr(f, n) for n in NAMES], case["iters"], TOL)
    _correct_exact(gen.pcorr_view(f, 0.7))
    return {**f.outputs(), **{n: getattr(f, n) for n in STEP_STATE}, "residual": res, "cg_residual": cg_res, "n_iter": it}
