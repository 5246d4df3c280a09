"""What a user of this framework runs: the cases by which its speed is measured.

listed() holds the cases, draw() gives more of the same ranges, prepare() makes what a
program has in hand before the call, run() is one pass through the public entry points
(the Python mirror, or the C ABI where the data stay on the device), work() the bytes and
operations a pass cannot do without, exact() the results in 64 bits by plain torch.

Every program of the path builds a mesh and an operator once and then evaluates T(k) at
many wavenumbers: one at a time (its own root finder), in sweeps, in the built-in searches,
for one large scatterer or a batch of uneven ones; behind T(k) come the dense, the
randomized and the Arnoldi sigma, the LU, the field of a transmission problem and, beside
them, the training of the proposal network.
"""
import ctypes
import math

import numpy as np
import torch

from helmholtzbem_gb300 import _capi as C
from helmholtzbem_gb300 import api, geometry


def listed():
    return [
        # the smallest calls: one layer set of a small circle of arcs, results on the host
        dict(name="layers_small", do="layers", shape="circle", N=24, p=7, d=0),
        # a program's own root finder: T, T', T'' at one wavenumber, then sigma and its derivatives
        dict(name="newton_point", do="point", shape="polygon", N=50, p=11),
        # sigma and both derivatives along a range of wavenumbers (the small scatterer's report)
        dict(name="sweep_derivatives", do="sweep", shape="polygon", N=48, p=11, nk=100, d=2),
        # the plain resonance search of the benchmark scatterer, a circle of arcs
        dict(name="search_circle", do="search", shape="circle", N=50, p=11, nk=200),
        # assembly at scale: T, T', T'' of a star polygon with 24 vertices on the device
        dict(name="scale_derivatives", do="batch", shape="polygon", N=1000, p=16, nk=1, d=2),
        # many scatterers of uneven size (polygons and Fourier curves) in one call
        dict(name="many_scatterers", do="multi", nops=8, N=100, p=11, nk=3, d=0),
        # sigma by the randomized SVD in FP64 along a few wavenumbers of a mid-sized scatterer
        dict(name="rsvd_fp64", do="rsvd", shape="fourier", N=401, p=11, nk=6, sketch=12, precision=0),
        # the largest matrices: complex-FP32 LU with FP64 refinement behind the sketch
        dict(name="rsvd_mixed", do="rsvd", shape="fourier", N=1500, p=11, nk=1, sketch=16, precision=1),
        # traces of the transmission problem and the total field on a grid through the scatterer
        dict(name="field", do="field", shape="graded", N=400, p=11, nx=201, ny=160, order=16),
        # Arnoldi sigma of a batch of small T(k) held on the device
        dict(name="arnoldi", do="arnoldi", N=50, p=11, nk=64, d=0),
        # batched LU and solves of device matrices, complex128
        dict(name="lu_solve", do="lu", n=1500, nmat=4, nrhs=8),
        # one gradient of the proposal network, batch and targets on the host
        dict(name="proposal_gradients", do="mlp", batch=256, width=512, depth=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["layers", "point", "sweep", "search", "batch", "multi", "rsvd", "rsvd", "field", "arnoldi", "lu",
                     "mlp"])
    shape = rng.choice(["circle", "polygon", "fourier"])
    p = rng.choice([7, 9, 11, 12])
    if do == "layers":
        return dict(do=do, shape=shape, N=_log_int(rng, 14, 120), p=p, d=rng.randrange(3))
    if do == "point":
        return dict(do=do, shape="polygon", N=_log_int(rng, 14, 150), p=p)
    if do == "sweep":   # derivatives where no two singular values (nearly) coincide: on the polygons
        d = rng.randrange(3)
        return dict(do=do, shape=shape if d == 0 else "polygon", N=rng.randint(16, 50), p=p,
                    nk=_log_int(rng, 3, 120), d=d)
    if do == "search":
        return dict(do=do, shape="circle", N=rng.randint(30, 50), p=11, nk=rng.randint(120, 200))
    if do == "batch":
        p = rng.choice([9, 11, 13, 16])
        return dict(do=do, shape=shape, N=_log_int(rng, 60, 900), p=p, nk=1, d=rng.randrange(3))
    if do == "multi":
        return dict(do=do, nops=rng.randint(2, 8), N=_log_int(rng, 20, 90), p=11, nk=rng.randint(1, 3),
                    d=rng.randrange(2))
    if do == "rsvd":
        return dict(do=do, shape=shape, N=_log_int(rng, 70, 500), p=11, nk=rng.randint(1, 6),
                    sketch=rng.randint(8, 16), precision=rng.randrange(2))
    if do == "field":
        return dict(do=do, shape=rng.choice(["graded", "circle"]), N=_log_int(rng, 40, 400), p=11,
                    nx=_log_int(rng, 20, 200), ny=_log_int(rng, 20, 160), order=rng.choice([8, 12, 16]))
    if do == "arnoldi":
        return dict(do=do, N=_log_int(rng, 20, 120), p=11, nk=_log_int(rng, 2, 32), d=0)
    if do == "lu":
        return dict(do=do, n=_log_int(rng, 60, 1500), nmat=rng.randint(1, 4), nrhs=rng.randint(1, 16))
    return dict(do=do, batch=_log_int(rng, 32, 256), width=rng.choice([128, 256, 512]), depth=rng.randint(2, 4))


# ------------------------------------------------------------------ inputs

def _mesh(shape, N, seed):
    """A mesh of N panels: the small scatterers (radius about 0.25) and the unit-sized ones."""
    rng = np.random.default_rng([seed, 1])
    if shape == "circle":
        return geometry.circle(0.25 * (1.0 + 0.04 * rng.uniform(-1, 1)), N)
    if shape == "polygon":
        x, y = geometry.star_polygon(12 if N < 100 else 24, int(seed) % 100000)
        return geometry.polygon(0.25 * x, 0.25 * y, N) if N < 100 else geometry.polygon(x, y, N)
    if shape == "graded":
        return geometry.polygon_graded(*geometry.star_polygon(24, int(seed) % 100000), N, 0.5)
    a, b = geometry.random_fourier_coeffs(int(seed) % 100000)
    kinds, par = geometry.fourier_curve(a, b, N)
    return (kinds, 0.25 * par) if N < 100 else (kinds, par)


def _range(case):
    """Wavenumbers in use: [0.5, 10] for the small scatterers, up to 30 for the large."""
    small = case.get("shape") == "circle" or case.get("N", 0) < 100
    return (0.5, 10.0) if small else (1.0, 30.0)


def _ks(case, seed, nk):
    lo, hi = _range(case)
    r = np.random.default_rng([seed, 2])
    return np.ascontiguousarray(np.linspace(lo, hi, nk) + r.uniform(0.0, 0.5, nk) if nk > 1 else r.uniform(lo, hi, 1))


def _sizes(case):
    """Uneven panel counts of the scatterers of one batch."""
    return [int(case["N"] * (1 + 0.45 * m)) + m for m in range(case["nops"])]


def _c_i(case, seed):
    hi = 23.4 if case.get("N", 0) < 100 or case.get("shape") == "circle" else 9.0
    return hi * (1.0 + 0.05 * float(np.random.default_rng([seed, 3]).uniform(-1, 1)))


def _inputs(case, seed):
    """The host-side inputs of a case: everything exact() needs as well."""
    s = dict(case=case, seed=seed)
    do = case["do"]
    if do == "multi":
        r = np.random.default_rng([seed, 4])
        s["meshes"], s["ks"], s["c_i"] = [], [], []
        for m in range(case["nops"]):
            N = _sizes(case)[m]
            s["meshes"].append(_mesh("polygon" if m % 2 else "fourier", N, seed + 17 * m))
            s["ks"].append(np.ascontiguousarray(r.uniform(*((1.0, 30.0) if N >= 100 else (0.5, 10.0)), case["nk"])))
            s["c_i"].append(float(r.uniform(2.0, 25.0)))
    elif do == "lu":
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        n, m = case["n"], case["nmat"]
        s["A"] = torch.randn((m, n, n), dtype=torch.complex128, device="cuda", generator=g) / math.sqrt(n)
        s["A"] += 0.5 * torch.eye(n, dtype=torch.complex128, device="cuda")
        s["X"] = torch.randn((m, case["nrhs"], n), dtype=torch.complex128, device="cuda", generator=g)
    elif do == "mlp":
        r = np.random.default_rng([seed, 5])
        s["X"] = r.normal(0.0, 0.7, (case["batch"], 34)).astype(np.float32)
        s["Y"] = r.normal(-1.0, 0.5, (case["batch"], 128)).astype(np.float32)
        dims = [34] + [case["width"]] * case["depth"] + [128]
        s["params"] = np.concatenate([np.concatenate([
            r.normal(0.0, math.sqrt(2.0 / i), o * i), r.normal(0.0, 0.02, o)]) for i, o in zip(dims[:-1], dims[1:])
        ]).astype(np.float32)
    else:
        s["mesh"] = _mesh(case.get("shape", "polygon"), case["N"], seed)
        s["c_i"] = _c_i(case, seed)
        if do == "field":
            r = np.random.default_rng([seed, 6])
            s["k"] = float(r.uniform(6.0, 10.0))
            s["angle"] = float(r.uniform(0.0, 2 * math.pi))
            s["c_i"] = 4.0
            h = (0.4 if case["shape"] == "circle" else 1.6) * (1.0 + 0.01 * float(r.uniform(-1, 1)))
            s["box"] = ((-h, -0.97 * h), (1.01 * h, h))
        elif do == "search":
            s["k0"], s["k1"] = 0.5, 10.0
        else:
            s["ks"] = _ks(case, seed, case.get("nk", 1))
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    do = case["do"]
    if do == "multi":
        s["ops"] = [api.SolutionsOperator(api.BuilderData(m, order=case["p"])) for m in s["meshes"]]
    elif do == "lu":
        pass
    elif do == "mlp":
        s["net"] = api.MLP(34, case["width"], case["depth"], 128)
        s["net"].set_params(s["params"])
    elif do == "arnoldi":
        s["T"] = torch.stack([_T(s["mesh"], case["p"], float(k), 1.0, s["c_i"], case["d"], True).transpose(-1, -2)
                              for k in s["ks"]]).contiguous()
        torch.cuda.synchronize()
    else:
        s["data"] = api.BuilderData(s["mesh"], order=case["p"])
        if do == "layers":
            s["builder"] = api.GalerkinBuilder(s["data"])
        else:
            s["op"] = api.SolutionsOperator(s["data"], proj=do != "field")
    return s


# ------------------------------------------------------------------ one pass

def run(s):
    case, do = s["case"], s["case"]["do"]
    if do == "layers":
        b, d = s["builder"], case["d"]
        b.assembleDense(float(s["ks"][0]), s["c_i"], d=d)
        return [(b.getDoubleLayer(t), b.getHypersingular(t), b.getSingleLayer(t)) for t in range(d + 1)]
    if do == "point":
        T = s["op"].gen_sol_op_2nd_der(float(s["ks"][0]), 1.0, s["c_i"])
        return {"T": list(T), "sigma": api.sv_dense([T], d=2)}
    if do == "sweep":
        return s["op"].sweep_sigma(s["ks"], 1.0, s["c_i"], d=case["d"])
    if do == "search":
        found, grid, _ = s["op"].find_resonances_plain(s["k0"], s["k1"], case["nk"], 1.0, s["c_i"])
        roots = np.full(64, np.nan)
        roots[:found.size] = found[:64]
        return {"roots": roots, "sigma": grid[:, 0].copy(), "slopes": grid[:, 1].copy()}
    if do == "batch":
        n, nk, d = 2 * case["N"], case["nk"], case["d"]
        T = torch.empty((nk, d + 1, n, n), dtype=torch.complex128, device="cuda")
        C.check(C.lib().hbem_gen_sol_op_batch_device(s["op"]._h, C.dptr(s["ks"]), nk, 1.0, s["c_i"], d,
                                                     ctypes.c_void_p(T.data_ptr())))
        return T
    if do == "multi":
        return api.gen_sol_op_multi_device(s["ops"], s["ks"], 1.0, s["c_i"], d=case["d"])
    if do == "rsvd":
        return s["op"].sigma_rsvd_sweep(s["ks"], 1.0, s["c_i"], sketch=case["sketch"], q=2,
                                        precision=case["precision"], seed=int(s["seed"]) % 1000)
    if do == "field":
        S, _, _ = api.tp_field_grid(s["op"], api.wave("Plane", 1.0, angle=s["angle"]), s["k"], 1.0, s["c_i"],
                                    case["order"], s["box"][0], s["box"][1], case["nx"], case["ny"], total_field=True)
        return S
    if do == "arnoldi":
        nk, d = case["nk"], case["d"]
        n = s["T"].shape[-1]
        out = np.zeros((nk, 1, d + 1))
        C.check(C.lib().hbem_arnoldi_sv_batch_device(n, nk, d, 1, 1e-12, ctypes.c_void_p(s["T"].data_ptr()),
                                                     (d + 1) * n * n, n * n, C.dptr(out), None, None))
        return out
    if do == "lu":
        n, m = case["n"], case["nmat"]
        A, X = s["A"].clone(), s["X"].clone()
        piv = torch.empty((m, n), dtype=torch.int32, device="cuda")
        C.check(C.lib().hbem_lu_factor_batch_device(n, m, ctypes.c_void_p(A.data_ptr()), n * n,
                                                    ctypes.c_void_p(piv.data_ptr()), None))
        C.check(C.lib().hbem_lu_solve_batch_device(n, m, 0, ctypes.c_void_p(A.data_ptr()), n * n,
                                                   ctypes.c_void_p(piv.data_ptr()), case["nrhs"],
                                                   ctypes.c_void_p(X.data_ptr()), case["nrhs"] * n))
        return X
    loss, grads = s["net"].gradients(s["X"], s["Y"])
    return {"loss": loss, "grads": grads}


# ------------------------------------------------------------------ what a pass cannot do without

def _points(N, p):
    """Quadrature points of one medium: general pairs, coincident and adjacent pairs."""
    nc = p * (p + 1) // 2 - 1
    return (N * (N + 1) // 2 - 2 * N) * p * p + 3 * N * nc * nc


def _assembly_flops(N, p, nk, d):
    # a Hankel pair (two orders, real and imaginary part, some ten terms each), the distance,
    # and per derivative order the moments of three kernels: about 100 + 40 per order
    return 2.0 * nk * _points(N, p) * (100.0 + 40.0 * d)


def work(case):
    do = case["do"]
    if do == "mlp":
        w, dep, b = case["width"], case["depth"], case["batch"]
        par = 34 * w + (dep - 1) * w * w + 128 * w
        return {"bytes": 8.0 * par + 4.0 * b * 162, "flops": 6.0 * b * par}
    if do == "lu":
        n, m = case["n"], case["nmat"]
        return {"bytes": 16.0 * m * (n * n + 2 * n * case["nrhs"]), "flops": m * (8 / 3 * n ** 3 + 8.0 * n * n * case["nrhs"])}
    if do == "arnoldi":
        n, m = 2 * case["N"], case["nk"]
        return {"bytes": 16.0 * m * n * n, "flops": m * 8 / 3 * n ** 3}
    if do == "multi":
        Ns = _sizes(case)
        return {"bytes": sum(16.0 * case["nk"] * (case["d"] + 1) * 4 * N * N for N in Ns),
                "flops": sum(_assembly_flops(N, case["p"], case["nk"], case["d"]) for N in Ns)}
    N, p, nk, d = case["N"], case["p"], case.get("nk", 1), case.get("d", 0)
    n = 2 * N
    lu = 8 / 3 * n ** 3
    if do == "layers":
        return {"bytes": 16.0 * 3 * (d + 1) * N * N, "flops": _assembly_flops(N, p, 1, d) / 2}
    if do == "point":
        return {"bytes": 16.0 * 3 * n * n, "flops": _assembly_flops(N, p, 1, 2) + lu}
    if do == "sweep":
        return {"bytes": 40.0 * N + 32.0 * nk, "flops": _assembly_flops(N, p, nk, d) + nk * lu}
    if do == "search":   # the grid, and some ten minima with two ends and about five Newton points each
        return {"bytes": 40.0 * N + 32.0 * nk,
                "flops": _assembly_flops(N, p, nk, 0) + _assembly_flops(N, p, 70, 2) + (nk + 50) * lu}
    if do == "batch":
        return {"bytes": 16.0 * nk * (d + 1) * n * n, "flops": _assembly_flops(N, p, nk, d)}
    if do == "rsvd":
        return {"bytes": 40.0 * N + 8.0 * nk, "flops": _assembly_flops(N, p, nk, 0) + nk * lu}
    G = case["nx"] * case["ny"]
    return {"bytes": 40.0 * N + 16.0 * G,
            "flops": _assembly_flops(N, p, 1, 0) * 1.5 + lu + 80.0 * G * N * case["order"]}


# ------------------------------------------------------------------ the same in 64 bits, by torch

def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 * (x + 1.0), 0.5 * w


def _composite(n):
    """The composite rule on [0, 1], graded towards 0: n points on [s, 1], n - 1 on [s^2, s], ..., two on the last."""
    sig = (math.sqrt(2.0) - 1.0) ** 2
    xs, ws, lo, hi = [], [], sig, 1.0
    for q in range(n, 1, -1):
        x, w = _gauss(q)
        xs.append((hi - lo) * x + lo)
        ws.append((hi - lo) * w)
        hi, lo = lo, lo * sig
    return np.concatenate(xs), np.concatenate(ws)


def _dev(a):
    return torch.as_tensor(np.asarray(a), device="cuda")


def _panel(kinds, par, t):
    """Points, tangents (d/dt on [0, 1]) and tangent norms; t broadcasts against the panels' leading axis."""
    line = (kinds == 0)
    a = par[3] + t * (par[4] - par[3])
    lx, ly = par[0] + t * (par[2] - par[0]), par[1] + t * (par[3] - par[1])
    dphi = par[4] - par[3]
    x = torch.where(line, lx, par[0] + par[2] * torch.cos(a))
    y = torch.where(line, ly, par[1] + par[2] * torch.sin(a))
    tx = torch.where(line, par[2] - par[0] + 0 * t, -par[2] * dphi * torch.sin(a))
    ty = torch.where(line, par[3] - par[1] + 0 * t, par[2] * dphi * torch.cos(a))
    return x, y, tx, ty, torch.sqrt(tx * tx + ty * ty)


def _hankel_taylor():
    """Taylor coefficients of H0 (degree 15) about the knots 2, 2.25, ..., 802 from Bessel's equation.
    H0 and H1 at a knot: Hankel's expansion from 26 on, below it the Taylor steps from the knot above.
    (torch.special.bessel_* are good to 1e-6 only beyond x = 5.)"""
    x = 2.0 + 0.25 * np.arange(3201)

    def taylor(x, h0, h1, deg):
        a = [h0, -h1]
        for m in range(deg - 1):
            a.append(-((m + 1) ** 2 * a[m + 1] + x * a[m] + (a[m - 1] if m else 0.0)) / (x * (m + 2) * (m + 1)))
        return a

    H = np.zeros((2, x.size), complex)
    big = x >= 26.0
    for nu in range(2):
        t, tot = np.ones(big.sum(), complex), np.ones(big.sum(), complex)
        for m in range(1, 45):
            t = t * (4.0 * nu - (2 * m - 1) ** 2) / (8.0 * m * x[big]) * 1j
            tot += np.where(np.abs(t) < 1e-18, 0.0, t) if m < 20 else 0.0
        s, c = np.sin(x[big]), np.cos(x[big])
        e = ((c + s) + 1j * (s - c)) / math.sqrt(2.0)              # exp(i (x - pi/4))
        H[nu, big] = np.sqrt(2.0 / (math.pi * x[big])) * (e if nu == 0 else -1j * e) * tot
    for j in range(int(big.argmax()) - 1, -1, -1):
        a = taylor(x[j + 1], H[0, j + 1], H[1, j + 1], 30)
        H[0, j] = sum(a[m] * (-0.25) ** m for m in range(31))
        H[1, j] = -sum(m * a[m] * (-0.25) ** (m - 1) for m in range(1, 31))
    return np.stack(taylor(x, H[0], H[1], 15))


_TABLE = []


def _hankel(x):
    """H0, H1 of x in 64 bits."""
    if not _TABLE:
        _TABLE.append(_dev(_hankel_taylor()))
    j = ((x - 2.0) * 4.0).round().clamp(0, 3200).long()
    h = x - (2.0 + 0.25 * j)
    c = _TABLE[0]
    h0, dh = c[15][j], 15.0 * c[15][j]
    for m in range(14, -1, -1):
        cm = c[m][j]
        h0 = h0 * h + cm
        if m:
            dh = dh * h + m * cm
    sp, y = torch.special, x.clamp(max=2.0)
    low = x < 2.0
    return (torch.where(low, torch.complex(sp.bessel_j0(y), sp.bessel_y0(y)), h0),
            torch.where(low, torch.complex(sp.bessel_j1(y), sp.bessel_y1(y)), -dh))


def _pair_blocks(P, Q, w, t, u, ks, c, d):
    """2 x 2 blocks of K, W, V and their derivatives: points P on the test panels (parameter t), Q on
    the trial panels (parameter u), weights w; sums over the last axis.  out[layer][order]: [..., 2, 2]."""
    zx, zy = P[0] - Q[0], P[1] - Q[1]
    r = torch.sqrt(zx * zx + zy * zy)
    zero = r == 0   # two mapped nodes of a pair may coincide to rounding: H0 = 1, H1 = 0 there, and no 1 / r
    h0, h1 = (torch.where(zero, v, h) for v, h in zip((1.0 + 0j, 0j), _hankel(ks * r + zero.double())))
    rc, rh = math.sqrt(c), r * h1
    cross = (zx * Q[3] - zy * Q[2]) * P[4]
    tt, tn = P[2] * Q[2] + P[3] * Q[3], P[4] * Q[4]
    k = ks / rc
    G = [h0, -rc * rh, -c * (r * r * h0 - rh / ks)]                    # the single-layer kernel by orders of d/dk
    H = [ks * h1 / (r + zero.double()), k * c * h0, c * (h0 - ks * rh)]                  # the double-layer kernel
    c2 = [ks * ks, 2 * ks * rc, 2 * c]                                 # ks^2 and its derivatives
    S = [c2[0] * G[0], c2[1] * G[0] + c2[0] * G[1], c2[2] * G[0] + 2 * c2[1] * G[1] + c2[0] * G[2]]
    ft, fu = (t, 1 - t), (u, 1 - u)
    out = [[], [], []]
    for o in range(d + 1):
        K, W, V = [], [], []
        for a in range(2):
            for b in range(2):
                f = w * ft[a] * fu[b]
                sg = 1.0 if a == b else -1.0
                K.append((f * cross * H[o]).sum(-1))
                W.append((sg * w * G[o] - f * tt * S[o]).sum(-1))
                V.append((f * tn * G[o]).sum(-1))
        for layer, x in zip(out, (K, W, V)):
            layer.append(torch.stack(x, -1).reshape(x[0].shape + (2, 2)))
    return out


def _layers(mesh, p, k, c, d):
    """[K, W, V][order] (N x N, continuous P1 spaces) of a closed mesh in panel order."""
    kinds, par = _dev(mesh[0]), _dev(mesh[1]).T.contiguous()
    N = kinds.shape[0]
    ks = k * math.sqrt(c)
    xg, wg = (_dev(v) for v in _gauss(p))
    xc, wc = (_dev(v) for v in _composite(p))
    A = [[torch.zeros((N, N, 2, 2), dtype=torch.complex128, device="cuda") for _ in range(d + 1)] for _ in range(3)]
    t, u = xg[:, None].expand(p, p).reshape(-1), xg[None, :].expand(p, p).reshape(-1)
    w = (wg[:, None] * wg[None, :]).reshape(-1)
    rows = max(1, (3 << 20) // (N * p * p))
    idx = torch.arange(N, device="cuda")
    Q = _panel(kinds[None, :, None], par[:, None, :, None], u[None, None, :])
    for i0 in range(0, N, rows):
        i = idx[i0:i0 + rows]
        P = _panel(kinds[i][:, None, None], par[:, i][:, :, None, None], t[None, None, :])
        gap = (i[:, None] - idx[None, :]) % N
        far = (gap > 1) & (gap < N - 1)
        ii, jj = torch.nonzero(far, as_tuple=True)
        sel = [v[ii, 0] for v in P]
        oth = [v[0, jj] for v in Q]
        for layer, got in zip(A, _pair_blocks(sel, oth, w, t, u, ks, c, d)):
            for o in range(d + 1):
                layer[o][i[ii], jj] = got[o]
    # coincident and adjacent pairs on the mapped composite rule
    a, b = (v.reshape(-1) for v in torch.meshgrid(xc, xc, indexing="ij"))
    wa, wb = (v.reshape(-1) for v in torch.meshgrid(wc, wc, indexing="ij"))
    s, big = a * (1 - b), a
    sets = (torch.cat([s, big]), torch.cat([big, s]), torch.cat([a * wa * wb] * 2))
    s2 = a * b
    adj = (torch.cat([s2, big]), torch.cat([big, s2]), torch.cat([a * wa * wb] * 2))
    step = max(1, (3 << 20) // (2 * xc.numel() ** 2))
    for q0 in range(0, N, step):
        i = idx[q0:q0 + step]
        j = (i + 1) % N
        pi = (kinds[i][:, None], par[:, i][:, :, None])
        pj = (kinds[j][:, None], par[:, j][:, :, None])
        todo = [(i, i, pi, pi, sets[0], sets[1], sets[2]),              # coincident
                (i, j, pi, pj, 1 - adj[0], adj[1], adj[2]),             # panel i ends where panel i + 1 begins
                (j, i, pj, pi, adj[1], 1 - adj[0], adj[2])]
        for m, n, pm, pn, tm, un, ww in todo:
            got = _pair_blocks(_panel(*pm, tm[None]), _panel(*pn, un[None]), ww, tm, un, ks, c, d)
            for layer, g in zip(A, got):
                for o in range(d + 1):
                    layer[o][m, n] = g[o]
    # local function 0 (t) of panel i belongs to degree of freedom i + 1, function 1 (1 - t) to i
    out = []
    for layer in A:
        out.append([0.25j * (torch.roll(B[:, :, 0, 0], (1, 1), (0, 1)) + torch.roll(B[:, :, 0, 1], 1, 0) +
                             torch.roll(B[:, :, 1, 0], 1, 1) + B[:, :, 1, 1]) for B in layer])
    return out


def _mass(mesh):
    P = _panel(_dev(mesh[0]), _dev(mesh[1]).T, torch.zeros(1, dtype=torch.float64, device="cuda"))
    L = P[4]
    i = torch.arange(L.shape[0], device="cuda")
    M = torch.zeros((L.shape[0],) * 2, dtype=torch.float64, device="cuda")
    M[i, i] = (L + torch.roll(L, 1)) / 3
    M[i, (i + 1) % L.shape[0]] += L / 6
    M[(i + 1) % L.shape[0], i] += L / 6
    return M


def _T(mesh, p, k, c_o, c_i, d, proj):
    """[d + 1, 2N, 2N]: the transmission operator and its derivatives."""
    Ki, Wi, Vi = _layers(mesh, p, k, c_i, d)
    Ko, Wo, Vo = _layers(mesh, p, k, c_o, d)
    M = _mass(mesh)
    out = []
    for o in range(d + 1):
        mm = M if o == 0 else 0 * M
        T = torch.cat([torch.cat([Ki[o] - Ko[o] + mm, Vo[o] - Vi[o]], 1),
                       torch.cat([Wo[o] - Wi[o], Ko[o] - Ki[o] + mm], 1)])
        if proj:
            F = torch.block_diag(*[torch.linalg.cholesky(M)] * 2).to(torch.complex128)
            T = torch.linalg.solve_triangular(F, T, upper=False)
            T = torch.linalg.solve_triangular(F, T.T, upper=False).T
        out.append(T)
    return torch.stack(out)


def _sigma(T, d):
    """sigma_min and its derivatives by perturbation of the whole SVD; [3] with zeros past order d."""
    U, S, Vh = (v.cpu().numpy() for v in torch.linalg.svd(T[0].cpu()))
    D = [m.cpu().numpy() for m in T]
    u, v, sg = U[:, -1], Vh[-1].conj(), S[-1]
    got = [sg, 0.0, 0.0]
    if d >= 1:
        got[1] = float(np.real(u.conj() @ D[1] @ v))
    if d == 2:
        a = U.conj().T @ (D[1] @ v)
        b = (Vh @ (D[1].conj().T @ u))
        val = float(np.real(u.conj() @ D[2] @ v))
        near = np.abs(S - sg) <= 1e-9 * sg
        val += 0.5 * float(np.sum((np.abs(a + b) ** 2)[~near] / (sg - S[~near])))
        got[2] = val + 0.5 * float(np.sum(np.abs(a - b) ** 2 / (sg + S)))
    return got


def _smallest(T):
    """sigma_min of a large matrix: subspace iteration on (T^H T)^-1."""
    n = T.shape[0]
    LU, piv = torch.linalg.lu_factor(T)
    g = torch.Generator(device="cuda").manual_seed(1)
    Q = torch.linalg.qr(torch.randn((n, min(24, n)), dtype=T.dtype, device="cuda", generator=g))[0]
    for _ in range(25):
        Q = torch.linalg.qr(torch.linalg.lu_solve(LU, piv, Q, adjoint=True))[0]
        Q = torch.linalg.qr(torch.linalg.lu_solve(LU, piv, Q))[0]
    return 1.0 / float(torch.linalg.matrix_norm(torch.linalg.lu_solve(LU, piv, Q, adjoint=True), 2))


def _akima(t, y):
    """Periodic Akima pieces y + h (b + h (c + h d)) of the values y[0..n-1] at the knots t[0..n]."""
    n = y.size
    m = (np.append(y[1:], y[0]) - y) / (t[1:] - t[:-1])
    w1, w2 = np.abs(np.roll(m, -1) - m), np.abs(np.roll(m, 1) - np.roll(m, 2))
    flat = (w1 + w2) == 0
    mid = np.where(flat, 0.0, (w1 * np.roll(m, 1) + w2 * m) / np.where(flat, 1.0, w1 + w2))
    left, right = np.where(flat, np.roll(m, 1), mid), np.where(flat, m, mid)
    h = t[1:] - t[:-1]
    end = np.append(left[1:], left[0])
    return np.stack([y, right, (3 * m - 2 * right - end) / h, (right + end - 2 * m) / (h * h)]).reshape(4, n)


def _exact_field(s):
    case, k, c_i = s["case"], s["k"], s["c_i"]
    kinds, par = _dev(s["mesh"][0]), _dev(s["mesh"][1]).T.contiguous()
    N = kinds.shape[0]
    T = _T(s["mesh"], case["p"], k, 1.0, c_i, 0, False)[0]
    K, W, V = (x[0] for x in _layers(s["mesh"], case["p"], k, 1.0, 0))
    M = _mass(s["mesh"]).to(torch.complex128)
    dx, dy = math.cos(s["angle"]), math.sin(s["angle"])

    def wave(x, y):
        return torch.exp(1j * k * (x * dx + y * dy))

    P = _panel(kinds, par, torch.zeros(1, dtype=torch.float64, device="cuda"))
    u = wave(P[0], P[1])
    un = 1j * k * u * (P[3] * dx - P[2] * dy) / P[4]
    rhs = torch.cat([(0.5 * M - K) @ u + V @ un, W @ u + (K.T + 0.5 * M) @ un])
    tr = torch.linalg.solve(T, rhs).cpu().numpy()
    length = torch.where(kinds == 0, P[4], par[2] * (par[4] - par[3]))
    knots = torch.cat([torch.zeros(1, dtype=torch.float64, device="cuda"), torch.cumsum(length, 0)])
    kn = knots.cpu().numpy()
    coef = [_dev(_akima(kn, tr[o:o + N].real) + 1j * _akima(kn, tr[o:o + N].imag)) for o in (0, N)]

    def nodes(i, t):
        """Points, outward normals, tangent norms and the traces inside / outside of panels i at t."""
        x, y, tx, ty, tn = _panel(kinds[i], par[:, i], t)
        h = t * length[i]
        val = [q[0][i] + h * (q[1][i] + h * (q[2][i] + h * q[3][i])) for q in coef]
        uu = wave(x, y)
        nx, ny = ty / tn, -tx / tn
        return x, y, nx, ny, tn, val, [val[0] - uu, val[1] - 1j * k * uu * (nx * dx + ny * dy)]

    def green(x, y, nd, w, inside):
        kap = k * (1.0 + inside.double() * (math.sqrt(c_i) - 1.0))
        zx, zy = x - nd[0], y - nd[1]
        r = torch.sqrt(zx * zx + zy * zy)
        h0, h1 = _hankel(kap * r)
        tD, tN = (torch.where(inside, a, b) for a, b in zip(nd[5], nd[6]))
        return ((h0 * tN - kap * h1 * tD * (zx * nd[2] + zy * nd[3]) / r) * nd[4] * w).sum(-1)

    (x0, y0), (x1, y1) = s["box"]
    nx, ny = case["nx"], case["ny"]
    gx = x0 + torch.arange(nx, dtype=torch.float64, device="cuda") * ((x1 - x0) / (nx - 1))
    gy = y0 + torch.arange(ny, dtype=torch.float64, device="cuda") * ((y1 - y0) / (ny - 1))
    X, Y = (v.reshape(-1) for v in torch.meshgrid(gx, gy, indexing="ij"))
    xg, wg = (_dev(v) for v in _gauss(case["order"]))
    pan = torch.arange(N, device="cuda").repeat_interleave(case["order"])
    nd = nodes(pan, xg.repeat(N))
    E = _panel(kinds, par, torch.ones(1, dtype=torch.float64, device="cuda"))
    S = torch.zeros(nx * ny, dtype=torch.complex128, device="cuda")
    step = max(1, (6 << 20) // (N * case["order"]))
    for g0 in range(0, nx * ny, step):
        x, y = X[g0:g0 + step, None], Y[g0:g0 + step, None]
        if case["shape"] == "circle":
            inside = (x - par[0, 0]) ** 2 + (y - par[1, 0]) ** 2 < par[2, 0] ** 2
            rho = torch.sqrt((x - par[0]) ** 2 + (y - par[1]) ** 2)
            th = torch.remainder(torch.atan2(y - par[1], x - par[0]) - par[3], 2 * math.pi) / (par[4] - par[3])
            on = th <= 1
            ends = [torch.sqrt((x - q[0]) ** 2 + (y - q[1]) ** 2) for q in (P, E)]
            t = torch.where(on, th, (ends[1] < ends[0]).double())
            dist = torch.where(on, torch.abs(rho - par[2]), torch.minimum(*ends))
        else:
            up, dn = (P[1] <= y) & (y < E[1]), (E[1] <= y) & (y < P[1])
            cut = (E[0] - P[0]) * (y - P[1]) / (E[1] - P[1]) + P[0]
            inside = (((up | dn) & (x < cut)).sum(-1, keepdim=True) % 2) == 1
            t = (((x - P[0]) * P[2] + (y - P[1]) * P[3]) / P[4] ** 2).clamp(0, 1)
            dist = torch.sqrt((x - P[0] - t * P[2]) ** 2 + (y - P[1] - t * P[3]) ** 2)
        val = green(x, y, nd, wg.repeat(N), inside)
        near = dist * k * (1.0 + inside.double() * (math.sqrt(c_i) - 1.0)) < 1e-2
        for q, i in torch.nonzero(near).tolist():
            # the panel's Gauss sum makes way for a rule graded towards the nearest point
            one = torch.full((case["order"],), i, device="cuda")
            val[q] -= green(x[q], y[q], nodes(one, xg), wg, inside[q])
            tm, g20 = float(t[q, i]), _gauss(20)
            for side, span in ((-1.0, tm), (1.0, 1.0 - tm)):
                if span > 0:
                    hi = span * 0.5 ** np.arange(45)
                    lo = np.append(hi[1:], 0.0)
                    tt = (tm + side * (lo[:, None] + (hi - lo)[:, None] * g20[0])).ravel()
                    ww = ((hi - lo)[:, None] * g20[1]).ravel()
                    tt = _dev(tt)
                    val[q] += green(x[q], y[q], nodes(torch.full(tt.shape, i, device="cuda"), tt), _dev(ww), inside[q])
        ins = inside[:, 0]
        S[g0:g0 + step] = torch.where(ins, 0.25j * val, -0.25j * val + wave(x[:, 0], y[:, 0]))
    return S.reshape(nx, ny)


def exact(case, seed):
    s = _inputs(case, seed)
    do = case["do"]
    if do == "layers":
        K, W, V = _layers(s["mesh"], case["p"], float(s["ks"][0]), s["c_i"], case["d"])
        return [(K[t], W[t], V[t]) for t in range(case["d"] + 1)]
    if do == "point":
        T = _T(s["mesh"], case["p"], float(s["ks"][0]), 1.0, s["c_i"], 2, True)
        return {"T": list(T), "sigma": np.array([_sigma(T, 2)])}
    if do == "sweep":
        return np.array([_sigma(_T(s["mesh"], case["p"], float(k), 1.0, s["c_i"], case["d"], True), case["d"])
                         for k in s["ks"]])
    if do == "search":   # the roots and the slopes come out of a search: the grid's sigma is what has a plain value
        ks = s["k0"] + (s["k1"] - s["k0"]) / (case["nk"] - 1) * np.arange(case["nk"])
        sig = [_sigma(_T(s["mesh"], case["p"], float(k), 1.0, s["c_i"], 0, True), 0)[0] for k in ks]
        return {"roots": None, "sigma": np.array(sig), "slopes": None}
    if do == "batch":
        return torch.stack([_T(s["mesh"], case["p"], float(k), 1.0, s["c_i"], case["d"], True).transpose(-1, -2)
                            for k in s["ks"]])
    if do == "multi":
        return [torch.stack([_T(m, case["p"], float(k), 1.0, c, case["d"], True).transpose(-1, -2) for k in ks])
                for m, ks, c in zip(s["meshes"], s["ks"], s["c_i"])]
    if do == "rsvd":   # what the randomized estimate stands for: sigma_min itself
        return np.array([_smallest(_T(s["mesh"], case["p"], float(k), 1.0, s["c_i"], 0, True)[0]) for k in s["ks"]])
    if do == "field":
        return _exact_field(s)
    if do == "arnoldi":
        return np.array([[[_smallest(_T(s["mesh"], case["p"], float(k), 1.0, s["c_i"], 0, True)[0])]] for k in s["ks"]])
    if do == "lu":
        return torch.linalg.solve(s["A"].transpose(-1, -2), s["X"].transpose(-1, -2)).transpose(-1, -2)
    # the network in float64 (the framework's products are bfloat16)
    par = _dev(s["params"]).double().requires_grad_()
    dims = [34] + [case["width"]] * case["depth"] + [128]
    h, off = _dev(s["X"]).double(), 0
    for l, (i, o) in enumerate(zip(dims[:-1], dims[1:])):
        h = h @ par[off:off + o * i].view(o, i).T + par[off + o * i:off + o * i + o]
        off += o * i + o
        h = torch.nn.functional.gelu(h) if l < len(dims) - 2 else h
    loss = torch.mean((h - _dev(s["Y"]).double()) ** 2)
    loss.backward()
    return {"loss": float(loss), "grads": par.grad}
