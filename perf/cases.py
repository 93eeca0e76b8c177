"""The framework's work as its users have it done, case by case, for timing.

A case is a dict of plain values.  ``kind`` says which public entry point it calls:

``mvp``         ``Operator.mvp_device``: one block matvec on device pointers, as a caller's own Krylov solver does it
                each iteration (``prec`` fp64, fp32 or df64; ``f`` 3 or 6; ``scaled``: with DIAG_A and the Jacobi scaling)
``mbt``         ``Operator.mbt_fft_mvp``: the reference's ``MBT_fft_mvp`` on a host cuboid vector
``solve``       ``solve`` / ``solve_device``: a block Krylov solve of one target
``batch``       ``batch_solve``: several uneven targets at once
``wavelength``  ``Operator.set_wavenumber`` and the first matvec after it: the step of a spectral sweep

Targets are seeded lattice aggregates (``bdda.aggregate``) at |m| k d = 0.5, wavelength 0.55 um.  The geometry belongs to
the case; the vectors, incident directions and wavenumbers come from the seed.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "block-dda_gb300"))
import bdda  # noqa: E402

K0 = 2 * np.pi / 0.55
PREC = {"fp64": bdda.PREC_FP64, "fp32": bdda.PREC_FP32, "df64": bdda.PREC_DF64}


def listed():
    return [
        # the smallest target of a batch (64 dipoles, one direction): five short launches, latency
        {"name": "mvp_fp64_n64_l2", "kind": "mvp", "prec": "fp64", "f": 3, "nocc": 64, "df": 2.8, "L": 2, "scaled": True},
        # a sparse soot-like aggregate with an odd number of right-hand sides, complex FP32
        {"name": "mvp_fp32_n1000_l3", "kind": "mvp", "prec": "fp32", "f": 3, "nocc": 1000, "df": 2.1, "L": 3, "scaled": True},
        # the matvec of the mixed-precision configuration (8 directions x 2 polarisations)
        {"name": "mvp_fp32_n16384_l16", "kind": "mvp", "prec": "fp32", "f": 3, "nocc": 16384, "df": 2.8, "L": 16, "scaled": True},
        # the matvec of the largest target: 65536 dipoles, 32 right-hand sides
        {"name": "mvp_fp32_n65536_l32", "kind": "mvp", "prec": "fp32", "f": 3, "nocc": 65536, "df": 2.8, "L": 32, "scaled": True},
        # the plain FP64 path's matvec at an ordinary size
        {"name": "mvp_fp64_n8192_l16", "kind": "mvp", "prec": "fp64", "f": 3, "nocc": 8192, "df": 2.8, "L": 16, "scaled": True},
        # the true-residual matvec of a mixed solve (double-float, no Jacobi scaling)
        {"name": "mvp_df64_n16384_l16", "kind": "mvp", "prec": "df64", "f": 3, "nocc": 16384, "df": 2.8, "L": 16, "scaled": False},
        # the reference's own entry point: one cuboid vector, host to host
        {"name": "mbt_33x47x29", "kind": "mbt", "nx": 33, "ny": 47, "nz": 29},
        # the plain configuration: 1024 dipoles, one direction, FP64 block COCG-RQ-Jacobi to 1e-8, host buffers
        {"name": "solve_fp64_n1024_l2", "kind": "solve", "prec": "fp64", "solver": "cocg_rq", "f": 3, "nocc": 1024, "df": 2.8,
         "L": 2, "mr": 1.95, "mi": 0.79},
        # electric and magnetic dipoles (f = 6), block BiCGSTAB-Jacobi as in the reference's recorded runs, FP64
        {"name": "solve_fp64_f6_n300_l4", "kind": "solve", "prec": "fp64", "solver": "bicgstab", "f": 6, "nocc": 300, "df": 2.8,
         "L": 4, "mr": 1.7, "mi": 0.5},
        # a mixed-precision solve with FP64 refinement on device buffers
        {"name": "solve_mixed_n8192_l16", "kind": "solve", "prec": "mixed", "solver": "cocg_rq", "f": 3, "nocc": 8192, "df": 2.8,
         "L": 16, "mr": 2.3, "mi": 0.6},
        # a batch of uneven targets solved concurrently (64 to 4096 dipoles, 2 to 16 right-hand sides)
        {"name": "batch_mixed_12", "kind": "batch", "count": 12, "nmin": 64, "nmax": 4096, "pick": 1},
        # the next wavelength of a sweep: rebuild the Green spectra, then the first matvec
        {"name": "wavelength_n4096_l4", "kind": "wavelength", "f": 3, "nocc": 4096, "df": 2.8, "L": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mvp", "mvp", "mvp", "mvp", "mbt", "solve", "solve", "batch", "wavelength"])
    if kind == "mbt":
        return {"kind": "mbt", "nx": _log(rng, 4, 60), "ny": _log(rng, 4, 60), "nz": _log(rng, 4, 60)}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(3, 12), "nmin": 64, "nmax": _log(rng, 400, 3000),
                "pick": rng.randint(2, 10 ** 6)}
    if kind == "mvp":
        prec = rng.choice(["fp64", "fp32", "df64"])
        f = rng.choice([3, 3, 3, 6])
        nocc = _log(rng, 64, {"fp64": 8192, "df64": 16384, "fp32": 60000}[prec] // (1 if f == 3 else 4))
        return {"kind": "mvp", "prec": prec, "f": f, "nocc": nocc, "df": round(rng.uniform(1.8 if nocc < 1500 else 2.6, 2.8), 2),
                "L": rng.randint(1, 32 if prec == "fp32" else 16), "scaled": rng.random() < 0.6}
    if kind == "wavelength":
        nocc = _log(rng, 64, 8000)
        return {"kind": "wavelength", "f": 3, "nocc": nocc, "df": round(rng.uniform(2.0 if nocc < 1500 else 2.6, 2.8), 2),
                "L": rng.randint(1, 8)}
    prec = rng.choice(["fp64", "mixed"])
    f = rng.choice([3, 3, 6]) if prec == "fp64" else 3
    nocc = _log(rng, 64, 400 if f == 6 else (1500 if prec == "fp64" else 8000))
    return {"kind": "solve", "prec": prec, "solver": "bicgstab" if f == 6 else "cocg_rq", "f": f, "nocc": nocc,
            "df": round(rng.uniform(2.5, 2.8), 2), "L": rng.randint(1, 8 if prec == "fp64" else 16),
            "mr": round(rng.uniform(1.3, 2.2), 2), "mi": round(rng.uniform(0.1, 0.9), 2)}


# ---------------------------------------------------------------- inputs

def _box(nocc, df, seed=1):
    n, addr = bdda.aggregate(nocc, 1.0, df, seed)
    return n, addr


def _spacing(m):
    return 0.5 / (abs(m) * K0)


def _gaussian(gen, shape):
    """Complex normal values, complex128 on the GPU."""
    r = torch.randn(shape + (2,), generator=gen, dtype=torch.float64, device="cuda")
    return torch.view_as_complex(r)


def _to_df(a):
    """complex128 -> double-float quadruples (re hi, re lo, im hi, im lo), float32."""
    v = torch.view_as_real(a.resolve_conj())
    hi = v.to(torch.float32)
    lo = (v - hi.to(torch.float64)).to(torch.float32)
    return torch.stack([hi[..., 0], lo[..., 0], hi[..., 1], lo[..., 1]], dim=-1).contiguous()


def _store(a, prec):
    return a if prec == "fp64" else a.to(torch.complex64) if prec == "fp32" else _to_df(a)


def _mvp_inputs(case, seed):
    """(n, address, spacing, x [L, f nocc], diag, jpre) in FP64, the values a solver's search block has."""
    n, addr = _box(case["nocc"], case["df"])
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rows = case["f"] * case["nocc"]
    x = _gaussian(gen, (case["L"], rows))
    lf = _spacing(1.78)
    diag = _gaussian(gen, (rows,)) * (0.1 / lf ** 3) + 4.0 / lf ** 3
    return n, addr, lf, x, diag, 1.0 / diag


def _mbt_inputs(case, seed):
    n = (case["nx"], case["ny"], case["nz"])
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((3 * n[0] * n[1] * n[2], 2))
    return n, _spacing(1.78), np.ascontiguousarray(x).view(np.complex128).ravel()


def _solve_inputs(nocc, df, m, L, f, seed, pick=1):
    """(n, address, spacing, diag, B): incident plane waves from seeded directions."""
    n, addr = _box(nocc, df, pick)
    lf = _spacing(m)
    r_eq = lf * (3.0 / (4.0 * np.pi)) ** (1.0 / 3.0)
    u, e = bdda.directions((L + 1) // 2, seed)
    rot = np.linalg.qr(np.random.default_rng(seed + 1).standard_normal((3, 3)))[0]  # the first direction is not always +z
    u, e = u[:L] @ rot, e[:L] @ rot
    if f == 3:
        a = bdda.polarizability(0.55, r_eq, m * m, K0)
        return n, addr, lf, bdda.diag_a(np.full(nocc, a)), bdda.incident_fields(n, lf, addr, K0, u, e)
    ae, ah = bdda.polarizabilities(0.55, r_eq, m * m, K0)
    diag = bdda.diag_a(np.full(nocc, ae), np.full(nocc, ah))
    return n, addr, lf, diag, bdda.incident_fields(n, lf, addr, K0, u, e, np.cross(u, e))


def _batch_inputs(case, seed):
    """[(n, address, spacing, diag, B)]: sizes log-uniform, shapes and materials as a batched study has them."""
    rng = np.random.default_rng(case["pick"])
    out = []
    for i in range(case["count"]):
        nocc = int(round(math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
        m = complex(rng.uniform(1.3, 2.2), rng.uniform(0.1, 0.9))
        L = int(rng.choice([2, 4, 8, 16]))
        out.append(_solve_inputs(nocc, rng.uniform(2.2, 2.8), m, L, 3, seed + 7 * i, int(rng.integers(1, 1000))))
    return out


def _opts(case):
    if case["prec"] == "mixed":
        # 1e-11 where a run would often ask for 1e-8: the solution is then settled well past any difference in rounding
        return bdda.solve_opts(case["solver"], jacobi=True, precision=bdda.SOLVE_MIXED, tol=1e-8, itermax=600, true_tol=1e-11)
    return bdda.solve_opts(case["solver"], jacobi=True, tol=1e-8 if case["f"] == 3 else 1e-6, itermax=600)


def _wavenumber(seed):
    return K0 * (0.8 + 0.4 * np.random.default_rng(seed).random())


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "mvp":
        n, addr, lf, x, diag, jpre = _mvp_inputs(case, seed)
        s["op"] = bdda.Operator(n, lf, K0, f=case["f"])
        s["op"].set_dipoles(addr)
        s["L"], s["rows"], s["prec"] = case["L"], x.shape[1], PREC[case["prec"]]
        s["x"] = _store(x, case["prec"])
        s["y"] = torch.zeros_like(s["x"])
        s["diag"] = _store(diag, case["prec"])
        s["jpre"] = _store(jpre, case["prec"]) if case["scaled"] else None
        s["stream"] = torch.cuda.Stream()
    elif kind == "mbt":
        n, lf, s["x"] = _mbt_inputs(case, seed)
        s["op"] = bdda.Operator(n, lf, K0)
    elif kind == "solve":
        n, addr, lf, diag, B = _solve_inputs(case["nocc"], case["df"], complex(case["mr"], case["mi"]), case["L"], case["f"], seed)
        s["op"] = bdda.Operator(n, lf, K0, f=case["f"])
        s["op"].set_dipoles(addr)
        s["opts"], s["mixed"] = _opts(case), case["prec"] == "mixed"
        if s["mixed"]:
            s["diag"], s["B"] = torch.from_numpy(diag).cuda(), torch.from_numpy(np.ascontiguousarray(B.T)).cuda()
            s["X"] = torch.zeros_like(s["B"])
            s["stream"] = torch.cuda.Stream()
        else:
            s["diag"], s["B"] = diag, B
    elif kind == "batch":
        s["problems"] = [bdda.Problem(n=n, lf=lf, address=a, k=K0, alpha=1.0 / d[::3], diag=d, B=B)
                         for n, a, lf, d, B in _batch_inputs(case, seed)]
        s["opts"] = bdda.solve_opts("cocg_rq", jacobi=True, precision=bdda.SOLVE_MIXED, tol=1e-8, itermax=600, true_tol=1e-11)
    else:
        n, addr, lf, x, diag, _ = _mvp_inputs(case, seed)
        s["op"] = bdda.Operator(n, lf, K0)
        s["op"].set_dipoles(addr)
        s["L"], s["rows"], s["k"] = case["L"], x.shape[1], _wavenumber(seed)
        s["x"], s["y"], s["diag"] = x, torch.zeros_like(x), diag
        s["stream"] = torch.cuda.Stream()
    torch.cuda.synchronize()  # the inputs are ready before a call on another stream reads them
    return s


def run(s):
    kind = s["kind"]
    if kind == "mvp":
        s["op"].mvp_device(s["x"].data_ptr(), s["y"].data_ptr(), s["L"], s["rows"], s["rows"], prec=s["prec"],
                           diag=s["diag"].data_ptr(), jpre=s["jpre"].data_ptr() if s["jpre"] is not None else None,
                           stream=s["stream"].cuda_stream)
        return s["y"]
    if kind == "mbt":
        return s["op"].mbt_fft_mvp(s["x"])
    if kind == "solve":
        if s["mixed"]:
            L, rows = s["B"].shape
            bdda.solve_device(s["op"], s["diag"].data_ptr(), s["B"].data_ptr(), rows, s["X"].data_ptr(), rows, L, s["opts"],
                              stream=s["stream"].cuda_stream, allow_not_converged=False)
            return s["X"]
        return bdda.solve(s["op"], s["diag"], s["B"], s["opts"], allow_not_converged=False)[0]
    if kind == "batch":
        return [X for X, _ in bdda.batch_solve(s["problems"], 8, 40e9, s["opts"])]
    s["op"].set_wavenumber(s["k"])
    s["op"].mvp_device(s["x"].data_ptr(), s["y"].data_ptr(), s["L"], s["rows"], s["rows"], diag=s["diag"].data_ptr(),
                       stream=s["stream"].cuda_stream)
    return s["y"]


# ---------------------------------------------------------------- the work and the values

def _padded(n):
    def smooth(v):
        while True:
            t = v
            for p in (2, 3, 5):
                while t % p == 0:
                    t //= p
            if t == 1:
                return v
            v += 1
    return tuple(smooth(2 * int(v)) for v in n)


def _mvp_work(n, nocc, L, f, size, scaled=True):
    """One block matvec: x, y, diag, jpre and the Green spectrum once each; the arithmetic of the pruned transforms and
    the product."""
    P = _padded(n)
    nc = 6 if f == 3 else 9
    data = (2 * f * L * nocc + (2 if scaled else 1) * f * nocc) * size + 4.0 * nocc + nc * P[0] * P[1] * P[2] * size

    def line(p):
        return 5.0 * p * math.log2(max(p, 2))
    fft = 2.0 * f * L * (n[1] * n[2] * line(P[0]) + P[0] * n[2] * line(P[1]) + P[0] * P[1] * line(P[2]))
    product = L * P[0] * P[1] * P[2] * (8.0 * f * f)
    return data, fft + product


def work(case):
    kind = case["kind"]
    if kind == "mbt":
        n = (case["nx"], case["ny"], case["nz"])
        b, fl = _mvp_work(n, n[0] * n[1] * n[2], 1, 3, 16)
        return {"bytes": b, "flops": fl}
    if kind == "batch":
        b = fl = 0.0
        for n, a, _, _, B in _batch_inputs(case, 0):
            x, y = _mvp_work(n, a.size, B.shape[1], 3, 8)
            b, fl = b + 20 * x, fl + 20 * y
        return {"bytes": b, "flops": fl}
    n, _ = _box(case["nocc"], case["df"])
    if kind == "mvp":
        b, fl = _mvp_work(n, case["nocc"], case["L"], case["f"], 8 if case["prec"] == "fp32" else 16, case["scaled"])
        return {"bytes": b, "flops": fl}
    if kind == "wavelength":
        b, fl = _mvp_work(n, case["nocc"], case["L"], 3, 16)
        P = _padded(n)
        g = float(P[0] * P[1] * P[2])
        # six components evaluated and transformed, written in each precision
        return {"bytes": b + 6 * g * 40, "flops": fl + 6 * g * (5 * math.log2(g) + 30)}
    # a solve: about 25 iterations of one matvec each, and the block algebra
    b, fl = _mvp_work(n, case["nocc"], case["L"], case["f"], 8 if case["prec"] == "mixed" else 16)
    return {"bytes": 25 * b, "flops": 25 * (fl + 8.0 * 6 * case["f"] * case["nocc"] * case["L"] ** 2)}


class _Exact:
    """diag o x + A x in complex128 by torch.fft: the dyadic Green tensor of vacuum on the padded circulant grid."""

    def __init__(self, n, lf, k, addr, f=3, device="cuda"):
        self.n, self.f, self.P = n, f, tuple(2 * int(v) for v in n)
        dev = torch.device(device)
        d = []
        ok = torch.ones((1, 1, 1), dtype=torch.bool, device=dev)
        for i in range(3):
            j = torch.arange(self.P[i], device=dev)
            off = torch.where(j < n[i], j, j - self.P[i]).to(torch.float64)
            shape = [1, 1, 1]
            shape[i] = self.P[i]
            d.append((off * lf).reshape(shape))
            ok = ok & (j != n[i]).reshape(shape)
        r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
        ok = ok & (r2 > 0)
        r = torch.sqrt(torch.where(ok, r2, torch.ones_like(r2)))
        e = torch.exp(1j * k * r) / r * ok
        u = [(v / r).expand(self.P) for v in d]
        self.g = {}
        for a in range(3):
            for b in range(a, 3):
                rr = u[a] * u[b]
                dl = 1.0 if a == b else 0.0
                g = -(k * k * (dl - rr) - (1.0 - 1j * k * r) / (r * r) * (dl - 3.0 * rr)) * e
                self.g[a, b] = self.g[b, a] = torch.fft.fftn(g)
        if f == 6:  # B = -F, F = -k^2 e^{ikr} / r (1 - 1 / (ikr)) [r^ x]
            c = -k * k * e * (1.0 - 1.0 / (1j * k * r))
            self.b = [torch.fft.fftn(c * v) for v in u]
        a = torch.as_tensor(np.asarray(addr, dtype=np.int64), device=dev)
        self.at = (a // (n[1] * n[2]), (a // n[2]) % n[1], a % n[2])

    def __call__(self, x, diag=None):
        """x [L, f nocc] -> [L, f nocc]."""
        out = torch.empty_like(x)
        f = self.f
        for l in range(x.shape[0]):
            h = []
            for c in range(f):
                grid = torch.zeros(self.P, dtype=torch.complex128, device=x.device)
                grid[self.at] = x[l, c::f]
                h.append(torch.fft.fftn(grid))
            y = [sum(self.g[a % 3, b] * h[b + 3 * (a // 3)] for b in range(3)) for a in range(f)]
            if f == 6:
                bz, by, bx = self.b[2], self.b[1], self.b[0]  # B_xy = fac u_z, B_xz = -fac u_y, B_yz = fac u_x
                for o, s, i in ((0, 1.0, 3), (3, -1.0, 0)):
                    y[o] = y[o] + s * (bz * h[i + 1] - by * h[i + 2])
                    y[o + 1] = y[o + 1] + s * (bx * h[i + 2] - bz * h[i])
                    y[o + 2] = y[o + 2] + s * (by * h[i] - bx * h[i + 1])
            for c in range(f):
                out[l, c::f] = torch.fft.ifftn(y[c])[self.at]
        return out if diag is None else out + diag * x


def _exact_solve(n, addr, lf, diag, B, f):
    """X of (diag + A) X = B by restarted GMRES on the torch operator, columns one by one, to the rounding of FP64."""
    op = _Exact(n, lf, K0, addr, f)
    dg = torch.as_tensor(diag, device="cuda")
    Bt = torch.as_tensor(np.ascontiguousarray(B.T), device="cuda")
    X = torch.zeros_like(Bt)
    for l in range(Bt.shape[0]):
        b = Bt[l:l + 1]
        x = torch.zeros_like(b)
        for _ in range(12):
            r = (b - op(x, dg)) / dg
            beta = float(torch.linalg.vector_norm(r))
            if beta <= 2e-15 * float(torch.linalg.vector_norm(b / dg)):
                break
            V, H = [r / beta], np.zeros((41, 40), complex)
            m = 40
            for j in range(40):
                w = op(V[j], dg) / dg
                for _ in range(2):
                    for i, v in enumerate(V):
                        h = torch.vdot(v[0], w[0])
                        H[i, j] += complex(h)
                        w = w - h * v
                H[j + 1, j] = float(torch.linalg.vector_norm(w))
                e1 = np.zeros(j + 2, complex)
                e1[0] = beta
                y, *_ = np.linalg.lstsq(H[:j + 2, :j + 1], e1, rcond=None)
                if np.linalg.norm(H[:j + 2, :j + 1] @ y - e1) < 1e-9 * beta:
                    m = j + 1
                    break
                V.append(w / H[j + 1, j].real)
            for i in range(m):
                x = x + complex(y[i]) * V[i]
        X[l] = x[0]
    return X


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mvp", "wavelength"):
        n, addr, lf, x, diag, jpre = _mvp_inputs(case, seed)
        P = _padded(n)
        if case["L"] * P[0] * P[1] * P[2] > 1.5e8:
            return None
        prec = case.get("prec", "fp64")
        if prec == "fp32":
            x, diag, jpre = (v.to(torch.complex64).to(torch.complex128) for v in (x, diag, jpre))
        y = _Exact(n, lf, K0 if kind == "mvp" else _wavenumber(seed), addr, case["f"])(x, diag)
        if case.get("scaled"):
            y = y * jpre
        return _to_df(y) if prec == "df64" else y
    if kind == "mbt":
        n, lf, x = _mbt_inputs(case, seed)
        op = _Exact(n, lf, K0, np.arange(n[0] * n[1] * n[2]))
        return op(torch.from_numpy(x).cuda()[None])[0].cpu().numpy()
    if kind == "solve":
        if case["nocc"] * case["L"] > 2e4:
            return None
        n, addr, lf, diag, B = _solve_inputs(case["nocc"], case["df"], complex(case["mr"], case["mi"]), case["L"], case["f"], seed)
        X = _exact_solve(n, addr, lf, diag, B, case["f"])
        return X if case["prec"] == "mixed" else X.T.cpu().numpy()
    return [_exact_solve(n, a, lf, d, B, 3).T.cpu().numpy() if a.size * B.shape[1] <= 4000 else None
            for n, a, lf, d, B in _batch_inputs(case, seed)]
