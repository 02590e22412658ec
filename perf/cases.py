"""The measured cases: what users of the SO(3) / S^2 transforms have the library do, through its public calls.

Four families, all through ``fftso3_gb300`` on device buffers (point evaluation takes its points and gives its values
in host memory, as the call is defined):

* ``so3`` / ``s2`` -- one forward transform of a batch of sampled functions and one inverse of a batch of coefficient
  vectors, on one plan that the program keeps.  Options: complex or real functions, the FP64, tensor-core and FP32
  precisions, and the refined forward with the exact inverse.
* ``uneven`` -- a batch of functions whose l_max differ, both directions, replayed from CUDA graphs.
* ``points`` -- a coefficient vector evaluated at given rotations or directions.

The samples are smooth random functions with measurement noise, the coefficients N(0,1) with a power-law decay in l.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from fftso3_gb300 import _lib

CDT = {True: torch.complex128, False: torch.complex64}
RDT = {True: torch.float64, False: torch.float32}


def _case(name, family, **kw):
    c = {"family": family, "real": False, "precision": "tc_bf16x3", "refined": False, "l_max": 0, "batch": 1}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one function of the default class configuration (FP64): the reference's own use, bound by latency
        _case("so3c_l16_fp64", "so3", precision="fp64", l_max=16),
        # one real function at the reference's largest published size, FP64
        _case("so3r_l127_fp64", "so3", precision="fp64", l_max=127, real=True),
        # a few small functions on the tensor cores: launches and gaps count
        _case("so3c_l31_b4", "so3", l_max=31, batch=4),
        # orientation maps at medium resolution, real
        _case("so3r_l63_b64", "so3", l_max=63, batch=64, real=True),
        # a batch of complex functions at the resolution of the reference's largest example
        _case("so3c_l127_b16", "so3", l_max=127, batch=16),
        # bandwidth whose grid has a large prime factor (N = 194 = 2 * 97)
        _case("so3c_l96_b64", "so3", l_max=96, batch=64),
        # the headline: refined forward and exact inverse at the largest resolution
        _case("so3c_l255_b4_refined", "so3", l_max=255, batch=4, refined=True),
        # refined forward and exact inverse of real functions on a grid that is no power of two (N = 160)
        _case("so3r_l79_b16_refined", "so3", l_max=79, batch=16, refined=True, real=True),
        # many real signals on the sphere at high resolution
        _case("s2r_l511_b512", "s2", l_max=511, batch=512, real=True),
        # a handful of spherical shapes in the default precision
        _case("s2c_l47_b8_fp64", "s2", precision="fp64", l_max=47, batch=8),
        # functions of mixed bandwidth in one batch, as a data set of shapes has them
        _case("uneven_r_l8to64_n1024", "uneven", l_min=8, l_max=64, batch=1024, real=True),
        # a fitted function evaluated at given rotations
        _case("points_so3c_l127_n2048", "points", l_max=127, n=2048, precision="fp64", sphere=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["so3", "so3", "so3", "refined", "s2", "s2", "uneven", "points", "fp64"])
    real = rng.random() < 0.5
    if family == "so3":
        l = _log(rng, 7, 160)
        most = max(1, min(64, int(1.0e9 / (8 * (2 * l + 2) ** 3))))
        return _case(None, "so3", l_max=l, batch=_log(rng, 1, most), real=real,
                     precision="tc_bf16x3" if rng.random() < 0.8 else "fp32")
    if family == "refined":
        l = _log(rng, 15, 140)
        most = max(1, min(32, int(0.5e9 / (8 * (2 * l + 2) ** 3))))
        return _case(None, "so3", l_max=l, batch=_log(rng, 1, most), real=real, refined=True)
    if family == "s2":
        l = _log(rng, 15, 511)
        return _case(None, "s2", l_max=l, batch=_log(rng, 1, 512), real=real,
                     precision="tc_bf16x3" if rng.random() < 0.8 else "fp32")
    if family == "uneven":
        return _case(None, "uneven", l_min=rng.randint(2, 16), l_max=rng.randint(24, 64), batch=_log(rng, 32, 1024),
                     real=real)
    if family == "points":
        sphere = rng.random() < 0.4
        return _case(None, "points", l_max=_log(rng, 8, 511 if sphere else 127), n=_log(rng, 1, 2048),
                     precision="fp64", real=real, sphere=sphere)
    l = _log(rng, 3, 100)
    if rng.random() < 0.4:
        return _case(None, "s2", precision="fp64", l_max=l, batch=_log(rng, 1, 64), real=real)
    most = max(1, min(16, int(6.0e7 / (2 * l + 2) ** 4)))
    return _case(None, "so3", precision="fp64", l_max=l, batch=_log(rng, 1, most), real=real)


# ------------------------------------------------------------------ inputs


def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + salt) % (1 << 62))


def _rand(shape, dtype, g):
    return torch.randn(shape, dtype=dtype, device="cuda", generator=g)


def _waves(b, r, N, real, g):
    """b x r smooth periodic functions of N points."""
    x = torch.arange(N, device="cuda", dtype=torch.float32) * (2 * math.pi / N)
    n = min(6, N // 4 + 1)
    ph = torch.arange(n, device="cuda", dtype=torch.float32)[:, None] * x
    c = _rand((2, b * r, n), torch.float32, g) / torch.arange(1, n + 1, device="cuda", dtype=torch.float32)
    v = c[0] @ torch.cos(ph) + c[1] @ torch.sin(ph)
    if not real:
        d = _rand((2, b * r, n), torch.float32, g) / torch.arange(1, n + 1, device="cuda", dtype=torch.float32)
        v = torch.complex(v, d[0] @ torch.cos(ph) + d[1] @ torch.sin(ph))
    return v.reshape(b, r, N)


def _samples(so3, L, b, real, fp64, g):
    """Samples of smooth random functions with 5% noise, flat, in the library's grid layout."""
    N = 2 * (L + 1)
    dt = torch.float32 if real else torch.complex64
    out = torch.empty((b,) + (N,) * (3 if so3 else 2), dtype=dt, device="cuda")
    for f0 in range(0, b, 64):
        nb = min(64, b - f0)
        o = out[f0:f0 + nb]
        A, B, C = (_waves(nb, 2, N, real, g) for _ in range(3))
        noise = _rand(o.shape, dt, g)
        for r in range(2):
            if so3:
                noise = noise.mul_(1.0 if r else 0.05).add_(
                    A[:, r, :, None, None] * B[:, r, None, :, None] * C[:, r, None, None, :])
            else:
                noise = noise.mul_(1.0 if r else 0.05).add_(A[:, r, :, None] * B[:, r, None, :])
        o.copy_(noise)
    return out.reshape(-1).to((RDT if real else CDT)[fp64])


def _degrees(so3, L):
    l = torch.arange(L + 1, device="cuda")
    return torch.repeat_interleave(l, (2 * l + 1) ** 2 if so3 else 2 * l + 1).to(torch.float32)


def _coeffs(so3, L, b, real, fp64, g):
    s = (_degrees(so3, L) + 1.0) ** (-1.5 if so3 else -1.0)
    v = _rand((b, s.numel()), torch.float32 if real else torch.complex64, g) * s
    return v.reshape(-1).to((RDT if real else CDT)[fp64])


def _uneven_l(case):
    r = np.random.Generator(np.random.PCG64(case["batch"] * 10007 + case["l_max"] * 101 + case["l_min"]))
    return [int(x) for x in r.integers(case["l_min"], case["l_max"] + 1, case["batch"])]


def _kind(case):
    so3 = case["family"] != "s2" and not case.get("sphere", False)
    return so3, (_lib.SO3_REAL if case["real"] else _lib.SO3_COMPLEX) if so3 else \
        (_lib.S2_REAL if case["real"] else _lib.S2_COMPLEX)


def _inputs(case, seed):
    """The pass's inputs, in the library's layouts and element types."""
    so3, _ = _kind(case)
    L, b, real, fp64 = case["l_max"], case["batch"], case["real"], case["precision"] == "fp64"
    if case["family"] == "points":
        r = np.random.Generator(np.random.PCG64(seed))
        n = case["n"]
        beta = np.arccos(r.uniform(-1.0, 1.0, n))
        ab = [r.uniform(0, 2 * np.pi, n) for _ in range(2)]
        pts = np.stack([beta, ab[0]] if case["sphere"] else [ab[0], beta, ab[1]], axis=1)
        return {"F": _coeffs(so3, L, 1, real, True, _gen(seed, 1)), "pts": np.ascontiguousarray(pts)}
    if case["family"] == "uneven":
        order = sorted(_uneven_l(case))  # the batch's layout: ascending l_max
        f = [_samples(True, l, 1, real, False, _gen(seed, 2 * i)) for i, l in enumerate(order)]
        F = [_coeffs(True, l, 1, real, False, _gen(seed, 2 * i + 1)) for i, l in enumerate(order)]
        return {"f": torch.cat(f), "F": torch.cat(F)}
    return {"f": _samples(so3, L, b, real, fp64, _gen(seed, 0)), "F": _coeffs(so3, L, b, real, fp64, _gen(seed, 1))}


def prepare(case, seed):
    so3, kind = _kind(case)
    s = _inputs(case, seed)
    s["stream"] = torch.cuda.current_stream().cuda_stream
    if case["family"] == "points":
        s["plan"] = _lib.Plan(kind, case["l_max"], 1, "fp64", "stable" if so3 else "reference")
        s["out"] = np.empty(case["n"], dtype=np.float64 if case["real"] else np.complex128)
        s["ptr"] = s["pts"].ctypes.data_as(_lib._dp)
        return s
    if case["family"] == "uneven":
        s["plan"] = _lib.Batch(kind, _uneven_l(case), case["precision"], "stable", _lib.FLAG_GRAPH)
    else:
        flags = _lib.FLAG_REFINE | _lib.FLAG_EXACT_INVERSE if case["refined"] else 0
        s["plan"] = _lib.Plan(kind, case["l_max"], case["batch"], case["precision"],
                              "stable" if so3 else "reference", flags)
    s["F_out"], s["f_out"] = torch.empty_like(s["F"]), torch.empty_like(s["f"])
    return s


def run(s):
    plan, st = s["plan"], s["stream"]
    if "pts" in s:
        plan.inverse_points(s["F"].data_ptr(), 0, s["ptr"], len(s["pts"]), s["out"].ctypes.data, st)
        return {"values": s["out"]}
    plan.forward(s["f"].data_ptr(), s["F_out"].data_ptr(), st)
    plan.inverse(s["F"].data_ptr(), s["f_out"].data_ptr(), st)
    return {"coeffs": s["F_out"], "grid": s["f_out"]}


# ------------------------------------------------------------------ the work of a pass


def _size(so3, L):
    B = L + 1
    return (8 * B ** 3, B * (4 * B * B - 1) // 3) if so3 else (4 * B * B, B * B)


def work(case):
    so3, _ = _kind(case)
    el = (8 if case["precision"] == "fp64" else 4) * (1 if case["real"] else 2)
    if case["family"] == "points":
        _, C = _size(so3, case["l_max"])
        out = 8 if case["real"] else 16
        return {"bytes": C * el + case["n"] * (out + (24 if so3 else 16)), "flops": 4.0 * C * case["n"]}
    ls = _uneven_l(case) if case["family"] == "uneven" else [case["l_max"]] * case["batch"]
    nbytes = flops = 0.0
    half = 0.5 if case["real"] else 1.0
    for l in ls:
        G, C = _size(so3, l)
        N = 2 * (l + 1)
        nbytes += 2 * el * (G + C)
        # both directions: the FFTs (5 log2 N flops a sample and axis) and the beta-sums (real times complex)
        flops += 2 * half * (5.0 * G * math.log2(N) * (2 if so3 else 1) + 4.0 * N * C)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ the same in 64 bits, by plain torch


def _beta(L):
    return (2 * torch.arange(2 * L + 2, device="cuda", dtype=torch.float64) + 1) * (math.pi / (4 * (L + 1)))


def _weights(so3, L):
    B = L + 1
    j = 2 * torch.arange(2 * B, device="cuda", dtype=torch.float64) + 1
    k = 2 * torch.arange(B, device="cuda", dtype=torch.float64) + 1
    s = (torch.sin(j[:, None] * k * (math.pi / (4 * B))) / k).sum(1) * torch.sin(j * (math.pi / (4 * B)))
    return s / (4.0 * B ** 3) if so3 else s * (2 * math.pi / B ** 2)


def _wigner(beta, L):
    """Yields (l, d) with d[k, m + l, n + l] = d^l_mn(beta_k): the three-term recursion in l, seeds in logarithms."""
    K, W = beta.numel(), 2 * L + 1
    m = torch.arange(-L, L + 1, device="cuda", dtype=torch.float64)[:, None].expand(W, W)
    n = m.T
    top = torch.maximum(m.abs(), n.abs())
    low = torch.where(m >= n.abs(), n, torch.where(-m >= n.abs(), -n, torch.where(n >= m.abs(), m, -m)))
    lg = torch.lgamma
    half = 0.5 * (lg(2 * top + 1) - lg(top + low + 1) - lg(top - low + 1))
    par = 1.0 - 2.0 * torch.remainder(m + n, 2)
    # seed of (top, low): (-1)^(top - low); swapping or negating one side gives (-1)^(m + n) once more
    keep = (m >= n.abs()) | (-n >= m.abs())
    sign = torch.where(keep, par, torch.ones_like(par))
    lc, ls = torch.log(torch.cos(beta / 2)), torch.log(torch.sin(beta / 2))
    cb = torch.cos(beta)[:, None, None]
    prev = torch.zeros((K, W, W), dtype=torch.float64, device="cuda")
    cur = torch.zeros_like(prev)
    for l in range(L + 1):
        # the entries that begin at this l: the border of the block
        b = slice(L - l, L + l + 1)
        for rows, cols in ((slice(L + l, L + l + 1), b), (slice(L - l, L - l + 1), b),
                           (b, slice(L + l, L + l + 1)), (b, slice(L - l, L - l + 1))):
            e = half[rows, cols] + lc[:, None, None] * (top + low)[rows, cols] + ls[:, None, None] * (top - low)[rows, cols]
            cur[:, rows, cols] = sign[rows, cols] * torch.exp(e)
        yield l, cur[:, b, b]
        if l == L:
            return
        if l == 0:
            prev[:, b, b], cur[:, b, b] = cur[:, b, b].clone(), cur[:, b, b] * cb
            continue
        mm, nn = m[b, b], n[b, b]
        s1 = torch.sqrt(((l + 1) ** 2 - mm * mm) * ((l + 1) ** 2 - nn * nn)) * l
        s0 = torch.sqrt((l * l - mm * mm) * (l * l - nn * nn)) * ((l + 1) / s1)
        new = ((2 * l + 1.0) / s1) * (l * (l + 1) * cb - mm * nn) * cur[:, b, b] - s0 * prev[:, b, b]
        prev[:, b, b] = new
        prev, cur = cur, prev


def _tmat(l):
    """Row a, column c of the complex-to-real basis: y_a = sum_c T_ac Y_c."""
    T = torch.zeros((2 * l + 1, 2 * l + 1), dtype=torch.complex128)
    T[l, l] = 1
    for a in range(1, l + 1):
        s = -math.sqrt(0.5) if a & 1 else math.sqrt(0.5)
        T[l - a, l - a], T[l - a, l + a] = 1j * math.sqrt(0.5), -1j * s
        T[l + a, l - a], T[l + a, l + a] = math.sqrt(0.5), s
    return T.cuda()


def _off(l):
    return l * (4 * l * l - 1) // 3


def _so3_complex_block(F, l, real):
    """The block [b, m, n] of degree l of packed coefficients (column-major), in the complex basis."""
    W = 2 * l + 1
    X = F[:, _off(l):_off(l + 1)].reshape(-1, W, W).transpose(1, 2).to(torch.complex128)
    if real:
        T = _tmat(l)
        X = T.conj().T @ X @ T
    return X


def _so3_exact(L, f, F, real):
    """(forward of the samples f, inverse of the coefficients F) of b functions."""
    N, W = 2 * L + 2, 2 * L + 1
    b = f.numel() // N ** 3
    f = f.reshape(b, N, N, N)
    F = F.reshape(b, -1)
    idx = torch.remainder(-torch.arange(-L, L + 1, device="cuda"), N)
    w = _weights(True, L)
    G = torch.empty((b, N, W, W), dtype=torch.complex128, device="cuda")
    for i in range(b):
        G[i] = torch.fft.fft2(f[i].to(torch.complex128))[:, idx][:, :, idx] * w[:, None, None]
    H = torch.zeros_like(G)
    out = torch.empty(F.shape, dtype=torch.float64 if real else torch.complex128, device="cuda")
    for l, d in _wigner(_beta(L), L):
        r = slice(L - l, L + l + 1)
        X = _so3_complex_block(F, l, real) * (2 * l + 1)
        Y = torch.empty_like(X)
        for i in range(b):
            Y[i] = (G[i, :, r, r] * d).sum(0)
            H[i, :, r, r] += X[i] * d
        if real:
            T = _tmat(l)
            Y = (T @ Y @ T.conj().T).real
        out[:, _off(l):_off(l + 1)] = Y.transpose(1, 2).reshape(b, -1)
    del G
    grid = torch.empty(f.shape, dtype=torch.float64 if real else torch.complex128, device="cuda")
    for i in range(b):
        P = torch.zeros((N, N, N), dtype=torch.complex128, device="cuda")
        P[:, idx[:, None], idx[None, :]] = H[i]  # e^{-i m alpha}: bin -m of an inverse DFT
        g = torch.fft.ifft2(P) * float(N * N)
        grid[i] = g.real if real else g
    return out.reshape(-1), grid.reshape(-1)


def _legendre(x, L):
    """nP[l, m, k], 0 <= m <= l."""
    P = torch.zeros((L + 1, L + 1, x.numel()), dtype=torch.float64, device="cuda")
    m = torch.arange(L + 1, device="cuda", dtype=torch.float64)
    lg = torch.lgamma
    # nP(m,m) = (-1)^m sqrt((2m+1)/(4 pi) (2m-1)!!/(2m)!!) sin^m
    e = 0.5 * (torch.log((2 * m + 1) / (4 * math.pi)) + lg(2 * m + 1) - 2 * m * math.log(2.0) - 2 * lg(m + 1))
    e = e[:, None] + m[:, None] * 0.5 * torch.log1p(-x * x)
    D = torch.exp(e) * (1.0 - 2.0 * torch.remainder(m, 2))[:, None]
    for l in range(L + 1):
        if l >= 1:
            mm = m[:l, None]
            a = torch.sqrt((4.0 * l * l - 1.0) / (l * l - mm * mm))
            P[l, :l] = a * x * P[l - 1, :l]
            if l >= 2:
                q = m[:l - 1, None]
                c = torch.sqrt((4.0 * (l - 1) ** 2 - 1.0) / ((l - 1) ** 2 - q * q))
                P[l, :l - 1] -= a[:l - 1] / c * P[l - 2, :l - 1]
        P[l, l] = D[l]
    return P


def _s2_basis(F, L, real, to_real):
    """Between the real and the complex basis, degree by degree; F [b, B^2]."""
    out = torch.empty(F.shape, dtype=torch.float64 if to_real else torch.complex128, device="cuda")
    T = _tmat(L)
    for l in range(L + 1):
        t = T[L - l:L + l + 1, L - l:L + l + 1]
        X = F[:, l * l:(l + 1) ** 2].to(torch.complex128)
        out[:, l * l:(l + 1) ** 2] = (X @ t.conj().T).real if to_real else X @ t
    return out


def _s2_exact(L, f, F, real):
    N = 2 * L + 2
    b = f.numel() // (N * N)
    f = f.reshape(b, N, N)
    F = F.reshape(b, -1)
    Fc = _s2_basis(F, L, real, False) if real else F.to(torch.complex128)
    G = torch.fft.fft(f.to(torch.complex128))
    w = _weights(False, L)
    P = _legendre(torch.cos(_beta(L)), L)
    H = torch.zeros((b, N, N), dtype=torch.complex128, device="cuda")
    out = torch.zeros((b, (L + 1) ** 2), dtype=torch.complex128, device="cuda")
    l = torch.arange(L + 1, device="cuda")
    for m in range(-L, L + 1):
        a = abs(m)
        sg = -1.0 if m < 0 and a & 1 else 1.0
        p = sg * P[a:, a]  # [l - a, k]
        g = torch.view_as_real(G[:, :, m] * w).permute(0, 2, 1).reshape(2 * b, N)
        at = l[a:] * (l[a:] + 1) + m
        y = (g @ p.T).reshape(b, 2, -1)
        out[:, at] = torch.complex(y[:, 0], y[:, 1])
        x = torch.view_as_real(Fc[:, at]).permute(0, 2, 1).reshape(2 * b, -1)
        y = (x @ p).reshape(b, 2, N)
        H[:, :, m] = torch.complex(y[:, 0], y[:, 1])
    grid = torch.fft.ifft(H) * N
    if real:
        return _s2_basis(out, L, real, True).reshape(-1), grid.real.reshape(-1).contiguous()
    return out.reshape(-1), grid.reshape(-1)


def _points_exact(case, s):
    L, real = case["l_max"], case["real"]
    p = torch.from_numpy(s["pts"]).cuda()
    F = s["F"].reshape(1, -1)
    m = torch.arange(-L, L + 1, device="cuda", dtype=torch.float64)
    if case["sphere"]:
        Fc = (_s2_basis(F, L, real, False) if real else F.to(torch.complex128))[0]
        P = _legendre(torch.cos(p[:, 0]), L)
        y = torch.zeros(case["n"], dtype=torch.complex128, device="cuda")
        l = torch.arange(L + 1, device="cuda")
        for q in range(-L, L + 1):
            a = abs(q)
            sg = -1.0 if q < 0 and a & 1 else 1.0
            c = Fc[l[a:] * (l[a:] + 1) + q]
            y += sg * (c[:, None] * P[a:, a]).sum(0) * torch.exp(1j * q * p[:, 1])
    else:
        parts = []
        for i in range(0, case["n"], 512):
            q = p[i:i + 512]
            S = torch.zeros((len(q), 2 * L + 1, 2 * L + 1), dtype=torch.complex128, device="cuda")
            for l, d in _wigner(q[:, 1].contiguous(), L):
                r = slice(L - l, L + l + 1)
                S[:, r, r] += _so3_complex_block(F, l, real) * (2 * l + 1) * d
            ea, eg = torch.exp(-1j * q[:, :1] * m), torch.exp(-1j * q[:, 2:] * m)
            parts.append(((S * ea[:, :, None]).sum(1) * eg).sum(1))
        y = torch.cat(parts)
    y = y.cpu().numpy()
    return y.real.copy() if real else y


def exact(case, seed):
    s = _inputs(case, seed)
    so3, _ = _kind(case)
    if case["family"] == "points":
        return {"values": _points_exact(case, s)}
    if case["family"] == "uneven":
        order = sorted(_uneven_l(case))
        F, f, c0, g0 = [], [], 0, 0
        for l in sorted(set(order)):
            n = order.count(l)
            G, C = _size(True, l)
            a, b = _so3_exact(l, s["f"][g0:g0 + n * G], s["F"][c0:c0 + n * C], case["real"])
            F.append(a)
            f.append(b)
            g0, c0 = g0 + n * G, c0 + n * C
        return {"coeffs": torch.cat(F), "grid": torch.cat(f)}
    F, f = (_so3_exact if so3 else _s2_exact)(case["l_max"], s["f"], s["F"], case["real"])
    return {"coeffs": F, "grid": f}
