"""The work that a program using this framework has it do, as measurable
cases: the calls, their inputs, what one call cannot do without, and its
result in 64 bits.

Sizes come from the five headline configurations of the 2D NFFT (plain 64^2,
polar raster 512^2, clustered 2048^2, uneven batch of 64, least squares
1024^2) and from the Knab regridding, PSO far-field and type-3 workloads of
the benchmark, with odd and small ones beside them.
"""
import math
import random

import numpy as np
import torch

from miscellaneous_gb300 import knab, nfft, nufft3

# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # one solver iteration (forward and adjoint on bound points) at the plain NDFT-comparison
        # size: an interactive or nested problem, where latency and launches count
        dict(name="solver 64^2, 4 k uniform", kind="solver", N1=64, N2=64, M=4096, K=6, points="uniform", precision="f32"),
        # the reference's drop-in call on new points each time (binning, spreading, FFT, crop), small
        dict(name="NFFT2_2D 64^2, 4 k", kind="nfft2", N1=64, N2=64, M=4096, K=6, points="uniform", precision="f32"),
        # the SAR back-projection shape: 512 spokes of 2048 samples, one solver iteration
        dict(name="solver 512^2, 1 M polar", kind="solver", N1=512, N2=512, M=1 << 20, K=6, points="polar", precision="f32"),
        # the same raster met once: the reference's forward call with its binning
        dict(name="NFFT1_2D 512^2, 1 M polar", kind="nfft1", N1=512, N2=512, M=1 << 20, K=6, points="polar", precision="f32"),
        # the headline configuration: the largest single transform, points in clusters
        dict(name="solver 2048^2, 16 M clustered", kind="solver", N1=2048, N2=2048, M=1 << 24, K=6, points="clustered",
             precision="f32"),
        # differentiable least squares: forward, adjoint and the gradient in the coordinates
        dict(name="lsq 1024^2, 4 M uniform", kind="lsq", N1=1024, N2=1024, M=1 << 22, K=6, points="uniform", precision="f32"),
        # a raster of no convenient size, an odd number of points, the narrow window (w = 4)
        dict(name="solver 250x378, 300 k, w 4", kind="solver", N1=250, N2=378, M=300007, K=4, points="clustered",
             precision="f32"),
        # double precision, the reference's second overload
        dict(name="solver 128^2, 100 k, f64", kind="solver", N1=128, N2=128, M=100003, K=6, points="uniform", precision="f64"),
        # 64 transforms of uneven size in one call
        dict(name="batch of 64 uneven", kind="batch", count=64, e_lo=7, e_hi=10, m_lo=10_000, m_hi=4_000_000, sizes=4, K=6),
        # one generation of the reflectarray synthesis: 250 particles, positions new each time
        dict(name="far field, 250 particles", kind="far_field", count=250, side=44),
        # regridding a SAR sub-image onto a finer, rotated raster
        dict(name="knab 1024^2 to 2048^2", kind="knab", N=1024, L=2048),
        # nonuniform points to nonuniform frequencies
        dict(name="type 3, 200 k to 150 k", kind="type3", M=200_000, N=150_001, eps=1e-6, precision="f32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi):
    """An even raster side: a power of two as often as not."""
    n = _log(rng, lo, hi)
    return 1 << int(round(math.log2(n))) if rng.random() < 0.5 else max(lo, n // 2 * 2)


def draw(rng):
    kind = rng.choice(["solver"] * 5 + ["nfft1", "nfft2", "lsq", "f64", "batch", "far_field", "knab", "type3"])
    points = rng.choice(["uniform", "polar", "clustered"])
    if kind in ("solver", "lsq", "nfft1", "nfft2"):
        N1 = _side(rng, 32, 1024 if kind != "solver" else 2048)
        N2 = N1 if rng.random() < 0.5 else min(2048, max(32, int(N1 * rng.uniform(0.5, 2)) // 2 * 2))
        M = _log(rng, 1000, {"solver": 1 << 24, "lsq": 1 << 22, "nfft1": 1 << 22, "nfft2": 1 << 22}[kind])
        K = rng.choice([4, 6, 6, 8]) if kind in ("solver", "lsq") else 6
        return dict(kind=kind, N1=N1, N2=N2, M=M, K=K if M <= 1 << 23 else min(K, 6), points=points, precision="f32")
    if kind == "f64":
        N1 = _side(rng, 32, 512)
        return dict(kind=rng.choice(["solver", "nfft1", "nfft2"]), N1=N1, N2=_side(rng, 32, 512), M=_log(rng, 1000, 500_000), K=6,
                    points=points, precision="f64")
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(8, 48), e_lo=7, e_hi=rng.randint(8, 10), m_lo=10_000,
                    m_hi=_log(rng, 100_000, 4_000_000), sizes=rng.randrange(1 << 20), K=rng.choice([4, 6]))
    if kind == "far_field":
        return dict(kind="far_field", count=rng.randint(20, 300), side=rng.randint(12, 52))
    if kind == "knab":
        N = 2 * _log(rng, 64, 512)
        return dict(kind="knab", N=N, L=int(N * rng.uniform(1.0, 2.0)))
    return dict(kind="type3", M=_log(rng, 2000, 400_000), N=_log(rng, 2000, 200_000), eps=rng.choice([1e-4, 1e-5, 1e-6]),
                precision=rng.choice(["f32", "f32", "f64"]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
_GRID = ("nfft1", "nfft2")  # calls that take coordinates in the reference's grid units
_PSO_LAMBDA = 3e8 / 14.25e9


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _real(n, g):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _normal(n, g):
    return torch.randn(n, generator=g, device="cuda", dtype=torch.float64)


def _cplx(shape, g, precision):
    dt = torch.complex64 if precision == "f32" else torch.complex128
    return torch.randn(shape, generator=g, device="cuda", dtype=dt) * math.sqrt(2.0)


def _points(points, M, g):
    """Unit coordinates in [-1/2, 1/2), 64 bits."""
    if points == "uniform":
        return _real(M, g) - 0.5, _real(M, g) - 0.5
    if points == "polar":
        spokes = max(1, int(math.sqrt(M / 4)))
        p = torch.arange(M, device="cuda")
        th = math.pi * (p % spokes).double() / spokes
        r = -0.5 + (p // spokes).double() / (-(-M // spokes))
        x1 = r * torch.cos(th) + 1e-3 * (2 * _real(M, g) - 1)
        x2 = r * torch.sin(th) + 1e-3 * (2 * _real(M, g) - 1)
    else:
        x1, x2 = 0.15 * _normal(M, g), 0.15 * _normal(M, g)
    return torch.remainder(x1 + 0.5, 1.0) - 0.5, torch.remainder(x2 + 0.5, 1.0) - 0.5


def _batch_sizes(case):
    r = random.Random(case["sizes"])
    ns = [1 << r.randint(case["e_lo"], case["e_hi"]) for _ in range(case["count"])]
    ms = [_log(r, case["m_lo"], case["m_hi"]) for _ in range(case["count"])]
    return ns, ms


def _knab_axes(N):
    T1, T2 = 0.15, 1.0 / N
    return T1, T2, 1000.0 + T1 * np.arange(N), -0.5 + T2 * np.arange(N), 0.45 / T1, 0.45 / T2


def _pso_scale(side):
    a_prime = float(np.float32((side - 1) * _PSO_LAMBDA))
    return nfft.pso_far_field_scales(side, side, a_prime, a_prime)


def _inputs(case, seed):
    """The arrays that the call is given, in the order of their making."""
    g, kind = _gen(seed), case["kind"]
    if kind in ("solver", "lsq", "nfft1", "nfft2"):
        prec = case["precision"]
        x1, x2 = _points(case["points"], case["M"], g)
        if kind in _GRID:
            x1, x2 = x1 * case["N1"], x2 * case["N2"]
        if prec == "f32":
            x1, x2 = x1.float(), x2.float()
        return dict(x1=x1, x2=x2, F=_cplx((case["N1"], case["N2"]), g, prec), f=_cplx(case["M"], g, prec))
    if kind == "batch":
        ns, ms = _batch_sizes(case)
        pts = [tuple(v.float() for v in _points("uniform", m, g)) for m in ms]
        return dict(x1=[p[0] for p in pts], x2=[p[1] for p in pts], F=[_cplx((n, n), g, "f32") for n in ns],
                    f=[_cplx(m, g, "f32") for m in ms])
    if kind == "far_field":
        side, P = case["side"], case["count"]
        at = (torch.arange(side, device="cuda", dtype=torch.float64) - (side - 1) / 2) * 0.6
        gy, gx = torch.meshgrid(at, at, indexing="ij")
        jit = lambda: 0.1 * _real(P * side * side, g).reshape(P, -1) - 0.05  # noqa: E731
        X = ((gx.reshape(1, -1) + jit()) * _PSO_LAMBDA).float()
        Y = ((gy.reshape(1, -1) + jit()) * _PSO_LAMBDA).float()
        ph = (2 * _real(P * side * side, g).reshape(P, -1) - 1) * math.pi
        u = torch.arange(-side, side, device="cuda", dtype=torch.float64)
        filt = (u[:, None] ** 2 + u[None, :] ** 2 <= (2.0 * (side - 1)) ** 2 / 4).float().reshape(-1)
        return dict(X=X, Y=Y, E=torch.polar(torch.ones_like(ph), ph).to(torch.complex64), filter=filt)
    if kind == "knab":
        N, L = case["N"], case["L"]
        T1, T2, rho, cosa, _, _ = _knab_axes(N)
        m = 24  # the window's reach inside the raster's edges
        u = torch.linspace(m, N - 1 - m, L, device="cuda", dtype=torch.float64)[None, :]
        v = torch.linspace(m, N - 1 - m, L, device="cuda", dtype=torch.float64)[:, None]
        th = 0.01 * (0.5 + float(_real(1, g)))
        rho_out = rho[0] + T1 * (math.cos(th) * u - math.sin(th) * v)
        cos_out = cosa[0] + T2 * (math.sin(th) * u + math.cos(th) * v)
        return dict(data=_cplx((N, N), g, "f32"), rho_out=rho_out.contiguous(), cos_out=cos_out.contiguous())
    M, N = case["M"], case["N"]  # type 3
    return dict(x=65 * _real(M, g) - 40, y=6 * _normal(M, g), s=7 * _real(N, g) - 3, t=5 * _real(N, g) - 2.5,
                f=_cplx(M, g, case["precision"]))


def prepare(case, seed):
    s = dict(_inputs(case, seed), case=case)
    kind = case["kind"]
    if kind in ("solver", "lsq"):  # a solver keeps its plan, with the points binned
        s["plan"] = nfft.Plan(case["N1"], case["N2"], sigma=2.0, K=case["K"], precision=case["precision"])
        s["plan"].set_points(s["x1"], s["x2"], units="unit")
    elif kind == "batch":
        ns, ms = _batch_sizes(case)
        s["plan"] = nfft.Batch([(n, n) for n in ns], sigma=2.0, K=case["K"])
        s["plan"].set_points(s["x1"], s["x2"], units="unit")
        s["f_out"] = torch.empty(sum(ms), dtype=torch.complex64, device="cuda")
        s["F_out"] = torch.empty(sum(n * n for n in ns), dtype=torch.complex64, device="cuda")
        s["f_outs"], s["F_outs"] = list(s["f_out"].split(ms)), list(s["F_out"].split([n * n for n in ns]))
    elif kind == "far_field":  # the swarm's buffers live as long as the optimisation
        n = 2 * case["side"]
        s["plan"] = nfft.Batch([(n, n)] * case["count"], sigma=2.0, K=6)
        s["out"] = torch.empty((case["count"], n * n), dtype=torch.complex64, device="cuda")
        s["outs"] = list(s["out"])
        s["Xs"], s["Ys"], s["Es"] = list(s["X"]), list(s["Y"]), list(s["E"])
        s["scale"] = _pso_scale(case["side"])
    elif kind == "knab":  # one geometry, many rasters
        _, _, rho, cosa, B1, B2 = _knab_axes(case["N"])
        s["plan"] = knab.Regridder(rho, cosa, B1, B2, precision="f32")
        s["plan"].set_points(s["rho_out"], s["cos_out"])
    return s


# ---------------------------------------------------------------------------
# one call
# ---------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "solver":
        return s["plan"].forward(s["F"]), s["plan"].adjoint(s["f"])
    if kind == "lsq":
        return s["plan"].forward(s["F"]), s["plan"].adjoint(s["f"]), *s["plan"].grad_x(s["F"], s["f"])
    if kind == "nfft1":
        return nfft.NFFT1_2D(s["F"], s["x1"], s["x2"])
    if kind == "nfft2":
        return nfft.NFFT2_2D(s["f"], s["x1"], s["x2"], case["N1"], case["N2"])
    if kind == "batch":
        s["plan"].forward(s["F"], s["f_outs"])
        s["plan"].adjoint(s["f"], s["F_outs"])
        return s["f_out"], s["F_out"]
    if kind == "far_field":
        s["plan"].far_field(s["Xs"], s["Ys"], s["Es"], s["scale"][0], s["scale"][1], s["filter"], s["outs"])
        return s["out"]
    if kind == "knab":
        return s["plan"](s["data"])
    return nufft3.NUFFT_2D(s["x"], s["y"], s["s"], s["t"], s["f"], case["eps"])


def _transform_work(N1, N2, M, K, c, ways):
    """Coordinates and values once a direction, coefficients once; window sums and the sigma = 2 FFT."""
    n = 4.0 * N1 * N2
    return dict(bytes=ways * (2 * c * M + c * N1 * N2), flops=ways * (4.0 * (2 * K + 1) ** 2 * M + 5.0 * n * math.log2(n)))


def work(case):
    kind = case["kind"]
    if kind in ("solver", "lsq", "nfft1", "nfft2"):
        c = 8 if case["precision"] == "f32" else 16
        return _transform_work(case["N1"], case["N2"], case["M"], case["K"], c, {"solver": 2, "lsq": 3}.get(kind, 1))
    if kind == "batch":
        each = [_transform_work(n, n, m, case["K"], 8, 2) for n, m in zip(*_batch_sizes(case))]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    if kind == "far_field":
        w = _transform_work(2 * case["side"], 2 * case["side"], case["side"] ** 2, 6, 8, 1)
        return {k: case["count"] * v for k, v in w.items()}
    if kind == "knab":
        n, L = 16.0 * case["N"] ** 2, case["L"]
        return dict(bytes=8 * case["N"] ** 2 + 16 * L * L, flops=4.0 * 169 * L * L + 5 * n * math.log2(n))
    msp = 2 + 2 * 4.84 * -math.log(case["eps"] / 76) / (math.pi * 2.84)
    taps = (2 * math.floor(msp - 2) + 1) ** 2
    c = 8 if case["precision"] == "f32" else 16
    return dict(bytes=(16 + c) * (case["M"] + case["N"]), flops=4.0 * taps * (case["M"] + case["N"]))


# ---------------------------------------------------------------------------
# the same in 64 bits: an NUFFT with the exp(sqrt) window of Barnett, Magland
# and af Klinteberg (16 taps, about 1e-14), direct sums where they are short
# ---------------------------------------------------------------------------
_W = 16
_BETA = 2.30 * _W
_CHUNK = 1 << 22


def _axis64(N, dev):
    n = max(2 * N, 2 * _W)
    q, w = np.polynomial.legendre.leggauss(120)
    k = np.arange(N) - N // 2
    phi = np.exp(_BETA * (np.sqrt(1 - q * q) - 1)) * w
    hat = (_W / 2) * (phi[None, :] * np.cos(2 * np.pi * k[:, None] * (q[None, :] * _W / 2) / n)).sum(1)
    return n, torch.tensor(1.0 / hat, device=dev), torch.tensor(k % n, device=dev)


def _taps64(x, n):
    u = x * n
    first = torch.ceil(u - _W / 2)
    z = (u - first)[None, :] - torch.arange(_W, device=x.device, dtype=torch.float64)[:, None]
    ph = torch.exp(_BETA * (torch.sqrt((1 - (2 * z / _W) ** 2).clamp_min(0)) - 1))
    cell = torch.remainder(first.long()[None, :] + torch.arange(_W, device=x.device)[:, None], n)
    return ph, cell


def _type2(F, x1, x2, sign):
    F = F.to(torch.complex128)
    n1, d1, r1 = _axis64(F.shape[0], F.device)
    n2, d2, r2 = _axis64(F.shape[1], F.device)
    G = torch.zeros((n1, n2), dtype=torch.complex128, device=F.device)
    G[r1[:, None], r2[None, :]] = F * d1[:, None] * d2[None, :]
    G = (torch.fft.fft2(G) if sign < 0 else torch.fft.ifft2(G) * (n1 * n2)).reshape(-1)
    out = torch.empty(x1.numel(), dtype=torch.complex128, device=F.device)
    for at in range(0, x1.numel(), _CHUNK):
        p1, c1 = _taps64(x1[at:at + _CHUNK], n1)
        p2, c2 = _taps64(x2[at:at + _CHUNK], n2)
        acc = torch.zeros(p1.shape[1], dtype=torch.complex128, device=F.device)
        for i in range(_W):
            row = torch.zeros_like(acc)
            for j in range(_W):
                row += p2[j] * G[c1[i] * n2 + c2[j]]
            acc += p1[i] * row
        out[at:at + _CHUNK] = acc
    return out


def _type1(f, x1, x2, N1, N2, sign):
    f = f.to(torch.complex128)
    n1, d1, r1 = _axis64(N1, f.device)
    n2, d2, r2 = _axis64(N2, f.device)
    re = torch.zeros(n1 * n2, dtype=torch.float64, device=f.device)
    im = torch.zeros_like(re)
    for at in range(0, x1.numel(), _CHUNK):
        p1, c1 = _taps64(x1[at:at + _CHUNK], n1)
        p2, c2 = _taps64(x2[at:at + _CHUNK], n2)
        v = f[at:at + _CHUNK]
        for i in range(_W):
            vr, vi = v.real * p1[i], v.imag * p1[i]
            for j in range(_W):
                cell = c1[i] * n2 + c2[j]
                re.index_add_(0, cell, vr * p2[j])
                im.index_add_(0, cell, vi * p2[j])
    G = torch.complex(re, im).reshape(n1, n2)
    G = torch.fft.fft2(G) if sign < 0 else torch.fft.ifft2(G) * (n1 * n2)
    return G[r1[:, None], r2[None, :]] * d1[:, None] * d2[None, :]


def _knab_window(T, B, P, N):
    """The Knab window over frequencies -kg .. kg: 1/N in the band, outside it the running integral of
    the convolution window, by Gauss-Legendre in theta after f = (B1/2) sin(theta)."""
    df = 1 / (N * T)
    kg = int(math.floor((1 / T - B / 2) / df))
    f = -df * kg + df * np.arange(kg + 1)
    B0, B1, beta = 1 / T, 1 / T - B, math.pi * (1 / T - B) * P * T
    q, w = np.polynomial.legendre.leggauss(200)
    den = B1 * math.sinh(beta) / beta
    G = np.zeros(2 * kg + 1)
    for k in range(kg + 1):
        hi = f[k] + B0 / 2
        if B1 / 2 <= hi:
            G[k] = 1
        elif hi > -B1 / 2:
            a, b = -math.pi / 2, math.asin(2 * hi / B1)
            c = np.cos((a + b) / 2 + (b - a) / 2 * q)
            G[k] = (b - a) / 2 * float((w * c * np.i0(beta * c)).sum()) * (B1 / 2) / den
    G = G + G[::-1]
    G[kg] -= 1
    return G / N, kg


def _knab64(case, d):
    N = case["N"]
    _, _, rho, cosa, B1, B2 = _knab_axes(N)
    T1, T2 = float(np.mean(np.diff(rho))), float(np.mean(np.diff(cosa)))
    Gn, kn = _knab_window(T1, B1, 18, N)
    Gm, km = _knab_window(T2, B2, 18, N)
    n = np.arange(-kn, kn + 1)
    m = np.arange(-km, km + 1)
    E = torch.fft.fft2(d["data"].to(torch.complex128))
    S = torch.zeros((2 * km + 2, 2 * kn + 2), dtype=torch.complex128, device=E.device)
    w = torch.tensor(Gm[:, None] * Gn[None, :], device=E.device)
    S[1:, 1:] = E[torch.tensor(m % N, device=E.device)[:, None], torch.tensor(n % N, device=E.device)[None, :]] * w
    x1, x2 = (d["cos_out"] - cosa[0]) / (N * T2), (d["rho_out"] - rho[0]) / (N * T1)
    out = _type2(S, x1.reshape(-1), x2.reshape(-1), 1).reshape(x1.shape)
    r, c = d["rho_out"][0], d["cos_out"][:, 0]
    out[:, (r < rho.min()) | (r > rho.max())] = 0
    out[(c < cosa.min()) | (c > cosa.max()), :] = 0
    return out


def _type3_64(d):
    out = torch.empty(d["s"].numel(), dtype=torch.complex128, device=d["x"].device)
    f = d["f"].to(torch.complex128)
    step = max(1, (1 << 26) // d["x"].numel())
    for at in range(0, out.numel(), step):
        ph = d["s"][at:at + step, None] * d["x"][None, :]
        ph.addcmul_(d["t"][at:at + step, None], d["y"][None, :])
        c = torch.cos(ph)
        s = torch.sin_(ph)
        out[at:at + step] = torch.complex(c @ f.real + s @ f.imag, c @ f.imag - s @ f.real)
    return out


def exact(case, seed):
    d, kind = _inputs(case, seed), case["kind"]
    if kind in ("solver", "lsq", "nfft1", "nfft2"):
        N1, N2 = case["N1"], case["N2"]
        x1, x2 = d["x1"].double(), d["x2"].double()
        if kind in _GRID:
            x1, x2 = x1 / N1, x2 / N2
        if kind == "nfft1":
            return _type2(d["F"], x1, x2, -1)
        if kind == "nfft2":
            return _type1(d["f"], x1, x2, N1, N2, -1)
        both = _type2(d["F"], x1, x2, -1), _type1(d["f"], x1, x2, N1, N2, 1)
        if kind == "solver":
            return both
        k1 = torch.arange(N1, device=x1.device, dtype=torch.float64)[:, None] - N1 // 2
        k2 = torch.arange(N2, device=x1.device, dtype=torch.float64)[None, :] - N2 // 2
        v = d["f"].to(torch.complex128).conj()
        return both + tuple((v * _type2(d["F"] * (-2j * math.pi * k), x1, x2, -1)).real for k in (k1, k2))
    if kind == "batch":
        ns, _ = _batch_sizes(case)
        each = [(F, f, x1.double(), x2.double(), n) for F, f, x1, x2, n in zip(d["F"], d["f"], d["x1"], d["x2"], ns)]
        return (torch.cat([_type2(F, x1, x2, -1) for F, f, x1, x2, n in each]),
                torch.cat([_type1(f, x1, x2, n, n, 1).reshape(-1) for F, f, x1, x2, n in each]))
    if kind == "far_field":
        n = 2 * case["side"]
        sx, sy = _pso_scale(case["side"])
        # the scaling is part of the call's definition and is done in 32 bits, as the reference does it
        x, y = (d["X"] * sx).double() / n, (d["Y"] * sy).double() / n
        k = torch.arange(n, device=x.device, dtype=torch.float64) - n // 2
        out = []
        for p in range(case["count"]):
            a, b = torch.outer(k, x[p]) * (-2 * math.pi), torch.outer(y[p], k) * (-2 * math.pi)
            e1, e2 = torch.polar(torch.ones_like(a), a), torch.polar(torch.ones_like(b), b)
            out.append(((e1 * d["E"][p].to(torch.complex128)) @ e2).reshape(-1) * d["filter"])
        return torch.stack(out)
    if kind == "knab":
        return _knab64(case, d)
    if case["M"] * case["N"] > 1 << 36:
        return None
    return _type3_64(d)
