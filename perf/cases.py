"""The work that a user of scarl_b200 has it do, as cases that can be timed.

A case is a dict of plain values.  `prepare` makes what a program holds before the call (decks,
device buffers, the context it keeps), `run` is one pass through the package's public entry points,
`exact` gives the same outputs in 64 bits from torch alone, `work` what one pass cannot do without.

Fields lie in device memory, x fastest: torch tensors of shape (L2, L1, L0).

Kinds of case:
  sample    one deck sample, end to end (`generate_sample`): the literal DCT generator in FP64 that
            the deck driver runs by default, or the padded periodic method in FP32, FP32 with the
            split-BF16 tensor-core pass, or FP64
  tile      one tile of the padded method without blending (`gen_padded`)
  steps     the reference's routines called one by one, as a host code that binds them does
  ensemble  many realisations of uneven grids (`gen_ensemble`)
  stat      the Stat_ScaRL step on one field: moments, directional spectra, correlation lengths
  cov       the streamed axis covariance of one field (`axis_cov`)
"""
import math
import random

import numpy as np
import torch

import scarl_b200 as S

DTYPES = {"f32": S.F32, "split": S.F32 | S.SPLIT_BF16, "f64": S.F64}
PAD_TOL = 1e-3
PI_REF = 3.1415926535898  # the reference's PI constant


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def _sample(name, gen, dtype, size, corr, ovlp, topo, mod=1, nu=0.5, margi=1, avg=0.0, std=1.0,
            policy="smooth", step=1.0, tuned=False):
    """corr, ovlp: correlation lengths and overlaps in grid points; size: grid points - 1."""
    c = dict(kind="sample", gen=gen, dtype=dtype, mod=mod, nu=nu, margi=margi, avg=avg, std=std,
             policy=policy, step=step, tuned=tuned)
    for d in range(3):
        c["n%d" % d], c["c%d" % d] = size[d], corr[d]
        c["o%d" % d], c["t%d" % d] = ovlp[d], topo[d]
    if name:
        c["name"] = name
    return c


def _grid(name, kind, size, **more):
    c = dict(kind=kind, **more)
    for d in range(3):
        c["n%d" % d] = size[d]
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the test deck (10 correlation lengths a side, 5 points each) on 8 ranks with the
        # driver's default generator: the smallest call, latency and launches
        _sample("deck_small", "dct", "f64", (40, 40, 40), (4, 4, 4), (4, 4, 4), (2, 2, 2), step=0.25),
        # the driver's default generator at the size of the benchmark deck
        _sample("deck_dct", "dct", "f64", (512, 512, 512), (40, 20, 10), (80, 40, 20), (2, 2, 2)),
        # a host code that binds the reference's routines one by one, odd FP64 tiles
        _grid("steps_f64", "steps", (95, 78, 83), o0=21, o1=16, o2=11, t0=2, t1=2, t2=2, c0=10, c1=8,
              c2=5),
        # the benchmark deck: exponential, lognormal, 2x2x2 tiles, tensor-core pass 1, tuned context
        _sample("deck_split", "padded", "split", (512, 512, 512), (40, 20, 10), (80, 40, 20), (2, 2, 2),
                mod=3, margi=2, avg=1.0, std=0.3, tuned=True),
        # an ordinary single-domain sample in FP32, von Karman, odd sizes
        _sample("sample_f32", "padded", "f32", (256, 210, 180), (16, 12, 9), (16, 12, 9), (1, 1, 1),
                mod=2, nu=1.5, margi=2, avg=1.0, std=0.5),
        # the call's defaults: FP32 on the reference's full padding, a few tiles
        _sample("sample_full", "padded", "f32", (250, 230, 200), (16, 16, 16), (32, 32, 32), (2, 2, 1),
                mod=3, margi=2, avg=1.0, std=0.3, policy="full"),
        # the padded method in the reference's precision on a few tiles
        _sample("sample_f64", "padded", "f64", (300, 260, 220), (20, 15, 10), (40, 30, 20), (2, 2, 1),
                mod=3),
        # one 128^3 tile on the reference's full padding (256^3), Gaussian model, FP32
        _grid("tile_f32", "tile", (128, 128, 128), dtype="f32", corr=10, mod=1, policy="full"),
        # Monte Carlo over uneven grids, one graph a draw, tuned context
        dict(name="ensemble", kind="ensemble", dtype="split", members=64, shapes=7, mod=3, tuned=True),
        # the Stat_ScaRL step on a sample file's FP64 field
        _grid("stat_f64", "stat", (241, 201, 163), dtype="f64", corr=12),
        # the same on the benchmark deck's FP32 field
        _grid("stat_513", "stat", (513, 513, 513), dtype="f32", corr=20),
        # axis covariance of a large field
        _grid("cov_large", "cov", (1024, 1024, 512), dtype="f32", corr=40, lag=256),
    ]


def draw(rng):
    kind = rng.choice(["dct", "dct", "padded", "padded", "padded", "tile", "steps", "ensemble", "stat", "cov"])

    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def box(lo, hi, most):
        while True:
            n = [log(lo, hi) for _ in range(3)]
            if n[0] * n[1] * n[2] <= most:
                return n

    def tiles(n):
        t = [rng.choice([1, 2, 2, 3]) if v >= 48 else rng.choice([1, 2]) for v in n]
        while t[0] * t[1] * t[2] > 12:
            t[rng.randrange(3)] = 1
        return t
    if kind in ("dct", "padded"):
        n = box(32, 512, 300 ** 3)
        c = [rng.randint(3, max(4, min(30, v // 8))) for v in n]
        o = [v * rng.choice([1, 2]) for v in c]
        if kind == "dct":
            return _sample(None, "dct", "f64", n, c, o, tiles(n), std=rng.choice([0.3, 1.0]))
        mod = rng.choice([1, 2, 3, 3])
        m = rng.choice([1, 2])
        small = max(n) <= 200
        return _sample(None, "padded", rng.choice(["f32", "split", "split", "f64"]), n, c, o, tiles(n), mod=mod,
                       nu=1.5 if mod == 2 else 0.5, margi=m, avg=1.0 if m == 2 else 0.0,
                       std=rng.choice([0.3, 0.5]), policy=rng.choice(["smooth", "smooth", "full"]) if small
                       else "smooth")
    if kind == "tile":
        n = box(16, 256, 160 ** 3)
        return _grid(None, "tile", n, dtype=rng.choice(["f32", "split", "f64"]), corr=rng.randint(3, 16),
                     mod=rng.choice([1, 3]), policy=rng.choice(["full", "smooth"]))
    if kind == "steps":
        n = box(24, 160, 100 ** 3)
        t = [rng.choice([1, 2]) for _ in range(3)]
        return _grid(None, "steps", n, o0=rng.randint(3, n[0] // 3), o1=rng.randint(3, n[1] // 3),
                     o2=rng.randint(3, n[2] // 3), t0=t[0], t1=t[1], t2=t[2], c0=rng.randint(3, 12),
                     c1=rng.randint(3, 12), c2=rng.randint(3, 12))
    if kind == "ensemble":
        return dict(kind="ensemble", dtype=rng.choice(["f32", "split", "f64"]), members=log(4, 64),
                    shapes=rng.randrange(1 << 20), mod=rng.choice([1, 3]), tuned=False)
    if kind == "stat":
        return _grid(None, "stat", box(24, 600, 300 ** 3), dtype=rng.choice(["f64", "f64", "f32"]),
                     corr=rng.randint(4, 20))
    n = box(48, 1100, 500 ** 3)
    if rng.random() < 0.5:
        n[0] = -(-n[0] // 16) * 16
    return _grid(None, "cov", n, dtype=rng.choice(["f32", "f32", "f64"]), corr=rng.randint(4, 20),
                 lag=rng.randint(8, min(min(n) - 1, 256)))


# ---------------------------------------------------------------------------
# What the program holds before the call
# ---------------------------------------------------------------------------
_contexts = {}


def _context(tuned=False):
    """The context a program keeps; a tuned one is kept apart."""
    if tuned not in _contexts:
        _contexts[tuned] = S.Context(0)
    return _contexts[tuned]


def _v(case, key):
    return [case["%s%d" % (key, d)] for d in range(3)]


def _deck(case, seed):
    h = case["step"]
    c = _v(case, "c")
    return S.make_sample(xMinGlob=(0, 0, 0), xMaxGlob=[n * h for n in _v(case, "n")], corrL=[v * h for v in c],
                         overlap=[o / v for o, v in zip(_v(case, "o"), c)],
                         pointsPerCorrL=[v + 1 for v in c], corrMod=case["mod"], margiFirst=case["margi"],
                         avg=case["avg"], std_dev=case["std"], seedBase=seed % 1000000007, nu=case["nu"])


def _layout(case):
    """Tile extents Np and blended extents L of a deck (SRC_F/main_ScaRL.f90:100-176)."""
    Np, L = [], []
    for n, o, t, c in zip(_v(case, "n"), _v(case, "o"), _v(case, "t"), _v(case, "c")):
        no = 1 + math.ceil((o / c) * float(c))
        p = math.ceil((n + 1 + (t - 1) * no) / t)
        if t == 2:
            p = max(p, no)
        if t >= 3:
            p = max(p, 2 * no)
        Np.append(p)
        L.append(p * t - (t - 1) * no)
    return Np, L, [1 + math.ceil((o / c) * float(c)) for o, c in zip(_v(case, "o"), _v(case, "c"))]


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _field(case, seed):
    """A correlated lognormal field, the input of the estimators."""
    n = _v(case, "n")[::-1]
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    x = torch.randn(n, generator=g, device=dev)
    h = torch.fft.rfftn(x)
    del x
    for d in range(3):
        f = torch.fft.rfftfreq(n[d], device=dev) if d == 2 else torch.fft.fftfreq(n[d], device=dev)
        h *= torch.exp(-1.5 * (case["corr"] * f) ** 2).reshape([-1 if i == d else 1 for i in range(3)])
    x = torch.fft.irfftn(h, s=n)
    del h
    x = torch.exp(x * (0.29 / x.std()) - 0.043)
    return (x.double() if case["dtype"] == "f64" else x).contiguous()


def _members(case):
    """Shapes (members, 3) and correlation lengths of an ensemble, from its own number."""
    r = random.Random(case["shapes"])
    Np = [[r.choice((64, 96, 128, 160, 192, 256)) for _ in range(3)] for _ in range(case["members"])]
    cl = [[v] * 3 for v in (r.uniform(4.0, 32.0) for _ in range(case["members"]))]
    return np.array(Np, dtype=np.int32), np.array(cl)


def _torch_type(case):
    return torch.float64 if case.get("dtype") == "f64" else torch.float32


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "seed": seed, "ctx": _context(case.get("tuned", False))}
    if kind == "sample":
        st["deck"] = _deck(case, seed)
        st["out"] = torch.empty(_layout(case)[1][::-1], dtype=_torch_type(case), device="cuda")
        st["topo"] = tuple(_v(case, "t"))
    elif kind == "tile":
        st["pad"] = _pads(case["policy"], case["mod"], 0.5, [case["corr"]] * 3, [1.0] * 3, _v(case, "n"))
        st["out"] = torch.empty(_v(case, "n")[::-1], dtype=_torch_type(case), device="cuda")
    elif kind == "steps":
        t = _v(case, "t")
        st["tiles"] = torch.empty([t[0] * t[1] * t[2]] + _v(case, "n")[::-1], dtype=torch.float64, device="cuda")
    elif kind == "ensemble":
        st["Np"], st["cl"] = _members(case)
        st["seeds"] = np.arange(case["members"], dtype=np.uint64) + np.uint64(seed * 4096)
        total = int(np.prod(st["Np"].astype(np.int64), axis=1).sum())
        st["out"] = torch.empty(total, dtype=_torch_type(case), device="cuda")
    else:
        st["field"] = _field(case, seed)
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(st):
    case, ctx, seed = st["case"], st["ctx"], st["seed"]
    kind = case["kind"]
    if kind == "sample":
        t = st["topo"]
        S.generate_sample(ctx, st["deck"], generator=S.GEN_DCT if case["gen"] == "dct" else S.GEN_PADDED,
                          dtype=DTYPES[case["dtype"]], nb_procs=t[0] * t[1] * t[2], topo=t,
                          pad_policy=S.PAD_FULL if case["policy"] == "full" else S.PAD_SMOOTH,
                          pad_tol=PAD_TOL, autotune=case["tuned"], out=st["out"])
        return st["out"]
    if kind == "tile":
        return S.gen_padded(ctx, _v(case, "n"), (1.0, 1.0, 1.0), [case["corr"]] * 3, case["mod"], pad=st["pad"],
                            seed=seed, dtype=DTYPES[case["dtype"]], out=st["out"])
    if kind == "steps":
        n, t, o, c = _v(case, "n"), _v(case, "t"), _v(case, "o"), _v(case, "c")
        tiles = st["tiles"]
        for r in range(t[0] * t[1] * t[2]):
            S.gen_std_gauss_FFT(ctx, n, [v - 1.0 for v in n], c, 1, seed=seed, rank=r, out=tiles[r])
            S.apply_UnityPartition_mtx(ctx, tiles[r], n, o, 1, S.get_topo_pos(r, t), t)
        S.add_overlap(ctx, tiles, n, o, t)
        S.multiVariateTransformation(ctx, 1.0, 0.5, 1, tiles)
        return tiles
    if kind == "ensemble":
        S.gen_ensemble(ctx, st["Np"], st["cl"], corrMod=case["mod"], pad_policy=S.PAD_SMOOTH, pad_tol=PAD_TOL,
                       seeds=st["seeds"], dtype=DTYPES[case["dtype"]], autotune=case["tuned"], out=st["out"])
        return st["out"]
    L = _v(case, "n")
    if kind == "stat":
        ea, es, ga, gs = S.calculate_average_and_stdVar(ctx, st["field"])
        sk = S.rebuild_Sk(ctx, st["field"], L, ga, gs)
        return {"avg": ea, "std": es, "Sk": sk, "corrL": S.rebuild_corrL(sk, L, (1.0, 1.0, 1.0))}
    mean, var, cov = S.axis_cov(ctx, st["field"], L, case["lag"])
    return {"mean": mean, "var": var, "cov": cov}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _fft_flops(P):
    m = float(P[0]) * P[1] * P[2]
    return 2.5 * m * math.log2(m)


def _padded_flops(P, n):
    """Half-spectrum synthesis (about 40 operations a mode) and the real inverse transform."""
    return _fft_flops(P) + 20.0 * P[0] * P[1] * P[2] + 4.0 * n


def work(case):
    kind = case["kind"]
    size = 8 if case.get("dtype") == "f64" or kind == "steps" else 4
    if kind == "sample":
        Np, L, _ = _layout(case)
        nb, n = math.prod(_v(case, "t")), math.prod(L)
        if case["gen"] == "dct":
            m = float(math.prod(Np))
            return {"bytes": n * size, "flops": nb * (2.5 * m * math.log2(m) + 10 * m / 8) + 4.0 * n}
        h = [case["step"]] * 3
        P = _pads(case["policy"], case["mod"], case["nu"], [c * case["step"] for c in _v(case, "c")], h, Np)
        return {"bytes": n * size, "flops": nb * _padded_flops(P, math.prod(Np))}
    if kind == "tile":
        P = _pads(case["policy"], case["mod"], 0.5, [case["corr"]] * 3, [1.0] * 3, _v(case, "n"))
        n = math.prod(_v(case, "n"))
        return {"bytes": n * size, "flops": _padded_flops(P, n)}
    if kind == "steps":
        m, nb = float(math.prod(_v(case, "n"))), math.prod(_v(case, "t"))
        # each routine hands its tiles on in memory: written, then read and written three times
        return {"bytes": 7 * nb * m * size, "flops": nb * (2.5 * m * math.log2(m) + 30 * m)}
    if kind == "ensemble":
        Np, cl = _members(case)
        f = 0.0
        for n, c in zip(Np.tolist(), cl.tolist()):
            f += _padded_flops(_pads("smooth", case["mod"], 0.5, c, [1.0] * 3, n), math.prod(n))
        return {"bytes": float(np.prod(Np.astype(np.int64), axis=1).sum()) * size, "flops": f}
    n = _v(case, "n")
    m = float(math.prod(n))
    lag = case.get("lag")
    f = 4.0 * m
    for v in n:
        p = 2 * v if kind == "stat" else v + lag
        f += m / v * (2.5 * p * math.log2(p) + 1.5 * p)
    return {"bytes": m * size, "flops": f}


# ---------------------------------------------------------------------------
# The same outputs in 64 bits, from torch alone
# ---------------------------------------------------------------------------
def _pads(policy, mod, nu, corr, step, Np):
    """Padded lengths: 2^ceil(log2 2 Np), or the smallest of 2^a and 3, 5, 7 x 2^a (2^a >= 16) whose
    nearest periodic image adds at most PAD_TOL to a covariance."""
    P = []
    for l, h, n in zip(corr, step, Np):
        if policy == "full":
            p = 1
            while p < 2 * n:
                p *= 2
            P.append(p)
            continue

        def corr_at(r):
            if mod == 1:
                return math.exp(-math.pi * r * r / (l * l))
            if mod == 3:
                return math.exp(-2.0 * r / l)
            x = r / (l * math.gamma(nu) / (2.0 * math.sqrt(math.pi) * math.gamma(nu + 0.5)))
            return (1.0 + x) * math.exp(-x)  # Matern of order 3/2
        good = sorted([1 << a for a in range(3, 12)] + [m << a for m in (3, 5, 7) for a in range(4, 11)])
        P.append(next(p for p in good if p <= 2048 and p >= n and corr_at((p - n + 1) * h) <= PAD_TOL))
    return P


def _philox(c0, c1, c2, c3, key):
    """Philox4x32-10 on int64 tensors of 32-bit words."""
    M = 0xFFFFFFFF
    k0, k1 = key & M, (key >> 32) & M
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = ((p1 >> 32) & M) ^ c1 ^ k0, p1 & M, ((p0 >> 32) & M) ^ c3 ^ k1, p0 & M
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return c0, c1, c2, c3


def _normal_pair(a, b):
    u1, u2 = (a.double() + 0.5) * 2.0 ** -32, (b.double() + 0.5) * 2.0 ** -32
    r = torch.sqrt(-2.0 * torch.log(u1))
    return torch.complex(r * torch.cos(2 * math.pi * u2), r * torch.sin(2 * math.pi * u2))


def _padded_exact(P, Np, step, corr, mod, nu, key):
    """One tile of the padded periodic method with normalised spectrum, shape (Np2, Np1, Np0)."""
    dev = _device()
    Hx = P[0] // 2 + 1
    f = [torch.arange(n, device=dev, dtype=torch.float64) for n in (Hx, P[1], P[2])]
    f = [torch.where(2 * k <= p, k, k - p) / (p * h) for k, p, h in zip(f, P, step)]
    f = [v.reshape([-1 if i == 2 - d else 1 for i in range(3)]) for d, v in enumerate(f)]
    if mod == 1:
        A = torch.exp(sum(-math.pi * (l * v) ** 2 / 2 for l, v in zip(corr, f)))
    else:
        v = 0.5 if mod == 3 else nu
        sc = math.gamma(v) / (2.0 * math.sqrt(math.pi) * math.gamma(v + 0.5))
        A = (1.0 + sum((2 * math.pi * l * sc * w) ** 2 for l, w in zip(corr, f))) ** (-(v + 1.5) / 2)
    w = torch.full((Hx,), 2.0, device=dev, dtype=torch.float64)
    w[0] = 1.0
    w[-1] = 1.0
    A = A * (torch.rsqrt(w) / torch.sqrt((w * A * A).sum()))
    H = torch.empty(P[2], P[1], Hx, dtype=torch.complex128, device=dev)
    half = P[2] // 2
    for z in range(0, half, 32):
        m = min(32, half - z)
        c = torch.arange(z * P[1] * Hx, (z + m) * P[1] * Hx, device=dev, dtype=torch.int64)
        o = _philox(c & 0xFFFFFFFF, c >> 32, torch.zeros_like(c), torch.zeros_like(c), key)
        H[z:z + m] = _normal_pair(o[0], o[1]).reshape(m, P[1], Hx)
        H[half + z:half + z + m] = _normal_pair(o[2], o[3]).reshape(m, P[1], Hx)
    H *= A
    del A
    t = torch.fft.ifft(H, dim=0, norm="forward")[:Np[2]]
    del H
    t = torch.fft.ifft(t, dim=1, norm="forward")[:, :Np[1]]
    return torch.fft.irfft(t, n=P[0], dim=2, norm="forward")[:, :, :Np[0]]


def _dct_exact(Np, xRange, corr, key):
    """One tile of the reference's active generator (DCT-III of the octant), shape (Np2, Np1, Np0)."""
    dev = _device()
    K = [n // 2 for n in Np]
    o = torch.arange(K[0] * K[1] * K[2], device=dev, dtype=torch.int64)
    zero = torch.zeros_like(o)
    w = _philox(o & 0xFFFFFFFF, o >> 32, zero, zero + 1, key)
    phi = ((w[0] << 20) | (w[1] >> 12)).double() * 2.0 ** -52 + 2.0 ** -53
    s = torch.cos(2.0 * PI_REF * phi).reshape(K[2], K[1], K[0])
    for d in range(3):
        dk = 1.0 / (xRange[d] / (Np[d] - 1)) / (Np[d] - 1)
        i = torch.arange(K[d], device=dev, dtype=torch.float64)
        e = torch.sqrt(corr[d] * torch.exp(-PI_REF * (i * dk / corr[d]) ** 2))
        s = s * e.reshape([-1 if a == 2 - d else 1 for a in range(3)])
    for d in range(3):
        i = torch.arange(K[d], device=dev, dtype=torch.int64)
        n = torch.arange(Np[d], device=dev, dtype=torch.int64)
        m = (i[:, None] * (2 * n[None, :] + 1)) % (4 * Np[d])
        C = 2.0 * torch.cos(math.pi * m.double() / (2.0 * Np[d]))
        C[0] = 1.0
        s = torch.movedim(torch.movedim(s, 2 - d, -1) @ C, -1, 2 - d)
    return s.contiguous()


def _pou(Np, No, pos, T):
    """Square root of an axis' partition-of-unity weight (SRC_F/main_ScaRL.f90:1216-1301)."""
    w = torch.ones(Np, dtype=torch.float64, device=_device())
    if No >= 2:
        p = (1.0 + torch.cos(PI_REF * torch.arange(No, device=w.device, dtype=torch.float64) / (No - 1))) / 2.0
        if pos > 0:
            w[:No] *= p.flip(0)
        if pos < T - 1:
            w[Np - No:] *= p
    return torch.sqrt(w)


def _weighted(tile, Np, No, pos, T):
    for d in range(3):
        tile = tile * _pou(Np[d], No[d], pos[d], T[d]).reshape([-1 if a == 2 - d else 1 for a in range(3)])
    return tile


def _marginal(f, margi, avg, std):
    if margi == 1:
        return f * std + avg
    v = math.log(1.0 + (std / avg) ** 2)
    return torch.exp(f * math.sqrt(v) + (math.log(avg) - v / 2.0))


def _positions(T):
    return [(r % T[0], (r // T[0]) % T[1], r // (T[0] * T[1])) for r in range(T[0] * T[1] * T[2])]


def _sample_exact(case, seed):
    Np, L, No = _layout(case)
    T, h = _v(case, "t"), case["step"]
    corr = [c * h for c in _v(case, "c")]
    key = seed % 1000000007 + 1
    out = torch.zeros(L[::-1], dtype=torch.float64, device=_device())
    P = None if case["gen"] == "dct" else _pads(case["policy"], case["mod"], case["nu"], corr, [h] * 3, Np)
    for r, pos in enumerate(_positions(T)):
        if P is None:
            t = _dct_exact(Np, [(n - 1) * h for n in Np], corr, key + r)
        else:
            t = _padded_exact(P, Np, [h] * 3, corr, case["mod"], case["nu"], key + r)
        a = [(Np[d] - No[d]) * pos[d] for d in range(3)]
        out[a[2]:a[2] + Np[2], a[1]:a[1] + Np[1], a[0]:a[0] + Np[0]] += _weighted(t, Np, No, pos, T)
        del t
    return _marginal(out, case["margi"], case["avg"], case["std"])


def _steps_exact(case, seed):
    n, o, T = _v(case, "n"), _v(case, "o"), _v(case, "t")
    L = [n[d] * T[d] - (T[d] - 1) * o[d] for d in range(3)]
    tiles = []
    whole = torch.zeros(L[::-1], dtype=torch.float64, device=_device())
    where = []
    for r, pos in enumerate(_positions(T)):
        t = _dct_exact(n, [v - 1.0 for v in n], _v(case, "c"), seed + r)
        a = [(n[d] - o[d]) * pos[d] for d in range(3)]
        at = (slice(a[2], a[2] + n[2]), slice(a[1], a[1] + n[1]), slice(a[0], a[0] + n[0]))
        whole[at] += _weighted(t, n, o, pos, T)
        where.append(at)
    for at in where:  # every tile holds the sum of all tiles over its points
        tiles.append(whole[at])
    return _marginal(torch.stack(tiles), 1, 1.0, 0.5)


def _lag_sums(f, dim, lags, window=None, mu=0.0, scale=1.0, circular=False):
    """Sums over lines of sum_i t_i t_{i+m}, m < lags, t = (f - mu) scale window, by FFT in slabs."""
    f = torch.movedim(f, dim, -1)
    n = f.shape[-1]
    M = n if circular else n + lags
    acc = 0.0
    for a in f.split(max(1, (1 << 25) // (f.shape[1] * n)), 0):
        t = (a.double() - mu) * scale
        if window is not None:
            t = t * window
        acc = acc + torch.fft.rfft(t, n=M, dim=-1).abs().square().sum(dim=(0, 1))
    return torch.fft.irfft(acc, n=M)[:lags]


def _stat_exact(case, seed):
    f = _field(case, seed)
    L = _v(case, "n")
    n = f.numel()
    s = sum(float(a.double().sum()) for a in f)
    s2 = sum(float(a.double().square().sum()) for a in f)
    avg = s / n
    std = math.sqrt(s2 / n - avg * avg)
    r = float(np.float32(0.1))
    sk, cl = [], []
    for d in range(3):
        ratio = torch.arange(L[d], device=f.device, dtype=torch.float64) / (L[d] - 1)
        w = torch.ones_like(ratio)
        w = torch.where(ratio < r, 0.5 * (1 + torch.cos(2 * PI_REF / r * (ratio - r / 2))), w)
        w = torch.where(ratio > r, 0.5 * (1 + torch.cos(2 * PI_REF / r * (ratio - 1 + r / 2))), w)
        c = _lag_sums(f, 2 - d, L[d] // 2, w, avg, 1.0 / std, True) / n
        sk.append(c)
    sk = torch.cat(sk)
    return {"avg": np.array([avg]), "std": np.array([std]), "Sk": sk.cpu().numpy(), "corrL": None}


def _cov_exact(case, seed):
    f = _field(case, seed)
    L, H = _v(case, "n"), case["lag"] + 1
    n = f.numel()
    mean = sum(float(a.double().sum()) for a in f) / n
    cov = []
    for d in range(3):
        pairs = (L[d] - torch.arange(H, device=f.device, dtype=torch.float64)) * (n // L[d])
        cov.append(_lag_sums(f, 2 - d, H, None, mean) / pairs)
    cov = torch.stack(cov).cpu().numpy()
    return {"mean": mean, "var": float(cov[0, 0]), "cov": cov}


def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":
        return _sample_exact(case, seed)
    if kind == "tile":
        n = _v(case, "n")
        P = _pads(case["policy"], case["mod"], 0.5, [case["corr"]] * 3, [1.0] * 3, n)
        return _padded_exact(P, n, [1.0] * 3, [case["corr"]] * 3, case["mod"], 0.5, seed).contiguous()
    if kind == "steps":
        return _steps_exact(case, seed)
    if kind == "ensemble":
        Np, cl = _members(case)
        return torch.cat([_padded_exact(_pads("smooth", case["mod"], 0.5, c, [1.0] * 3, n), n, [1.0] * 3, c,
                                        case["mod"], 0.5, seed * 4096 + i).reshape(-1)
                          for i, (n, c) in enumerate(zip(Np.tolist(), cl.tolist()))])
    return _stat_exact(case, seed) if kind == "stat" else _cov_exact(case, seed)
