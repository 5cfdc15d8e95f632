"""Workloads whose speed this framework is judged by.

A user solves the vibrational problem of a triatomic molecule: a deck and a surface go in, the
lowest levels come out (`Context.solve`). The cases span the two coordinate families (Radau,
Jacobi), the three precision forms, few and many levels, J = 0 and single k blocks of J > 0, and
final matrices of order 120 to 12202; beside them stand the fit (`Context.solve_batch`), the whole
job with its second variational step through files (`Context.run_deck`, `rotlev3b_pair`), and the
batched eigensolver on device blocks (`dvr3d_b200_diag_batched`).

Every surface is seeded: the Morse + bend family of `dvr3d_b200.configs` with its parameters moved
a little, as the trial surfaces of a fit are. `exact` restates a J = 0 or single-block solve in
numpy / torch FP64 with quadratures of its own (Golub-Welsch).
"""
from __future__ import annotations

import ctypes
import math
import random
import tempfile
from pathlib import Path

import numpy as np
import torch

import dvr3d_b200
from dvr3d_b200 import _abi, configs

PRECISION = {"fp64": dvr3d_b200.DVR3D_PREC_FP64, "mixed": dvr3d_b200.DVR3D_PREC_MIXED_DAVIDSON,
             "split": dvr3d_b200.DVR3D_PREC_SPLIT_BF16}


def listed() -> list[dict]:
    return [
        # a quick look at a surface: the smallest useful grid, where latency counts
        dict(name="radau_10_15_fp64", kind="radau", npnt=10, nalf=15, emax2=0.0, max3d=120, neval=20, precision="fp64"),
        # the reference's water example sizes, default precision form
        dict(name="radau_21_40_fp64", kind="radau", npnt=21, nalf=40, emax2=40000.0, max3d=924, neval=200,
             precision="fp64"),
        # a production water-like run (final basis about 4000), default form
        dict(name="radau_30_64_fp64", kind="radau", npnt=30, nalf=64, emax2=62000.0, max3d=3984, neval=300,
             precision="fp64"),
        # the same by the iterative form for many levels
        dict(name="radau_30_64_mixed", kind="radau", npnt=30, nalf=64, emax2=62000.0, max3d=3984, neval=300,
             precision="mixed"),
        # odd sizes, few levels, split-BF16 form
        dict(name="radau_27_51_split", kind="radau", npnt=27, nalf=51, emax2=0.0, max3d=2499, neval=24,
             precision="split"),
        # the benchmark workload (H3+-like, 40 x 40 x 80), default form: the largest call
        dict(name="jacobi_40_80_fp64", kind="jacobi", npnt1=40, npnt2=40, nalf=80, emax1=50000.0, emax2=40000.0,
             max3d=12202, neval=500, precision="fp64"),
        # the benchmark workload as the benchmark runs it
        dict(name="jacobi_40_80_mixed", kind="jacobi", npnt1=40, npnt2=40, nalf=80, emax1=50000.0, emax2=40000.0,
             max3d=12202, neval=500, precision="mixed"),
        # the same matrix, only the band origins that a spectroscopist first looks at
        dict(name="jacobi_40_80_low24", kind="jacobi", npnt1=40, npnt2=40, nalf=80, emax1=50000.0, emax2=40000.0,
             max3d=12202, neval=24, precision="mixed"),
        # one k block of a J = 2 run on an H/C/N surface, odd sizes, basis by count (`choose`)
        dict(name="hcn_j2_k1_mixed", kind="hcn", npnt1=43, npnt2=27, nalf=71, emax1=60000.0, emax2=0.0, max3d=7001,
             neval=401, k=1, precision="mixed"),
        # trial surfaces of a fit, solved as one batch
        dict(name="fit_batch_12", kind="batch", problems=12, sizes=2024, neval=100, precision="mixed"),
        # J = 2, both parities: first step with its wavefunction file, then ROTLEV3B
        dict(name="rovib_j2_job", kind="rovib", jrot=2, npnt=21, nalf=40, max3d=924, nvib=150, neval=150),
        # 1D / 2D DVR blocks of uneven order, all eigenpairs, on device memory
        dict(name="diag_blocks_57", kind="diag", blocks=57, nmin=61, nmax=463, sizes=7),
    ]


def _logint(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    kind = rng.choices(("radau", "jacobi", "hcn", "batch", "rovib", "diag"), (8, 6, 3, 2, 2, 3))[0]
    if kind == "diag":
        nmax = _logint(rng, 30, 700)
        return dict(kind=kind, blocks=_logint(rng, 5, 150), nmin=max(2, nmax // rng.randint(2, 8)), nmax=nmax,
                    sizes=rng.randrange(1 << 16))
    if kind == "batch":
        return dict(kind=kind, problems=rng.randint(3, 12), sizes=rng.randrange(1 << 16), neval=100,
                    precision=rng.choice(("mixed", "fp64")))
    if kind == "rovib":
        npnt, nalf = rng.randint(10, 21), rng.randint(14, 40)
        max3d = min(_logint(rng, 200, 1000), npnt * npnt * nalf // 8)
        return dict(kind=kind, jrot=rng.choice((1, 2)), npnt=npnt, nalf=nalf, max3d=max3d,
                    nvib=max(10, max3d // 8), neval=max(10, max3d // 8))
    precision = rng.choices(("fp64", "mixed", "split"), (5, 6, 1))[0]
    if kind == "radau":
        npnt, nalf = rng.randint(9, 32), rng.randint(13, 72)
        states = npnt * (npnt + 1) // 2 * nalf
        case = dict(kind=kind, npnt=npnt, nalf=nalf, emax2=0.0, max3d=min(_logint(rng, 100, 4500), states // 4))
    else:
        npnt1, npnt2, nalf = rng.randint(14, 43), rng.randint(12, 30), rng.randint(17, 81)
        top = min(12000, npnt1 * npnt2 * nalf // 12)
        case = dict(kind=kind, npnt1=npnt1, npnt2=npnt2, nalf=nalf, emax1=45000.0, emax2=0.0,
                    max3d=_logint(rng, min(500, top), top))
        if kind == "hcn":
            case["k"] = rng.randint(0, 2)
            case["emax1"] = 60000.0
    most = min(24 if precision == "split" else 500, max(8, case["max3d"] // 8))
    return dict(case, neval=_logint(rng, 8, most), precision=precision)


# ------------------------------------------------------------------ decks and surfaces
def _moved(seed: int, pes: np.ndarray) -> np.ndarray:
    """A trial surface near `pes`: well depths and ranges by up to 0.3 %, bend and couplings by up
    to 5 %; the minimum stays put."""
    g = np.random.default_rng(seed)
    out = pes.copy()
    out[[0, 3]] *= 1.0 + 0.003 * g.uniform(-1, 1)
    out[[1, 4]] *= 1.0 + 0.003 * g.uniform(-1, 1)
    out[6] *= 1.0 + 0.05 * g.uniform(-1, 1)
    out[8] *= 1.0 + 0.05 * g.uniform(-1, 1)
    out[9:11] *= 1.0 + 0.05 * g.uniform(-1, 1, 2)
    return out


def _hcn(c: dict) -> configs.Workload:
    """One k block of the J = 2 Jacobi H/C/N workload of `configs.config5` at other sizes."""
    ur1, ur2 = configs.reduced_masses(configs.HCN_MASSES, 1)
    m1, m2 = (2.18, 0.30, 0.0095), (3.19, 0.20, 0.0150)
    deck = configs.deck_text(title="Jacobi HCN-like J=2", npnt2=c["npnt2"], jrot=2, neval=c["neval"], nalf=c["nalf"],
                             max2d=1500, max3d=c["max3d"], idia=1, kmin=1, npnt1=c["npnt1"], ipar=0,
                             masses=configs.HCN_MASSES, emax1=c["emax1"], emax2=c["emax2"], morse1=m1, morse2=m2,
                             flags={"ZCUT": c["emax2"] > 0, "ZTHETA": False, "ZR2R1": False, "ZEMBED": False,
                                    "ZROT": True, "ZLIN": True})
    pes = configs.pes_row(m1[1], configs.morse_beta(m1[2], ur1, m1[1]), m1[0],
                          m2[1], configs.morse_beta(m2[2], ur2, m2[1]), m2[0], kb=0.05, c0=1.0)
    return configs.Workload("hcn", deck, pes, c["neval"])


def _workload(c: dict) -> configs.Workload:
    if c["kind"] == "hcn":
        return _hcn(c)
    if c["kind"] == "jacobi":
        w = configs.jacobi_h3p_like(c["npnt1"], c["npnt2"], c["nalf"], c["emax1"], c["emax2"], c["neval"],
                                    max3d=40000 if c["emax2"] > 0 else c["max3d"])
        if not c["emax2"] > 0:
            w.deck = w.deck.replace("ZCUT=.TRUE.", "ZCUT=.FALSE.")
        return w
    return configs.radau_water_like(c["npnt"], c["nalf"], c["emax2"], c["neval"], zcut=c["emax2"] > 0,
                                    max3d=20000 if c["emax2"] > 0 else c["max3d"])


def _fit(c: dict) -> list[configs.Workload]:
    """Problems with the sizes of `configs.config3`; `sizes` fixes the sizes, not the surfaces."""
    return configs.config3(seed=c["sizes"], nprob=c["problems"])


def _rovib(c: dict) -> tuple[configs.Workload, str]:
    """First step (KMIN = 2, ZROT, ZTRAN) and second step decks of a J > 0 run of both parities."""
    w = configs.radau_water_like(c["npnt"], c["nalf"], 0.0, c["nvib"], zcut=False, max3d=c["max3d"])
    lines = w.deck.splitlines()
    card = list(lines[2])
    card[5:10] = f"{c['jrot']:5d}"
    card[35:40] = f"{2:5d}"
    lines[2] = "".join(card)
    w.deck = "\n".join(lines).replace("ZPMIN=.TRUE.", "ZPMIN=.TRUE., ZROT=.TRUE., ZTRAN=.TRUE., ZLIN=.TRUE.") + "\n"
    card2 = "".join(f"{v:5d}" for v in (c["nvib"], c["neval"], 2, 0, c["neval"], 0))
    return w, " &PRT zdcore=.true. /\n" + card2 + "\n ROTLEV3B both parities\n" + f"{4500.0:20.6f}\n"


def _block_sizes(c: dict) -> list[int]:
    return [int(n) for n in np.random.default_rng(c["sizes"]).integers(c["nmin"], c["nmax"] + 1, c["blocks"])]


def _dvr_blocks(c: dict, seed: int) -> list[torch.Tensor]:
    """One-dimensional sinc-DVR Hamiltonians (kinetic energy + Morse well + ripple), each of its
    own order, spacing and well."""
    g = np.random.default_rng(seed)
    out = []
    for n in _block_sizes(c):
        h, de, a, x0 = 12.0 / (n + 1), g.uniform(4, 8), g.uniform(0.5, 0.8), g.uniform(1.5, 2.5)
        x = h * torch.arange(1, n + 1, dtype=torch.float64, device="cuda")
        i = torch.arange(n, device="cuda")
        d = (i[:, None] - i[None, :]).to(torch.float64)
        sign = 1.0 - 2.0 * ((i[:, None] + i[None, :]) % 2).to(torch.float64)
        t = sign / torch.where(d == 0, 1.0, d) ** 2
        t.fill_diagonal_(math.pi ** 2 / 6)
        v = de * (1 - torch.exp(-a * (x - x0))) ** 2 + 0.3 * torch.cos(g.uniform(1, 3) * x + g.uniform(0, 6))
        out.append(t / h ** 2 + torch.diag(v))
    return out


# ------------------------------------------------------------------ one pass
def prepare(case: dict, seed: int) -> dict:
    ctx = dvr3d_b200.Context(0)
    s = {"case": case, "ctx": ctx}
    if case["kind"] == "diag":
        # the library works on the stream that the program fills its blocks on
        s["stream"] = torch.cuda.Stream()
        ctx.set_stream(s["stream"].cuda_stream)
        blocks = _dvr_blocks(case, seed)
        n = [b.shape[0] for b in blocks]
        s["flat"] = torch.cat([b.reshape(-1) for b in blocks])
        s["vec"] = torch.empty_like(s["flat"])
        s["val"] = torch.empty(sum(n), dtype=torch.float64, device="cuda")
        nb = len(n)
        s["n"] = (ctypes.c_int * nb)(*n)
        s["off"] = (ctypes.c_longlong * nb)(*np.concatenate([[0], np.cumsum(np.square(n))[:-1]]).tolist())
        s["woff"] = (ctypes.c_longlong * nb)(*np.concatenate([[0], np.cumsum(n)[:-1]]).tolist())
        torch.cuda.synchronize()
    elif case["kind"] == "batch":
        ws = _fit(case)
        s["decks"] = [dvr3d_b200.parse_deck(w.deck) for w in ws]
        s["pes"] = np.stack([_moved(seed * 1009 + i, w.pes) for i, w in enumerate(ws)])
    elif case["kind"] == "rovib":
        w, s["rot"] = _rovib(case)
        s["deck"], s["pes"], s["dir"] = w.deck, _moved(seed, w.pes), tempfile.TemporaryDirectory()
    else:
        w = _workload(case)
        s["deck"], s["pes"] = dvr3d_b200.parse_deck(w.deck), _moved(seed, w.pes)
    return s


def run(s: dict):
    case, ctx = s["case"], s["ctx"]
    if case["kind"] == "diag":
        with torch.cuda.stream(s["stream"]):
            s["vec"].copy_(s["flat"])
            rc = _abi.load_library().dvr3d_b200_diag_batched(
                ctx._h, len(s["n"]), s["n"], s["off"], s["woff"], ctypes.c_void_p(s["vec"].data_ptr()),
                ctypes.c_void_p(s["val"].data_ptr()), 1)
            if rc != 0:
                raise dvr3d_b200.DVR3DError(rc, "diag_batched")
            # probability densities on the DVR points (an eigenvector's sign is free)
            return {"levels": s["val"], "density": s["vec"].square()}
    if case["kind"] == "batch":
        rs = ctx.solve_batch(s["decks"], s["pes"], precision=PRECISION[case["precision"]])
        return [{"levels": r.eval, "selected": r.iv2, "order": r.nham3} for r in rs]
    ctx.set_pes(s["pes"])
    if case["kind"] == "rovib":
        wave = str(Path(s["dir"].name) / "fort.26")
        ctx.run_deck(s["deck"], wave_path=wave)
        even, odd, _ = ctx.rotlev3b_pair(s["rot"], wave)
        return {"e": even, "f": odd}
    r = ctx.solve(s["deck"], case.get("k"), precision=PRECISION[case["precision"]])
    return {"levels": r.eval, "selected": r.iv2, "order": r.nham3}


def _solve_flops(n3: float, p: float, neval: float, precision: str) -> float:
    """Assembly of the contracted matrix (lower triangle), then a tridiagonalisation (default form)
    or a Cholesky factorisation and 4 solves per level, or 20 products per level for few levels."""
    f = n3 * n3 * p
    if precision == "fp64":
        return f + 4.0 / 3.0 * n3 ** 3
    if neval <= 32:
        return f + 40.0 * n3 * n3 * neval
    return f + n3 ** 3 / 3.0 + 8.0 * n3 * n3 * neval


def work(case: dict) -> dict:
    k = case["kind"]
    if k == "diag":
        n = np.array(_block_sizes(case), dtype=np.float64)
        return {"bytes": 8.0 * float((2 * n * n + n).sum()), "flops": float((16.0 / 3.0 * n ** 3).sum())}
    if k == "batch":
        f = b = 0.0
        for w in _fit(case):
            d = dvr3d_b200.parse_deck(w.deck)
            n = d.npnt2 * (d.npnt2 + 1) / 2
            f += d.nalf * 4.0 / 3.0 * n ** 3 + _solve_flops(d.max3d, n, case["neval"], case["precision"])
            b += 8.0 * (13 + case["neval"])
        return {"bytes": b, "flops": f}
    if k in ("radau", "rovib"):
        n = case["npnt"] * (case["npnt"] + 1) / 2
        one = case["nalf"] * 4.0 / 3.0 * n ** 3
        if k == "radau":
            return {"bytes": 8.0 * (13 + case["neval"]),
                    "flops": one + _solve_flops(case["max3d"], n, case["neval"], case["precision"])}
        blocks = case["jrot"] + 2
        wave = 8.0 * case["npnt"] ** 2 * case["nalf"] * case["nvib"] * blocks / 2
        both = (case["nvib"] * (case["jrot"] + 1.0)) ** 3 + (case["nvib"] * float(case["jrot"])) ** 3
        return {"bytes": 2 * wave, "flops": blocks * (one + _solve_flops(case["max3d"], n, case["nvib"], "fp64"))
                + 4.0 / 3.0 * both}
    n2 = min(case["npnt1"] * case["npnt2"], case["max3d"] * 3.0 / case["nalf"])
    return {"bytes": 8.0 * (13 + case["neval"]),
            "flops": case["nalf"] * 4.0 / 3.0 * n2 ** 3
            + _solve_flops(case["max3d"], case["npnt1"] * case["npnt2"], case["neval"], case["precision"])}


# ------------------------------------------------------------------ the same in plain FP64
def _eigh(a: torch.Tensor):
    return torch.linalg.eigh(a)


def _morse_radial(n: int, re: float, de: float, we: float, mu: float):
    """DVR points and kinetic matrix of n Morse-oscillator functions: Gauss-Laguerre points and the
    transform from the Jacobi matrix, the analytic kinetic energy in the basis between."""
    beta, a = we * math.sqrt(0.5 * mu / de), 4.0 * de / we
    iu = int(a + 0.5)
    i = np.arange(n, dtype=np.float64)
    off = -np.sqrt(i[1:] * (i[1:] + iu))
    y, u = np.linalg.eigh(np.diag(2 * i + iu + 1) + np.diag(off, 1) + np.diag(off, -1))
    fke = beta * beta / (8.0 * mu)
    h = np.diag(fke * (2 * i * (i + 1 + iu) + iu + 1))
    m = i[:-2] + 1
    band = -fke * np.sqrt((iu + m + 1) * (iu + m) * (m + 1) * m)
    h += np.diag(band, 2) + np.diag(band, -2)
    return re + np.log(a / y) / beta, u.T @ h @ u


def _angular(n: int, k: int):
    """Gauss points of the weight (1 - x^2)^k and the matrix of l(l+1), l = k..k+n-1."""
    i = np.arange(1, n, dtype=np.float64)
    off = np.sqrt(i * (i + 2 * k) / ((2 * i + 2 * k - 1) * (2 * i + 2 * k + 1)))
    x, u = np.linalg.eigh(np.diag(off, 1) + np.diag(off, -1))
    l = np.arange(k, k + n, dtype=np.float64)
    return x, u.T @ np.diag(l * (l + 1)) @ u


def _surface(q: np.ndarray, r1, r2, x):
    m1, m2 = 1 - np.exp(-q[1] * (r1 - q[2])), 1 - np.exp(-q[4] * (r2 - q[5]))
    return (q[0] * m1 ** 2 + q[3] * m2 ** 2 + q[6] * (x - q[7]) ** 2 + q[8] * (r1 - q[2]) * (r2 - q[5])
            + q[9] * x + q[10] * (3 * x ** 2 - 1) / 2 + q[11] * (5 * x ** 2 - 3) * x / 2
            + q[12] * (35 * x ** 4 - 30 * x ** 2 + 3) / 8)


def _kept(vals: list, emax: float, most: int) -> list[int]:
    """States kept per block: those below `emax`, or the `most` lowest of all (emax = 0)."""
    if emax <= 0:
        every = np.sort(np.concatenate(vals))
        last = every[min(most, len(every)) - 1]
        return [int(np.sum(v <= last)) for v in vals]
    return [int(np.sum(v < emax / configs.AUTOCM)) for v in vals]


def _contracted(vecs: list, vals: list, keep: list[int], w: np.ndarray, t: np.ndarray, neval: int):
    """Lowest levels of (V' W V) o T + diag(e) over the kept states of every angle."""
    g = np.repeat(np.arange(len(keep)), keep)
    sw = torch.tensor(np.sqrt(w), device="cuda")[:, None]
    v = torch.cat([vecs[b][:, :m] for b, m in enumerate(keep) if m], 1) * sw
    h = (v.T @ v) * torch.tensor(t, device="cuda")[g][:, g]
    h.diagonal().add_(torch.tensor(np.concatenate([vals[b][:m] for b, m in enumerate(keep)]), device="cuda"))
    e = torch.linalg.eigvalsh(h).cpu().numpy()[:neval]
    return {"levels": e, "selected": np.array(keep, dtype=np.int32), "order": len(g)}


def _exact_radau(c: dict, deck, q: np.ndarray, neval: int):
    mu = configs.reduced_masses(configs.H2O_MASSES, -2)[0]
    r, t = _morse_radial(deck.npnt2, deck.re1, deck.diss1, deck.we1, mu)
    x, lmat = _angular(deck.nalf, 0)
    n = len(r)
    a, b = np.array([(i, j) for j in range(n) for i in range(j + 1)]).T
    pick = np.zeros((n * n, len(a)))
    pick[a * n + b, np.arange(len(a))] += np.sqrt(0.5)
    pick[b * n + a, np.arange(len(a))] += np.sqrt(0.5)
    pick[:, a == b] *= np.sqrt(0.5)
    kin = pick.T @ (np.kron(t, np.eye(n)) + np.kron(np.eye(n), t)) @ pick
    pot = np.stack([_surface(q, r[a], r[b], xi) for xi in x])
    h = torch.tensor(kin, device="cuda")[None] + torch.diag_embed(torch.tensor(pot, device="cuda"))
    e, v = _eigh(h)
    vals = list(e.cpu().numpy())
    keep = _kept(vals, deck.emax2 if deck.zcut else 0.0, deck.max3d)
    return _contracted(list(v), vals, keep, 0.5 / mu * (1 / r[a] ** 2 + 1 / r[b] ** 2), lmat, neval)


def _exact_jacobi(c: dict, deck, q: np.ndarray, neval: int):
    hcn = c["kind"] == "hcn"
    mu1, mu2 = configs.reduced_masses(configs.HCN_MASSES if hcn else configs.H3P_MASSES, 1)
    r1, t1 = _morse_radial(deck.npnt1, deck.re1, deck.diss1, deck.we1, mu1)
    r2, t2 = _morse_radial(deck.npnt2, deck.re2, deck.diss2, deck.we2, mu2)
    k = c.get("k", 0)
    x, lmat = _angular(deck.nalf, k)
    # first coordinate contracted first: r1 for H/C/N (z along r1), r2 for the H3+-like deck
    ra, rb, ta, tb = (r1, r2, t1, t2) if hcn else (r2, r1, t2, t1)
    vals, vecs = [], []
    extra = 0.5 * (2 * 3 - 2 * k * k) / (ra ** 2 * mu1) if hcn else 0.0
    for xi in x:
        pot = _surface(q, ra[:, None], rb, xi) if hcn else _surface(q, rb, ra[:, None], xi)
        e1, u1 = np.linalg.eigh(ta + np.stack([np.diag(p + extra) for p in pot.T]))
        low = [int(np.sum(e < deck.emax1 / configs.AUTOCM)) for e in e1]
        u = np.zeros((len(ra), len(rb), sum(low)))
        bi = np.repeat(np.arange(len(rb)), low)
        u[:, bi, np.arange(sum(low))] = np.concatenate([u1[j][:, :m].T for j, m in enumerate(low)]).T
        flat = np.concatenate([u1[j][:, :m] for j, m in enumerate(low)], 1)
        h2 = torch.tensor((flat.T @ flat) * tb[bi][:, bi] + np.diag(np.concatenate([e1[j][:m] for j, m in enumerate(low)])),
                          device="cuda")
        e2, v2 = _eigh(h2)
        vals.append(e2.cpu().numpy())
        vecs.append(torch.tensor(u.reshape(-1, sum(low)), device="cuda") @ v2[:, :600])
    keep = _kept(vals, deck.emax2 if deck.zcut else 0.0, deck.max3d)
    w = 0.5 / (ra[:, None] ** 2 * (mu1 if hcn else mu2)) + 0.5 / (rb ** 2 * (mu2 if hcn else mu1))
    return _contracted(vecs, vals, keep, w.reshape(-1), lmat, neval)


def exact(case: dict, seed: int):
    k = case["kind"]
    if k == "rovib":  # files in between: no short restatement
        return None
    if k == "diag":
        pairs = [torch.linalg.eigh(b) for b in _dvr_blocks(case, seed)]
        return {"levels": torch.cat([e for e, _ in pairs]),
                # column-major blocks: eigenvectors one after another
                "density": torch.cat([v.T.reshape(-1) for _, v in pairs]).square()}
    if k == "batch":
        out = []
        for i, w in enumerate(_fit(case)):
            deck = dvr3d_b200.parse_deck(w.deck)
            out.append(_exact_radau(case, deck, _moved(seed * 1009 + i, w.pes), case["neval"]) if i < 3 else None)
        return out
    w = _workload(case)
    deck, q = dvr3d_b200.parse_deck(w.deck), _moved(seed, w.pes)
    return (_exact_radau if k == "radau" else _exact_jacobi)(case, deck, q, case["neval"])
