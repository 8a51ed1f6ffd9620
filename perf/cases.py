"""What this framework is timed on: calls a user's program makes, over the sizes it is used at.

The package finds motifs in DNA: it trains convolutional dictionaries (the ADMM), turns
their codes into filter pairs and count matrices, and refines the motifs by scanning.
Four kinds of case, each through the package's public calls:

train   one outer iteration of a training from its initial draws (init_state, then
        code_update + update_best + dict_update by run_outer, then code_threshold) and
        the learned dictionary read back.  One iteration, because the recursion amplifies
        float32 rounding by a third per iteration whichever way it is evaluated.  The data
        is loaded before; the initial state is drawn inside, so that every pass runs the
        same training.  Scalars come back as plain numbers: they are float64 sums of a
        float32 state.
round   one refinement round over the data: two-strand scan, non-overlapping selection,
        extension with new count matrices, masked trim with new score thresholds.
hits    the forward scan of candidate motifs, their count matrices, and the filter that
        compares their hits with those on shuffled sequences.
pairs   the codes of two trainings recorded as activations, counted as filter pairs, and
        the frequent pairs' weighted count matrices.
"""
from __future__ import annotations

import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG_DIR = os.path.join(ROOT, "cdlmotif.jl_gb300")

# CDL_setup's own penalties, and those of the benchmark's trainings
DEFAULTS = dict(lam=0.01, rho=100.0, sigma=100.0)
BENCH = dict(lam=0.1, rho=1.0, sigma=100.0)

# float32 codes (N, M, Lg) are read back with the rest up to this many values, the
# reconstruction (N, Lg) up to this many sequences; larger trainings leave them on the
# device, where the next step reads them
CODES_READ = 2_000_000
RECON_READ = 2_000


def _pkg():
    """The package, by path (its directory's name is no Python identifier)."""
    name = "cdlmotif_gb300"
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            name, os.path.join(PKG_DIR, "__init__.py"), submodule_search_locations=[PKG_DIR])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _train(name, N, L, M, W, pen, residuals=False):
    return dict(name=name, kind="train", N=N, L=L, M=M, W=W, residuals=residuals, **pen)


def listed():
    return [
        # a handful of short sequences with the package's default filters: launches and latency
        _train("train_n200_l50_k10_w4", 200, 50, 10, 4, DEFAULTS),
        # the small benchmark training: N = 1000 sequences of 100 bases, 16 filters of 12
        _train("train_n1000_l100_k16_w12", 1000, 100, 16, 12, BENCH),
        # the package's defaults (10 filters of 4 bases) on an ordinary peak set
        _train("train_n5000_l200_k10_w4", 5000, 200, 10, 4, DEFAULTS),
        # sizes that divide nothing: odd L, M and W, with the residual record kept
        _train("train_n1500_l137_k25_w9", 1500, 137, 25, 9, BENCH, residuals=True),
        # the headline benchmark: N = 20000, L = 200, 64 filters of 16 bases
        _train("train_n20000_l200_k64_w16", 20000, 200, 64, 16, BENCH),
        # long sequences of the batched mix (L = 500, 32 filters of 16 bases)
        _train("train_n5000_l500_k32_w16", 5000, 500, 32, 16, BENCH),
        # the longest sequences that the server takes
        _train("train_n500_l1000_k32_w16", 500, 1000, 32, 16, BENCH),
        # a refinement round on the headline data with 32 motifs, and on a small set
        dict(name="round_n20000_l200_k32", kind="round", N=20000, L=200, K=32),
        dict(name="round_n1000_l100_k16", kind="round", N=1000, L=100, K=16),
        # candidate motifs against the first 10000 records of a file, which is what is read
        dict(name="hits_n10000_l200_k24", kind="hits", N=10000, L=200, K=24),
        # two trainings' activations into pairs
        dict(name="pairs_n5000_l200_k32", kind="pairs", N=5000, L=200, M=32, W=16),
        dict(name="pairs_n1000_l100_k10", kind="pairs", N=1000, L=100, M=10, W=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: 200-20000 sequences of 50-1000 bases, 4-64
    filters of 3-16 bases, 4-40 motifs, any of them odd."""
    kind = rng.choice(["train"] * 6 + ["round"] * 2 + ["hits", "pairs"])
    L = _log(rng, 50, 1000)
    if kind == "train":
        M, W = _log(rng, 4, 64), rng.randint(3, 16)
        most = 250_000_000 // ((4 * L + 8 * W) * M)      # values of the codes
        N = _log(rng, 200, max(250, min(20000, most)))
        return dict(kind=kind, N=N, L=L, M=M, W=W, residuals=rng.random() < 0.2,
                    **(DEFAULTS if rng.random() < 0.4 else BENCH))
    if kind == "pairs":
        L = min(L, 400)
        M = _log(rng, 4, 40)
        N = _log(rng, 200, min(10000, 40_000_000 // (L * M)))
        return dict(kind=kind, N=N, L=L, M=M, W=rng.randint(4, 16))
    N = _log(rng, 200, min(20000, 4_000_000 // L))
    return dict(kind=kind, N=N, L=L, K=rng.randint(4, 40))


# ---------------------------------------------------------------------------- inputs
def _bases(rng, N, L, motifs, occupancy):
    """i.i.d. bases with the motifs planted at the given occupancy on a random strand."""
    bases = rng.integers(0, 4, size=(N, L), dtype=np.uint8)
    for pfm, occ in zip(motifs, occupancy):
        w = pfm.shape[1]
        rows = np.flatnonzero(rng.random(N) < occ)
        u = rng.random((len(rows), w))
        site = np.minimum((u[:, None, :] > np.cumsum(pfm, axis=0)[None]).sum(axis=1), 3).astype(np.uint8)
        rc = rng.random(len(rows)) < 0.5
        site[rc] = 3 - site[rc][:, ::-1]
        pos = rng.integers(0, L - w + 1, size=len(rows))
        bases[rows[:, None], pos[:, None] + np.arange(w)[None]] = site
    return bases


def _onehot(bases):
    out = np.zeros(bases.shape + (4,), np.float32)
    np.put_along_axis(out, bases[..., None].astype(np.int64), 1.0, axis=2)
    return out.reshape(bases.shape[0], -1)


def _dataset(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    widths = rng.integers(8, 21, size=5)
    motifs = [rng.dirichlet(0.1 * np.ones(4), size=int(w)).T for w in widths]
    return rng, motifs, _bases(rng, case["N"], case["L"], motifs, rng.uniform(0.1, 0.4, 5))


def _pwms(rng, motifs, K):
    """The planted motifs' cores and other motifs of 8 to 16 columns, K in all."""
    pfms = [m[:, 2:-2] for m in motifs if m.shape[1] >= 12][:K]
    while len(pfms) < K:
        pfms.append(rng.dirichlet(np.ones(4), size=int(rng.integers(8, 17))).T)
    return [np.log2(((p + 0.05) / 1.2) / 0.25).astype(np.float32) for p in pfms]


def _codes(case, seed):
    """Codes of two trainings (N, M, L): heavy-tailed, a few in a hundred above their own
    threshold, with filter pairs that fire together."""
    rng = np.random.Generator(np.random.PCG64([seed, 3]))
    N, L, M, W = case["N"], case["L"], case["M"], case["W"]
    pairs = [(int(rng.integers(M)), int(rng.integers(M)), int(rng.integers(1, W))) for _ in range(12)]
    codes = []
    for t in range(2):
        z = rng.standard_normal((N, M, L), dtype=np.float32)
        codes.append(np.where(z > 0, np.exp(1.5 * rng.standard_normal((N, M, L), dtype=np.float32)), 0))
    for a, b, d in pairs:
        rows = np.flatnonzero(rng.random(N) < 0.2)
        p = rng.integers(0, L - 2 * W, size=len(rows))
        codes[0][rows, a, p] = rng.uniform(30, 60, len(rows))
        codes[1][rows, b, p + d] = rng.uniform(30, 60, len(rows))
    return [c.astype(np.float32) for c in codes]


def _active(codes):
    """Codes above the deviation of the positive ones."""
    return [c > np.float32(c[c > 0].std(ddof=1, dtype=np.float64)) for c in codes]


def _pair_threshold(case, active):
    """Pairs counted well above what chance gives at this density."""
    chance = case["N"] * case["L"] * active[0].mean() * active[1].mean()
    return int(chance + 6 * math.sqrt(chance) + 0.1 * case["N"])


def _setup(case, **kw):
    return _pkg().CDLSetup(M=case["M"], filter_size=case["W"], **kw)


def prepare(case, seed):
    pkg = _pkg()
    state = {"case": dict(case), "seed": seed}
    rng, motifs, bases = _dataset(case, seed)
    S = _onehot(bases)
    if case["kind"] == "train":
        c = pkg.CDL(_setup(case, lambda_=case["lam"], rho=case["rho"], sigma=case["sigma"],
                           track_residuals=case["residuals"]))
        c.load_data(S)
        state["cdl"] = c
    elif case["kind"] == "pairs":
        state["trainings"] = []
        trained = _codes(case, seed)
        for codes in trained:
            c = pkg.CDL(_setup(case))
            c.load_data(S)
            X = np.zeros((c.N, c.M, c.Lg), np.float32)
            X[:, :, c.gamma:c.gamma + c.L:4] = codes
            c.init_state(X0=X)
            state["trainings"].append(c)
        state["threshold"] = _pair_threshold(case, _active(trained))
    else:
        c = pkg.CDL(pkg.CDLSetup(M=2, filter_size=2))
        c.load_data(S)
        state["cdl"] = c
        state["pwms"] = _pwms(rng, motifs, case["K"])
        state["lens"] = np.array([p.shape[1] for p in state["pwms"]], np.int32)
        state["thresh"] = pkg.get_thresh(c, state["pwms"])
        if case["kind"] == "hits":
            c.make_background(k=3, seed=seed)
    return state


# ---------------------------------------------------------------------------- one pass
def run(state):
    return {"train": _run_train, "round": _run_round, "hits": _run_hits,
            "pairs": _run_pairs}[state["case"]["kind"]](state)


def _run_train(state):
    pkg, c = _pkg(), state["cdl"]
    c.init_state(seed=state["seed"])
    objs = pkg.run_outer(c, 1)
    out = {"objective": float(objs[0]), "threshold": pkg.code_threshold(c),
           "G1": c.get("G1"), "G3": c.get("G3"), "D_best": c.get("D_best")}
    if c.N <= RECON_READ:
        out["DX"] = c.get("DX")
    if c.N * c.M * c.Lg <= CODES_READ:
        out["codes"] = c.get("X_best")
    if state["case"]["residuals"]:
        out["residuals"] = c.residuals().astype(np.float32)
    return out


def _rows(a, rows, cols):
    """The first entries of a (rows, cols) array of zeros: what a pass finds differs in
    number from data to data."""
    out = np.zeros((max(rows, len(a)), cols) if cols else max(rows, len(a)), a.dtype)
    if cols:
        out[:len(a), :a.shape[1]] = a
    else:
        out[:len(a)] = a
    return out


def _matrices(pfms, count, width, dtype=np.float32):
    """Count matrices (4, w) side by side."""
    out = np.zeros((max(count, len(pfms)), 4, width), dtype)
    for k, p in enumerate(pfms):
        out[k, :, :p.shape[1]] = p
    return out


MAX_WIDTH = 64          # columns of a motif after its extension
MAX_PAIRS = 64          # filter pairs that are frequent enough


def _run_round(state):
    pkg, c, lens = _pkg(), state["cdl"], state["lens"]
    pos, score, comp = pkg.overlapping_scan(c, state["pwms"], state["thresh"])
    out = {"position": pos, "score": score, "strand": comp}
    pos, score, comp = pkg.non_overlap_scan(c, pos, score, lens, comp)
    ext = pkg.extend(c, pos, lens, 4, use_comp=comp, smoothing=False)
    trim = pkg.masked_trim(ext["pfms"], 4, ext["positions"], ext["use_comp"], c=c)
    N, K = pos.shape
    thresh = trim["thresh"] if trim["thresh"] is not None else np.zeros(0, np.float32)
    out.update(extended=_rows(ext["positions"], N, K), lens=_rows(ext["lens"], K, 0),
               pfms=_matrices(ext["pfms"], K, MAX_WIDTH), front=_rows(trim["front"], K, 0),
               back=_rows(trim["back"], K, 0), thresh=_rows(thresh, K, 0))
    return out


def _run_hits(state):
    pkg, c = _pkg(), state["cdl"]
    pos = pkg.scan_w_gpu(c, state["pwms"], state["thresh"])
    pfms = pkg.posdicts2pfms(c, pos, state["lens"])
    kept = pkg.filter_using_evalue(c, state["pwms"], state["thresh"], pos)
    return {"position": pos, "pfms": _matrices(pfms, pos.shape[1], MAX_WIDTH), "evalues": kept["evalues"],
            "hits": kept["hits"], "hits_bg": kept["hits_bg"]}


def _run_pairs(state):
    pkg, case, (c1, c2) = _pkg(), state["case"], state["trainings"]
    W = case["W"]
    with pkg.ActivationRecord(case["N"], case["L"], case["M"], T=2) as record:
        for t, c in enumerate((c1, c2)):
            pkg.record_training_result(c, pkg.code_threshold(c), record, t + 1, W)
        over, non_over, next_to = pkg.get_spatial_info(record)
        pairs, spans, pfms = pkg.get_pair_pfms(record, c1, over, state["threshold"], W)
    return {"over": over, "non_over": non_over, "next_to": next_to,
            "pairs": _rows(pairs, MAX_PAIRS, 3), "spans": _rows(spans, MAX_PAIRS, 0),
            "pfms": _matrices(pfms, MAX_PAIRS, 2 * W)}


# ---------------------------------------------------------------------------- the least work
def work(case):
    N, L = case["N"], case["L"]
    if case["kind"] == "train":
        # the data read and the training's state written once: X, y2, y3 and the
        # dictionary copies d, g1 of every sequence; 15 sparse-coding steps of a forward
        # and an inverse transform and two products per code, one dictionary step
        Lg, M = 4 * L + 8 * case["W"], case["M"]
        codes = Lg * M * N
        return {"bytes": 16.0 * L * N + 20.0 * codes + 24.0 * Lg * N,
                "flops": 15.0 * codes * (5 * math.log2(Lg) + 16) + codes * (2.5 * math.log2(Lg) + 40)}
    if case["kind"] == "pairs":
        M, W = case["M"], case["W"]
        acts = 2 * M * L * 0.035
        return {"bytes": 2.0 * 4 * N * M * L + 16.0 * N * L + 4.0 * (2 * M) ** 2 * (L + W),
                "flops": N * acts * acts / 2}
    K = case["K"]
    strands = 2 if case["kind"] == "round" else 1
    passes = 1 if case["kind"] == "round" else 2            # the data, and the background
    return {"bytes": passes * (16.0 * N * L + 9.0 * N * K),
            "flops": passes * strands * 12.0 * N * max(1, L - 11) * K}


# ---------------------------------------------------------------------------- 64 bits
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _mix(x):
    """splitmix64 on uint64 arrays."""
    with np.errstate(over="ignore"):
        x = x + np.uint64(0x9E3779B97F4A7C15)
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return x ^ (x >> np.uint64(31))


def _mix_t(x):
    """The same on int64 tensors, whose products wrap alike; shifts made logical."""
    def s64(v):
        return v - (1 << 64) if v >> 63 else v

    def shr(v, k):
        return (v >> k) & ((1 << (64 - k)) - 1)
    x = x + s64(0x9E3779B97F4A7C15)
    x = (x ^ shr(x, 30)) * s64(0xBF58476D1CE4E5B9)
    x = (x ^ shr(x, 27)) * s64(0x94D049BB133111EB)
    return x ^ shr(x, 31)


def _seeded(seed):
    return (seed * 0x2545F4914F6CDD1D) & (2 ** 64 - 1)


def _init_codes(seed, n0, n1, M, Lg, dev):
    """The library's standard-normal codes of sequences n0..n1: on every fourth row, drawn
    from the row's own index."""
    base = _seeded(seed)
    idx = torch.arange(n0 * M * Lg, n1 * M * Lg, 4, dtype=torch.int64, device=dev)
    h = _mix_t(idx ^ (base - (1 << 64) if base >> 63 else base))
    u1 = (((h >> 40) & 0xFFFFFF).float() + 0.5).double() / 16777216.0
    u2 = ((h & 0xFFFFFF).float() + 0.5).double() / 16777216.0
    X = torch.zeros((n1 - n0, M, Lg), dtype=torch.float64, device=dev)
    X[..., ::4] = (torch.sqrt(-2 * torch.log(u1)) * torch.cos(2 * math.pi * u2)).view(n1 - n0, M, Lg // 4)
    return X


def _init_filters(seed, M, flen, Lg):
    i = np.arange(M * flen, dtype=np.uint64) + np.uint64(0x9E37)
    h = _mix(np.uint64(_seeded(seed)) ^ i)
    u1 = ((h >> np.uint64(11)).astype(np.float64) + 0.5) / 2.0 ** 53
    u2 = ((_mix(h) >> np.uint64(11)).astype(np.float64) + 0.5) / 2.0 ** 53
    v = (np.sqrt(-2 * np.log(u1)) * np.cos(2 * np.pi * u2)).reshape(M, flen)
    D = np.zeros((M, Lg))
    D[:, :flen] = (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)
    return D


def exact(case, seed):
    return {"train": _exact_train, "round": _exact_round, "hits": _exact_hits,
            "pairs": _exact_pairs}[case["kind"]](case, seed)


def _exact_train(case, seed):
    """The outer iteration in float64, some sequences at a time: only the objective, the
    deviation of the positive codes and the dictionary's means join them."""
    dev = _dev()
    N, L, M, W = case["N"], case["L"], case["M"], case["W"]
    lam, rho, sigma = case["lam"], case["rho"], case["sigma"]
    L4, gamma, flen = 4 * L, 4 * W, 4 * W
    Lg = L4 + 2 * gamma
    bases = _dataset(case, seed)[2]
    D = torch.from_numpy(_init_filters(seed, M, flen, Lg)).to(dev)
    Dh = torch.fft.rfft(D)
    A = (Dh.abs() ** 2).sum(0)
    win = torch.zeros(Lg, dtype=torch.float64, device=dev)
    win[gamma:gamma + L4] = 1

    def shrink(t):
        return torch.sign(t) * (t.abs() - lam).clamp(min=0)

    def kept(t):
        o = torch.zeros_like(t)
        o[..., ::4] = t[..., ::4]
        return o

    fit0 = fit1 = abs0 = abs1 = cnt = tot = sq = 0.0
    sum_d = torch.zeros((M, Lg), dtype=torch.float64, device=dev)
    recon, codes, pos_codes = [], [], 0
    step = max(1, min(N, 40_000_000 // (M * Lg)))
    for n0 in range(0, N, step):
        n1 = min(N, n0 + step)
        S = torch.zeros((n1 - n0, Lg), dtype=torch.float64, device=dev)
        S[:, gamma:gamma + L4] = torch.from_numpy(_onehot(bases[n0:n1])).to(dev)
        X = _init_codes(seed, n0, n1, M, Lg, dev)
        DX = torch.fft.irfft((Dh * torch.fft.rfft(X)).sum(1), n=Lg)
        DX0 = DX
        fit0 += float((((DX - S) * win) ** 2).sum())
        abs0 += float(X.abs().sum())
        y2, y3 = torch.zeros_like(X), torch.zeros_like(X)
        y1, Y1 = torch.zeros_like(DX), torch.zeros_like(DX)
        for _ in range(15):
            y1 = y1 + DX - Y1
            Uh = torch.fft.rfft(Y1 - y1)
            Y2, Y3 = shrink(X + y2), kept(X + y3)
            y2, y3 = y2 + X - Y2, y3 + X - Y3
            Vh = torch.fft.rfft((Y2 - y2) + (Y3 - y3))
            P = (Dh * Vh).sum(1)
            Wh = Uh - (A * Uh + P) / (A + 2)
            X = torch.fft.irfft((Vh + Dh.conj() * Wh[:, None]) / 2, n=Lg)
            DX = torch.fft.irfft((P + A * Wh) / 2, n=Lg)
            Y1 = (S + rho * (DX + y1)) / (win + rho)
        fit1 += float((((DX - S) * win) ** 2).sum())
        abs1 += float(X.abs().sum())
        p = X[X > 0]
        cnt, tot, sq = cnt + p.numel(), tot + float(p.sum()), sq + float((p * p).sum())
        # dictionary step: d of every sequence, from G2 = DX at the start
        Yh = torch.fft.rfft(kept(X))
        H, Zh = 2 * Dh, torch.fft.rfft(DX0)
        B, Q = (Yh.abs() ** 2).sum(1), (Yh * H).sum(1)
        beta = (Zh * B + Q) / (B + 2)
        sum_d += torch.fft.irfft(H + Yh.conj() * (Zh - beta)[:, None], n=Lg).sum(0)
        recon.append(DX.cpu().numpy() if N <= RECON_READ else None)
        codes.append(X.cpu().numpy() if N * M * Lg <= CODES_READ else None)
    if not (0.5 * fit1 + lam * abs1 < 0.5 * fit0 + lam * abs0):
        return None
    v = (2 * sum_d / N - D).cpu().numpy()
    G3 = np.zeros((M, Lg))
    G3[:, :flen] = v[:, :flen].clip(0, 1)
    G1 = np.zeros((M, Lg))
    for l in range(flen):
        i = 4 * ((l + 1) // 4)
        G1[:, l] = v[:, l] - 0.25 * (v[:, i:i + 4].sum(axis=1) - 1)
    out = {"objective": 0.5 * fit1 + lam * abs1,
           "threshold": math.sqrt(max(0.0, sq - tot * tot / cnt) / (cnt - 1)),
           "G1": G1, "G3": G3, "D_best": D.cpu().numpy()}
    if N <= RECON_READ:
        out["DX"] = np.concatenate(recon)
    if N * M * Lg <= CODES_READ:
        out["codes"] = np.concatenate(codes)
    if case["residuals"]:
        out["residuals"] = None
    return out


def _scan(bases, pwms, thresh, both):
    """Best window of every sequence and motif in float64: position (1-based, 0 none),
    score and strand, each (N, K)."""
    dev = _dev()
    N, L = bases.shape
    onehot = torch.from_numpy(_onehot(bases)).to(dev).double().view(N, L, 4).transpose(1, 2)
    pos, score, comp = (np.zeros((N, len(pwms)), t) for t in (np.int64, np.float64, np.int64))
    for k, p in enumerate(pwms):
        if p.shape[1] > L:
            continue
        best = []
        for q in (p, p[::-1, ::-1].copy()):
            windows = onehot.unfold(2, q.shape[1], 1)                       # (N, 4, places, w)
            s = torch.einsum("njpk,jk->np", windows, torch.from_numpy(q.copy()).to(dev).double())
            best.append([t.cpu().numpy() for t in s.max(dim=1)])
        (sf, pf), (sc, pc) = best
        fwd = (sf >= sc) if both else np.ones(N, bool)
        s, i = np.where(fwd, sf, sc), np.where(fwd, pf, pc) + 1
        hit = s > np.float64(thresh[k])
        pos[:, k], score[:, k], comp[:, k] = np.where(hit, i, 0), np.where(hit, s, 0), hit & ~fwd
    return pos, score, comp


def _thresholds(pwms, pval=2.7e-4):
    """Score at which fewer than pval of random windows lie, in steps of 0.1."""
    out = []
    for p in pwms:
        steps = np.floor(np.asarray(p, np.float64) / 0.1).astype(np.int64)
        low = steps.min(axis=0)
        q = np.ones(1)
        for col in (steps - low).T:
            nxt = np.zeros(len(q) + int(col.max()))
            for s in col:
                nxt[s:s + len(q)] += 0.25 * q
            q = nxt
        tail = np.cumsum(q[::-1])[::-1]
        k = np.flatnonzero((tail < pval) & (q > 0))
        k = k[0] if len(k) else np.flatnonzero(q > 0)[-1]
        out.append(0.1 * (k + low.sum()))
    return np.array(out)


def _select(pos, score, comp, lens):
    """Per sequence the best motifs whose spans do not meet."""
    N, K = pos.shape
    left = np.where(pos > 0, score, 0.0)
    kept = np.zeros((N, K), bool)
    rows = np.arange(N)
    for _ in range(K):
        b = left.argmax(axis=1)
        live = left[rows, b] != 0
        s, e = pos[rows, b], pos[rows, b] + lens[b] - 1
        meets = (kept & (pos <= e[:, None]) & (s[:, None] <= pos + lens[None] - 1)).any(axis=1)
        kept[rows, b] |= live & ~meets
        left[rows, b] = 0
    return np.where(kept, pos, 0), np.where(kept, comp, 0)


def _extend(bases, pos, comp, lens):
    """Columns added to each motif while they carry information."""
    L = bases.shape[1]
    pos, lens = pos.copy(), lens.astype(np.int64).copy()
    for k in range(len(lens)):
        rows = np.flatnonzero(pos[:, k])
        start, rc, w = pos[rows, k], comp[rows, k] != 0, lens[k]
        inc = np.ones(len(rows), bool)
        grown = {False: 0, True: 0}
        going = {False: True, True: True}
        while going[False] or going[True]:
            for right in (False, True):
                if not going[right]:
                    continue
                off = grown[right] + 1
                at = np.where(right != rc, start + w - 1 + off, start - off)
                inside = (at >= 1) & (at <= L)
                use = inc & inside
                b = bases[rows[use], at[use] - 1].astype(np.int64)
                col = np.bincount(np.where(rc[use], 3 - b, b), minlength=4) + 5.0
                p = col / col.sum()
                if (p * np.log2(p / 0.25)).sum() <= 0.075:
                    going[right] = False
                else:
                    inc &= inside
                    grown[right] += 1
            if len(rows) <= math.floor(0.95 * len(rows)) or max(grown.values()) > 2 * L:
                break
        if grown[False] or grown[True]:
            pos[rows, k] = np.where(inc, np.where(rc, start - grown[True], start - grown[False]), 0)
        lens[k] = w + grown[False] + grown[True]
    return pos, lens


def _pfms(bases, pos, comp, lens, smoothing):
    out = []
    for k, w in enumerate(lens):
        rows = np.flatnonzero(pos[:, k])
        win = bases[rows[:, None], pos[rows, k][:, None] - 1 + np.arange(w)[None]].astype(np.int64)
        rc = comp[rows, k] != 0
        win[rc] = 3 - win[rc][:, ::-1]
        counts = np.stack([(win == a).sum(axis=0) for a in range(4)]).astype(np.float64)
        ps = 0.0295 * len(rows) if smoothing else 5.0
        out.append((counts + ps) / (len(rows) + 4 * ps))
    return out


def _search_inputs(case, seed):
    rng, motifs, bases = _dataset(case, seed)
    pwms = _pwms(rng, motifs, case["K"])
    return bases, pwms, np.array([p.shape[1] for p in pwms], np.int64), _thresholds(pwms).astype(np.float32)


def _exact_round(case, seed):
    bases, pwms, lens, thresh = _search_inputs(case, seed)
    pos, score, comp = _scan(bases, pwms, thresh, both=True)
    out = dict.fromkeys(("position", "strand", "extended", "lens", "front", "back", "thresh"))
    out["score"] = score
    pos, comp = _select(pos, score, comp, lens)
    pos, lens = _extend(bases, pos, comp, lens)
    keep = np.flatnonzero((pos > 0).any(axis=0) & (lens > 6))
    out["pfms"] = _matrices(_pfms(bases, pos[:, keep], comp[:, keep], lens[keep], smoothing=False),
                              case["K"], MAX_WIDTH, np.float64)
    return out


def _exact_hits(case, seed):
    bases, pwms, lens, thresh = _search_inputs(case, seed)
    pos, _, _ = _scan(bases, pwms, thresh, both=False)
    pos[pos == 1] = 0                                  # a best window at position 1 reads as none
    out = dict.fromkeys(("position", "evalues", "hits", "hits_bg"))
    with np.errstate(invalid="ignore"):                # a motif without a hit divides by nothing
        pfms = _pfms(bases, pos, np.zeros_like(pos), lens, smoothing=True)
    out["pfms"] = _matrices(pfms, case["K"], MAX_WIDTH, np.float64)
    return out


def _exact_pairs(case, seed):
    N, L, M, W = case["N"], case["L"], case["M"], case["W"]
    bases = _dataset(case, seed)[2]
    onehot = _onehot(bases).reshape(N, L, 4)
    codes = _codes(case, seed)
    on = _active(codes)
    least = _pair_threshold(case, on)
    # every filter fires in at least one sequence, so filter k is (training, m) in order
    found = {}
    for o in range(1, W + 1):
        for t in (0, 1):                               # the pair's first filter is of training t
            d = W - o                                  # and the second starts d bases after
            if d == 0:                                 # at one place the pair is not counted
                continue
            a = np.ascontiguousarray(on[t][:, :, :L - d].transpose(1, 0, 2)).reshape(M, -1)
            b = np.ascontiguousarray(on[1 - t][:, :, d:].transpose(1, 0, 2)).reshape(M, -1)
            n = torch.from_numpy(a).to(_dev()).float() @ torch.from_numpy(b).to(_dev()).float().T
            for fr, fc in np.argwhere(n.cpu().numpy() > least):
                found[(o, (1 - t) * M + int(fc), t * M + int(fr))] = (t, int(fr), int(fc), d)
    pfms = []
    for key in sorted(found):
        t, fr, fc, d = found[key]
        o = key[0]
        span = o if o >= W else 2 * W - o
        n, p = np.nonzero(on[t][:, fr, :L - d] & on[1 - t][:, fc, d:])
        n, p = n[p + span <= L], p[p + span <= L]
        avg = (codes[t][n, fr, p].astype(np.float64) + codes[1 - t][n, fc, p + d]) / 2
        msa = (avg[:, None, None] * onehot[n[:, None], p[:, None] + np.arange(span)[None]]).sum(axis=0) + 0.1
        pfms.append((msa / msa[0].sum()).T)
    out = dict.fromkeys(("over", "non_over", "next_to", "pairs", "spans"))
    out["pfms"] = _matrices(pfms, MAX_PAIRS, 2 * W, np.float64)
    return out
