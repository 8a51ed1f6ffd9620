"""The filtered scans (csrc/scan.cu: integer tables of four columns, exact sums for the
windows near the best) against the oracle, bit for bit, where the filter could lose a
window or a tie: motif widths around the segments of four, the last and the first window,
repeated windows (ties), scores close together, thresholds inside, below and above the
scores, palindromes (equal strands), columns that are not one base, sequences of one
32-position word, of more than the registers hold, and of more motifs than a CTA's tables."""
import numpy as np
import pytest

from oracle import search_oracle as SO

pytestmark = pytest.mark.gpu


def _check(pkg, S, pwms, thresh, fwd=True):
    lens = np.array([p.shape[1] for p in pwms], np.int32)
    with pkg.CDL(pkg.CDLSetup(M=2, filter_size=2)) as c:
        c.load_data(S)
        pos, score, comp = pkg.overlapping_scan(c, pwms, thresh)
        rp, rs, rc = SO.overlapping_scan(S, pwms, lens, thresh)
        np.testing.assert_array_equal(pos.T, rp)
        np.testing.assert_array_equal(score.T, rs)
        np.testing.assert_array_equal(comp.T, rc)
        if fwd:
            pad = np.zeros((len(pwms), 4, int(lens.max())), np.float32)
            for k, p in enumerate(pwms):
                pad[k, :, : lens[k]] = p
            np.testing.assert_array_equal(pkg.scan_w_gpu(c, pwms, thresh).T,
                                          SO.scan_w_gpu_positions(pad, S, lens, thresh))


@pytest.mark.parametrize("N,L,K,lo,hi,scale", [(40, 32, 5, 1, 9, 1.0), (20, 33, 6, 3, 6, 1.0),
                                              (12, 257, 9, 15, 18, 1.0), (9, 700, 40, 29, 33, 1.0),
                                              (33, 100, 12, 7, 17, 1e-5), (33, 100, 12, 7, 17, 100.0),
                                              (3, 1500, 3, 4, 9, 1.0)])
def test_random_scores_bit_exact(pkg, built_lib, N, L, K, lo, hi, scale):
    rng = np.random.default_rng(N + L + K)
    S = pkg.synth.onehot(rng.integers(0, 4, (N, L)).astype(np.uint8))
    pwms = [(scale * np.log2(rng.dirichlet(np.ones(4), size=int(rng.integers(lo, hi))).T / 0.25 + 1e-2)).astype(np.float32)
            for _ in range(K)]
    top = np.array([p.max(axis=0).sum() for p in pwms], np.float32)
    for f in (0.0, 0.3, 0.6, 2.0, -1.0):
        _check(pkg, S, pwms, (f * top).astype(np.float32), fwd=f >= 0)


def test_ties_near_ties_and_odd_columns(pkg, built_lib):
    rng = np.random.default_rng(5)
    N, L, w = 24, 90, 12
    bases = rng.integers(0, 4, (N, L)).astype(np.uint8)
    word = rng.integers(0, 4, w).astype(np.uint8)
    for n in range(N):                       # the same window at several places, both strands
        for p in rng.permutation(L // w)[: 1 + n % 4]:
            bases[n, p * w:(p + 1) * w] = word if n % 2 else (3 - word)[::-1]
    bases[0, :w] = word
    bases[1, L - w:] = word
    S = pkg.synth.onehot(bases)
    pwm = np.full((4, w), -1.0, np.float32)
    pwm[word, np.arange(w)] = 1.0
    near = pwm.copy()
    near[word[0], 0] = np.float32(1.0 + 2.0 ** -20)      # decided far below a table's step
    pal = np.tile(np.array([[1, -1, -1, 1]], np.float32).T, (1, w))
    flat = np.zeros((4, 7), np.float32)
    pwms = [pwm, near, pal, flat, -pwm]
    for th in (0.0, 5.0, 11.9999, 12.0, -3.0, -np.inf, np.inf, np.nan):
        _check(pkg, S, pwms, np.full(len(pwms), th, np.float32), fwd=th >= 0)
    S = S.reshape(N, L, 4).copy()
    S[2, 10] = 0                              # a column with no base
    S[3, 20] = [1, 0, 1, 0]                   # and one with two
    S[4] = 0
    _check(pkg, S.reshape(N, 4 * L), pwms, np.full(len(pwms), 1.0, np.float32))
