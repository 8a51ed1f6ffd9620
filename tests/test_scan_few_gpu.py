"""Scans of few sequences (csrc/scan.cu: the motifs cut over more CTAs than their tables ask
for) against the oracle, bit for bit: every value is an integer or an ordered float32 sum."""
import numpy as np
import pytest

from oracle import search_oracle as SO

pytestmark = pytest.mark.gpu


# one sequence; one CTA's 16 and one more; as many CTAs as leave two and one motif per cut
@pytest.mark.parametrize("N,L,K", [(1, 40, 1), (1, 130, 35), (16, 33, 5), (17, 290, 3), (160, 50, 60), (2000, 24, 7)])
def test_scans(pkg, built_lib, N, L, K):
    rng = np.random.default_rng(N + L + K)
    S = pkg.synth.onehot(rng.integers(0, 4, (N, L)).astype(np.uint8))
    pwms = [np.log2(rng.dirichlet(np.ones(4), size=int(rng.integers(3, 21))).T / 0.25 + 1e-2).astype(np.float32)
            for _ in range(K)]
    lens = np.array([p.shape[1] for p in pwms], np.int32)
    thresh = np.array([0.4 * p.max(axis=0).sum() for p in pwms], np.float32)
    pad = np.zeros((K, 4, int(lens.max())), np.float32)
    for k, p in enumerate(pwms):
        pad[k, :, : lens[k]] = p
    with pkg.CDL(pkg.CDLSetup(M=2, filter_size=2)) as c:
        c.load_data(S)
        for got, want in zip(pkg.overlapping_scan(c, pwms, thresh), SO.overlapping_scan(S, pwms, lens, thresh)):
            np.testing.assert_array_equal(got.T, want)
        np.testing.assert_array_equal(pkg.scan_w_gpu(c, pwms, thresh).T, SO.scan_w_gpu_positions(pad, S, lens, thresh))
