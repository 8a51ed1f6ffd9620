"""Both scans through the C interface with motifs in an array wider than any of them (the
interface allows zero padding past lens[k]): the results of the array that just fits, and
the oracle's.  What the scan kernels keep per motif goes by the motifs' own widths."""
import ctypes as C

import numpy as np
import pytest

from oracle import search_oracle as SO

pytestmark = pytest.mark.gpu


def _scans(pkg, c, pwms, lens, thresh, maxlen):
    from cdlmotif_gb300._lib import lib, ptr
    K = len(pwms)
    arr = np.zeros((maxlen, 4, K), np.float32)
    for k, p in enumerate(pwms):
        arr[:lens[k], :, k] = p.T
    pos, score, comp = (np.zeros((c.N, K), t) for t in (np.int32, np.float32, np.uint8))
    fwd = np.zeros((c.N, K), np.int32)
    args = (ptr(arr, C.c_float), ptr(lens, C.c_int32), ptr(thresh, C.c_float), K, maxlen)
    assert lib().cdlgb_scan_both(c._h, *args, ptr(pos, C.c_int32), ptr(score, C.c_float), ptr(comp, C.c_uint8)) == 0
    assert lib().cdlgb_scan_fwd(c._h, *args, ptr(fwd, C.c_int32)) == 0
    return pos, score, comp, fwd


# (K, widest motif, columns of the array): a little and far wider, many narrow motifs in one
# CTA's tables, one motif, the widest array that the filtered scans take and one past it
@pytest.mark.parametrize("K,width,maxlen", [(24, 8, 24), (32, 10, 32), (104, 4, 32), (24, 8, 32), (1, 1, 32), (7, 13, 14),
                                            (6, 9, 40)])
def test_padded_motifs(pkg, built_lib, K, width, maxlen):
    rng = np.random.default_rng(K + maxlen)
    S = pkg.synth.onehot(rng.integers(0, 4, (40, 90)).astype(np.uint8))
    lens = rng.integers(max(1, width - 3), width + 1, K).astype(np.int32)
    lens[K // 2] = width
    pwms = [np.log2(rng.dirichlet(np.ones(4), size=int(w)).T / 0.25 + 1e-2).astype(np.float32) for w in lens]
    thresh = np.array([0.4 * p.max(axis=0).sum() for p in pwms], np.float32)
    with pkg.CDL(pkg.CDLSetup(M=2, filter_size=2)) as c:
        c.load_data(S)
        wide = _scans(pkg, c, pwms, lens, thresh, maxlen)
        fits = _scans(pkg, c, pwms, lens, thresh, width)
    for a, b in zip(wide, fits):
        np.testing.assert_array_equal(a, b)
    for a, b in zip(wide, SO.overlapping_scan(S, pwms, lens, thresh)):
        np.testing.assert_array_equal(a.T, b)
    assert wide[0].any() and wide[3].any()
