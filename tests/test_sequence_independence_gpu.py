"""A sequence's state does not depend on the others of its dataset: the same bits, whatever
the number of sequences makes of the kernels' grids.  The initial reconstruction (ranges of a
sequence per CTA, csrc/init.cu), and the convolution X-step (csrc/xconv.cu) in the form for
datasets that are resident at once, in the one that takes a launch per part, and in that one
over more sequences than one chunk of its scratch holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("X", "y2", "y3", "y1", "Y1", "DX")


def _setup(pkg, M, W):
    return pkg.CDLSetup(M=M, filter_size=W, lambda_=0.1, rho=1.0, sigma=100.0)


def _data(pkg, N, L):
    return pkg.synth.onehot(np.random.default_rng(N + L).integers(0, 4, (N, L)).astype(np.uint8))


# (N, L, M, W): sequences cut into ranges, by more when they are few
@pytest.mark.parametrize("shape", [(400, 500, 32, 16), (500, 300, 33, 5), (240, 1000, 7, 13)])
def test_initial_reconstruction(pkg, built_lib, shape):
    N, L, M, W = shape
    S = _data(pkg, N, L)
    with pkg.init_cdl(_setup(pkg, M, W), S, seed=3) as c:
        X, D, DX, G2 = c.X, c.G1, c.DX, c.G2
    for n in (1, 7, 160):
        with pkg.init_cdl(_setup(pkg, M, W), S[:n], seed=3) as c:         # the same draws
            np.testing.assert_array_equal(c.X, X[:n])
            np.testing.assert_array_equal(c.DX, DX[:n])
        with pkg.init_cdl(_setup(pkg, M, W), S[-n:], X0=X[-n:], D0=D) as c:
            np.testing.assert_array_equal(c.DX, DX[-n:])
            np.testing.assert_array_equal(c.G2, G2[-n:])


# (N, L, M, W): one to sixteen pairs of filters, which the form with a launch per part splits
# over CTAs; N is past what is resident at once
@pytest.mark.parametrize("shape", [(1500, 100, 10, 4), (1500, 100, 11, 4), (1500, 101, 16, 4), (1500, 60, 25, 9),
                                   (1500, 101, 32, 5), (900, 250, 13, 3), (1100, 61, 31, 2)])
def test_convolution_xstep_forms(pkg, built_lib, shape):
    N, L, M, W = shape
    S = _data(pkg, N, L)
    Lg = 4 * L + 8 * W
    X0, D0 = pkg.synth.init_X0(9, N, M, Lg), pkg.synth.init_D0_unit_norm(9, M, Lg, 4 * W)
    out = {}
    for n in (N, 300, 7):
        with pkg.init_cdl(_setup(pkg, M, W), S[:n], X0=X0[:n], D0=D0) as c:
            pkg.code_update(c, 15)
            out[n] = {f: c.get(f)[:7] for f in FIELDS}
    for n in (300, 7):
        for f in FIELDS:
            np.testing.assert_array_equal(out[N][f], out[n][f], err_msg=f"{f} {n}")


def test_convolution_xstep_in_chunks(pkg, built_lib):
    """About 556 sequences of this size to a chunk: the sequences of the second one read and
    write their own rows of the state, and the scratch's first rows again."""
    N, L, M, W = 600, 1500, 64, 4
    S = _data(pkg, N, L)
    pick = np.array([0, 1, 554, 556, 560, N - 1])
    with pkg.init_cdl(_setup(pkg, M, W), S, seed=5) as c:
        X0, D0 = c.X[pick], c.G1
        pkg.code_update(c, 4)
        many = {f: c.get(f)[pick] for f in FIELDS}
    with pkg.init_cdl(_setup(pkg, M, W), S[pick], X0=X0, D0=D0) as c:
        pkg.code_update(c, 4)
        for f in FIELDS:
            np.testing.assert_array_equal(many[f], c.get(f), err_msg=f)
