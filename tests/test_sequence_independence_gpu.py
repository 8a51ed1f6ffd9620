"""A sequence's state does not depend on the others of its dataset: the same bits, whatever
the number of sequences makes of the kernels' grids: the initial reconstruction (ranges of a
sequence per CTA, csrc/init.cu)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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
