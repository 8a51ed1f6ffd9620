"""The initial objective's sum |X| (csrc/init.cu) over a given X0 is a float64 sum, whatever
the sizes of the codes.  With filters of zeros the fit is exactly the number of bases, so
what is left of the objective is that sum: within 4 units in the last place, 2^-51, of the
sum in extended precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _initial(pkg, X0, S, M, W, lam):
    Lg = X0.shape[2]
    D0 = np.zeros((M, Lg), np.float32)
    setup = pkg.CDLSetup(M=M, filter_size=W, lambda_=lam, rho=1.0, sigma=100.0)
    with pkg.init_cdl(setup, S, X0=X0, D0=D0) as c:
        return c.obj_best


# ones and 2^-25 + 2^-48, of which a float32 pair drops the last bit at every addition; codes
# whose float32 sum would overflow
@pytest.mark.parametrize("sizes", [(1.0, 2.0 ** -25 * (1 + 2.0 ** -23)), (3e38, 1e30)])
@pytest.mark.parametrize("shape", [(2, 200, 64, 4), (7, 61, 33, 9), (1, 500, 128, 16)])
def test_sum_of_given_codes(pkg, built_lib, shape, sizes):
    N, L, M, W = shape
    rng = np.random.default_rng(L)
    S = pkg.synth.onehot(rng.integers(0, 4, (N, L)).astype(np.uint8))
    X0 = np.zeros((N, M, 4 * L + 8 * W), np.float32)
    X0[:, :, ::4] = rng.choice(np.array(sizes, np.float32), X0[:, :, ::4].shape)
    X0[:, :, ::4] *= rng.choice(np.array([-1, 1], np.float32), X0[:, :, ::4].shape)
    want = np.longdouble(N * L) / 2 + np.abs(X0).astype(np.longdouble).sum()
    got = _initial(pkg, X0, S, M, W, 1.0)
    assert abs(np.longdouble(got) - want) <= 2.0 ** -51 * want
