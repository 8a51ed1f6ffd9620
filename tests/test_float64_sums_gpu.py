"""The objective's and the threshold's sums, evaluated in runs of float32 sums with their
errors (csrc/admm.cu), keep float64: against the state that is read back, summed in extended
precision.  What is left is the rounding of the last few float64 additions, the root and
the quotient: within 4 units in the last place, 2^-51 (a run that lost 2^-48 of its terms
would be past it, its loss being much the same for every run)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(200, 50, 4, 3), (200, 50, 10, 4), (60, 137, 25, 9), (20, 701, 9, 16)])
def test_objective_and_threshold(pkg, built_lib, shape):
    N, L, M, W = shape
    lam = 1e-3
    S = pkg.synth.onehot(np.random.default_rng(L + M).integers(0, 4, (N, L)).astype(np.uint8))
    setup = pkg.CDLSetup(M=M, filter_size=W, lambda_=lam, rho=1.0, sigma=100.0)
    for seed in range(4):
        with pkg.init_cdl(setup, S, seed=seed) as c:
            pkg.code_update(c, 3)
            obj, X, DX = pkg.objective(c), c.X, c.DX
            pkg.update_best(c)
            thr, best = pkg.code_threshold(c), c.X_best
        x = best[best > 0].astype(np.longdouble)
        want = np.sqrt(((x - x.sum() / len(x)) ** 2).sum() / (len(x) - 1))
        assert abs(np.longdouble(thr) - want) <= 2.0 ** -51 * want
        g = np.abs(X).reshape(-1, 4)                      # groups of four codes in float32
        absx = ((g[:, 0] + g[:, 1]) + (g[:, 2] + g[:, 3])).astype(np.longdouble).sum()
        fit = ((DX[:, 4 * W:4 * W + 4 * L].astype(np.longdouble) - S.reshape(N, -1)) ** 2).sum()
        want = fit / 2 + np.longdouble(np.float32(lam)) * absx
        assert abs(np.longdouble(obj) - want) <= 2.0 ** -51 * want
