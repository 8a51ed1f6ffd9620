"""The objective behind the convolution X-step: sum |X| comes from its last pass, which adds
groups of four neighbouring codes in float32, as a pass over X does, and the groups in
float64.  From the state that is read back, with the same groups, the objective is then
known to rounding in float64 (n terms: n 2^-53 at most; the fit's float32 pairs, 2^-46)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (N, L, M, W): one long sequence of few filters (most codes per thread), odd M, both forms of
# the launch, several CTAs per sequence
@pytest.mark.parametrize("shape", [(1, 3900, 2, 4), (2, 1500, 3, 8), (5, 50, 10, 4), (40, 137, 25, 9), (900, 50, 10, 4)])
def test_sum_of_codes(pkg, built_lib, shape):
    N, L, M, W = shape
    lam = 0.1
    S = pkg.synth.onehot(np.random.default_rng(L).integers(0, 4, (N, L)).astype(np.uint8))
    setup = pkg.CDLSetup(M=M, filter_size=W, lambda_=lam, rho=1.0, sigma=100.0)
    with pkg.init_cdl(setup, S, seed=4) as c:
        pkg.code_update(c, 5)
        obj, X, DX = pkg.objective(c), np.abs(c.X), c.DX
    g = X.reshape(-1, 4)
    four = (g[:, 0] + g[:, 1]) + (g[:, 2] + g[:, 3])
    assert four.dtype == np.float32
    fit = DX[:, 4 * W:4 * W + 4 * L].astype(np.float64) - S.reshape(N, -1)
    want = 0.5 * (fit ** 2).sum() + float(np.float32(lam)) * four.astype(np.float64).sum()
    assert obj == pytest.approx(want, rel=2.0 ** -44)
