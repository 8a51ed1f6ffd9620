"""What the convolution X-step keeps between its steps (t = X + y2 and u = X + y3, U and y1')
is what it would form again from the arrays it leaves behind: a code update of several X-steps
and as many of one X-step give the same bits, in both launch forms.  And the scalars that the
last block of a pass adds up, at sizes around a block's share, call after call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("X", "y2", "y3", "y1", "Y1", "DX")


@pytest.mark.parametrize("shape", [(3, 13, 2, 3), (5, 50, 10, 4), (2, 137, 25, 9), (700, 11, 4, 4), (2, 114, 34, 12)])
def test_one_update_of_three_steps_is_three_of_one(pkg, built_lib, shape):
    N, L, M, W = shape
    S = pkg.synth.onehot(np.random.default_rng(L).integers(0, 4, size=(N, L)).astype(np.uint8))
    got = []
    for split in ([3], [1, 1, 1], [1, 2]):
        with pkg.init_cdl(pkg.CDLSetup(M=M, filter_size=W, lambda_=0.1, rho=1.0), S, seed=8) as c:
            for n in split:
                pkg.code_update(c, n)
            got.append([c.get(f) for f in FIELDS])
    for other in got[1:]:
        for f, a, b in zip(FIELDS, got[0], other):
            assert np.array_equal(a, b), f


# values per pass: less than a block's share of 4096 (objective) and 8192 (threshold), just
# that, one block more, and more than all blocks' first round
@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (1, 1024, 1, 4), (4, 1024, 1, 4), (5, 1023, 2, 4), (700, 1500, 2, 3)])
def test_scalars_added_by_the_last_block(pkg, built_lib, shape):
    N, L, M, W = shape
    S = pkg.synth.onehot(np.random.default_rng(L).integers(0, 4, size=(N, L)).astype(np.uint8))
    with pkg.init_cdl(pkg.CDLSetup(M=M, filter_size=W, lambda_=0.25), S, seed=8) as c:
        X, DX = c.X.astype(np.float64), c.DX.astype(np.float64)
        fit = DX[:, 4 * W:4 * W + 4 * L] - S.reshape(N, -1)
        want = 0.5 * (fit ** 2).sum() + 0.25 * np.abs(X).sum()
        p = X[X > 0]
        # sums in float64, or in pairs of float32 exact to 2^-48: both far below this
        for _ in range(3):
            assert pkg.objective(c) == pytest.approx(want, rel=1e-11)
            if len(p) > 1:
                assert pkg.code_threshold(c) == pytest.approx(p.std(ddof=1), rel=1e-10)
