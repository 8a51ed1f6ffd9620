"""The initial state (csrc/init.cu): the drawn filters and codes against their definition on
the host, and the reconstruction DX of drawn and of given codes, which is convolved from the
filters' taps, against float64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (N, L, M, W): the smallest; rows a = Lg / 4 modulo the 8 of a thread, W modulo the 4 and 8
# taps of a step; fewer filters than parts and more than a pass; a sequence cut into ranges,
# also into one longer than a CTA; more taps than a pass; more ranges than CTAs
SHAPES = [(1, 1, 1, 1), (2, 8, 3, 2), (3, 13, 2, 3), (5, 50, 10, 4), (2, 61, 65, 5), (2, 137, 25, 9), (1, 200, 64, 16),
          (3, 500, 33, 16), (2, 1000, 7, 13), (1, 2100, 2, 8), (1, 5003, 3, 4), (2, 300, 2, 260), (1500, 9, 3, 7)]
U = 2.0 ** -24


def _mix(x):
    with np.errstate(over="ignore"):
        x = np.asarray(x, np.uint64) + np.uint64(0x9E3779B97F4A7C15)
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return x ^ (x >> np.uint64(31))


def _key(seed, mul):
    return np.uint64(seed * mul & 0xFFFFFFFFFFFFFFFF)


def _drawn(seed, N, M, Lg, W):
    """The draws in float64: X per kept row, D per filter's first 4 W rows."""
    j = np.arange(N * M * Lg // 4, dtype=np.uint64)
    h = _mix(_key(seed, 0x2545F4914F6CDD1D) ^ (np.uint64(4) * j))
    # the two uniforms are float32 values: u + 0.5 is rounded above 2^23
    u1 = ((h >> np.uint64(40)).astype(np.float32) + np.float32(0.5)).astype(np.float64) / 2 ** 24
    u2 = ((h & np.uint64(0xFFFFFF)).astype(np.float32) + np.float32(0.5)).astype(np.float64) / 2 ** 24
    X = np.zeros((N, M, Lg))
    X[:, :, ::4] = (np.sqrt(-2 * np.log(u1)) * np.cos(2 * np.pi * u2)).reshape(N, M, -1)
    h = _mix(_key(seed, 0x2545F4914F6CDD1D) ^ (np.arange(M * 4 * W, dtype=np.uint64) + np.uint64(0x9E37)))
    v = [((a >> np.uint64(11)).astype(np.float64) + 0.5) / 2 ** 53 for a in (h, _mix(h))]
    D = (np.sqrt(-2 * np.log(v[0])) * np.cos(2 * np.pi * v[1])).reshape(M, 4 * W)
    out = np.zeros((M, Lg))
    out[:, :4 * W] = D / np.linalg.norm(D, axis=1, keepdims=True)
    return X, out


@pytest.mark.parametrize("given", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_initial_state(pkg, built_lib, shape, given):
    N, L, M, W = shape
    Lg = 4 * L + 8 * W
    rng = np.random.default_rng(N + L + M + W)
    S = pkg.synth.onehot(rng.integers(0, 4, size=(N, L)).astype(np.uint8))
    X0 = D0 = None
    if given:
        X0 = rng.standard_normal((N, M, Lg)).astype(np.float32)          # masked to every fourth row
        D0 = rng.standard_normal((M, Lg)).astype(np.float32)             # and to the first 4 W
    with pkg.init_cdl(pkg.CDLSetup(M=M, filter_size=W, lambda_=0.5), S, X0=X0, D0=D0, seed=77) as c:
        X, D, DX, obj = c.X, c.G1, c.DX, c.obj_best
        for f in ("y2", "y3", "Y1", "y1", "g2", "Td", "g1", "g3"):
            assert not c.get(f).any(), f
        for f in ("G3", "D_best"):
            assert np.array_equal(c.get(f), D)
        assert np.array_equal(c.G2, DX) and np.array_equal(c.X_best, X)
    if given:
        want = np.zeros_like(X0)
        want[:, :, ::4] = X0[:, :, ::4]
        assert np.array_equal(X, want)
        want = np.zeros_like(D0)
        want[:, :4 * W] = D0[:, :4 * W]
        assert np.array_equal(D, want)
    else:
        wx, wd = _drawn(77, N, M, Lg, W)
        # a float32 logarithm, root, cosine and product, a few units in the last place each
        # (of the cosine: of 1)
        assert np.abs(X - wx).max() <= 16 * U * 6.0
        assert np.abs(D - wd).max() <= 2 * U
    # a sum of M W products in float32, in any order
    X64, D64 = X.astype(np.float64), D.astype(np.float64)
    fx, fd = np.fft.rfft(X64), np.fft.rfft(D64)
    exact = np.fft.irfft((fx * fd[None]).sum(1), Lg)
    size = np.fft.irfft((np.fft.rfft(np.abs(X64)) * np.fft.rfft(np.abs(D64))[None]).sum(1), Lg)
    assert (np.abs(DX - exact) <= (M * W + 8) * U * size + 1e-12 * np.abs(size).max()).all()
    fit = DX[:, 4 * W:4 * W + 4 * L].astype(np.float64) - S.reshape(N, -1)
    # sums of |X| from the pass that draws it
    assert obj == pytest.approx(0.5 * (fit ** 2).sum() + 0.5 * np.abs(X64).sum(), rel=1e-5)
