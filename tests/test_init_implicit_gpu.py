"""The initial duals y2 = y3 = 0 and the initial dictionary spectra, which the first steps
take as known instead of reading: a training whose initial arrays were written first (by a
reader, or by the tuner) runs on the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("X", "y2", "y3", "y1", "Y1", "DX", "G1", "G3", "d", "g1", "g3", "g2", "Td", "D_best")

# (N, L, M, W, fft_mode): the fused kernels over clusters and per warp, the one-step kernel
# of other lengths, the convolution form's two launches, cuFFT transforms, more filters than
# the pipelined D-step holds, an odd M
SHAPES = [(40, 50, 10, 4, 0), (12, 200, 64, 16, 0), (9, 137, 25, 9, 0), (5, 40, 70, 3, 0), (30, 100, 16, 12, 2),
          (6, 100, 15, 12, 2), (6, 61, 5, 4, 1), (700, 11, 4, 4, 0)]


def _training(pkg, shape, before):
    N, L, M, W, mode = shape
    S = pkg.synth.onehot(np.random.default_rng(3).integers(0, 4, size=(N, L)).astype(np.uint8))
    setup = pkg.CDLSetup(M=M, filter_size=W, lambda_=0.1, rho=1.0, sigma=100.0, track_residuals=True)
    with pkg.init_cdl(setup, S, seed=5, fft_mode=mode) as c:
        out = []
        for again in range(2):                   # the second time over a used state
            before(c)
            pkg.code_update(c, 3)
            pkg.update_best(c)
            pkg.dict_update(c, 2)
            pkg.code_update(c, 2)
            out.append([c.get(f) for f in FIELDS] + [c.residuals()])
            c.init_state(seed=6)
        return out


@pytest.mark.parametrize("shape", SHAPES)
def test_arrays_written_first_change_nothing(pkg, built_lib, shape):
    def read(c):
        for f in ("y2", "y3", "d", "g1", "g3"):
            a = c.get(f)
            assert f == "d" or not a.any()

    plain, written = _training(pkg, shape, lambda c: None), _training(pkg, shape, read)
    for p, w in zip(plain, written):
        for f, a, b in zip(FIELDS + ("residuals",), p, w):
            assert np.array_equal(a, b), f


def test_dictionary_step_before_any_code_update(pkg, built_lib):
    """y3 is read by the time-domain dictionary step only, and zero then."""
    S = pkg.synth.onehot(np.random.default_rng(4).integers(0, 4, size=(7, 40)).astype(np.uint8))
    got = []
    for mode in (0, 1):
        with pkg.init_cdl(pkg.CDLSetup(M=4, filter_size=5), S, seed=5, fft_mode=mode) as c:
            pkg.dict_update(c, 1)
            got.append((c.G1, c.get("g1"), c.get("y2"), c.get("y3")))
    # both forms of one linear step on values of order one, transforms of 200 rows
    np.testing.assert_allclose(got[0][0], got[1][0], atol=2e-6)
    np.testing.assert_allclose(got[0][1], got[1][1], atol=2e-5)
    assert not got[0][2].any() and not got[1][3].any()
