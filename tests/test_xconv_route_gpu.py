"""Which X-step the automatic choice takes: the convolution (csrc/xconv.cu) up to 64 taps and
Lg = 4128 unless a multi-iteration kernel's filter slots are well filled, past that only where
it is the cheaper one.  The two forms round differently, so the codes' bits show the route."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _codes(pkg, monkeypatch, N, L, M, W, form):
    S = pkg.synth.onehot(np.random.default_rng(L).integers(0, 4, (N, L)).astype(np.uint8))
    setup = pkg.CDLSetup(M=M, filter_size=W, lambda_=0.1, rho=1.0, sigma=100.0)
    if form is None:
        monkeypatch.delenv("CDLGB_XCONV", raising=False)
    else:
        monkeypatch.setenv("CDLGB_XCONV", form)
    with pkg.init_cdl(setup, S, seed=6) as c:
        pkg.code_update(c, 3)
        return c.X


# (L, M, W, taken): odd M on the lengths of the one-X-step register FFTs; powers of two and other
# smooth lengths of cuFFT, with up to 64 taps and with more; lengths that cuFFT or the
# in-kernel transforms are slow at; the multi-iteration kernel's lengths with few filters of
# many taps and of few, and with as many filters as it has slots for
@pytest.mark.parametrize("L,M,W,taken", [(200, 17, 16, True), (100, 33, 12, True), (92, 5, 16, True), (992, 9, 16, True),
                                         (1000, 9, 16, True), (448, 9, 32, False), (2000, 32, 24, False),
                                         (836, 9, 32, False), (1360, 9, 24, False), (4032, 2, 32, False),
                                         (224, 17, 4, True), (120, 25, 2, True), (200, 63, 16, True), (480, 32, 16, True),
                                         (500, 32, 16, True), (1000, 25, 16, True), (50, 10, 4, True), (137, 25, 9, True),
                                         (701, 9, 24, True), (8, 1, 1, True), (200, 8, 16, True), (200, 10, 16, True),
                                         (100, 10, 12, True), (100, 10, 4, True), (200, 10, 4, True), (108, 4, 8, True),
                                         (200, 12, 16, False), (100, 16, 12, False), (200, 64, 16, False)])
def test_route(pkg, built_lib, monkeypatch, L, M, W, taken):
    default, fft = (_codes(pkg, monkeypatch, 3, L, M, W, form) for form in (None, "0"))
    assert np.array_equal(default, fft) != taken
