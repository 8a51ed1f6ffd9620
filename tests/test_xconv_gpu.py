"""The convolution X-step (csrc/xconv.cu: short convolutions of the codes with the filters'
taps, one row per sequence through a padded transform) against the FP64 oracle, at the
sizes where its layout can go wrong, and against the FFT form of the same context
(CDLGB_XCONV=0), whose route it replaces in the automatic choice."""
import numpy as np
import pytest

from oracle import cdl_oracle as O

from conftest import rel

pytestmark = pytest.mark.gpu

TOL_X = 1e-4          # the parity tolerance after a fixed iteration count
TOL_OBJ = 1e-5
FIELDS = ("X", "y2", "y3", "y1", "Y1", "DX")

# (N, L, M, W): rows modulo the 16 of a thread (Lg % 16 = 0, 4, 8, 12), pairs of filters
# per CTA and CTAs per sequence (M = 1, odd, one more than a CTA's), blocks of 16 taps
# (4 taps to 80), transform lengths 2^a 3^b 5^c, N of one and more sequences than are
# resident at once (the two forms of the launch), and the reference's defaults
SHAPES = [(1, 8, 1, 1), (3, 13, 2, 3), (3, 9, 3, 2), (5, 50, 10, 4), (4, 61, 11, 4), (2, 137, 25, 9),
          (2, 30, 33, 5), (2, 114, 34, 12), (2, 500, 6, 16), (1, 1000, 4, 16), (2, 70, 9, 20), (700, 11, 4, 4),
          (1300, 15, 5, 3), (3, 200, 10, 4)]


def _case(pkg, N, L, M, W):
    synth = pkg.synth
    bases, _, _ = synth.plant_dataset(31, N, L, [min(6, L), min(8, L)], [0.4, 0.4])
    Lg = 4 * L + 8 * W
    return synth.onehot(bases), synth.init_X0(9, N, M, Lg), synth.init_D0_unit_norm(9, M, Lg, 4 * W)


@pytest.mark.parametrize("shape", SHAPES)
def test_convolution_xstep_against_oracle(pkg, built_lib, shape, monkeypatch):
    """Two code updates around a dictionary step (15 and 4 X-steps) from one initial state:
    every field the X-step writes within the parity tolerance of FP64, the objective, the
    residual record and sum |X| behind them, and the FFT form's other rounding (the route)."""
    N, L, M, W = shape
    S, X0, D0 = _case(pkg, N, L, M, W)
    setup = pkg.CDLSetup(M=M, filter_size=W, lambda_=0.1, rho=1.0, sigma=100.0, track_residuals=True)
    ref = O.init_cdl(S, M, W, 1.0, 100.0, 0.1, X0=X0, D0=D0)
    got = {}
    for form in ("1", "0"):
        monkeypatch.setenv("CDLGB_XCONV", form)
        with pkg.init_cdl(setup, S, X0=X0, D0=D0) as c:
            pkg.code_update(c, 15)
            got[form] = {f: c.get(f) for f in FIELDS}
            got[form]["obj"] = pkg.objective(c)
            got[form]["res"] = c.residuals()[:5]
            pkg.update_best(c)
            pkg.dict_update(c, 1)
            pkg.code_update(c, 4)
            got[form]["X2"], got[form]["best"] = c.X, c.X_best
    O.code_update(ref, 15)
    for f in FIELDS:
        want = getattr(ref, f)
        e = rel(got["1"][f], want) if np.linalg.norm(want) else np.abs(got["1"][f]).max()
        assert e < TOL_X, (f, e, rel(got["0"][f], want))
    assert got["1"]["obj"] == pytest.approx(O.objective(ref), rel=TOL_OBJ)
    np.testing.assert_allclose(got["1"]["res"], got["0"]["res"], rtol=1e-3, atol=1e-6)
    O.update_best(ref)
    O.dict_update(ref, 1)
    O.code_update(ref, 4)
    assert rel(got["1"]["X2"], ref.X) < TOL_X and rel(got["1"]["best"], ref.X_best) < TOL_X
    assert not np.array_equal(got["1"]["X"], got["0"]["X"])


def test_sequences_do_not_depend_on_each_other(pkg, built_lib):
    """A sequence's codes are the same bits alone and among others, in both launch forms."""
    N, L, M, W = 900, 13, 4, 4
    S, X0, D0 = _case(pkg, N, L, M, W)
    setup = pkg.CDLSetup(M=M, filter_size=W, lambda_=0.1, rho=1.0, sigma=100.0)
    out = {}
    for n in (N, 450, 7):
        with pkg.init_cdl(setup, S[:n], X0=X0[:n], D0=D0) as c:
            pkg.code_update(c, 15)
            out[n] = {f: c.get(f)[:7] for f in FIELDS}
    for n in (450, 7):
        for f in FIELDS:
            np.testing.assert_array_equal(out[N][f], out[n][f], err_msg=f"{f} {n}")


def test_autotune_keeps_a_convolution_training(pkg, built_lib):
    """The autotuner counts the convolution X-step among its candidates and leaves the state
    as it was, whichever it keeps (M = 10 at the reference's default W = 4)."""
    S, X0, D0 = _case(pkg, 40, 100, 10, 4)
    setup = pkg.CDLSetup(M=10, filter_size=4, lambda_=0.1, rho=1.0, sigma=100.0)
    with pkg.init_cdl(setup, S, X0=X0, D0=D0) as c:
        info = c.autotune()
        best = info["candidates"][info["chosen"]]
        assert best["ms_per_xstep"] == min(x["ms_per_xstep"] for x in info["candidates"])
        assert any(x["filters_per_cta"] == 10 for x in info["candidates"])
        objs = pkg.run_outer(c, 2)
        X = c.X
    ref = O.init_cdl(S, 10, 4, 1.0, 100.0, 0.1, X0=X0, D0=D0)
    np.testing.assert_allclose(objs, O.run_outer(ref, 2), rtol=TOL_OBJ)
    assert rel(X, ref.X) < TOL_X
