"""cdlgb_autotune with room for exactly the transform candidates: the convolution X-step is
one more where it is in use, and does not turn the call away."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _autotune(c, room):
    from cdlmotif_gb300._lib import lib, ptr
    ms = np.zeros(16, np.float64)
    kind, cs, mc = (np.zeros(16, np.int32) for _ in range(3))
    n, chosen = C.c_int32(), C.c_int32()
    st = lib().cdlgb_autotune(c._h, room, ptr(ms, C.c_double), ptr(kind, C.c_int32), ptr(cs, C.c_int32),
                              ptr(mc, C.c_int32), C.byref(n), C.byref(chosen))
    return st, n.value, chosen.value


def test_room_for_the_transforms_only(pkg, built_lib, monkeypatch):
    N, L, M, W = 40, 100, 10, 4                # Lg = 432, where both kinds exist
    S = pkg.synth.onehot(np.random.default_rng(1).integers(0, 4, (N, L)).astype(np.uint8))
    setup = pkg.CDLSetup(M=M, filter_size=W, lambda_=0.1, rho=1.0, sigma=100.0)
    count = {}
    for form in ("0", "1"):
        monkeypatch.setenv("CDLGB_XCONV", form)
        with pkg.init_cdl(setup, S, seed=2) as c:
            st, count[form], _ = _autotune(c, 16)
            assert st == 0
    assert count["1"] == count["0"] + 1
    with pkg.init_cdl(setup, S, seed=2) as c:
        st, n, chosen = _autotune(c, count["0"])
        assert (st, n) == (0, count["0"]) and 0 <= chosen < n
        assert np.isfinite(pkg.run_outer(c, 2)).all()
    with pkg.init_cdl(setup, S, seed=2) as c:
        assert _autotune(c, count["0"] - 1)[0] != 0
