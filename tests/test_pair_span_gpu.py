"""The span limit of the pair matrices (the last pass holds a matrix in 48 KB of float64):
the widest filter size that fits is taken, one more is refused before anything runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_widest_filters(pkg, built_lib):
    N, L, M = 40, 30, 3
    rng = np.random.default_rng(3)
    S = pkg.synth.onehot(rng.integers(0, 4, (N, L)).astype(np.uint8))
    with pkg.CDL(pkg.CDLSetup(M=M, filter_size=5)) as c, pkg.ActivationRecord(N, L, M, T=2) as ar:
        c.load_data(S)
        X = np.zeros((N, M, c.Lg), np.float32)
        for t in (1, 2):
            X[:, :, c.gamma:c.gamma + 4 * L:4] = np.where(rng.random((N, M, L)) < 0.2, 1 + rng.random((N, M, L)), 0)
            c.init_state(X0=X)
            pkg.record_training_result(c, 0.5, ar, t, 5)
        over = pkg.get_spatial_info(ar)[0]
        want = pkg.get_pair_pfms(ar, c, over, 0, 5)[2]
        with pytest.raises(pkg.CDLGBError, match="769.*1536") as e:
            pkg.get_pair_pfms(ar, c, over, 0, 769)
        assert e.value.status == -1
        got = pkg.get_pair_pfms(ar, c, over, 0, 768)[2]
    assert len(want) > 0 and all(np.array_equal(a, b) for a, b in zip(want, got))
