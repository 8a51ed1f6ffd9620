"""Activation records of few sequences (csrc/record.cu) against the oracle, counts equal: rows cut
over warps, activation lists filled to their last entry, sequences cut into the chunks that
leave fewest SMs idle."""
import numpy as np
import pytest

from oracle import search_oracle as SO

pytestmark = pytest.mark.gpu


# a row's last word of 256 positions and one past it; lists that 16 full words fill, and that
# take 32 words at a time; 30 tiles over the chunks of 70 sequences
@pytest.mark.parametrize("N,L,M,sizes,density", [(2, 256, 3, (4, 4), 1.0), (3, 257, 2, (5, 5), 0.6), (2, 520, 2, (3, 9), 1.0),
                                                 (3, 1030, 2, (8, 8), 0.02), (70, 40, 3, (3, 3, 4, 5, 3, 6), 0.1)])
def test_records(pkg, built_lib, N, L, M, sizes, density):
    rng = np.random.default_rng(N * L)
    S = pkg.synth.onehot(rng.integers(0, 4, (N, L)).astype(np.uint8))
    codes = np.where(rng.random((len(sizes), N, M, L)) < density, 2.0, 0.1).astype(np.float32)
    codes[:, -1, :, -1] = 2.0
    with pkg.ActivationRecord(N, L, M, T=len(sizes)) as ar:
        for t, fs in enumerate(sizes):
            with pkg.CDL(pkg.CDLSetup(M=M, filter_size=fs)) as c:
                c.load_data(S)
                X = np.zeros((N, M, c.Lg), np.float32)
                X[:, :, c.gamma:c.gamma + 4 * L:4] = codes[t]
                c.init_state(X0=X)
                assert pkg.record_training_result(c, 1.0, ar, t + 1, fs) == M
        u, tn, fl = ar.info()
        on = np.stack([codes[tn[k] - 1][:, u[k] - 1, :] > 1.0 for k in range(len(u))], axis=1)
        for got, want in zip(pkg.get_spatial_info(ar), SO.activation_topology(on, tn, fl, L)):
            np.testing.assert_array_equal(got, want)
