"""The filter-pair topology's tiles and bit masks (csrc/record.cu) against the oracle where
they can go wrong: sequences of a word of positions, one more and several; more filters
than a tile's lanes; filters of unequal lengths (same-place pairs count) and of three
trainings; windows at the ends of a sequence.  Integer counts bit-exact, pair PFMs 1e-5."""
import numpy as np
import pytest

from oracle import search_oracle as SO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,L,M,sizes,density", [(9, 32, 3, (3, 3), 0.2), (17, 33, 5, (4, 6), 0.15),
                                                 (40, 96, 40, (5, 5), 0.05), (5, 250, 4, (16, 7, 16), 0.3),
                                                 (3, 65, 2, (1, 9), 1.0)])
def test_topology_and_pairs_against_oracle(pkg, built_lib, N, L, M, sizes, density):
    rng = np.random.default_rng(N * L)
    S = pkg.synth.onehot(rng.integers(0, 4, (N, L)).astype(np.uint8))
    T = len(sizes)
    codes = np.where(rng.random((T, N, M, L)) < density, rng.uniform(1, 3, (T, N, M, L)), 0).astype(np.float32)
    codes[:, 0, :, -1] = 2.5                     # windows that would leave the sequence
    ctxs = []
    try:
        with pkg.ActivationRecord(N, L, M, T=T) as ar:
            for t, fs in enumerate(sizes):
                c = pkg.CDL(pkg.CDLSetup(M=M, filter_size=fs))
                ctxs.append(c)
                c.load_data(S)
                X = np.zeros((N, M, c.Lg), np.float32)
                X[:, :, c.gamma:c.gamma + 4 * L:4] = codes[t]
                c.init_state(X0=X)
                assert pkg.record_training_result(c, 0.5, ar, t + 1, fs) == M
            u, tn, fl = ar.info()
            on = np.stack([codes[tn[k] - 1][:, u[k] - 1, :] > 0.5 for k in range(len(u))], axis=1)
            over, non_over, next_to = pkg.get_spatial_info(ar)
            ro, rn, rx = SO.activation_topology(on, tn, fl, L)
            np.testing.assert_array_equal(over, ro)
            np.testing.assert_array_equal(non_over, rn)
            np.testing.assert_array_equal(next_to, rx)
            if len(set(sizes)) > 1:
                return                            # get_pair_pfms takes one filter size
            thr = int(np.sort(over.ravel())[-40])
            pairs, spans, pfms = pkg.get_pair_pfms(ar, ctxs[0], over, thr, sizes[0])
            rp, rs, rf = SO.pair_msas(over, on, fl, tn, u, codes, S, thr, sizes[0])
            assert [tuple(int(v) for v in p) for p in pairs] == rp and len(rp) > 0
            np.testing.assert_array_equal(spans, rs)
            for a, b in zip(pfms, rf):
                np.testing.assert_allclose(a, b, rtol=1e-5, atol=1e-6)
    finally:
        for c in ctxs:
            c.close()


@pytest.mark.parametrize("longest", [5, 384, 768])
def test_pair_pfms_with_room_for_long_spans(pkg, built_lib, longest):
    """The span limit sets the shared memory of the pair sums (up to the 48 KB of float64 that
    the last pass takes), not their values."""
    N, L, M = 300, 60, 4
    rng = np.random.default_rng(2)
    S = pkg.synth.onehot(rng.integers(0, 4, (N, L)).astype(np.uint8))
    with pkg.CDL(pkg.CDLSetup(M=M, filter_size=5)) as c, pkg.ActivationRecord(N, L, M, T=2) as ar:
        c.load_data(S)
        X = np.zeros((N, M, c.Lg), np.float32)
        for t in (1, 2):                              # pairs are between trainings
            X[:, :, c.gamma:c.gamma + 4 * L:4] = np.where(rng.random((N, M, L)) < 0.1, rng.uniform(1, 3, (N, M, L)), 0)
            c.init_state(X0=X)
            pkg.record_training_result(c, 0.5, ar, t, 5)
        over = pkg.get_spatial_info(ar)[0]
        thr = 0                                       # every pair that occurs
        pairs, spans, pfms = pkg.get_pair_pfms(ar, c, over, thr, 5)
        wide = pkg.get_pair_pfms(ar, c, over, thr, longest)
    assert np.array_equal(pairs, wide[0]) and np.array_equal(spans, wide[1]) and len(pairs) > 0
    for a, b in zip(pfms, wide[2]):
        assert np.array_equal(a, b)
