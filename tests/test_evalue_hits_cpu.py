"""filter_using_evalue counts the entries > 0 of any array of positions, not of integers alone
(the scan of the background is replaced here; it needs a GPU)."""
import contextlib

import numpy as np
import pytest


@pytest.fixture
def hits(pkg, built_lib, monkeypatch):
    class Context:
        N = 4

        def on_background(self):
            return contextlib.nullcontext()

    monkeypatch.setattr(pkg, "scan_w_gpu", lambda *a, **k: np.zeros((4, 3), np.int32))
    pwms = [np.zeros((4, 8), np.float32)] * 3
    return lambda pos: pkg.filter_using_evalue(Context(), pwms, np.zeros(3), pos)["hits"]


ENTRIES = np.array([[3, 0, 7], [0, 0, 2], [5, 0, 0], [1, 0, 9]])


@pytest.mark.parametrize("kind", [np.int32, np.int64, np.uint8, np.float32, np.float64, bool, object, list])
def test_types(hits, kind):
    pos = ENTRIES.tolist() if kind is list else ENTRIES.astype(kind)
    np.testing.assert_array_equal(hits(pos), [3, 0, 3])


def test_negative_and_missing(hits):
    pos = ENTRIES.copy()
    pos[pos == 0] = -1
    np.testing.assert_array_equal(hits(pos), [3, 0, 3])
    pos = np.where(ENTRIES > 0, ENTRIES * 0.25, np.nan)
    np.testing.assert_array_equal(hits(pos), [3, 0, 3])
