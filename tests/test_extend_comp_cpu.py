"""extend()'s use_comp: its kept motifs' columns as a C-order copy, and a use_comp without a
column for a kept motif refused (the device part of extend() is replaced here)."""
import numpy as np
import pytest


@pytest.fixture
def extend(pkg, monkeypatch):
    pos = np.array([[3, 0, 7], [0, 0, 2]], np.int32)

    def run(lens, use_comp):
        monkeypatch.setattr(pkg, "extension", lambda *a, **k: (pos, np.array(lens, np.int32), None, None))
        return pkg.extend(None, pos, lens, 8, use_comp, re_evaluate_pfm=False)
    return run


def test_use_comp_without_a_kept_column(extend):
    with pytest.raises(IndexError):
        extend([12, 12, 12], np.zeros((2, 2), np.uint8))


@pytest.mark.parametrize("order", ["C", "F"])
@pytest.mark.parametrize("columns", [3, 5])
def test_use_comp_columns(extend, monkeypatch, pkg, order, columns):
    uc = np.arange(2 * columns, dtype=np.uint8).reshape(2, columns).copy(order=order)
    for all_kept in (False, True):
        if all_kept:
            monkeypatch.setattr(pkg, "_any_entry", lambda pos: np.ones(3, bool))
        out = extend([12, 12, 12], uc)["use_comp"]
        np.testing.assert_array_equal(out, uc[:, :3] if all_kept else uc[:, [0, 2]])
        assert out.flags["C_CONTIGUOUS"] and not np.shares_memory(out, uc)
