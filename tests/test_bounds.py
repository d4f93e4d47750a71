"""Bounds of a hierarchy: any six numbers, whatever their type and layout."""
import numpy as np
import pytest

from operatorgraph_gb300 import engine

WANT = [-1.0, -2.0, -3.0, 4.0, 5.0, 6.0]


@pytest.mark.parametrize("form", ["list", "rows", "float64", "column", "every_second", "reversed", "columns_first",
                                  "read_only"])
def test_bounds_in_any_layout(form):
    six = np.array(WANT, np.float32)
    table = np.zeros((6, 3), np.float32)
    table[:, 1] = six
    wide = np.zeros(12, np.float32)
    wide[::2] = six
    frozen = six.copy()
    frozen.flags.writeable = False
    b = engine._bounds({
        "list": WANT, "rows": [WANT[:3], WANT[3:]], "float64": six.astype(np.float64), "column": table[:, 1],
        "every_second": wide[::2], "reversed": six[::-1].copy()[::-1],
        "columns_first": np.asfortranarray(six.reshape(2, 3)), "read_only": frozen}[form])
    assert list(b.min) + list(b.max) == WANT


def test_other_counts_are_refused():
    for bad in (WANT[:5], WANT + [7.0], 1.0):
        with pytest.raises(ValueError):
            engine._bounds(bad)
