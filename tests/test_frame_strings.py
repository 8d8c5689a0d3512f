"""String columns of the data frames: single bases by lookup, longer fields by conversion."""
import numpy as np
import pytest

from process_gb300 import _lib
from process_gb300.engine import _sid_strings


@pytest.mark.parametrize("fields", [
    [], ["A"], [""], ["ACGT"], ["A", "", "T", "N"], ["A", "AC", "G" * _lib.SID_CHARS, "", "C"], ["AT"] * 3,
])
def test_sid_strings(fields):
    buf = np.zeros(len(fields) * _lib.SID_CHARS, np.uint8)
    for i, f in enumerate(fields):
        buf[i * _lib.SID_CHARS:i * _lib.SID_CHARS + len(f)] = list(f.encode())
    out = _sid_strings(buf, len(fields))
    assert out.dtype == object and out.tolist() == fields
    assert all(type(x) is str for x in out)
