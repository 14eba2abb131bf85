"""engine._arrow against pa.array for the arrays a PSM table can be built of, and the table's columns and types."""
import numpy as np
import pyarrow as pa
import pytest


@pytest.mark.parametrize("dtype", ["i1", "u1", "<i2", "<u2", "<i4", "<u4", "<i8", "<u8", "<f4", "<f8", ">i4", ">f8", "?"])
@pytest.mark.parametrize("form", ["plain", "empty", "strided", "slice", "readonly"])
def test_arrow_equals_pa_array(dtype, form):
    from vulcan.gpu.engine import _arrow
    a = (np.arange(40) % 5).astype(dtype)
    if a.dtype.kind == "f":
        a[3], a[4] = np.nan, np.inf
    a = {"plain": a, "empty": a[:0], "strided": a[::2], "slice": a[7:31], "readonly": a.copy()}[form]
    if form == "readonly":
        a.flags.writeable = False
    try:
        want = pa.array(a)
    except (pa.ArrowException, NotImplementedError, ValueError, TypeError) as e:
        with pytest.raises(type(e)):
            _arrow(a)
        return
    got = _arrow(a)
    assert got.type == want.type and len(got) == len(want) and got.null_count == want.null_count == 0
    assert got.to_numpy(zero_copy_only=False).tobytes() == want.to_numpy(zero_copy_only=False).tobytes()
