"""The host columns of a PSM table: scan numbers and retention times of any kind that pa.array takes; and the Searcher
on runs whose arrays are of other array types."""
import datetime

import numpy as np
import pyarrow as pa
import pytest

T0 = datetime.datetime(2024, 5, 1)


@pytest.mark.parametrize("scan,rt", [
    (np.array([7, 8, 9, 10], np.uint32), np.array([.1, .2, .3, .4])),
    (np.array(["scan=7", "scan=8", "scan=9", "scan=10"], object), np.array([.1, .2, None, .4], object)),
    (np.array(["a", "bb", "c", "d"]), np.array([b"1", b"2", b"3", b"4"])),
    (np.array([7, None, 9, 10], object), np.array([T0] * 4, "M8[ms]")),
], ids=["numbers", "object", "text", "mixed"])
def test_table_takes_every_column_kind(scan, rt):
    from vulcan.gpu import engine as E
    from vulcan.gpu.host import Spectra
    sp = Spectra("r", scan, np.arange(4), rt, np.zeros(4), np.zeros(4, np.int8), np.zeros(0, np.float32),
                 np.zeros(0, np.float32), np.zeros(5, np.int64))
    s = np.array([3, 1, 2], np.int32)
    rec = {k: np.arange(3, dtype=np.int32) for k in E._PSM_TABLE}
    rec["spec_idx"] = s
    t = E._table(sp, rec)
    assert t.column("scan").combine_chunks() == pa.array(scan[s])
    assert t.column("rt").combine_chunks() == pa.array(rt[s])
    assert t.num_rows == 3 and t.column("run").to_pylist() == ["r"] * 3


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["list", "series", "arrow"])
def test_searcher_takes_offsets_of_any_array_type(mini, kind):
    import dataclasses

    import pandas as pd
    from vulcan.gpu import engine as E
    from vulcan.gpu.host import SearchParams
    l1, sp, _ = mini
    p = SearchParams(fragment_ppm=(-0.02, 0.02), fragment_unit="da", max_fragment_charge=1)
    gi = E.GpuIndex(l1, p, {"C": 57.021464}, {"M": 15.9949})
    off = {"list": list, "series": pd.Series, "arrow": pa.array}[kind](sp.offsets.tolist())
    want = E.Searcher(gi, l1, p).search(sp)[0]
    assert want.num_rows > 0
    assert E.Searcher(gi, l1, p).search(dataclasses.replace(sp, offsets=off))[0].equals(want)
