"""The dense K2 kernel (vk_k2_spectra) over rows of no and of one residue -- which have no ions -- among rows whose
lists are full, against the thread-per-candidate kernel (vk_k2_cands), bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("charges", [2, 4])
@pytest.mark.parametrize("where", ["inside", "zero", "end"])   # the offsets of the empty rows
def test_rows_without_ions(charges, where):
    import torch
    from vulcan.gpu import _lib as K
    from vulcan.gpu import engine as E
    rng = np.random.default_rng(4)
    letters = np.frombuffer(b"GASPVTCLINDQKEMHFRYW", np.uint8)
    n_rows, n_spec, n_c = 300, 12, 70
    lengths = rng.choice(np.array([0, 1, 2, 30, 60, 65]), n_rows, p=[.25, .15, .1, .2, .2, .1])
    lengths[[0, -1]] = 0
    res = letters[rng.integers(0, 20, int(lengths.sum()))]
    off = np.concatenate([[0], np.cumsum(lengths)[:-1]]).astype(np.int64)
    off[lengths == 0] = {"inside": off[lengths == 0], "zero": 0, "end": len(res)}[where]
    mask = rng.integers(0, 1 << 62, n_rows).astype(np.uint64) | np.uint64(1 << 63)
    fp = E.frag_params({"C": 57.021464}, {"M": 15.9949, "^": 42.010565}, "da")
    mono = np.array(fp.mono[:], np.float32)
    mass = np.array([18.010565 + mono[res[o:o + n] - 65].sum() for o, n in zip(off, lengths)], np.float32)
    n_pk = 512
    pm = np.sort(rng.uniform(20.0, 2300.0, (n_spec, n_pk)).astype(np.float32), 1)
    pi = rng.uniform(1.0, 1e3, (n_spec, n_pk)).astype(np.float32)
    rows = rng.integers(0, n_rows, (n_spec, n_c)).astype(np.int32)
    rows[0] = np.flatnonzero(lengths == 0)[rng.integers(0, (lengths == 0).sum(), n_c)]   # nothing but empty rows
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    tot = n_spec * n_c
    args = [up(np.arange(n_spec + 1, dtype=np.int64) * n_c), up(rows.ravel()), up(np.full(tot, charges, np.int8)),
            up(np.arange(n_spec + 1, dtype=np.int64) * n_pk), up(pm.ravel()), up(pi.ravel()), up(off),
            up(lengths.astype(np.uint8)), up(mask.view(np.int64)), up(mass), up(res)]
    outs = []
    for dense in (True, False):
        o = E._k2_outputs(tot, torch.device("cuda"))
        common = (C.byref(fp), n_spec, *[K.ptr(t) for t in args], -1.5, 1.5)   # most ions meet a peak
        if dense:
            K.check(K.lib().vk_k2_spectra(*common, None, *E._k2_ptrs(o), K.stream()), "k2_spectra")
        else:
            K.check(K.lib().vk_k2_cands(*common, *E._k2_ptrs(o), K.stream()), "k2_cands")
        torch.cuda.synchronize()
        outs.append({k: v.cpu().numpy() for k, v in o.items()})
    for k in outs[0]:
        assert np.array_equal(outs[0][k], outs[1][k], equal_nan=outs[0][k].dtype.kind == "f"), k
    none = lengths[rows.ravel()] < 2
    assert not outs[0]["matched_b"][none].any() and not outs[0]["matched_y"][none].any()
    assert int(outs[0]["matched_b"].astype(int).sum()) > 0
