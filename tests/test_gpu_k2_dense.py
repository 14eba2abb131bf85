"""The dense K2 kernel (vk_k2_spectra: presence bitmap, listed ions, warp-wide lookup) against the thread-per-candidate
kernel (vk_k2_cands: one binary search per ion), bit for bit, at the sizes where the dense one changes its path."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _table(rng, lengths):
    letters = np.frombuffer(b"GASPVTCLINDQKEMHFRYW", np.uint8)
    res = letters[rng.integers(0, 20, int(lengths.sum()))]
    off = np.concatenate([[0], np.cumsum(lengths)[:-1]]).astype(np.int64)
    mask = np.where(rng.random(len(lengths)) < 0.5, rng.integers(0, 1 << 62, len(lengths)), 0).astype(np.uint64)
    mask[::7] |= np.uint64(1 << 63)   # N-terminal modification
    return res, off, mask


@pytest.mark.parametrize("case", [
    # name, rows' lengths, peaks per spectrum, candidates per spectrum, (tolerance, Da), fragment charges + 1
    ("usual", (7, 31), (40, 300), (0, 1, 31, 32, 33, 95, 96, 97, 200), (0.02, 1), (2, 2)),
    ("ppm", (7, 31), (40, 300), (5, 64, 130), (20.0, 0), (2, 2)),
    ("charges", (7, 51), (100, 300), (5, 64, 130), (20.0, 0), (1, 5)),
    ("mask_edge", (60, 71), (40, 300), (40, 97), (0.02, 1), (2, 2)),      # 64 ions fit the marks, 65 do not
    ("longest", (200, 256), (40, 300), (33,), (0.02, 1), (2, 3)),
    ("lists_overflow", (7, 51), (300, 512), (33, 97), (1.5, 1), (2, 2)),  # most ions marked
    ("wide_ppm", (7, 31), (40, 200), (33, 97), (900000.0, 0), (2, 2)),    # every bucket marked
    ("few_peaks", (2, 31), (0, 3), (1, 33), (0.5, 1), (2, 2)),
    ("peak_limit", (7, 31), (511, 515), (33, 97), (0.02, 1), (2, 2)),     # only the first 512 peaks count
], ids=lambda c: c[0])
@pytest.mark.parametrize("shift", [0, 1])   # the residue table at an odd address
def test_dense_equals_sparse(case, shift):
    import torch
    from vulcan.gpu import _lib as K
    from vulcan.gpu import engine as E
    _, (l0, l1), (n0, n1), cands, (tol, da), (z0, z1) = case
    rng = np.random.default_rng(17 + shift)
    n_rows, n_spec = 400, 24
    lengths = rng.integers(l0, l1, n_rows)
    res, off, mask = _table(rng, lengths)
    fp = E.frag_params({"C": 57.021464}, {"M": 15.9949, "S": 79.966331, "^": 42.010565}, "da" if da else "ppm")
    mono = np.array(fp.mono[:], np.float32)
    mass = np.array([18.010565 + mono[res[o:o + n] - 65].sum() for o, n in zip(off, lengths)], np.float32)
    pk_off, pm, pi = [0], [], []
    for s in range(n_spec):
        k = int(rng.integers(n0, n1))
        own = []
        for r in rng.integers(0, n_rows, 3):   # fragments of a few rows among the noise
            b = np.cumsum(mono[res[off[r]:off[r] + lengths[r]] - 65])[:-1]
            own += [b[b < 2300], (mass[r] - b)[(mass[r] - b) < 2300]]
        x = np.concatenate(own + [rng.uniform(20.0, 2300.0, max(k, 1))])
        x = np.sort(rng.permutation(x)[:k].astype(np.float32))
        pm.append(x)
        pi.append(rng.choice(np.array([0.0, 1.0, 1.0, 250.5, 3e4], np.float32), len(x)))
        pk_off.append(pk_off[-1] + len(x))
    n_c = np.array([cands[s % len(cands)] for s in range(n_spec)])
    cand_off = np.concatenate([[0], np.cumsum(n_c)]).astype(np.int64)
    tot = int(cand_off[-1])
    dev = torch.device("cuda")
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    res_d = torch.zeros(len(res) + shift, dtype=torch.uint8, device=dev)
    res_d[shift:] = up(res)
    res_d = res_d[shift:]
    args = [up(cand_off), up(rng.integers(0, n_rows, tot).astype(np.int32)),
            up(rng.integers(z0, z1 + 1, tot).astype(np.int8)), up(np.array(pk_off, np.int64)),
            up(np.concatenate(pm + [np.zeros(1, np.float32)])), up(np.concatenate(pi + [np.zeros(1, np.float32)])),
            up(off), up(lengths.astype(np.uint8)), up(mask.view(np.int64)), up(mass), res_d]
    outs = []
    for dense in (True, False):
        o = E._k2_outputs(tot, dev)
        common = (C.byref(fp), n_spec, *[K.ptr(t) for t in args], -tol, tol)
        if dense:
            K.check(K.lib().vk_k2_spectra(*common, None, *E._k2_ptrs(o), K.stream()), "k2_spectra")
        else:
            K.check(K.lib().vk_k2_cands(*common, *E._k2_ptrs(o), K.stream()), "k2_cands")
        torch.cuda.synchronize()
        outs.append({k: v.cpu().numpy() for k, v in o.items()})
    for k in outs[0]:
        assert np.array_equal(outs[0][k], outs[1][k], equal_nan=outs[0][k].dtype.kind == "f"), k
    if case[0] != "few_peaks":
        assert int(outs[0]["matched_b"].astype(int).sum()) > 0
