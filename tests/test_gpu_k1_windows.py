"""K1 at the widths and sizes where the filter and the queue change their path: tolerance windows from a fraction of a
bitmap bit to many words and several coarse bins, peak counts around the words a warp tests at once, fragment charges
beyond the precomputed ones.  Dense counts against vk_k1_brute; hit lists and intensity sums against the dense form."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STATIC, VAR = {"C": 57.021464}, {"M": 15.9949}
PEAKS = (15, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 191, 193, 300, 511, 512)


def _spectra(l1):
    """A spectrum per peak count, its precursor a row of the index, half its peaks on that row's fragments."""
    from vulcan.gpu.host import Spectra
    from vulcan.synth import fragment_ladders
    rng = np.random.default_rng(3)
    mz, it, off, pmz, ch = [], [], [0], [], []
    for n in PEAKS:
        r = int(rng.integers(len(l1.mass32) // 4, len(l1.mass32)))
        z = int(rng.integers(2, 5))
        seq = l1.residues[l1.seq_off[r]:l1.seq_off[r] + l1.length[r]].tobytes()
        ions = np.concatenate(fragment_ladders(seq, int(l1.mask[r]), STATIC, VAR)) + 1.0072764
        ions = ions[(ions > 151) & (ions < 1999)][:n // 2]
        x = np.sort(np.concatenate([ions, rng.uniform(151, 1999, n - len(ions))]).astype(np.float32))
        mz.append(x)
        it.append(rng.uniform(1, 1000, n).astype(np.float32))
        off.append(off[-1] + n)
        pmz.append((float(l1.mass32[r]) + z * 1.0072764) / z)
        ch.append(z)
    k = len(PEAKS)
    ids = np.arange(k, dtype=np.uint32)
    return Spectra("windows", ids, ids, np.zeros(k), np.array(pmz), np.array(ch, np.int8), np.concatenate(mz),
                   np.concatenate(it), np.array(off, np.int64))


@pytest.mark.parametrize("unit,tol", [("da", 1e-4), ("da", 0.02), ("da", 0.3), ("da", 4.0), ("da", 60.0), ("ppm", 2.0),
                                      ("ppm", 20.0), ("ppm", 800.0), ("ppm", 40000.0)])
@pytest.mark.parametrize("charge", [1, 0])   # 0: up to the precursor's charge less one (the third is not precomputed)
@pytest.mark.parametrize("rows,warps", [(128, 4), (32, 1), (256, 3)])
def test_counts_at_every_window_width(mini, unit, tol, charge, rows, warps):
    import torch
    from vulcan.gpu import engine as E
    from vulcan.gpu.host import SearchParams, make_hypotheses
    l1 = mini[0]
    p = SearchParams(fragment_unit=unit, fragment_ppm=(-tol, tol), max_fragment_charge=charge or None, max_peaks=512,
                     precursor_ppm=(-2000.0, 2000.0), tile_rows=rows, k1_warps=warps)
    gi = E.GpuIndex(l1, p, STATIC, VAR)
    sp = _spectra(l1)
    st = E.Stats()
    peaks = E.k0_preprocess(sp, p, gi.dev, st)
    hyp = make_hypotheses(sp, peaks["valid"], l1.mass32, p)
    assert len(hyp["spec"]) > 0
    h, r = E.window_candidates(hyp, gi.dev)
    o = torch.argsort(h * (1 << 28) + r)
    h, r = h[o], r[o]
    want = E.k1_brute(gi, hyp, peaks, h, r, p)
    dh = E._as_dev(hyp, gi.dev)
    n_h = len(hyp["spec"])
    win_off, cnt, status, isum = E._k1_dense(gi, dh, peaks, p, n_h, isum=True)
    total = int(win_off[-1])
    assert int(status.item()) == 0 and total == len(want)
    assert torch.equal(cnt[:total], want)
    plain = E._k1_dense(gi, dh, peaks, p, n_h)[1]
    assert torch.equal(plain[:total], want)
    thr = 2
    for with_isum in (True, False):
        k1h = E._k1_hits(gi, dh, peaks, p, n_h, thr, isum=with_isum)
        dh2 = dict(dh, n_max=n_h, spec_off=torch.searchsorted(dh["spec"].long(), torch.arange(len(sp.scan) + 1,
                                                                                              device=gi.dev)))
        cand, sums = E._shortlist_hits(gi, dataclasses.replace(p, topk=1000), len(sp.scan), dh2, k1h, 1000)
        n_c = int(cand["cand_off"][-1])
        keep = want >= thr
        if int(torch.bincount(dh["spec"].long()[h[keep]], minlength=1).max()) <= 1000:
            # (spectrum, row) order; no row is reached by two hypotheses of a spectrum within +-2000 ppm at these masses
            key = dh["spec"].long()[h[keep]] * (1 << 28) + r[keep]
            s = torch.argsort(key)
            if len(torch.unique(key)) == len(key):
                assert torch.equal(cand["c_row"][:n_c], r[keep][s])
                assert torch.equal(cand["c_cnt"][:n_c], want[keep][s].long())
                if with_isum:
                    assert torch.equal(cand["c_isum"][:n_c], isum[:total][keep][s])
        scored = torch.zeros(n_h, dtype=torch.int64, device=gi.dev).index_add_(0, h, (want > 0).long())
        matched = torch.zeros(n_h, dtype=torch.int64, device=gi.dev).index_add_(0, h, want.long())
        assert torch.equal(sums["hyp_scored"][:n_h].long(), scored)
        assert torch.equal(sums["hyp_matched"][:n_h], matched)
    assert bool((isum[:total][want == 0] == 0).all())
