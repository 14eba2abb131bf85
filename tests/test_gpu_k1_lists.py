"""The rows, counts and intensity sums of K1's hit lists at every tolerance window width, one hypothesis per spectrum (so
that no row is reached twice): the dense counts (vk_k1_brute) and the dense sums above the threshold, in row order."""
import dataclasses

import pytest

from tests.test_gpu_k1_windows import STATIC, VAR, _spectra

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unit,tol", [("da", 1e-4), ("da", 0.02), ("da", 0.3), ("da", 4.0), ("da", 60.0), ("ppm", 2.0),
                                      ("ppm", 20.0), ("ppm", 800.0), ("ppm", 40000.0)])
@pytest.mark.parametrize("charge", [1, 0])
@pytest.mark.parametrize("rows,warps", [(128, 4), (32, 1), (256, 3)])
def test_hit_list_contents(mini, unit, tol, charge, rows, warps):
    import torch
    from vulcan.gpu import engine as E
    from vulcan.gpu.host import SearchParams, make_hypotheses
    l1 = mini[0]
    p = SearchParams(fragment_unit=unit, fragment_ppm=(-tol, tol), max_fragment_charge=charge or None, max_peaks=512,
                     precursor_ppm=(-2000.0, 2000.0), isotope_errors=(0, 0), tile_rows=rows, k1_warps=warps)
    gi = E.GpuIndex(l1, p, STATIC, VAR)
    sp = _spectra(l1)
    peaks = E.k0_preprocess(sp, p, gi.dev, E.Stats())
    hyp = make_hypotheses(sp, peaks["valid"], l1.mass32, p)
    n, n_h = len(sp), len(hyp["spec"])
    assert n_h == len(set(hyp["spec"].tolist())) > 0
    h, r = E.window_candidates(hyp, gi.dev)
    o = torch.argsort(h * (1 << 28) + r)          # hypotheses are in spectrum order: the order of the lists
    h, r = h[o], r[o]
    want = E.k1_brute(gi, hyp, peaks, h, r, p)
    dh = E._as_dev(hyp, gi.dev)
    win_off, _, status, isum = E._k1_dense(gi, dh, peaks, p, n_h, isum=True)
    assert int(status.item()) == 0 and int(win_off[-1]) == len(want)
    spec = dh["spec"].long()
    dh = dict(dh, n_max=n_h, spec_off=torch.searchsorted(spec, torch.arange(n + 1, device=gi.dev)))
    for thr in (1, 2, 4):
        keep = want >= thr
        per = torch.bincount(spec[h[keep]], minlength=n)
        assert 0 < int(per.max()) <= 1000
        for with_isum in (True, False):
            k1h = E._k1_hits(gi, dh, peaks, p, n_h, thr, isum=with_isum)
            cand, _ = E._shortlist_hits(gi, dataclasses.replace(p, topk=1000), n, dh, k1h, 1000)
            assert int(k1h["status"].item()) == 0
            assert torch.equal(cand["cand_off"][1:n + 1] - cand["cand_off"][:n], per)
            m = int(per.sum())
            assert torch.equal(cand["c_hyp"][:m], h[keep])
            assert torch.equal(cand["c_row"][:m], r[keep])
            assert torch.equal(cand["c_cnt"][:m], want[keep].long())
            if with_isum:
                assert torch.equal(cand["c_isum"][:m], isum[:len(want)][keep])
