"""K1 at the shared-memory limit of its shape: tile, bitmap and histograms up to 200 KB beside queues of 64 entries a warp."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warps", [1, 4, 16])
@pytest.mark.parametrize("isum", [False, True])
def test_largest_shape(mini, warps, isum):
    import torch
    from vulcan.gpu import engine as E
    from vulcan.gpu.host import SearchParams, make_hypotheses
    l1, sp, _ = mini
    static, var = {"C": 57.021464}, {"M": 15.9949}
    p = SearchParams(k1_warps=warps)
    gi = E.GpuIndex(l1, p, static, var)
    peaks = E.k0_preprocess(sp, p, gi.dev, E.Stats())
    hyp = make_hypotheses(sp, peaks["valid"], l1.mass32, p)
    dh, n_h = E._as_dev(hyp, gi.dev), len(hyp["spec"])

    def run():
        out = E._k1_dense(gi, dh, peaks, p, n_h, isum=isum)
        hits = E._k1_hits(gi, dh, peaks, p, n_h, 2, isum=isum)
        assert int(out[2].item()) == 0 and int(hits["status"].item()) == 0
        n = int(out[0][-1])
        return [out[1][:n]] + ([out[3][:n]] if isum else []) + [hits["hyp_scored"], hits["hyp_matched"]]
    want = run()
    assert int(want[0].sum()) > 0
    # the bytes beside the postings, then as many postings as reach the limit (room only: the tiles stay as they are)
    nb, T = 1 << gi.tix.cbin_bits, 1 << gi.tix.tile_shift
    other = ((nb + 1 + 7) & ~7) * 2 + nb * 8 + warps * (T * 4 * (2 if isum else 1) + 64 * 4)
    most = (200 * 1024 - other) // 4 & ~3
    assert most > gi.tix.max_tile_postings
    gi.tix.max_tile_postings = most
    for a, b in zip(run(), want):
        assert torch.equal(a, b)
    gi.tix.max_tile_postings = most + 4
    with pytest.raises(RuntimeError):
        E._k1_dense(gi, dh, peaks, p, n_h, isum=isum)
    with pytest.raises(RuntimeError):
        E._k1_hits(gi, dh, peaks, p, n_h, 2, isum=isum)
