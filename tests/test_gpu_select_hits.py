"""vk_select_hits on hit lists of every size it routes (registers, one warp's shared memory, a CTA over the lists in
global memory) against the oracle's select_topk, with the intensity sum of each row's lowest hypothesis."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHIFT = 7


def _spectra(rng, n_rows):
    """Hypothesis windows: small disjoint ones, and open ones that overlap each other and the small ones."""
    out = []
    for n in (0, 1, 300, 520, 1500, 6000):
        a = int(rng.integers(0, 100))
        out.append([(a, a + n), (a + n, a + 2 * n)])                      # touching
        out.append([(a + 200, a + 230), (a, a + 2 * n), (a + 40, a + n + 50)])   # overlapping
    out.append([(17 * i, 17 * i + 900) for i in range(40)])                # more than a warp of hypotheses
    out.append([(5000, 5001)] * 1100)                                      # more hypotheses on a row than fit
    out.append([])
    out.append([(0, n_rows), (0, n_rows)])
    return out


@pytest.mark.parametrize("counts", ["small", "equal", "tall", "huge", "sparse"])
@pytest.mark.parametrize("topk,closure", [(1, True), (8, False), (33, False), (100, True), (200, False), (512, True)])
def test_select_hits_equals_oracle(counts, topk, closure):
    import torch
    from oracle import oracle as O
    from vulcan.gpu import _lib as K
    n_rows, thr = 14000, 2
    rng = np.random.default_rng(9)
    specs = _spectra(rng, n_rows)
    wins = [(s, a, b) for s, w in enumerate(specs) for a, b in w]
    spec, lo, hi = (np.array([w[k] for w in wins]) for k in range(3))
    n_spec, n = len(specs), hi - lo
    win_off = np.concatenate([[0], np.cumsum(n)]).astype(np.int64)
    total = int(win_off[-1])
    cnt = {"small": rng.geometric(0.35, total), "equal": np.full(total, 2), "tall": rng.integers(0, 900, total),
           "huge": rng.integers(900, 40000, total), "sparse": np.where(rng.random(total) < 0.02, 3, 0)
           }[counts].astype(np.int64)
    w8 = rng.integers(0, 1 << 24, total).astype(np.uint32)
    # the lists K1 writes: per (tile, hypothesis) segment the kept rows in order, their number at its first slot
    rc, isum = np.zeros(total, np.uint64), np.zeros(total, np.uint32)
    seg = np.zeros(total, np.uint32)
    for h in range(len(lo)):
        r = np.arange(lo[h], hi[h])
        keep = cnt[win_off[h]:win_off[h + 1]] >= thr
        for t in range(lo[h] >> SHIFT, (hi[h] - 1 >> SHIFT) + 1 if n[h] else lo[h] >> SHIFT):
            m = keep & (r >> SHIFT == t)
            at = win_off[h] + max(lo[h], t << SHIFT) - lo[h]
            k = np.flatnonzero(m) + win_off[h]
            rc[at:at + len(k)] = (cnt[k].astype(np.uint64) << np.uint64(32)) | r[m].astype(np.uint64)
            isum[at:at + len(k)] = w8[k]
            seg[at] = len(k)
    partner = (np.arange(n_rows) ^ 1).astype(np.int64)
    hyp = {"lo": lo, "hi": hi}
    o_h, o_r, o_c = O.k1_appended(hyp, win_off, cnt, thr)
    want = O.select_topk(o_h, o_r, o_c, spec, partner, topk, closure)
    cap = (2 if closure else 1) * topk
    dev = torch.device("cuda")
    up = lambda a, t: torch.from_numpy(np.ascontiguousarray(a, t)).to(dev)  # noqa: E731
    sc = np.array([(cnt[a:b] > 0).sum() for a, b in zip(win_off[:-1], win_off[1:])])
    mt = np.array([cnt[a:b].sum() for a, b in zip(win_off[:-1], win_off[1:])])
    spec_off = np.searchsorted(spec, np.arange(n_spec + 1))
    args = [up(spec_off, np.int64), up(lo, np.int64), up(hi, np.int64), up(win_off, np.int64),
            up(np.where(n > 0, SHIFT, 0), np.int8), up(seg.view(np.int32), np.int32), up(rc.view(np.int64), np.int64),
            up(isum.view(np.int32), np.int32), up(sc, np.int32), up(mt, np.int64)]
    part = up(partner, np.int64)
    slots = [torch.full((n_spec * cap,), -7, dtype=torch.int64, device=dev) for _ in range(3)]
    s_isum = torch.zeros(n_spec * cap, dtype=torch.int32, device=dev)
    n_cand, s_sc, s_mt = (torch.full((n_spec,), -9, dtype=torch.int64, device=dev) for _ in range(3))
    K.check(K.lib().vk_select_hits(n_spec, *[K.ptr(t) for t in args], topk, int(closure), K.ptr(part), cap,
                                   *[K.ptr(t) for t in slots], K.ptr(s_isum), K.ptr(n_cand), K.ptr(s_sc), K.ptr(s_mt),
                                   K.stream()), "select_hits")
    torch.cuda.synchronize()
    m = n_cand.cpu().numpy()
    assert np.array_equal(m, np.bincount(spec[want[0]], minlength=n_spec))
    sel = (np.arange(cap)[None, :] < m[:, None]).ravel()
    for got, ref in zip(slots, want):
        assert np.array_equal(got.cpu().numpy()[sel], ref)
    # the sum of the hit itself where the row's lowest hypothesis took it, 0 for a partner that was not taken
    key = lambda h, r: h.astype(np.int64) * n_rows + r  # noqa: E731
    s2 = spec[o_h]
    o = np.lexsort((o_h, -o_r, -np.minimum(o_c, 32767), s2))
    first = np.searchsorted(s2[o], s2[o], side="left")
    taken = o[np.arange(len(o)) - first < topk]
    sums = dict(zip(key(o_h[taken], o_r[taken]).tolist(),
                    w8[win_off[o_h[taken]] + o_r[taken] - lo[o_h[taken]]].tolist()))
    ref = np.array([sums.get(k, 0) for k in key(want[0], want[1]).tolist()], np.uint32)
    assert np.array_equal(s_isum.cpu().numpy().view(np.uint32)[sel], ref)
    assert np.array_equal(s_sc.cpu().numpy(), np.bincount(spec, weights=sc, minlength=n_spec).astype(np.int64))
    assert np.array_equal(s_mt.cpu().numpy(), np.bincount(spec, weights=mt, minlength=n_spec).astype(np.int64))
