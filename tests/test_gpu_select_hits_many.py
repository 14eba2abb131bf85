"""vk_select_hits over many spectra: lists past one warp's shared memory streamed by the warp (few and many ties, rows
in and out of order, a list as long as the buffer), and more lists left to CTAs than CTAs are launched, against the
oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHIFT, THR = 7, 2


def _lists(lo, hi, win_off, cnt, weight):
    """What K1 writes: per (tile, hypothesis) segment the kept rows in order, their number at its first slot."""
    h = np.repeat(np.arange(len(lo)), hi - lo)
    row = np.arange(len(cnt)) - win_off[h] + lo[h]
    first = win_off[h] + np.maximum(lo[h], row >> SHIFT << SHIFT) - lo[h]     # the segment's first slot
    keep = np.flatnonzero(cnt >= THR)
    f = first[keep]
    new = np.concatenate([[True], f[1:] != f[:-1]])
    start = np.flatnonzero(new)
    at = f + np.arange(len(f)) - start[np.cumsum(new) - 1]
    rc, isum, seg = np.zeros(len(cnt), np.uint64), np.zeros(len(cnt), np.uint32), np.zeros(len(cnt), np.uint32)
    rc[at] = (cnt[keep].astype(np.uint64) << np.uint64(32)) | row[keep].astype(np.uint64)
    isum[at] = weight[keep]
    seg[f[start]] = np.diff(np.concatenate([start, [len(f)]]))
    return rc, isum, seg


def _check(specs, counts, topk, closure, copies, n_rows):
    import torch
    from oracle import oracle as O
    from vulcan.gpu import _lib as K
    rng = np.random.default_rng(31)
    wins = [(s, a, b) for s, w in enumerate(specs) for a, b in w]
    spec, lo, hi = (np.array([w[k] for w in wins]) for k in range(3))
    n_spec, n_h, n = len(specs), len(lo), hi - lo
    win_off = np.concatenate([[0], np.cumsum(n)]).astype(np.int64)
    total = int(win_off[-1])
    cnt = {"small": rng.geometric(0.35, total), "equal": np.full(total, 3), "tall": rng.integers(0, 900, total),
           "sparse": np.where(rng.random(total) < 0.02, 3, 0)}[counts].astype(np.int64)
    weight = rng.integers(0, 1 << 24, total).astype(np.uint32)
    rc, isum, seg = _lists(lo, hi, win_off, cnt, weight)
    partner = (np.arange(n_rows) ^ 1).astype(np.int64)
    o_h, o_r, o_c = O.k1_appended({"lo": lo, "hi": hi}, win_off, cnt, THR)
    want = O.select_topk(o_h, o_r, o_c, spec, partner, topk, closure)
    sc = np.array([(cnt[a:b] > 0).sum() for a, b in zip(win_off[:-1], win_off[1:])])
    mt = np.array([cnt[a:b].sum() for a, b in zip(win_off[:-1], win_off[1:])])
    cap, n_t = (2 if closure else 1) * topk, n_spec * copies
    up = lambda a, t: torch.from_numpy(np.ascontiguousarray(a, t)).cuda()  # noqa: E731

    def rep(a, t, step=0):   # the spectra's arrays once per copy, each shifted by step
        x = up(a, t)
        return (x[None, :] + step * torch.arange(copies, device="cuda", dtype=x.dtype)[:, None]).reshape(-1)
    spec_off = np.searchsorted(spec, np.arange(n_spec + 1))
    args = [torch.cat([rep(spec_off[:-1], np.int64, n_h), up([n_h * copies], np.int64)]), rep(lo, np.int64),
            rep(hi, np.int64), torch.cat([rep(win_off[:-1], np.int64, total), up([total * copies], np.int64)]),
            rep(np.where(n > 0, SHIFT, 0), np.int8), rep(seg.view(np.int32), np.int32),
            rep(rc.view(np.int64), np.int64), rep(isum.view(np.int32), np.int32), rep(sc, np.int32), rep(mt, np.int64)]
    part = up(partner, np.int64)
    slots = [torch.full((n_t * cap,), -7, dtype=torch.int64, device="cuda") for _ in range(3)]
    s_isum = torch.zeros(n_t * cap, dtype=torch.int32, device="cuda")
    n_cand, s_sc, s_mt = (torch.full((n_t,), -9, dtype=torch.int64, device="cuda") for _ in range(3))
    K.check(K.lib().vk_select_hits(n_t, *[K.ptr(t) for t in args], topk, int(closure), K.ptr(part), cap,
                                   *[K.ptr(t) for t in slots], K.ptr(s_isum), K.ptr(n_cand), K.ptr(s_sc), K.ptr(s_mt),
                                   K.stream()), "select_hits")
    torch.cuda.synchronize()
    want_m = np.bincount(spec[want[0]], minlength=n_spec)
    assert bool((n_cand.view(copies, -1) == up(want_m, np.int64)).all())
    sel = up((np.arange(cap)[None, :] < want_m[:, None]).ravel(), bool)
    for got, ref, step in zip(slots, want, (n_h, 0, 0)):
        g = got.view(copies, -1)[:, sel] - step * torch.arange(copies, device="cuda")[:, None]
        assert bool((g == up(ref, np.int64)).all())
    # the sum of the hit itself where the row's lowest hypothesis took it, 0 for a partner that was not taken
    key = lambda h, r: h.astype(np.int64) * n_rows + r  # noqa: E731
    s2 = spec[o_h]
    o = np.lexsort((o_h, -o_r, -np.minimum(o_c, 32767), s2))
    taken = o[np.arange(len(o)) - np.searchsorted(s2[o], s2[o], side="left") < topk]
    at = win_off[o_h[taken]] + o_r[taken] - lo[o_h[taken]]
    sums = dict(zip(key(o_h[taken], o_r[taken]).tolist(), weight[at].tolist()))
    ref = np.array([sums.get(k, 0) for k in key(want[0], want[1]).tolist()], np.uint32)
    assert bool((s_isum.view(copies, -1)[:, sel] == up(ref.view(np.int32), np.int32)).all())
    assert bool((s_sc.view(copies, -1) == up(np.bincount(spec, weights=sc, minlength=n_spec), np.int64)).all())
    assert bool((s_mt.view(copies, -1) == up(np.bincount(spec, weights=mt, minlength=n_spec), np.int64)).all())


# 12 spectra, so 60, 660, 1,320 and 4,800 of them: lists are left to a CTA from 1,024, 4,096, 16,384 and 65,536 rows
@pytest.mark.parametrize("counts", ["small", "equal", "tall", "sparse"])
@pytest.mark.parametrize("topk,closure", [(1, True), (33, False), (100, True), (256, True), (385, False), (512, False),
                                          (900, False)])
@pytest.mark.parametrize("copies", [5, 55, 110, 400])
def test_long_lists_of_many_spectra(counts, topk, closure, copies):
    specs = []
    for n in (511, 513, 640, 1000, 4097):
        specs.append([(37, 37 + n)])                                           # in row order
        specs.append([(600 + n, 600 + 2 * n), (20, 20 + n // 2), (9, 9 + n)])  # overlapping, not in row order
    specs.append([(17 * i, 17 * i + 60) for i in range(40)])                   # more than a warp of hypotheses
    specs.append([(5000, 5001)] * 700)                                         # one row, more hypotheses than fit
    _check(specs, counts, topk, closure, copies, 14000)


@pytest.mark.parametrize("topk,closure", [(40, False), (100, True)])
def test_more_lists_left_than_ctas(topk, closure):
    _check([[(128, 70128)], [(40, 65580), (100, 130)], [(3, 90)]], "sparse", topk, closure, 400, 71000)


@pytest.mark.parametrize("topk,closure", [(40, False), (100, True)])
def test_several_lists_per_cta(topk, closure):
    specs = [[(300, 300 + n), (100, 90 + n)] for n in (2100, 2600, 4500)] + [[(3, 90)]]
    _check(specs, "small", topk, closure, 290, 14000)
