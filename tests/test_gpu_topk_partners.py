"""vk_select_topk where closure partners lie outside their row's window -- beside it, in another hypothesis' window, far
away, shared by several rows, more of them than are kept aside -- against the oracle's select_topk."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N_ROWS = 20000


def _windows(rng):
    """Spectra of disjoint windows, the hypotheses in random row order; odd and even starts, touching and apart."""
    spec, lo, hi, s = [], [], [], 0
    for sizes in ((1,), (33,), (64, 64), (5, 700, 31), (300, 0, 280, 1), (900, 1100, 950), (40,) * 31, (6, 2) * 16,
                  (4000,)):
        for gap in (0, 1, 40):
            at, wins = int(rng.integers(1, 60)), []
            for n in sizes:
                wins.append((at, at + n))
                at += n + gap
            wins = [wins[k] for k in rng.permutation(len(wins))]
            spec += [s] * len(wins)
            lo += [a for a, _ in wins]
            hi += [b for _, b in wins]
            s += 1
    return np.array(spec), np.array(lo), np.array(hi), s


def _partner(kind, rng):
    p = np.arange(N_ROWS) ^ 1
    if kind == "beside":                                   # the other row of a pair, at most 3 rows off
        o = np.argsort(np.arange(N_ROWS) + rng.uniform(0, 3, N_ROWS), kind="stable")
        p[o[0::2]], p[o[1::2]] = o[1::2], o[0::2]
    elif kind == "some":                                   # 3% anywhere: other windows, between windows, far
        a = rng.permutation(4000)[:120]
        b = np.concatenate([rng.permutation(4000)[:80], rng.integers(4000, N_ROWS, 40)])
        p[a] = b
    elif kind == "shared":                                 # 5% with one of six partners
        a = rng.permutation(4000)[:200]
        p[a] = rng.choice(np.array([0, 2, 77, 640, 1201, N_ROWS - 1]), 200)
    elif kind == "anywhere":                               # more than a warp keeps aside
        o = rng.permutation(N_ROWS)
        p[o[0::2]], p[o[1::2]] = o[1::2], o[0::2]
    return p.astype(np.int64)


# copies of the spectra: the launch over the left-over ones at 1, 2 and 4 of them a warp
@pytest.mark.parametrize("kind,topk,copies",
                         [(k, t, 1) for k in ("beside", "some", "shared", "anywhere") for t in (1, 7, 40, 300, 512)] +
                         [(k, 40, c) for k in ("beside", "anywhere") for c in (320, 700)])
def test_partners_outside_their_window(kind, topk, copies):
    import torch
    from oracle import oracle as O
    from vulcan.gpu import _lib as K
    rng = np.random.default_rng(23)
    spec, lo, hi, n_spec = _windows(rng)
    partner = _partner(kind, rng)
    n = hi - lo
    win_off = np.concatenate([[0], np.cumsum(n)]).astype(np.int64)
    total = int(win_off[-1])
    cnt = (rng.geometric(0.4, total) - 1).astype(np.int32)
    if copies > 1:   # the same spectra again and again: 27 x 320 and 27 x 700 of them
        k = np.arange(copies)
        so = (k[:, None] * n_spec + spec[None, :]).ravel()
        wo = np.concatenate([(k[:, None] * total + win_off[None, :-1]).ravel(), [copies * total]])
        lo_t, hi_t, cnt_t, n_t = np.tile(lo, copies), np.tile(hi, copies), np.tile(cnt, copies), n_spec * copies
    else:
        so, wo, lo_t, hi_t, cnt_t, n_t = spec, win_off, lo, hi, cnt, n_spec
    want = O.select_topk(*O.k1_appended({"lo": lo, "hi": hi}, win_off, cnt, 1), spec, partner, topk, True)
    up = lambda a, t: torch.from_numpy(np.ascontiguousarray(a, t)).cuda()  # noqa: E731
    cap = 2 * topk
    slots = [torch.full((n_t * cap,), -7, dtype=torch.int64, device="cuda") for _ in range(3)]
    n_cand, s_sc, s_mt = (torch.full((n_t,), -9, dtype=torch.int64, device="cuda") for _ in range(3))
    h_sc = torch.zeros(len(so), dtype=torch.int32, device="cuda")
    h_mt = torch.zeros(len(so), dtype=torch.int64, device="cuda")
    args = [up(np.searchsorted(so, np.arange(n_t + 1)), np.int64), up(lo_t, np.int64), up(hi_t, np.int64),
            up(wo, np.int64), up(cnt_t, np.int32)]
    part = up(partner, np.int64)
    K.check(K.lib().vk_select_topk(n_t, *[K.ptr(t) for t in args], len(cnt_t), K.ptr(part), 1, topk, 1, cap,
                                   *[K.ptr(t) for t in slots], K.ptr(n_cand), K.ptr(h_sc), K.ptr(h_mt), K.ptr(s_sc),
                                   K.ptr(s_mt), K.stream()), "select_topk")
    torch.cuda.synchronize()
    m = n_cand.cpu().numpy().reshape(copies, n_spec)
    want_m = np.bincount(spec[want[0]], minlength=n_spec)
    assert (m == want_m).all()
    sel = (np.arange(cap)[None, :] < want_m[:, None]).ravel()
    for got, ref, per in zip(slots, want, (len(spec), 0, 0)):
        g = got.cpu().numpy().reshape(copies, -1)[:, sel] - np.arange(copies)[:, None] * per
        assert (g == ref).all()
