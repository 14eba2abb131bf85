"""vk_select_topk over every kind of window it routes (disjoint windows: bitmap kernel; the rest: key kernel) against
the oracle's select_topk: candidates, counts and the K1 statistics, exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _windows(rng, n_rows):
    """Hypothesis windows of a few spectra per kind."""
    spec, lo, hi = [], [], []
    s = 0

    def add(wins):
        nonlocal s
        for a, b in wins:
            spec.append(s)
            lo.append(a)
            hi.append(b)
        s += 1
    for sizes in ((0,), (1,), (31, 32, 33), (255, 256, 257), (300, 0, 280), (1023, 1025), (5000, 7288), (5000, 7289),
                  (13000,), (40,) * 32, (40,) * 33):
        for order in (1, -1):                      # disjoint, rows ascending or descending over the hypotheses
            at, wins = int(rng.integers(0, 50)), []
            for n in sizes:
                wins.append((at, at + n))
                at += n + int(rng.integers(0, 3))  # neighbours may touch
            add(wins[::order])
    add([])                                        # no hypothesis
    add([(10, 400), (300, 700)])                   # overlapping
    add([(10, 400), (10, 400), (900, 950)])        # twice the same
    add([(500, 400), (20, 90)])                    # empty by order
    return np.array(spec), np.array(lo), np.array(hi), s


@pytest.mark.parametrize("counts", ["small", "equal", "tall", "huge"])
@pytest.mark.parametrize("thr,topk,closure", [(1, 100, True), (1, 50, False), (2, 7, True), (1, 1, True),
                                              (3, 512, True), (1, 513, False), (8, 25, True), (254, 20, False),
                                              (255, 20, True), (0, 30, True)])
def test_select_topk_equals_oracle(counts, thr, topk, closure):
    import torch
    from oracle import oracle as O
    from vulcan.gpu import _lib as K
    n_rows = 16000
    rng = np.random.default_rng(5)
    spec, lo, hi, n_spec = _windows(rng, n_rows)
    n = np.maximum(hi - lo, 0)
    win_off = np.concatenate([[0], np.cumsum(n)]).astype(np.int64)
    total = int(win_off[-1])
    cnt = {"small": rng.geometric(0.45, total) - 1, "equal": np.full(total, 3), "tall": rng.integers(0, 255, total),
           "huge": np.where(rng.random(total) < 0.001, rng.integers(200, 40000, total), rng.geometric(0.4, total) - 1)
           }[counts].astype(np.int32)
    partner = (np.arange(n_rows) ^ 1).astype(np.int64)                      # mostly a neighbour, some far away
    far = rng.choice(n_rows // 2, 40, replace=False) * 2
    partner[far[:20]], partner[far[20:]] = far[20:], far[:20]
    keep = cnt.size - 37                                                     # the last windows end past the buffer
    hyp = {"lo": lo, "hi": np.where(win_off[1:] <= keep, hi, lo)}
    n_in = np.maximum(hyp["hi"] - lo, 0)
    off_in = np.concatenate([[0], np.cumsum(n_in)]).astype(np.int64)
    cnt_in = np.concatenate([cnt[a:a + m] for a, m in zip(win_off[:-1], n_in)])
    want = O.select_topk(*O.k1_appended(hyp, off_in, cnt_in, thr), spec, partner, topk, closure)
    dev = torch.device("cuda")
    up = lambda a, t: torch.from_numpy(np.ascontiguousarray(a, t)).to(dev)  # noqa: E731
    cap = (2 if closure else 1) * topk
    spec_off = np.searchsorted(spec, np.arange(n_spec + 1)).astype(np.int64)
    slots = [torch.full((n_spec * cap,), -7, dtype=torch.int64, device=dev) for _ in range(3)]
    n_cand, s_sc, s_mt = (torch.full((n_spec,), -9, dtype=torch.int64, device=dev) for _ in range(3))
    h_sc = torch.zeros(len(spec), dtype=torch.int32, device=dev)
    h_mt = torch.zeros(len(spec), dtype=torch.int64, device=dev)
    args = [up(spec_off, np.int64), up(lo, np.int64), up(hi, np.int64), up(win_off, np.int64), up(cnt[:keep], np.int32)]
    part = up(partner, np.int64)
    K.check(K.lib().vk_select_topk(n_spec, *[K.ptr(t) for t in args], keep, K.ptr(part), thr, topk, int(closure), cap,
                                   *[K.ptr(t) for t in slots], K.ptr(n_cand), K.ptr(h_sc), K.ptr(h_mt), K.ptr(s_sc),
                                   K.ptr(s_mt), K.stream()), "select_topk")
    torch.cuda.synchronize()
    m = n_cand.cpu().numpy()
    assert np.array_equal(m, np.bincount(spec[want[0]], minlength=n_spec))
    sel = (np.arange(cap)[None, :] < m[:, None]).ravel()
    for got, ref in zip(slots, want):
        assert np.array_equal(got.cpu().numpy()[sel], ref)
    sums = lambda v: np.array([v[a:a + k].sum() for a, k in zip(off_in[:-1], n_in)])  # noqa: E731
    assert np.array_equal(h_sc.cpu().numpy(), sums(cnt_in > 0))
    assert np.array_equal(h_mt.cpu().numpy(), sums(cnt_in.astype(np.int64)))
    for got, v in ((s_sc, cnt_in > 0), (s_mt, cnt_in.astype(np.int64))):
        assert np.array_equal(got.cpu().numpy(), np.bincount(spec, weights=sums(v), minlength=n_spec).astype(np.int64))
