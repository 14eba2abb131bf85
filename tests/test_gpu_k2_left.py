"""The dense K2 kernel's ways around its walk -- a warp per candidate for spectra of few, for the few long or crowded
candidates of 32, lanes side by side for many -- and CTAs that take several spectra, against the thread-per-candidate
kernel (vk_k2_cands), bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _equal(rng, lengths, pick, n_c, n_pk, tol, da, charges, intensities):
    """n_c[s] candidates of spectrum s, rows chosen by pick(s, n), n_pk peaks each."""
    import torch
    from vulcan.gpu import _lib as K
    from vulcan.gpu import engine as E
    letters = np.frombuffer(b"GASPVTCLINDQKEMHFRYW", np.uint8)
    res = letters[rng.integers(0, 20, int(lengths.sum()))]
    off = np.concatenate([[0], np.cumsum(lengths)[:-1]]).astype(np.int64)
    mask = np.where(rng.random(len(lengths)) < 0.5, rng.integers(0, 1 << 62, len(lengths)), 0).astype(np.uint64)
    mask[::5] |= np.uint64(1 << 63)
    fp = E.frag_params({"C": 57.021464}, {"M": 15.9949, "S": 79.966331, "^": 42.010565}, "da" if da else "ppm")
    mono = np.array(fp.mono[:], np.float32)
    mass = np.array([18.010565 + mono[res[o:o + n] - 65].sum() for o, n in zip(off, lengths)], np.float32)
    n_spec, tot = len(n_c), int(n_c.sum())
    rows = np.concatenate([pick(s, n) for s, n in enumerate(n_c)]).astype(np.int32)
    pm = rng.uniform(100.0, 2200.0, (n_spec, n_pk))
    for s in range(n_spec):   # a third of the peaks on fragments of the spectrum's first row
        r = rows[n_c[:s].sum()] if n_c[s] else 0
        b = np.cumsum(mono[res[off[r]:off[r] + lengths[r]] - 65])[:-1]
        own = np.concatenate([b, mass[r] - b])
        own = own[(own > 100) & (own < 2200)][:n_pk // 3]
        pm[s, :len(own)] = own
    pm = np.sort(pm.astype(np.float32), 1)
    pi = rng.choice(np.array(intensities, np.float32), (n_spec, n_pk))
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    args = [up(np.concatenate([[0], np.cumsum(n_c)]).astype(np.int64)), up(rows),
            up(rng.integers(1, charges + 2, tot).astype(np.int8)), up(np.arange(n_spec + 1, dtype=np.int64) * n_pk),
            up(pm.ravel()), up(pi.ravel()), up(off), up(lengths.astype(np.uint8)), up(mask.view(np.int64)), up(mass),
            up(res)]
    outs = []
    for dense in (True, False):
        o = E._k2_outputs(tot, torch.device("cuda"))
        common = (C.byref(fp), n_spec, *[K.ptr(t) for t in args], -tol, tol)
        if dense:
            K.check(K.lib().vk_k2_spectra(*common, None, *E._k2_ptrs(o), K.stream()), "k2_spectra")
        else:
            K.check(K.lib().vk_k2_cands(*common, *E._k2_ptrs(o), K.stream()), "k2_cands")
        torch.cuda.synchronize()
        outs.append({k: v.cpu().numpy() for k, v in o.items()})
    for k in outs[0]:
        assert np.array_equal(outs[0][k], outs[1][k], equal_nan=outs[0][k].dtype.kind == "f"), k
    assert n_pk == 1 or int(outs[0]["matched_b"].astype(int).sum()) > 0


@pytest.mark.parametrize("tol,da,n_pk", [(0.02, 1, 150), (20.0, 0, 150), (1.5, 1, 512), (0.02, 1, 1)])
@pytest.mark.parametrize("charges", [1, 3, 40])
@pytest.mark.parametrize("values", [(1.0, 250.5, 3e4), (0.0, -0.0, -1.0, 1.0, 7.0, np.inf, np.nan)])
def test_few_and_left_candidates(tol, da, n_pk, charges, values):
    rng = np.random.default_rng(n_pk + charges)
    lengths = np.concatenate([rng.integers(2, 31, 200), rng.integers(60, 71, 60), rng.integers(200, 256, 60), [0, 1]])
    short, long = np.arange(200), np.arange(200, len(lengths))
    n_c = np.array([0, 1, 2, 3, 4, 5, 31, 32, 33, 40, 96, 97, 130] * 3)

    def pick(s, n):
        kind = s // 13   # all long; a few long among short ones (at most 8 of 32, or around that); all short
        r = rng.choice(long if kind == 0 else short, n)
        if kind == 1:
            put = rng.random(n) < (0.2 if s % 2 else 0.28)
            r[put] = rng.choice(long, int(put.sum()))
        return r
    _equal(rng, lengths, pick, n_c, n_pk, tol, da, charges, values)


@pytest.mark.parametrize("charges", [1, 2])
def test_several_spectra_per_cta(charges):
    """More spectra than the grid has CTAs: a CTA's tables are built anew for each of its spectra."""
    rng = np.random.default_rng(8)
    lengths = np.concatenate([rng.integers(7, 31, 300), rng.integers(66, 100, 6)])
    n_c = rng.choice(np.array([0, 1, 2, 4, 7, 33, 100]), 21000, p=[.1, .2, .2, .2, .2, .08, .02])
    _equal(rng, lengths, lambda s, n: rng.integers(0, len(lengths), n), n_c, 60, 0.02, 1, charges, (1.0, 250.5, 3e4))
