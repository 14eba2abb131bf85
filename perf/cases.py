"""The work that a program using this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values; ``prepare`` makes what the program holds before the call (spectra in pinned host
memory, the resident index, a search handle, a pruner), ``run`` is one call through the public entry points, ``work``
the bytes and operations it cannot do without, ``exact`` the floating results in 64 bits.

Indexes are random tryptic-like peptides of the repository's workload shapes (length 7-30, up to two missed cleavages,
Swiss-Prot composition, CAM-C, variable Met-ox, and S/T/Y phospho for "mods"), each with its pseudo-reversed decoy:
"small" ~0.16M peptidoforms, "human" ~5.5M, "mods" ~12M.  They depend on nothing but their name, as a program's
index does; everything else comes from the seed.  Runs are simulated like ``vulcan.synth``: b/y ions present with
probability 0.6, Gaussian ppm error, uniform noise peaks, log-normal intensities and peak counts.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vulcan-proteomics_b200"))

from vulcan.gpu import engine as E  # noqa: E402
from vulcan.gpu import prune as PR  # noqa: E402
from vulcan.gpu.host import SearchParams, Spectra  # noqa: E402
from vulcan.ptm import search as PTM  # noqa: E402

DEV = torch.device("cuda")
PROTON, NEUTRON, H2O = 1.0072764, 1.00335, 18.010565
MONO = {"A": 71.03711, "C": 103.00919, "D": 115.02694, "E": 129.04259, "F": 147.0684, "G": 57.02146, "H": 137.05891,
        "I": 113.08406, "K": 128.09496, "L": 113.08406, "M": 131.0405, "N": 114.04293, "P": 97.05276, "Q": 128.05858,
        "R": 156.1011, "S": 87.03203, "T": 101.04768, "V": 99.06841, "W": 186.07932, "Y": 163.06332}
PERCENT = {"A": 8.25, "N": 4.06, "D": 5.45, "C": 1.37, "Q": 3.93, "E": 6.75, "G": 7.07, "H": 2.27, "I": 5.96,
           "L": 9.66, "M": 2.42, "F": 3.86, "P": 4.70, "S": 6.56, "T": 5.34, "W": 1.08, "Y": 2.92, "V": 6.87}
STATIC = {"C": 57.021464}
OXIDATION = {"M": 15.9949}
PHOSPHO = {"M": 15.9949, "S": 79.966331, "T": 79.966331, "Y": 79.966331}
# target peptides and variable modifications of each index
INDEXES = {"small": (60_000, OXIDATION), "human": (2_040_000, OXIDATION), "mods": (1_760_000, PHOSPHO)}
ROWS = {"small": 160_000, "human": 5_460_000, "mods": 12_000_000}   # about; for work()
MAX_LEN = 30


# ---------------------------------------------------------------------------------------------------- index
class Peptidoforms:
    """The columns of a built index (those of ``vulcan.index.build.L1Index``)."""

    def __len__(self):
        return len(self.pf_id)


def _table(values, dtype):
    t = torch.zeros(26, dtype=dtype)
    for r, v in values.items():
        t[ord(r) - 65] = v
    return t


@functools.lru_cache(maxsize=None)
def _index(name):
    """(columns on the host, the same on the device): one unmodified form per peptide and one per variable site,
    targets and pseudo-reversed decoys, in (mass, id) order."""
    n, var = INDEXES[name]
    g = torch.Generator(device=DEV).manual_seed(20400)
    # tryptic lengths: the digest's negative-binomial pieces with 0, 1 or 2 missed cleavages
    w, cut = [], 0.109
    for m in range(3):
        for ln in range(7, MAX_LEN + 1):
            w.append(math.comb(ln - 1, m) * cut ** (m + 1) * (1 - cut) ** (ln - m - 1))
    pick = torch.multinomial(torch.tensor(w, device=DEV), n, replacement=True, generator=g)
    span = MAX_LEN - 6
    length, missed = pick % span + 7, pick // span
    letters = torch.tensor([ord(c) for c in PERCENT], device=DEV, dtype=torch.uint8)
    share = torch.tensor(list(PERCENT.values()), device=DEV)
    seq = letters[torch.multinomial(share, n * MAX_LEN, replacement=True, generator=g)].view(n, MAX_LEN)
    at = torch.arange(MAX_LEN, device=DEV)[None, :]
    kr = torch.tensor([ord("K"), ord("R")], device=DEV, dtype=torch.uint8)
    for m in range(3):   # the C-terminus, then the missed sites
        where = (length - 1) if m == 0 else (torch.rand(n, device=DEV, generator=g) * (length - 1)).long()
        hit = (at == where[:, None]) & (missed >= m)[:, None]
        seq = torch.where(hit, kr[torch.randint(2, (n, 1), device=DEV, generator=g)], seq)
    inside = at < length[:, None]
    seq = torch.where(inside, seq, torch.zeros_like(seq))
    aa = (seq.long() - 65).clamp(min=0)
    base = torch.where(inside, (_table(MONO, torch.float64) + _table(STATIC, torch.float64)).to(DEV)[aa],
                       torch.zeros((), dtype=torch.float64, device=DEV)).sum(1) + H2O
    pep, site = torch.nonzero(_table(var, torch.float64).to(DEV)[aa].ne(0) & inside, as_tuple=True)
    delta = _table(var, torch.float64).to(DEV)[aa[pep, site]] - _table(STATIC, torch.float64).to(DEV)[aa[pep, site]]
    pep_f = torch.cat([torch.arange(n, device=DEV), pep])
    mask_t = torch.cat([torch.zeros(n, dtype=torch.int64, device=DEV), torch.ones_like(site) << site])
    site_d = torch.where(site == length[pep] - 1, site, length[pep] - 2 - site)   # the decoy keeps its C-terminus
    mask_d = torch.cat([torch.zeros(n, dtype=torch.int64, device=DEV), torch.ones_like(site) << site_d])
    mass = torch.cat([base, base[pep] + delta]).float()
    nf = len(pep_f)
    order_d = torch.where(at < length[:, None] - 1, length[:, None] - 2 - at, at)
    seq_d = torch.gather(seq, 1, order_d.clamp(min=0))
    pf_id = torch.arange(1, 2 * nf + 1, device=DEV) * -7046029254386353131   # odd: all different
    mass2 = torch.cat([mass, mass])
    o = torch.argsort(pf_id, stable=True)
    o = o[torch.argsort(mass2[o], stable=True)]
    rank = torch.empty_like(o)
    rank[o] = torch.arange(2 * nf, device=DEV)
    form, side = o % nf, o // nf
    d = Peptidoforms()
    d.pf_id = pf_id[o]
    d.mass32 = mass2[o]
    d.partner = rank[torch.where(o < nf, o + nf, o - nf)]
    pe = pep_f[form]
    d.length = length[pe].to(torch.uint8)
    d.missed = missed[pe].to(torch.uint8)
    d.mask = torch.where(side == 0, mask_t[form], mask_d[form])
    d.n_var = (d.mask != 0).to(torch.uint8)
    d.seq_off = torch.cumsum(d.length.long(), 0) - d.length.long()
    parts = []
    for i in range(0, 2 * nf, 1 << 21):   # residues row by row
        p, s = pe[i:i + (1 << 21)], side[i:i + (1 << 21), None]
        rows = torch.where(s == 0, seq[p], seq_d[p])
        parts.append(rows[rows > 0])
    d.residues = torch.cat(parts)
    d.decoy = side == 1
    h = Peptidoforms()
    for k in ("mass32", "partner", "length", "missed", "n_var", "seq_off", "residues"):
        setattr(h, k, getattr(d, k).cpu().numpy())
    h.pf_id = d.pf_id.cpu().numpy().view(np.uint64)
    h.mask = d.mask.cpu().numpy().view(np.uint64)
    return h, d


@functools.lru_cache(maxsize=None)
def _gpu_index(name, unit):
    return E.GpuIndex(_index(name)[0], SearchParams(fragment_unit=unit), STATIC, INDEXES[name][1], device=DEV)


# ---------------------------------------------------------------------------------------------------- spectra
def _padded(d, rows):
    at = torch.arange(MAX_LEN, device=DEV)[None, :]
    ln = d.length[rows].long()[:, None]
    ix = (d.seq_off[rows][:, None] + at).clamp(max=len(d.residues) - 1)
    return torch.where(at < ln, d.residues[ix].long() - 65, torch.full_like(ix, -1)), at, ln


def _simulate(case, seed, run, n):
    """One simulated run of n spectra of the case's index, as host arrays."""
    _, d = _index(case["index"])
    var = INDEXES[case["index"]][1]
    g = torch.Generator(device=DEV).manual_seed(1_000_003 * (seed + 1) + run)
    rnd = lambda *s: torch.rand(*s, device=DEV, generator=g)  # noqa: E731
    nrm = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    rows = torch.randint(len(d.mass32), (n,), device=DEV, generator=g)
    rows = torch.where(d.decoy[rows], d.partner[rows], rows)   # targets
    aa, at, ln = _padded(d, rows)
    on = ((d.mask[rows][:, None] >> at) & 1).bool()
    delta = torch.where(on, _table(var, torch.float64).to(DEV)[aa.clamp(min=0)],
                        _table(STATIC, torch.float64).to(DEV)[aa.clamp(min=0)])
    res = torch.where(aa >= 0, _table(MONO, torch.float64).to(DEV)[aa.clamp(min=0)] + delta, torch.zeros_like(delta))
    b = torch.cumsum(res, 1)
    ions = torch.cat([b, H2O + res.sum(1, keepdim=True) - b], 1) + PROTON
    # each ion with probability 0.6, and at least ten of those in the fragment range: a spectrum has a match
    chance = torch.where((at < ln - 1).repeat(1, 2), rnd(n, 2 * MAX_LEN), 2.0)
    seen = (ions >= 150) & (ions <= 2000)
    first = torch.where(seen, chance, 2.0)
    is_ion = (chance < 0.6) | ((first <= torch.sort(first, 1).values[:, 9:10]) & (first < 2.0))
    if case["peaks"]:
        total = torch.exp(math.log(case["peaks"]) + 0.5 * nrm(n)).round().clamp(24, 600).long()
    else:
        total = is_ion.sum(1) + 100
    keep = is_ion & (torch.cumsum(is_ion, 1) <= total[:, None])
    noise = torch.arange(600, device=DEV)[None, :] < (total - (keep & seen).sum(1))[:, None]   # total: in range
    mz = torch.cat([ions * (1 + 5e-6 * nrm(n, 2 * MAX_LEN)), 150 + 1850 * rnd(n, 600)], 1).float()
    it = torch.exp(torch.cat([math.log(3000) + 0.8 * nrm(n, 2 * MAX_LEN), math.log(1000) + nrm(n, 600)], 1)).float()
    have = torch.cat([keep, noise], 1)
    key = torch.where(have, mz, torch.full_like(mz, math.inf))
    if case.get("shuffled", 0.0):   # spectra whose peaks come in no order
        mixed = rnd(n) < case["shuffled"]
        key = torch.where(have & mixed[:, None], rnd(n, key.shape[1]), key)
    o = torch.argsort(key, 1)
    have = torch.gather(have, 1, o)
    mz, it = torch.gather(mz, 1, o)[have], torch.gather(it, 1, o)[have]
    off = torch.cat([torch.zeros(1, dtype=torch.int64, device=DEV), torch.cumsum(have.sum(1), 0)])
    z = torch.randint(2, 5, (n,), device=DEV, generator=g)
    iso = torch.multinomial(torch.tensor([0.85, 0.12, 0.03], device=DEV), n, replacement=True, generator=g)
    zf = z.double()
    pmz = (d.mass32[rows].double() + iso * NEUTRON + zf * PROTON) / zf * (1 + 1e-6 * nrm(n).double())
    charge = z.to(torch.int8)
    unknown = int(n * case.get("unknown", 0.0))   # this many precursors carry no charge
    if unknown:
        charge[torch.randperm(n, device=DEV, generator=g)[:unknown]] = 0
    ids = np.arange(n, dtype=np.uint32)
    return Spectra("run%d" % run, ids, ids, np.linspace(0.0, 120.0, n), pmz.cpu().numpy(), charge.cpu().numpy(),
                   mz.cpu().numpy(), it.cpu().numpy(), off.cpu().numpy())


def _run_sizes(case):
    """Spectra of each run of the case: equal, or (batches) uneven between half and one and a half of the mean."""
    n, k = case["spectra"], case["runs"]
    if case["call"] != "batch":
        return [n] * k
    return [max(1, int(n * (0.5 + (0.61803 * i) % 1.0))) for i in range(k)]


# ---------------------------------------------------------------------------------------------------- handles
def _params(case):
    da = case["unit"] == "da"
    return SearchParams(fragment_unit=case["unit"], fragment_ppm=(-0.02, 0.02) if da else (-20.0, 20.0),
                        topk=case["topk"], max_peaks=case["max_peaks"], isotope_errors=(case["iso_lo"], case["iso_hi"]),
                        max_fragment_charge=case["fragment_charge"] or None, peak_mode=case["peak_mode"])


@functools.lru_cache(maxsize=None)
def _pruner():
    """A pruner whose logit grows with the K1 count and the matched intensity (as a trained one's does): about two of
    the at most eight shortlisted hits of a spectrum are kept."""
    g = torch.Generator().manual_seed(7)
    pr = PR.Pruner(DEV, seed=7)
    w = {k: v.cpu().numpy() for k, v in pr.w.items()}
    w1 = 0.3 * torch.randn(256, 16, generator=g)
    w1[:, 6:] = 0
    w2 = 0.02 * torch.randn(256, 256, generator=g)
    w3 = 0.02 * torch.randn(256, generator=g)
    for j, (up, down) in enumerate([(1.0, -1.0), (0.8, -0.8), (-0.2, -0.2)]):   # count, intensity, |ppm|
        for k, (sign, out) in enumerate(((1.0, up), (-1.0, down))):
            u = 2 * j + k
            w1[u], w2[u], w2[:, u] = 0.0, 0.0, 0.0
            w1[u, j] = sign
            w2[u, u] = 1.0
            w3[u] = out
    w.update(W1=w1.numpy(), W2=w2.numpy(), w3=w3.numpy())
    mu, sd = np.zeros(16, np.float32), np.ones(16, np.float32)
    mu[:6] = [4.0, 0.05, 0.0, 3.0, 14.0, 0.8]
    sd[:6] = [3.0, 0.08, 5.0, 0.8, 5.0, 0.8]
    sel = np.array([-0.25, 1, 128, 2, 8], np.float64)   # tau, min_keep, max_keep, min_count, shortlist_k
    return pr.load_state_dict({**w, "mu": mu, "sd": sd, "sel": sel})


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


@functools.lru_cache(maxsize=4)
def _searcher(key):
    """The search handle that a program keeps for all its runs, used once (on a run of its own) so that its buffers
    and its captured pass are there."""
    case = dict(key)
    h = E.Searcher(_gpu_index(case["index"], case["unit"]), _index(case["index"])[0], _params(case),
                   pruner=_pruner() if case["pruned"] else None)
    runs = [E.pin_spectra(_simulate(case, -1, i, n)) for i, n in enumerate(_run_sizes(case))]
    _search(h, case["call"], runs)
    return h


def _search(h, call, runs):
    if call == "search":
        return [h.search(runs[0])[0]]
    found = h.search_batch(runs) if call == "batch" else h.search_many(runs)
    return [t for t, _ in found]


# ---------------------------------------------------------------------------------------------------- the cases
def _case(name, call, index, spectra, *, runs=1, peaks=150, topk=100, max_peaks=512, unit="da", pruned=False,
          fragment_charge=1, iso_lo=0, iso_hi=2, peak_mode="global", unknown=0.0, shuffled=0.0, offsets=0,
          open_window=False):
    c = dict(call=call, index=index, spectra=spectra, runs=runs, peaks=peaks, topk=topk, max_peaks=max_peaks,
             unit=unit, pruned=pruned, fragment_charge=fragment_charge, iso_lo=iso_lo, iso_hi=iso_hi,
             peak_mode=peak_mode, unknown=unknown, shuffled=shuffled, offsets=offsets, open_window=open_window)
    return {"name": name, **c} if name else c


def listed():
    return [
        # a handful of spectra looked up while a program waits: launches and latency
        _case("query_32", "search", "small", 32, peaks=0, topk=50, max_peaks=150),
        # the small workload: 5,000 spectra of ~130 peaks against a small proteome
        _case("run_small", "search", "small", 5000, peaks=0, topk=50, max_peaks=150),
        # the human workload, plain exhaustive search, runs one after another
        _case("runs_human", "many", "human", 40_000, runs=2),
        # the same through the learned pruner, the headline path
        _case("runs_human_pruned", "many", "human", 40_000, runs=2, pruned=True),
        # runs of uneven size packed into batches
        _case("batch_human", "batch", "human", 14_001, runs=9),
        # one call of the reference's entry point with its default knobs: ppm tolerance, 500 candidates and 150 peaks
        # per spectrum, some precursors without a charge, some peak lists out of order
        _case("run_defaults_ppm", "engine", "human", 10_001, topk=500, max_peaks=150, unit="ppm", unknown=0.3,
              shuffled=0.05),
        # the window peak view, fragment charges up to z - 1, a wider isotope range
        _case("run_window_charges", "search", "human", 8191, unit="ppm", peaks=250, fragment_charge=0, iso_lo=-1,
              iso_hi=3, peak_mode="window"),
        # an index with phosphorylation: wide row windows, longer candidate lists
        _case("run_mods", "search", "mods", 16_384, topk=200),
        _case("runs_mods_pruned", "many", "mods", 32_768, runs=2, topk=200, pruned=True),
        # mass-offset and open search of a small run
        _case("run_open", "modes", "small", 777, topk=50, max_peaks=150, peaks=120, offsets=3, open_window=True),
        # training data of the pruner: shortlist, features, labels from the rescoring of every window row
        _case("pruner_data", "collect", "human", 4000, max_peaks=512),
        # one epoch of the pruner's training (forward, backward, Adam), 8,192 hits a step
        {"name": "pruner_fit", "call": "fit", "hits": 262_144, "batch": 8192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "many", "many", "batch", "engine", "modes", "collect", "fit"])
    if kind == "fit":
        batch = rng.choice([4096, 8192])
        return {"call": "fit", "hits": _log(rng, batch, 262_144), "batch": batch}
    unit = rng.choice(["da", "ppm"])
    more = dict(topk=rng.choice([50, 100, 150, 200]), max_peaks=rng.choice([150, 150, 300, 512]), unit=unit,
                peaks=rng.randint(80, 250))
    if kind == "modes":
        return _case("", kind, "small", _log(rng, 50, 777), offsets=rng.randint(0, 4), open_window=rng.random() < 0.7,
                     **more)
    if kind == "collect":
        return _case("", kind, rng.choice(["small", "human"]), _log(rng, 300, 4000), **more)
    index = rng.choice(["small", "human", "human", "mods"])
    pruned = kind in ("search", "many", "batch") and rng.random() < 0.5
    if kind == "many":
        return _case("", kind, index, _log(rng, 1000, 16_000 if index == "mods" else 40_000), runs=rng.randint(1, 2),
                     pruned=pruned, **more)
    if kind == "batch":
        return _case("", kind, rng.choice(["small", "human"]), _log(rng, 1000, 14_000), runs=rng.randint(3, 9),
                     pruned=pruned, **more)
    if kind == "engine":
        return _case("", kind, rng.choice(["small", "human"]), _log(rng, 20, 10_000), unknown=rng.choice([0.0, 0.3]),
                     shuffled=rng.choice([0.0, 0.05]), **dict(more, topk=rng.choice([100, 500])))
    return _case("", kind, index, _log(rng, 20, 16_000), pruned=pruned, fragment_charge=rng.choice([1, 1, 2, 0]),
                 iso_hi=rng.choice([0, 1, 2, 3]), iso_lo=rng.choice([0, 0, -1]),
                 peak_mode=rng.choice(["global", "global", "window"]), **more)


# ---------------------------------------------------------------------------------------------------- measuring
def _fit_inputs(case, seed):
    """Standardised features (BF16), labels that depend on them, and the initial weights."""
    g = torch.Generator(device=DEV).manual_seed(1_000_003 * (seed + 1))
    x = torch.zeros(case["hits"], 16, device=DEV)
    x[:, :6] = torch.randn(case["hits"], 6, device=DEV, generator=g)
    s = 1.5 * x[:, 0] + x[:, 1] - 0.5 * x[:, 2].abs() - 3.0
    y = (torch.rand(case["hits"], device=DEV, generator=g) < torch.sigmoid(s)).float()
    cpu = torch.Generator().manual_seed(seed + 5)
    w = {"W1": torch.zeros(256, 16), "b1": torch.zeros(256), "W2": torch.randn(256, 256, generator=cpu) / 11.3,
         "b2": torch.zeros(256), "w3": torch.randn(256, generator=cpu) / 16.0, "b3": torch.zeros(1)}
    w["W1"][:, :6] = torch.randn(256, 6, generator=cpu) / 1.73
    return x.to(torch.bfloat16), y, w


def prepare(case, seed):
    if case["call"] == "fit":
        x, y, w = _fit_inputs(case, seed)
        start = {k: v.numpy() for k, v in w.items()}
        start.update(mu=np.zeros(16, np.float32), sd=np.ones(16, np.float32), sel=np.array([0.0, 1, 128, 1, 0]))
        return {"case": case, "x": x, "y": y, "start": start, "pruner": PR.Pruner(DEV)}
    h = None
    if case["call"] in ("search", "many", "batch"):
        h = _searcher(_key(case))
    runs = [_simulate(case, seed, i, n) for i, n in enumerate(_run_sizes(case))]
    if h is not None:
        runs = [E.pin_spectra(r) for r in runs]
    s = {"case": case, "runs": runs, "handle": h, "p": _params(case), "l1": _index(case["index"])[0],
         "gi": _gpu_index(case["index"], case["unit"]), "out": {}}
    if case["call"] == "modes":
        s["modes"] = PTM.ModeParams(offsets=(79.966331, 0.984016, -17.026549, 42.010565)[:case["offsets"]],
                                    open_da=(-150.0, 500.0) if case["open_window"] else None)
    if case["call"] == "collect":
        s["pruner"] = PR.Pruner(DEV)
    return s


def _pad(t, n):
    return torch.nn.functional.pad(t, (0, 0) * (t.dim() - 1) + (0, n - len(t)))


def _columns(tables, sizes):
    """The PSM tables' columns of numbers, a row per spectrum (zeros after the last where a spectrum has no PSM)."""
    found = [{c: t.column(c).to_numpy() for c in t.column_names if c != "run"} for t in tables]
    return [{c: v if len(v) == n else np.pad(v, (0, n - len(v))) for c, v in q.items()} for q, n in zip(found, sizes)]


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "fit":
        pr = state["pruner"].load_state_dict(state["start"])
        pr.step = 0
        losses = pr.fit(state["x"], state["y"], epochs=1, batch=case["batch"], lr=2e-3, seed=3)
        return {"loss": losses[0], **{k: v.clone() for k, v in pr.w.items()}}
    sizes = _run_sizes(case)
    if call == "engine":
        return _columns([E.search(state["runs"][0], state["gi"], state["l1"], state["p"])[0]], sizes)
    if call == "modes":
        tbl, _ = PTM.search_modes(state["runs"][0], state["gi"], state["l1"], state["p"], state["modes"])
        return _columns([tbl], sizes)
    if call == "collect":
        d = PR.collect(state["runs"][0], state["gi"], state["p"], state["pruner"])
        slots = len(state["runs"][0].scan) * state["p"].topk   # the hits in their slots' number of rows
        hits = {k: _pad(d[k], slots) for k in ("feat", "y", "spec", "row", "cnt")}
        return {**hits, "top1": d["top1"], "n_rescored_plain": d["n_rescored_plain"]}
    tables = _search(state["handle"], call, state["runs"])
    if call != "batch":
        return _columns(tables, sizes)
    parts, out = _columns(tables, sizes), state["out"]   # many runs: their rows together, in arrays kept for it
    for c in parts[0]:
        if c not in out:
            out[c] = np.empty(sum(sizes), parts[0][c].dtype)
        np.concatenate([q[c] for q in parts], out=out[c])
    return out


def work(case):
    if case["call"] == "fit":
        steps = case["hits"] // case["batch"]
        return {"bytes": case["hits"] * 36 + 70_000 * 8.0,
                "flops": 6.0 * steps * case["batch"] * (16 * 256 + 256 * 256 + 256)}
    n = sum(_run_sizes(case))
    peaks = n * ((case["peaks"] * 1.13) or 117)
    rows = ROWS[case["index"]]
    z = 1 + 2 * case["unknown"]
    hyps = n * z * (case["iso_hi"] - case["iso_lo"] + 1 + case["offsets"])
    window = hyps * max(1.0, rows * 5.2e-5) + (n * z * rows * 0.4 if case["open_window"] else 0)
    # spectra once, the fragments (4 bytes, 24 a row) of the rows in their windows once, a PSM row per spectrum
    return {"bytes": peaks * 8 + n * (25 + 132) + min(window, float(rows)) * 24 * 4, "flops": 0.0}


# ---------------------------------------------------------------------------------------------------- 64 bits
def exact(case, seed):
    """The floating outputs by plain torch: which peaks, rows and candidates count is decided by the search's 32-bit
    comparisons (they define it), the values are 64-bit.  No value for the searches whose candidates depend on the
    pruner's BF16 network, and for the mass-offset and open ones, whose scores depend on a site that 32-bit running
    sums choose.  Training is recomputed step by step in 64 bits."""
    if case["call"] == "fit":
        return _exact_fit(case, seed)
    if case["pruned"] or case["call"] == "modes":
        return None
    runs = [_exact_search(case, _simulate(case, seed, i, n)) for i, n in enumerate(_run_sizes(case))]
    if case["call"] == "collect":
        return runs[0]
    return {k: np.concatenate([r[k] for r in runs]) for k in runs[0]} if case["call"] == "batch" else runs


def _ranges(off, n):
    """(owner, value) of the concatenated ranges off[i], off[i] + 1, ..., n[i] values each."""
    who = torch.repeat_interleave(torch.arange(len(n), device=DEV), n)
    first = torch.cumsum(n, 0) - n
    return who, off[who] + torch.arange(len(who), device=DEV) - first[who]


def _bounds(m, p):
    lo, hi = p.fragment_ppm
    if p.fragment_unit == "da":
        return m + lo, m + hi
    return m + (m * lo) / 1e6, m + (m * hi) / 1e6


def _ladder(d, var, rows):
    """Per ion step k: (b mass, y mass) of every row in 32 bits, and whether the step exists."""
    aa, at, ln = _padded(d, rows)
    on = ((d.mask[rows][:, None] >> at) & 1).bool()
    a = aa.clamp(min=0)
    tab = lambda t: _table(t, torch.float32).to(DEV)[a]  # noqa: E731
    res = tab(MONO) + torch.where(on, tab(var), tab(STATIC))
    b, y = torch.zeros(len(rows), device=DEV), d.mass32[rows].clone()
    for k in range(MAX_LEN - 1):
        b, y = b + res[:, k], y - res[:, k]
        yield k, b, y, k + 1 < ln[:, 0]


def _exact_search(case, sp):
    p = _params(case)
    _, d = _index(case["index"])
    var = INDEXES[case["index"]][1]
    n, f64 = len(sp.scan), torch.float64
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
    off = up(sp.offsets)
    mz, it = up(sp.mz), up(sp.intensity)
    spec = torch.repeat_interleave(torch.arange(n, device=DEV), off[1:] - off[:-1])
    ok = (mz >= p.fragment_min_mz) & (mz <= p.fragment_max_mz)
    spec, mass, it = spec[ok], mz[ok] - PROTON, it[ok]
    o = torch.argsort(mass, descending=True, stable=True)
    o = o[torch.argsort(it[o], descending=True, stable=True)]
    wide = p.peak_mode == "window"   # the top peaks of every window instead of the whole spectrum
    group = spec * 1000 + (mz[ok] * (1.0 / p.window_th)).long() if wide else spec
    o = o[torch.argsort(group[o], stable=True)]
    first = torch.searchsorted(group[o], group[o])
    o = o[torch.arange(len(o), device=DEV) - first < (p.window_k if wide else p.max_peaks)]
    o = o[torch.argsort(mass[o], stable=True)]
    o = o[torch.argsort(spec[o], stable=True)]
    spec, mass, it = spec[o], mass[o], it[o]
    first = torch.searchsorted(spec, torch.arange(n + 1, device=DEV))
    tic = torch.zeros(n, dtype=f64, device=DEV).index_add_(0, spec, it.double())
    valid = (first[1:] - first[:-1]) >= p.min_peaks
    # hypotheses, in (spectrum, charge, isotope) order
    pm0, charge = up(sp.precursor_mz).float() - PROTON, up(sp.charge).long()
    cols = [(z, i) for z in range(1, 8) for i in range(p.isotope_errors[0], p.isotope_errors[1] + 1)]
    hs = torch.arange(n, device=DEV).repeat_interleave(len(cols))
    hz = torch.tensor([c[0] for c in cols], device=DEV).repeat(n)
    hi_ = torch.tensor([c[1] for c in cols], device=DEV).repeat(n)
    known = charge[hs] > 0
    use = valid[hs] & torch.where(known, hz == charge[hs],
                                  (hz >= p.precursor_charge[0]) & (hz <= p.precursor_charge[1]))
    hs, hz, hi_ = hs[use], hz[use], hi_[use]
    pm = pm0[hs] * hz.float()
    ie = hi_.float() * NEUTRON
    M = pm - ie
    mfc = p.max_fragment_charge or 0
    mfz = (hz.clamp(max=mfc + 1) if mfc else hz).clamp(min=2)   # fragment charges 1 .. mfz - 1
    lo = torch.searchsorted(d.mass32, M + (M * p.precursor_ppm[0]) / 1e6)
    hi = torch.searchsorted(d.mass32, M + (M * p.precursor_ppm[1]) / 1e6, right=True)
    # shared-peak counts of every window row, keeping those over the threshold
    lift = lambda s, x: s.to(f64) * 8192.0 + x.to(f64)  # noqa: E731  (exact: 32-bit masses under 8192)
    edges = {z: [lift(spec, x) for x in _bounds(mass * z, p)] for z in range(1, int(mfz.max()))}
    csum = torch.cat([torch.zeros(1, dtype=f64, device=DEV), torch.cumsum(it.double(), 0)])

    def peaks_at(h, m, z):
        """First and one past the last of the peaks whose window (at fragment charge z) holds mass m."""
        ka, kb = edges[z]
        q = lift(hs[h], m)
        return torch.searchsorted(kb, q), torch.searchsorted(ka, q, right=True)

    def counted(h, r):
        """(peak range, whether it counts) of every fragment of rows r that the index holds."""
        ln = d.length[r].long()
        for k, b, y, there in _ladder(d, var, r):
            for m, far in ((b, k + 1 > p.min_ion_index), (y, ln - 1 - k > p.min_ion_index)):
                t = there & far & (m >= p.fragment_min_mz) & (m <= p.fragment_max_mz)
                for z in edges:
                    yield peaks_at(h, m, z), t & (z < mfz[h])

    scored = torch.zeros(n, dtype=f64, device=DEV)
    matched = torch.zeros(n, dtype=f64, device=DEV)
    keep = []
    step, ends = 1_500_000, torch.cumsum(hi - lo, 0).cpu().numpy()
    i = 0
    while i < len(hs):
        j = max(i + 1, int(np.searchsorted(ends, (ends[i - 1] if i else 0) + step, side="right")))
        h, r = _ranges(lo[i:j], (hi - lo)[i:j])
        h = h + i
        c = torch.zeros(len(r), dtype=torch.int64, device=DEV)
        for (j0, j1), t in counted(h, r):
            c += torch.where(t, j1 - j0, 0)
        scored.index_add_(0, hs[h], (c > 0).to(f64))
        matched.index_add_(0, hs[h], c.to(f64))
        t = c >= p.k1_threshold
        keep.append((h[t], r[t], c[t]))
        i = j
    h, r, c = (torch.cat(x) for x in zip(*keep))
    o = torch.argsort(h, stable=True)
    o = o[torch.argsort(r[o], descending=True, stable=True)]
    o = o[torch.argsort(c[o], descending=True, stable=True)]
    o = o[torch.argsort(hs[h[o]], stable=True)]
    at = torch.searchsorted(hs[h[o]], torch.arange(n, device=DEV))
    o = o[torch.arange(len(o), device=DEV) - at[hs[h[o]]] < p.topk]
    h, r, c = h[o], r[o], c[o]
    if case["call"] == "collect":   # the hits' features: count, share of the TIC, ppm, charge, length, missed sites
        o = torch.argsort(h, stable=True)
        o = o[torch.argsort((hs[h] * (1 << 28) + r)[o], stable=True)]
        h, r, c = h[o], r[o], c[o]
        share = torch.zeros(len(r), dtype=f64, device=DEV)
        for (j0, j1), t in counted(h, r):
            share += torch.where(t, csum[j1] - csum[j0], 0)
        calc = d.mass32[r].to(f64)
        feat = torch.zeros(len(r), 16, dtype=f64, device=DEV)
        feat[:, :6] = torch.stack([c.to(f64), share / tic[hs[h]], (M[h].to(f64) - calc) / calc * 1e6, hz[h].to(f64),
                                   d.length[r].to(f64), d.missed[r].to(f64)], 1)
        return {"feat": _pad(feat, n * p.topk)}
    h, r = torch.cat([h, h]), torch.cat([r, d.partner[r]])
    o = torch.argsort(h, stable=True)
    o = o[torch.argsort((hs[h] * (1 << 28) + r)[o], stable=True)]
    h, r = h[o], r[o]
    new = torch.ones(len(h), dtype=torch.bool, device=DEV)
    new[1:] = (hs[h][1:] != hs[h][:-1]) | (r[1:] != r[:-1])
    h, r = h[new], r[new]
    # rescoring: the most intense peak of each ion's window (the last of equals)
    n_c = len(h)
    tot = {k: torch.zeros(n_c, dtype=f64, device=DEV) for k in ("b", "y", "ppm", "nb", "ny", "ly", "run")}
    km = lift(spec, mass)
    for k, b, y, there in _ladder(d, var, r):
        for kind, mass_k in (("b", b), ("y", y)):
            any_hit = torch.zeros(n_c, dtype=torch.bool, device=DEV)
            for z in edges:
                m = mass_k / z
                wa, wb = _bounds(m, p)
                j0, j1 = torch.searchsorted(km, lift(hs[h], wa)), torch.searchsorted(km, lift(hs[h], wb), right=True)
                j1 = torch.where(there & (z < mfz[h]), j1, j0)
                best = torch.full_like(j0, -1)
                top = torch.zeros(n_c, device=DEV)
                for t in range(int((j1 - j0).max())):
                    v = torch.where(j0 + t < j1, it[(j0 + t).clamp(max=len(it) - 1)], -1.0)
                    best, top = torch.where(v >= top, j0 + t, best), torch.maximum(v, top)
                hit = best >= 0
                x, g = it[best.clamp(min=0)].to(f64), mass[best.clamp(min=0)].to(f64)
                tot[kind] += torch.where(hit, x, 0)
                tot["n" + kind] += hit
                tot["ppm"] += torch.where(hit, x * (m.to(f64) - g).abs() * 2e6 / (m.to(f64) + g), 0)
                any_hit |= hit
            if kind == "y":
                tot["run"] = torch.where(any_hit, tot["run"] + 1, 0) if k else tot["run"]   # Sage's: not ion 0
                tot["ly"] = torch.maximum(tot["ly"], tot["run"])

    def lnfact(x):
        s = x.clamp(min=1)
        return torch.where(x == 0, 1.0, s * s.log() - s + 0.5 * s.log() + 0.5 * (2 * math.pi * s).log())
    score = ((tot["b"] + 1) * (tot["y"] + 1)).log() + lnfact(tot["nb"]) + lnfact(tot["ny"])
    ok = tot["nb"] + tot["ny"] >= p.min_matched_peaks
    idx = torch.nonzero(ok)[:, 0]
    o = idx[torch.argsort(score[idx], descending=True, stable=True)]   # rows ascend within a spectrum already
    o = o[torch.argsort(hs[h[o]], stable=True)]
    s = hs[h[o]]
    lead = torch.ones(len(s), dtype=torch.bool, device=DEV)
    lead[1:] = s[1:] != s[:-1]
    nxt = torch.cat([score[o][1:], torch.zeros(1, dtype=f64, device=DEV)])
    nxt = torch.where(torch.cat([lead[1:], torch.ones(1, dtype=torch.bool, device=DEV)]), 0.0, nxt)[lead]
    w, s = o[lead], s[lead]
    hh, rr = h[w], r[w]
    e, calc, shift = pm[hh].to(f64), d.mass32[rr].to(f64), ie[hh].to(f64)
    kk, lam = tot["nb"][w] + tot["ny"][w], matched[s] / scored[s]
    total = tot["b"][w] + tot["y"][w]
    out = {"expmass": e, "calcmass": calc, "delta_mass_ppm": (e - calc - shift).abs() * 2e6 / (e - shift + calc),
           "hyperscore": score[w], "delta_next": score[w] - nxt, "delta_best": torch.zeros_like(e),
           "summed_intensity": total, "matched_intensity_pct": 100 * total / tic[s],
           "average_ppm": tot["ppm"][w] / total, "longest_y_pct": tot["ly"][w] / d.length[rr].to(f64),
           "poisson": (kk * lam.log() - lam - lnfact(kk)) / math.log(10.0),
           "rt": up(sp.rt)[s]}
    return {k: np.pad(v.cpu().numpy(), (0, n - len(s))) for k, v in out.items()}


def _exact_fit(case, seed):
    x, y, w = _fit_inputs(case, seed)
    f64, names = torch.float64, ("W1", "b1", "W2", "b2", "w3", "b3")
    x, y = x.to(f64), y.to(f64)
    w = {k: w[k].to(DEV, f64) for k in names}
    m, v = ({k: torch.zeros_like(w[k]) for k in names} for _ in range(2))
    short = lambda t: t.to(torch.bfloat16).to(f64)  # noqa: E731  (the network's own 16-bit weights and activations)
    g = torch.Generator(device=DEV).manual_seed(3)
    perm = torch.randperm(len(y), generator=g, device=DEV)
    size = min(case["batch"], len(y))
    steps, loss = len(y) // size, 0.0
    for i in range(steps):
        at = perm[i * size:(i + 1) * size]
        xb, yb, w1, w2 = x[at], y[at], short(w["W1"]), short(w["W2"])
        h1 = short((xb @ w1.T + w["b1"]).clamp(min=0))
        h2 = (h1 @ w2.T + w["b2"]).clamp(min=0)
        z = h2 @ w["w3"] + w["b3"]
        loss += float((torch.nn.functional.softplus(z) - z * yb).sum()) / size
        dz = (torch.sigmoid(z) - yb) / size
        d2 = dz[:, None] * w["w3"] * (h2 > 0)
        d1 = (d2 @ w2) * (h1 > 0)
        grad = {"w3": h2.T @ dz, "b3": dz.sum()[None], "W2": d2.T @ h1, "b2": d2.sum(0), "W1": d1.T @ xb,
                "b1": d1.sum(0)}
        lr = 2e-3 * 0.5 * (1.0 + math.cos(math.pi * i / steps))
        for k in names:
            m[k] = 0.9 * m[k] + 0.1 * grad[k]
            v[k] = 0.999 * v[k] + 0.001 * grad[k] ** 2
            w[k] = w[k] - lr * (m[k] / (1 - 0.9 ** (i + 1))) / ((v[k] / (1 - 0.999 ** (i + 1))).sqrt() + 1e-8)
    return {"loss": loss / steps, **w}
