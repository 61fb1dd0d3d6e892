"""The work users of the engine have it do, as timed cases.

Profiles and proteins are synthetic, with the shapes of the benchmark
configurations (sentinel-x_b200/sxhmm/synth.py): match emissions Dirichlet over
the BLOSUM62 background, Dirichlet transitions, background proteins with
planted homologs, STATS calibrated on the device by simulation.  Lengths are
the quantiles of their distributions in a seeded order, so the work of a case
does not depend on the seed.

Kinds of case:
  search  every profile x every target through Engine.search: filters, rows,
          domain definition, report.  `upload` makes the target set from host
          residues in the pass, as a caller streaming batches of proteins does;
          otherwise the set stays on the device.  `filters` False is
          hmmsearch --max.
  many    single-profile sets against one target set, Engine.search_many
  score   stage scores of explicit pairs, Engine.score_pairs
  grad    lnZ and its gradients for explicit pairs, Engine.posterior_grad
"""
import functools
import math
import os
import sys
from statistics import NormalDist

import numpy as np
import torch

# the engine drives up to 31 streams; hardware queues for all of them
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")
sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sentinel-x_b200"))

import sxhmm  # noqa: E402
from sxhmm import _capi, synth  # noqa: E402

STAR, NSYM = 24, 25
MEMBERS = {20: (2, 11), 21: (7, 9), 22: (3, 13), 23: tuple(range(20))}  # B J Z X


def _search(name, profiles, m_lo, m_hi, m_med, targets, l_lo, l_hi, l_med, planted, cutoff="evalue", filters=True,
            upload=False, domains=1):
    return {"name": name, "kind": "search", "profiles": profiles, "m_lo": m_lo, "m_hi": m_hi, "m_med": m_med,
            "targets": targets, "l_lo": l_lo, "l_hi": l_hi, "l_med": l_med, "planted": planted, "domains": domains,
            "cutoff": cutoff, "filters": filters, "upload": upload}


def listed():
    """Medians of 0 mean uniform lengths between the bounds."""
    return [
        # one profile against a small proteome that stays loaded: the plain hmmsearch call, the smallest
        _search("search_single", 1, 100, 100, 0, 1000, 100, 500, 0, 0.05),
        # a handful of short and mid profiles against a few hundred freshly called proteins
        _search("search_ragged", 13, 20, 333, 0, 777, 30, 900, 250, 0.03, upload=True),
        # marker-set completeness (BUSCO, EukCC): 250 markers against one genome's proteins, gathering cutoffs
        _search("search_markers", 250, 200, 1500, 0, 4000, 30, 4000, 280, 0.06, cutoff="ga", upload=True),
        # viral screen (CheckV): many profiles against short viral proteins
        _search("search_viral", 800, 30, 800, 180, 20000, 40, 1500, 150, 0.01, upload=True),
        # Pfam-scale annotation, the headline workload and the largest
        _search("search_pfam", 1000, 20, 1000, 150, 50000, 30, 3000, 300, 0.02, upload=True),
        # hmmsearch --max over multi-domain homologs: every pair reaches domain definition
        _search("search_max", 4, 300, 300, 0, 512, 400, 400, 0, 0.75, cutoff="bits", filters=False, domains=3),
        # models of long proteins, past the 2048 columns the batched kernels hold
        _search("search_long", 2, 2100, 2500, 0, 300, 60, 3000, 350, 0.03),
        # BUSCO's one search per marker file, batched
        {"name": "search_many", "kind": "many", "profiles": 64, "m_lo": 60, "m_hi": 700, "m_med": 250,
         "targets": 3000, "l_lo": 30, "l_hi": 2500, "l_med": 280, "planted": 0.02, "domains": 1},
        # calibration: every stage's score of random L = 100 sequences against each new profile
        {"name": "score_calibrate", "kind": "score", "profiles": 40, "m_lo": 30, "m_hi": 300, "m_med": 150,
         "targets": 200, "l_lo": 100, "l_hi": 100, "l_med": 0, "planted": 0.0, "domains": 1, "pairs": 8000},
        # rescoring a list of hits: mixed lengths, homologs among them
        {"name": "score_hits", "kind": "score", "profiles": 41, "m_lo": 33, "m_hi": 650, "m_med": 200,
         "targets": 501, "l_lo": 40, "l_hi": 1200, "l_med": 300, "planted": 0.6, "domains": 1, "pairs": 501},
        # profile training steps: expected counts of every emission and transition, a small and a full batch
        {"name": "grad_small", "kind": "grad", "profiles": 3, "m_lo": 121, "m_hi": 121, "m_med": 0,
         "targets": 37, "l_lo": 90, "l_hi": 400, "l_med": 0, "planted": 0.8, "domains": 1, "pairs": 37},
        {"name": "grad_batch", "kind": "grad", "profiles": 16, "m_lo": 300, "m_hi": 300, "m_med": 0,
         "targets": 4096, "l_lo": 400, "l_hi": 400, "l_med": 0, "planted": 0.75, "domains": 3, "pairs": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search"] * 5 + ["max", "long", "many", "score", "score", "grad", "grad"])
    if kind == "search":
        m_lo, l_lo = rng.choice([20, 30, 101, 200]), rng.choice([30, 41, 100])
        m_hi, l_hi = rng.choice([333, 800, 1000, 1500]), rng.choice([500, 1500, 3000, 4000])
        m_med, l_med = rng.choice([0, 150, 180, 249]) if m_lo < 150 else 0, rng.choice([150, 233, 280, 300])
        c = _search("", _log_int(rng, 1, 500), m_lo, m_hi, m_med, _log_int(rng, 100, 20000), l_lo, l_hi, l_med,
                    rng.choice([0.01, 0.02, 0.05]), cutoff=rng.choice(["evalue", "evalue", "ga", "bits"]),
                    upload=rng.random() < 0.6)
        cells = c["profiles"] * _mean(m_lo, m_hi, m_med) * c["targets"] * _mean(l_lo, l_hi, l_med)
        if cells > 1.0e12:
            c["targets"] = max(100, int(c["targets"] * 1.0e12 / cells))
    elif kind == "max":
        m = _log_int(rng, 40, 400)
        c = _search("", rng.randint(1, 4), m, m, 0, _log_int(rng, 20, 400), 60, 450, 0, 0.5, cutoff="bits",
                    filters=False, domains=rng.randint(1, 3))
    elif kind == "long":
        m = rng.randint(2049, 2500)
        c = _search("", rng.randint(1, 2), m, m + 37, 0, _log_int(rng, 40, 250), 60, 1500, 300, 0.02)
    elif kind == "many":
        c = {"kind": "many", "profiles": _log_int(rng, 3, 100), "m_lo": 60, "m_hi": rng.choice([433, 700]), "m_med": 0,
             "targets": _log_int(rng, 200, 3000), "l_lo": 30, "l_hi": 2000, "l_med": 280, "planted": 0.02, "domains": 1}
    elif kind == "score":
        n = _log_int(rng, 5, 4000)
        c = {"kind": "score", "profiles": rng.randint(1, 40), "m_lo": rng.choice([1, 20, 65]),
             "m_hi": rng.choice([129, 400, 650]), "m_med": 0, "targets": max(1, n // 4), "l_lo": rng.choice([1, 50]),
             "l_hi": rng.choice([100, 400, 700]), "l_med": 0, "planted": rng.choice([0.0, 0.5]), "domains": 1,
             "pairs": n}
    else:
        m, n = _log_int(rng, 20, 400), _log_int(rng, 4, 1500)
        c = {"kind": "grad", "profiles": rng.randint(1, 16), "m_lo": m, "m_hi": m, "m_med": 0, "targets": n,
             "l_lo": 50, "l_hi": rng.choice([200, 401, 600]), "l_med": 0, "planted": 0.7,
             "domains": rng.randint(1, 2), "pairs": n}
    c.pop("name", None)
    return c


# ---- inputs --------------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _quantiles(n, lo, hi, median):
    """n lengths at the quantiles of the distribution: uniform, or log-normal clipped to [lo, hi]."""
    q = (np.arange(n) + 0.5) / n
    if median == 0:
        return np.minimum(lo + np.floor(q * (hi - lo + 1)), hi).astype(np.int64)
    z = NormalDist()
    sigma = synth.SIGMA_M if median < 200 else synth.SIGMA_L
    v = [math.exp(math.log(median) + sigma * z.inv_cdf(x)) for x in q]
    return np.clip(np.rint(v), lo, hi).astype(np.int64)


def _mean(lo, hi, median):
    return float(_quantiles(257, lo, hi, median).mean())


def _lengths(case):
    return (_quantiles(case["profiles"], case["m_lo"], case["m_hi"], case["m_med"]),
            _quantiles(case["targets"], case["l_lo"], case["l_hi"], case["l_med"]))


class Models:
    """Probability-space models in flat arrays: profile i has rows
    start[i] .. start[i] + M (nodes 0..M) of mat [rows, 20] and t [rows, 7]."""

    def __init__(self, ms, rng):
        self.ms = ms
        self.start = np.concatenate([[0], np.cumsum(ms + 1)]).astype(np.int64)
        rows = int(self.start[-1])
        g = rng.standard_gamma(0.5 * synth.BLOSUM_BG, (rows, 20))
        g = np.maximum(g / np.maximum(g.sum(1, keepdims=True), 1e-300), 1e-30)
        self.mat = g / g.sum(1, keepdims=True)
        c = synth.CONC

        def dirichlet(*alpha):
            v = np.maximum(rng.standard_gamma(c * np.array(alpha), (rows, len(alpha))), 1e-30)
            return v / v.sum(1, keepdims=True)
        self.t = np.concatenate([dirichlet(0.9, 0.05, 0.05), dirichlet(0.6, 0.4), dirichlet(0.6, 0.4)], axis=1)
        first, last = self.start[:-1], self.start[1:] - 1
        self.t[first, 5], self.t[first, 6] = 1.0, 0.0
        mm_mi = self.t[last, 0] + self.t[last, 1]
        self.t[last, 0] /= mm_mi
        self.t[last, 1] /= mm_mi
        self.t[last, 2], self.t[last, 5], self.t[last, 6] = 0.0, 1.0, 0.0

    def homologs(self, which, rng):
        """Residues of one local path through each of the profiles `which`:
        entry in the first tenth of the nodes, exit in the last tenth."""
        n = len(which)
        m, base = self.ms[which], self.start[which]
        k = 1 + (rng.random(n) * np.maximum(1, m // 10)).astype(np.int64)
        kend = np.maximum(k, m - (rng.random(n) * (np.minimum(m // 10, m - 1) + 1)).astype(np.int64))
        state = np.zeros(n, np.int8)  # 0 match, 1 insert, 2 delete
        out = np.zeros((n, 3 * int(m.max()) + 100), np.uint8)
        pos = np.zeros(n, np.int64)
        live = np.arange(n)
        bg = np.cumsum(synth.BG / synth.BG.sum())
        while len(live):
            s, row = state[live], base[live] + k[live]
            u, v = rng.random(len(live)), rng.random(len(live))
            match = (np.cumsum(self.mat[row], axis=1) < u[:, None]).sum(1)
            res = np.minimum(np.where(s == 0, match, np.searchsorted(bg, u)), 19)
            emits = s != 2
            out[live[emits], pos[live[emits]]] = res[emits]
            pos[live[emits]] += 1
            t = self.t[row]
            to_m = np.where(s == 0, t[:, 0], np.where(s == 1, t[:, 3], t[:, 5]))
            nxt = np.where(v < to_m, 0, np.where(s == 0, np.where(v < t[:, 0] + t[:, 1], 1, 2), s))
            go = (k[live] < kend[live]) & (pos[live] < out.shape[1])
            live, nxt = live[go], nxt[go]
            state[live] = nxt
            k[live] += nxt != 1
        return [out[i, :pos[i]] for i in range(n)]

    def arrays(self, cutoffs=True):
        """Configured profiles, as Engine.load_arrays takes them."""
        n, w = len(self.ms), int(self.ms.max()) + 1
        rows = len(self.mat)
        bg = synth.BG.astype(np.float32).astype(np.float64)
        sc = np.full((rows, NSYM), -np.inf, np.float32)
        sc[:, :20] = np.log(self.mat / bg)
        for code, members in MEMBERS.items():
            b = bg[list(members)]
            sc[:, code] = (sc[:, list(members)].astype(np.float64) * b).sum(1) / b.sum()
        occ = np.zeros((n, w))
        node = lambda k: np.minimum(self.start[:-1] + k, rows - 1)  # noqa: E731
        t0 = self.t[node(0)]
        occ[:, 1] = t0[:, 0] + t0[:, 1]
        for k in range(2, w):
            t = self.t[node(k - 1)]
            occ[:, k] = np.where(k <= self.ms, occ[:, k - 1] * (t[:, 0] + t[:, 1]) + (1 - occ[:, k - 1]) * t[:, 5], 0)
        out = []
        with np.errstate(divide="ignore"):
            lt = np.log(self.t).astype(np.float32)
        for i, m in enumerate(self.ms):
            m, a = int(m), int(self.start[i])
            msc = np.ascontiguousarray(sc[a:a + m + 1].T)
            msc[:, 0] = -np.inf
            t = np.full((8, m + 1), -np.inf, np.float32)
            t[:7, 1:m] = lt[a + 1:a + m].T
            t[5:7, min(1, m)] = -np.inf
            o = occ[i, 1:m + 1]
            t[7, 1:] = np.log(o / (o * np.arange(m, 0, -1)).sum())
            compo = (o[:, None] * self.mat[a + 1:a + m + 1]).sum(0)
            p = {"name": f"p{i}", "m": m, "msc": msc, "mo": np.exp(msc), "t": t, "p": np.exp(t),
                 "compo": (compo / compo.sum()).astype(np.float32), "msv_tbm": np.float32(math.log(2.0 / (m * (m + 1.0))))}
            if cutoffs:
                p.update(ga=(25.0, 20.0), tc=(30.0, 25.0), nc=(20.0, 15.0))
            out.append(p)
        return out


def _residues(n, rng):
    """n background residues (frequencies to 2^-16)."""
    edges = np.rint(np.cumsum(synth.BG / synth.BG.sum()) * 65536).astype(np.int64)
    lut = np.searchsorted(edges, np.arange(65536), side="right").clip(0, 19).astype(np.uint8)
    return lut[rng.integers(0, 65536, n, dtype=np.uint16)]


def _inputs(case, seed):
    """Configured profiles, packed targets (residues, offsets, lengths) and, for explicit pairs, their indices."""
    rng = np.random.default_rng([seed, 20260])
    ms, lens = _lengths(case)
    ms, lens = rng.permutation(ms), rng.permutation(lens)
    models = Models(ms, rng)
    carriers = rng.choice(len(lens), size=int(round(case["planted"] * len(lens))), replace=False)
    if case["kind"] in ("score", "grad"):
        # every target's first pair is the profile its homologs come from
        own = np.arange(len(lens)) % len(ms)
    else:
        own = rng.integers(0, len(ms), len(lens))
    copies = rng.integers(1, case["domains"] + 1, len(carriers))
    doms = models.homologs(np.repeat(own[carriers], copies), rng) if len(carriers) else []
    lens, at, placed = lens.copy(), 0, []
    for t, c in zip(carriers, copies):
        ds = doms[at:at + c]
        at += c
        need = sum(map(len, ds))
        lens[t] = max(lens[t], need + c)
        cuts = np.sort(rng.integers(0, lens[t] - need + 1, c))
        placed.append((t, cuts, ds))
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.int64)
    seq = _residues(int(lens.sum()), rng)
    for t, cuts, ds in placed:
        o = offs[t]
        for c, d in zip(cuts, ds):
            seq[o + c:o + c + len(d)] = d
            o += len(d)
    pairs = None
    if case["kind"] in ("score", "grad"):
        k = np.arange(case["pairs"])
        pt = (k % len(lens)).astype(np.int32)
        pp = ((own[pt] + k // len(lens)) % len(ms)).astype(np.int32)
        pairs = (pp, pt)
    return models.arrays(), (seq, offs, lens), pairs


def _calibrate(engine, profiles, rng, n=100, length=100):
    """STATS by simulation: Gumbel fits of the stage scores of random sequences."""
    seqs = _residues(n * length, rng)
    ps = engine.load_arrays(profiles)
    ts = engine.targets_digital(seqs, np.arange(n) * length, np.full(n, length))
    pp, pt = np.repeat(np.arange(len(profiles)), n), np.tile(np.arange(n), len(profiles))
    sc = engine.score_pairs(ps, ts, pp, pt, stages=("msv", "viterbi", "forward"))
    ps.close()
    ts.close()
    null = length * math.log(length / (length + 1.0)) - math.log(length + 1.0)
    lam = synth.LN2
    tau = (math.log(0.04) - math.log(-math.log(0.96))) / lam
    mu = {s: [synth.gumbel_mu_known_lambda((row - null) / lam, lam)
              for row in v.astype(np.float64).reshape(len(profiles), n)] for s, v in sc.items()}
    for i, p in enumerate(profiles):
        p.update(msv=(mu["msv"][i], lam), viterbi=(mu["viterbi"][i], lam), forward=(mu["forward"][i] + tau, lam))


@functools.lru_cache(maxsize=1)
def _engine():
    return sxhmm.default_engine()


def prepare(case, seed):
    """Profile sets on the device; targets on the device, or in host memory where each pass uploads them."""
    eng = _engine()
    profiles, targets, pairs = _inputs(case, seed)
    state = {"engine": eng, "case": case}
    if case["kind"] in ("search", "many"):
        if case.get("filters", True):
            _calibrate(eng, profiles, np.random.default_rng([seed, 7]))
        cut = {"evalue": sxhmm.Cutoff.evalue(), "ga": sxhmm.Cutoff.gathering(),
               "bits": sxhmm.Cutoff.bits(0.0, 0.0)}[case.get("cutoff", "evalue")]
        state["cfg"] = sxhmm.SearchConfig(cut, sxhmm.PipelineConfig(filters=case.get("filters", True))).to_c()
    if case["kind"] == "many":
        state["sets"] = [eng.load_arrays([p]) for p in profiles]
    else:
        state["profiles"] = eng.load_arrays(profiles)
    if case.get("upload"):
        state["host"] = targets
    else:
        state["targets"] = eng.targets_digital(*targets)
    state["pairs"] = pairs
    if case["kind"] == "grad":  # gradient buffers that a training loop keeps
        n, w = case["pairs"], case["m_lo"] + 1
        state["out"] = (np.zeros(n), np.zeros((n, 25, w), np.float32), np.zeros((n, 25, w), np.float32),
                        np.zeros((n, 8, w), np.float32))
    return state


def _table(records, kind, rows):
    """ctypes records as one array per field, in a table of `rows` rows (how many are found varies with the inputs)."""
    a = np.zeros(rows, np.dtype(kind))
    if len(records) > rows:
        raise ValueError(f"{len(records)} records for a table of {rows}")
    if records:
        a[:len(records)] = np.frombuffer((kind * len(records))(*records), dtype=a.dtype)
    return {f: a[f] for f in a.dtype.names if f != "reserved"}


def _found(case, hits, doms):
    rows = 1024 + 12 * case["profiles"] + int(4 * case["planted"] * case["targets"])
    if not case.get("filters", True):
        rows = case["profiles"] * case["targets"]
    return {"n": np.array([len(hits), len(doms)]), "hits": _table(hits, _capi.SxHit, rows),
            "domains": _table(doms, _capi.SxDomain, 8 * rows)}


def run(state):
    case, eng = state["case"], state["engine"]
    if case["kind"] == "search":
        ts = eng.targets_digital(*state["host"]) if case["upload"] else state["targets"]
        found = eng.search(state["profiles"], ts, state["cfg"])
        if case["upload"]:
            ts.close()
        return _found(case, *found)
    if case["kind"] == "many":
        got = eng.search_many(state["sets"], state["targets"], state["cfg"])
        out = _found(case, [h for hits, _ in got for h in hits], [d for _, doms in got for d in doms])
        out["per_set"] = np.array([len(hits) for hits, _ in got])
        return out
    pp, pt = state["pairs"]
    if case["kind"] == "score":
        return eng.score_pairs(state["profiles"], state["targets"], pp, pt)
    return dict(zip(("lnz", "d_msc", "d_isc", "d_trans"),
                    eng.posterior_grad(state["profiles"], state["targets"], pp, pt, case["m_lo"], out=state["out"])))


def work(case):
    """Lane operations of the recurrences (MSV 3 a cell, Viterbi 16, Forward 12, Backward 14, counts 20) over the
    cells that cannot be skipped: every pair's MSV in a filtered search, Forward and Backward of every pair in an
    unfiltered one.  Bytes: residues, the profiles' scores, the results."""
    ms, lens = _lengths(case)
    profile_bytes = float((25 + 8) * 4 * (ms + 1).sum())
    if case["kind"] in ("search", "many"):
        cells = float(ms.sum()) * float(lens.sum())
        ops = 3 if case.get("filters", True) else 26
        hits = case["planted"] * len(lens) if ops == 3 else len(ms) * len(lens)
        return {"bytes": float(lens.sum()) + profile_bytes + 100 * hits, "flops": ops * cells}
    cells = case["pairs"] * float(ms.mean()) * float(lens.mean())
    if case["kind"] == "score":
        return {"bytes": float(lens.sum()) + profile_bytes + 20 * case["pairs"], "flops": 45 * cells}
    w = case["m_lo"] + 1
    return {"bytes": float(lens.sum()) + profile_bytes + case["pairs"] * (8 + 58 * 4 * w), "flops": 46 * cells}


# ---- 64-bit values ---------------------------------------------------------------
class Batch:
    """Padded 64-bit tensors of explicit pairs; rows step through every pair at once."""

    def __init__(self, case, seed):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        profiles, (seq, offs, lens), (pp, pt) = _inputs(case, seed)
        w = max(p["m"] for p in profiles) + 1
        f64 = dict(dtype=torch.float64, device=dev)

        def stack(key, rows, pad):
            a = np.full((len(profiles), rows, w), pad)
            for i, p in enumerate(profiles):
                a[i, :, :p["m"] + 1] = p[key]
            return torch.tensor(a, **f64)
        self.pp, self.pt = torch.tensor(pp, device=dev).long(), torch.tensor(pt, device=dev).long()
        self.msc, self.mo = stack("msc", NSYM, -np.inf), stack("mo", NSYM, 0.0)
        self.t, self.p = stack("t", 8, -np.inf)[self.pp], stack("p", 8, 0.0)[self.pp]
        self.m = torch.tensor([p["m"] for p in profiles], device=dev)[self.pp]
        self.tbm = torch.tensor([float(p["msv_tbm"]) for p in profiles], **f64)[self.pp]
        self.compo = torch.tensor(np.array([p["compo"] for p in profiles]), **f64)[self.pp]
        self.len = torch.tensor(lens, device=dev)[self.pt]
        self.rows = int(lens[pt].max())
        dsq = np.full((len(lens), int(lens.max())), STAR, np.uint8)
        for i, (o, n) in enumerate(zip(offs, lens)):
            dsq[i, :n] = seq[o:o + n]
        self.x = torch.tensor(dsq, device=dev).long()[self.pt]
        k = torch.arange(w, device=dev)
        self.col = (k >= 1) & (k <= self.m[:, None])      # columns 1..M
        self.ins = (k >= 1) & (k < self.m[:, None])       # insert columns 1..M-1
        self.k, self.w, self.n, self.dev, self.f64 = k, w, len(pp), dev, f64


def _shift(v, fill):
    return torch.cat([torch.full_like(v[:, :1], fill), v[:, :-1]], dim=1)


def _exact_scores(b):
    neg = -math.inf
    L = b.len.double()
    out = {}
    # MSV
    loop, move, ln2 = torch.log(L / (L + 3)), torch.log(3 / (L + 3)), math.log(2.0)
    prev = torch.full((b.n, b.w), neg, **b.f64)
    xj, final = torch.full((b.n,), neg, **b.f64), torch.full((b.n,), neg, **b.f64)
    xb = move.clone()
    for i in range(b.rows):
        prev = b.msc[b.pp, b.x[:, i]] + torch.maximum(_shift(prev, neg), (xb + b.tbm)[:, None])
        prev = prev.masked_fill(~b.col, neg)
        xj = torch.maximum(xj + loop, prev.amax(1) - ln2)
        xb = torch.maximum((i + 1) * loop, xj) + move
        final = torch.where(b.len == i + 1, xj + move, final)
    out["msv"] = final
    # Viterbi; D by prefix sums: D[k] = cum[k] + max_j (a_j - cum[j])
    mm, mi, md, im, ii, dm, dd, bm = (b.t[:, q] for q in range(8))
    ddl = torch.nan_to_num(_shift(dd, 0.0), neginf=0.0)
    cum = torch.cumsum(ddl, 1)
    m = i_ = d = torch.full((b.n, b.w), neg, **b.f64)
    xj, final = torch.full((b.n,), neg, **b.f64), torch.full((b.n,), neg, **b.f64)
    xb = move.clone()
    for i in range(b.rows):
        best = torch.maximum(torch.maximum(_shift(m + mm, neg), _shift(i_ + im, neg)),
                             torch.maximum(_shift(d + dm, neg), xb[:, None] + bm))
        m2 = (best + b.msc[b.pp, b.x[:, i]]).masked_fill(~b.col, neg)
        i_ = torch.maximum(m + mi, i_ + ii).masked_fill(~b.ins, neg)
        m = m2
        d = (torch.cummax(_shift(m + md, neg) - cum, 1).values + cum).masked_fill(~b.col, neg)
        xj = torch.maximum(xj + loop, torch.maximum(m, d).amax(1) - ln2)
        xb = torch.maximum((i + 1) * loop, xj) + move
        final = torch.where(b.len == i + 1, xj + move, final)
    out["viterbi"] = final
    out["forward"] = out["backward"] = _log_z(b, b.p, lambda i: b.mo[b.pp, b.x[:, i]], lambda i: 1.0)
    # composition bias: a two-state filter
    e1 = torch.ones((b.n, NSYM), **b.f64)
    bg = torch.tensor(synth.BG.astype(np.float32), **b.f64)
    e1[:, :20] = b.compo / bg
    l1 = b.m.double() / 8
    t00, t01, t10, t11 = 400 / 401, 1 / 401, 1 / (l1 + 1), l1 / (l1 + 1)
    take = lambda i: e1.gather(1, b.x[:, i:i + 1])[:, 0]  # noqa: E731
    d0, d1 = torch.full((b.n,), 0.999, **b.f64), 0.001 * take(0)
    logs = torch.zeros(b.n, **b.f64)
    for i in range(b.rows):
        if i:
            d0, d1 = d0 * t00 + d1 * t10, (d0 * t01 + d1 * t11) * take(i)
        live = b.len > i
        top = torch.maximum(d0, d1)
        logs += torch.where(live, torch.log(top), 0)
        d0, d1 = d0 / top, d1 / top
        if i == 0:
            s0, s1 = d0, d1
        s0, s1 = torch.where(live, d0, s0), torch.where(live, d1, s1)
    p1 = L / (L + 1)
    out["bias"] = logs + torch.log(s0 + s1) + L * torch.log(p1) + torch.log(1 - p1)
    return {k: v.cpu().numpy() for k, v in out.items()}


def _log_z(b, p, emit, ins):
    """lnZ of every pair, rows rescaled by constants; p [n, 8, w], emit(i) and ins(i) the odds of row i."""
    mm, mi, md, im, ii, dm, dd, bm = (p[:, q] for q in range(8))
    L = b.len.double()
    move = 3 / (L + 3)
    loop = 1 - move
    ddl = _shift(dd, 1.0)
    chain = torch.cumprod(torch.where(ddl > 0, ddl, torch.ones_like(ddl)), 1)  # D[k] = chain[k] sum_j a_j / chain[j]
    zero = torch.zeros((b.n, b.w), **b.f64)
    m = i_ = d = zero
    xn, xj, xb = torch.ones(b.n, **b.f64), torch.zeros(b.n, **b.f64), move
    logs, lnz = torch.zeros(b.n, **b.f64), torch.zeros(b.n, **b.f64)
    for i in range(b.rows):
        m2 = (xb[:, None] * bm + _shift(m * mm + i_ * im + d * dm, 0.0)) * emit(i)
        i_ = torch.where(b.ins, (m * mi + i_ * ii) * ins(i), zero)
        m = torch.where(b.col, m2, zero)
        d = torch.where(b.col, torch.cumsum(_shift(m * md, 0.0) / chain, 1) * chain, zero)
        xe = (m + d).sum(1)
        xj = xj * loop + xe * 0.5
        xn = xn * loop
        xb = (xn + xj) * move
        s = 1 / torch.maximum(torch.maximum(xe, xn), xj).detach()
        m, i_, d, xn, xj, xb = m * s[:, None], i_ * s[:, None], d * s[:, None], xn * s, xj * s, xb * s
        logs = logs - torch.log(s)
        lnz = torch.where(b.len == i + 1, torch.log(xj * move) + logs, lnz)
    return lnz


def _exact_grad(b):
    """lnZ and its derivatives by automatic differentiation of the 64-bit recurrence."""
    ident = torch.zeros((b.n, 8, b.w), requires_grad=True, **b.f64)       # log transitions, as offsets
    em = torch.zeros((b.rows, b.n, b.w), requires_grad=True, **b.f64)     # log match odds of each row
    en = torch.zeros((b.rows, b.n, b.w), requires_grad=True, **b.f64)     # log insert odds of each row
    lnz = _log_z(b, b.p * torch.exp(ident), lambda i: b.mo[b.pp, b.x[:, i]] * torch.exp(em[i]),
                 lambda i: torch.exp(en[i]))
    lnz.sum().backward()
    d_msc, d_isc = (torch.zeros((b.n, NSYM, b.w), **b.f64) for _ in range(2))
    who = torch.arange(b.n, device=b.dev)
    for i in range(b.rows):
        d_msc.index_put_((who, b.x[:, i]), em.grad[i], accumulate=True)
        d_isc.index_put_((who, b.x[:, i]), en.grad[i], accumulate=True)
    return lnz, d_msc, d_isc, ident.grad


def exact(case, seed):
    if case["kind"] not in ("score", "grad"):
        return None  # a whole search; its stages have their own cases
    if case["kind"] == "grad" and case["pairs"] * case["m_lo"] * case["l_hi"] > 2.0e7:
        return None
    b = Batch(case, seed)
    if case["kind"] == "score":
        return _exact_scores(b)
    lnz, d_msc, d_isc, d_trans = _exact_grad(b)
    return {"lnz": lnz.detach().cpu().numpy(), "d_msc": d_msc.cpu().numpy(), "d_isc": d_isc.cpu().numpy(),
            "d_trans": d_trans.cpu().numpy()}
