"""Requests of the domain passes whose matrices alone exceed the scratch
budget: the host answers them, with the same hits as an engine with room."""
import numpy as np
import pytest

import sxhmm
from sxhmm import synth

pytestmark = pytest.mark.gpu

CFG = sxhmm.SearchConfig(sxhmm.Cutoff.bits(-1e9, -1e9), sxhmm.PipelineConfig(filters=False)).to_c()


def _search(m, targets, **opts):
    """Raw records of the search and the counters of envelopes and regions the
    device answered."""
    text = synth.profile_text(synth.sample_profile(np.random.default_rng(m), m, f"big{m}"))
    lens = np.array([len(t) for t in targets])
    e = sxhmm.Engine(**opts)
    try:
        ps = e.load_text(text)
        ts = e.targets_digital(np.concatenate(targets), np.concatenate([[0], np.cumsum(lens)[:-1]]), lens)
        hits, doms = e.search(ps, ts, CFG)
        st = e.stats()
        return ([bytes(h) for h in hits], [bytes(d) for d in doms]), st["pairs_out"][5], st["pairs_out"][6]
    finally:
        e.close()


def _consensus(m, first, last):
    p = synth.sample_profile(np.random.default_rng(m), m, f"big{m}")
    return p.mat[first:last + 1].argmax(1).astype(np.uint8)


def test_envelope_above_the_budget():
    """256 MB is the smallest budget of the envelope passes: 5 planes of 4,001
    rows of 4,096 columns take 328, those of the second target 31."""
    m = 4000
    rng = np.random.default_rng(1)
    targets = [_consensus(m, 1, m), np.concatenate([synth.background_seq(rng, 40), _consensus(m, 700, 1000)])]
    small, env, _ = _search(m, targets, batch_bytes=1)
    roomy, env_all, _ = _search(m, targets)
    assert env_all >= 2 and env == env_all - 1
    assert small == roomy and len(small[1]) >= 2


def test_region_above_the_budget():
    """1 GB is the smallest budget of the trace passes: a region of 2,800
    residues of M = 8,192 takes 1.08 GB, one of 602 0.86.  (Two sampled homologs
    end to end; with these seeds each target is one region of two domains.)"""
    m = 8192
    p = synth.sample_profile(np.random.default_rng(m), m, f"big{m}")
    targets = []
    for seed, n in ((1, 1400), (2, 301)):
        rng = np.random.default_rng(seed)
        targets.append(np.concatenate([synth.emit_homolog(rng, p)[:n] for _ in range(2)]))
    small, _, regions = _search(m, targets, batch_bytes=1, envelopes="device", traces="device")
    roomy, _, regions_all = _search(m, targets, envelopes="device", traces="device")
    assert regions_all == 2 and regions == 1
    assert small == roomy and len(small[1]) == 4


def test_survivor_lists_within_the_budget(capfd, monkeypatch):
    """420 small profiles x 20,000 short targets reserve 68 MB of survivor
    lists: more than an engine with the smallest budget (64 MB) holds at once,
    so it searches in blocks, with the same hits."""
    rng = np.random.default_rng(3)
    profs = [synth.sample_profile(rng, 12, f"s{q}") for q in range(420)]
    targets = [synth.background_seq(rng, int(n)) for n in rng.integers(10, 40, 19900)]
    targets += [synth.plant(rng, 40, [synth.emit_homolog(rng, profs[4 * q])]) for q in range(100)]
    lens = np.array([len(t) for t in targets])
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]])
    cfg = sxhmm.SearchConfig(sxhmm.Cutoff.evalue(10.0, 10.0)).to_c()
    text, got, blocks = None, [], []
    for opts in ({}, {"batch_bytes": 1}):
        e = sxhmm.Engine(**opts)
        try:
            if text is None:
                synth.calibrate(profs, synth.engine_scorer(e), np.random.default_rng(7), nseq=40)
                text = "".join(synth.profile_text(p) for p in profs)
            ps, ts = e.load_text(text), e.targets_digital(np.concatenate(targets), offs, lens)
            capfd.readouterr()
            monkeypatch.setenv("SXHMM_PROFILE", "1")
            hits, doms = e.search(ps, ts, cfg)
            monkeypatch.delenv("SXHMM_PROFILE")
            blocks.append(capfd.readouterr().err.count("_cascade="))
            got.append(([bytes(h) for h in hits], [bytes(d) for d in doms], e.stats()["pairs_out"][:4]))
        finally:
            e.close()
    assert blocks[0] == 1 and blocks[1] >= 3
    assert got[0] == got[1] and len(got[0][0]) > 0
