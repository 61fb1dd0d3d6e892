"""Exact Forward/Backward row passes (csrc/exact_rows.cuh) and the envelope
passes built on them (csrc/envelope.cuh) at the edges of their shapes, against
the oracle with `==`: every team width, profiles whose
D chain carries from one warp into the next (delete-extend 0.9995), and
targets of one and two residues and with '*' and degenerate codes."""
import numpy as np
import pytest

from oracle import oracle as O
import sxhmm
from sxhmm import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    e = sxhmm.Engine()
    yield e
    e.close()


def _text(m, dd, seed):
    rng = np.random.default_rng(seed)
    p = synth.sample_profile(rng, m, f"rows{m}")
    if dd is not None and m > 2:
        p.t[1:m, 5:7] = [1.0 - dd, dd]
        p.t[1:m, 0:3] = [0.6, 0.1, 0.3]
    return synth.profile_text(p), p


@pytest.mark.parametrize("dd", [None, 0.9995])
@pytest.mark.parametrize("m", [1, 4, 127, 128, 129, 256, 257, 512, 513, 769, 1025, 1537, 2048])
def test_scores_equal_the_oracle(engine, m, dd):
    text, p = _text(m, dd, 40 + m)
    rng = np.random.default_rng(m)
    hom = synth.emit_homolog(rng, p)
    targets = [synth.background_seq(rng, n) for n in (1, 2, 17, 90)]
    targets.append(synth.plant(rng, len(hom) + 20, [hom]))
    targets.append(np.array([24, 3, 24, 24, 20, 21, 22, 23, 5, 24], np.uint8))
    lens = np.array([len(t) for t in targets])
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]])
    ps = engine.load_text(text)
    ts = engine.targets_digital(np.concatenate(targets), offs, lens)
    got = engine.score_pairs(ps, ts, np.zeros(len(targets), np.int32), np.arange(len(targets)),
                             stages=("forward", "backward"))
    o = O.Oracle(text=text)
    for i, t in enumerate(targets):
        assert got["forward"][i] == np.float32(o.forward(0, t)), (m, i)
        assert got["backward"][i] == np.float32(o.backward(0, t)), (m, i)


@pytest.mark.parametrize("dd", [None, 0.9995])
@pytest.mark.parametrize("m", [2049, 3072, 3073, 4096, 4097, 8192, 8193])
def test_wide_scores_equal_the_oracle(engine, m, dd):
    """M above the lane-group kernels' columns (csrc/wide.cuh and the widest
    row shapes), and the first M past those (csrc/long.cuh)."""
    text, p = _text(m, dd, 40 + m)
    rng = np.random.default_rng(m)
    hom = synth.emit_homolog(rng, p)[:150]
    targets = [synth.background_seq(rng, n) for n in (1, 2, 33)]
    targets.append(synth.plant(rng, len(hom) + 20, [hom]))
    targets.append(np.array([24, 3, 24, 24, 20, 21, 22, 23, 5, 24], np.uint8))
    lens = np.array([len(t) for t in targets])
    ps = engine.load_text(text)
    ts = engine.targets_digital(np.concatenate(targets), np.concatenate([[0], np.cumsum(lens)[:-1]]), lens)
    got = engine.score_pairs(ps, ts, np.zeros(len(targets), np.int32), np.arange(len(targets)),
                             stages=("msv", "viterbi", "forward", "backward"))
    o = O.Oracle(text=text)
    for i, t in enumerate(targets):
        for stage in got:
            assert got[stage][i] == np.float32(getattr(o, stage)(0, t)), (m, i, stage)


def _hits(hits, doms):
    """Hits with their domains, from either side's records."""
    out = []
    for h in hits:
        first = h.domain_offset if hasattr(h, "domain_offset") else h.dom_offset
        n = h.ndomains if hasattr(h, "ndomains") else h.ndom
        ds = [(d.score, d.bias, d.hmm_from, d.hmm_to, d.ali_from, d.ali_to, d.env_from, d.env_to, bool(d.reported))
              for d in doms[first:first + n]]
        out.append((h.target_index, h.score, h.bias, h.nexpected, ds))
    return out


@pytest.fixture(scope="module")
def device_engine():
    e = sxhmm.Engine(envelopes="device", traces="device")
    yield e
    e.close()


@pytest.mark.parametrize("gappy", [False, True])
@pytest.mark.parametrize("m", [3, 5, 127, 128, 129, 256, 257, 513, 1025, 1537, 2048, 2049, 3073, 4100])
def test_device_envelopes_equal_the_oracle(device_engine, m, gappy):
    """Envelope matrices, null2 and insert sums, optimal accuracy and its
    traceback (runs of matches, inserts, deletes) on the team widths, for
    homologs of well-behaved and of gap-rich models, alone and twice."""
    rng = np.random.default_rng(900 + m)
    p = synth.sample_profile(rng, m, f"env{m}")
    if gappy:
        p.t[1:m, 0:3] = [0.7, 0.12, 0.18]
        p.t[1:m, 3:5] = [0.5, 0.5]
        p.t[1:m, 5:7] = [0.3, 0.7]
    homs = [synth.emit_homolog(rng, p) for _ in range(4)]
    targets = [synth.plant(rng, len(homs[0]) + 7, homs[:1]), synth.plant(rng, len(homs[1]) + 90, homs[1:2]),
               synth.plant(rng, len(homs[2]) + len(homs[3]) + 40, homs[2:]), synth.background_seq(rng, 60)]
    lens = np.array([len(t) for t in targets])
    text = synth.profile_text(p)
    ps = device_engine.load_text(text)
    ts = device_engine.targets_digital(np.concatenate(targets), np.concatenate([[0], np.cumsum(lens)[:-1]]), lens)
    cfg = sxhmm.SearchConfig(sxhmm.Cutoff.bits(-1e9, -1e9), sxhmm.PipelineConfig(filters=False)).to_c()
    got = _hits(*device_engine.search(ps, ts, cfg))
    o = O.Oracle(text=text)
    want = _hits(*o.search(O.TargetBatch(targets), O.make_cfg(cutoff="T", seq=-1e9, dom=-1e9, filters=False)))
    assert got == want
    assert any(len(h[4]) for h in got)
