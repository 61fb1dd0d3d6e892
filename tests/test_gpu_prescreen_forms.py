"""The packed pre-screens' decisions over the forms they have: tiles that
follow J and tiles that do not (F1 up to 1), lane widths at their edges,
profile pairs with and without a second profile, targets of every length
modulo the block of four, without any scoring residue, and repeated homologs
that raise J again and again.  Searches with and without the pre-screen must
keep the same pairs at every stage and report the same hits."""
import numpy as np
import pytest

import sxhmm
from sxhmm import synth

pytestmark = pytest.mark.gpu

MS = (1, 5, 32, 33, 64, 100, 129, 208, 256, 300, 513, 1024, 1025, 1536, 1601)


def _workload():
    rng = np.random.default_rng(77)
    profs = [synth.sample_profile(rng, m, f"f{m}_{q}") for m in MS for q in range(2 + m % 2)]
    targets = [synth.background_seq(rng, n) for n in list(range(1, 18)) + [60, 127, 256, 333]]
    targets += [np.full(n, 24, np.uint8) for n in (1, 4, 37)] + [np.full(23, 23, np.uint8)]
    targets.append(np.concatenate([np.full(40, 24, np.uint8), synth.background_seq(rng, 50), np.full(41, 24, np.uint8)]))
    for p in profs[::3]:
        h = synth.emit_homolog(rng, p)
        targets.append(synth.plant(rng, len(h) + 11, [h]))
        targets.append(synth.plant(rng, 3 * len(h) + 50, [h, h, h]))
    return profs, targets


@pytest.fixture(scope="module")
def engines():
    es = [sxhmm.Engine(), sxhmm.Engine(prescreen=False)]
    yield es
    for e in es:
        e.close()


@pytest.mark.parametrize("f1", [1e-4, 0.02, 0.6, 1.0])
def test_same_pairs_at_every_stage(engines, f1):
    profs, targets = _workload()
    synth.calibrate(profs, synth.engine_scorer(engines[0]), np.random.default_rng(7), nseq=60)
    text = "".join(synth.profile_text(p) for p in profs)
    lens = np.array([len(t) for t in targets])
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]])
    cfg = sxhmm.SearchConfig(sxhmm.Cutoff.evalue(10.0, 10.0), sxhmm.PipelineConfig(f1=f1, f2=max(f1, 1e-3))).to_c()
    got = []
    for e in engines:
        ps, ts = e.load_text(text), e.targets_digital(np.concatenate(targets), offs, lens)
        hits, doms = e.search(ps, ts, cfg)
        st = e.stats()
        got.append(([bytes(h) for h in hits], [bytes(d) for d in doms], st["pairs_out"][:4]))
    assert got[0] == got[1]
    assert got[0][2][0] > 0
