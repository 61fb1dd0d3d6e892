"""One search over several sets reads every set's device images where they are:
repeated sets, an empty one, sets allocated in any order and profiles of every
size class give what each set's own search gives, byte for byte."""
import numpy as np
import pytest

import sxhmm
from sxhmm import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    e = sxhmm.Engine()
    yield e
    e.close()


def _raw(res):
    hits, doms = res
    return [bytes(h) for h in hits], [bytes(d) for d in doms]


def test_views_of_the_sets(engine):
    rng = np.random.default_rng(7)
    lengths = (30, 700, 2100, 120, 1500)
    profs = [synth.sample_profile(rng, m, f"p{i}") for i, m in enumerate(lengths)]
    for p in profs:
        p.stats = (-9.0, -10.0, -4.0, float(np.log(2.0)))
    texts = [synth.profile_text(p) for p in profs]
    spare = engine.load_text(texts[1])
    sets = [engine.load_text("".join(texts[3:])), engine.load_arrays([]), engine.load_text(texts[2]),
            engine.load_text(texts[0])]
    del spare
    sets.append(engine.load_text(texts[1]))  # may lie below the others
    sets += [sets[2], sets[0]]
    targets = [synth.plant(rng, 3000, [synth.emit_homolog(rng, p)]) for p in profs for _ in range(3)]
    targets += [synth.background_seq(rng, n) for n in (1, 7, 350, 900)]
    lens = np.array([len(x) for x in targets], np.int32)
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.int64)
    ts = engine.targets_digital(np.concatenate(targets), offs, lens)
    for f1 in (0.02, 0.3):
        cfg = sxhmm.SearchConfig(sxhmm.Cutoff.evalue(10.0, 10.0)).to_c()
        cfg.f1 = f1
        many = engine.search_many(sets, ts, cfg)
        assert [len(h) > 0 for h, _ in many] == [True, False, True, True, True, True, True]
        for s, got in zip(sets, many):
            assert _raw(got) == _raw(engine.search(s, ts, cfg))
