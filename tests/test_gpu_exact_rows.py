"""Exact Forward/Backward row passes (csrc/exact_rows.cuh) at the edges of
their shapes, against the oracle with `==`: every team width, profiles whose
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
