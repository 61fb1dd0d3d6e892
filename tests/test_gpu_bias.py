"""Composition-bias scores (bias_kernel, csrc/kernels.cuh) at the edges of its
16-residue words, against the oracle, within the 2 f32 ulps that two f64
evaluations rounded to f32 may differ by."""
import numpy as np
import pytest

from oracle import oracle as O
import sxhmm
from sxhmm import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 60, 300])
def test_bias_scores(m):
    rng = np.random.default_rng(70 + m)
    profs = [synth.sample_profile(rng, m, f"b{m}"), synth.sample_profile(rng, m, f"c{m}")]
    text = "".join(synth.profile_text(p) for p in profs)
    targets = [synth.background_seq(rng, n) for n in (1, 2, 15, 16, 17, 31, 32, 33, 64, 100, 5000)]
    targets += [np.full(40, 24, np.uint8), np.full(700, 1, np.uint8), np.array([20, 21, 22, 23, 24, 24], np.uint8)]
    lens = np.array([len(x) for x in targets], np.int32)
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.int64)
    pp = np.repeat(np.arange(2, dtype=np.int32), len(targets))
    pt = np.tile(np.arange(len(targets), dtype=np.int32), 2)
    e = sxhmm.Engine()
    try:
        got = e.score_pairs(e.load_text(text), e.targets_digital(np.concatenate(targets), offs, lens), pp, pt,
                            stages=("bias",))["bias"]
    finally:
        e.close()
    o = O.Oracle(text=text)
    want = np.array([o.bias(int(p), targets[t]) for p, t in zip(pp, pt)], np.float32)
    assert np.all(np.abs(got.astype(np.float64) - want) <= 2 * np.spacing(np.abs(want)))
