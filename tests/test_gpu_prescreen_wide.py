"""The packed Viterbi pre-screen on its two widest shapes (M 513 to 1,536, one
word of two targets a lane), which sx_score_prescreens does not report.  Their
bounds are read off searches: F1 = 1 sends every pair to the pre-screen, and
its count of passing pairs just below and just above each bound of the CPU
model (tests/_prescreen_model.py) must step by one.  A cell's unit is 2^-9 nat
or 2.8e-3 bits, the special states' 1.4e-6 bits and the f32 statistic's 7.6e-6
below 128 bits, so a step of 1e-4 bits to either side pins the bound's integers."""
import numpy as np
import pytest

import _prescreen_model as model
import sxhmm
from oracle import oracle as O
from sxhmm import synth

pytestmark = pytest.mark.gpu

LN2 = 0.693147182464599609375
SLACK, STEP, LAM = 1e-3, 1e-4, 0.69315


@pytest.fixture(scope="module")
def engine():
    e = sxhmm.Engine()
    yield e
    e.close()


def _targets(rng, p):
    ts = [synth.background_seq(rng, n) for n in list(range(1, 10)) + [30, 41, 90, 130, 333]]
    ts += [np.full(5, 24, np.uint8), np.array([24, 3, 24, 24, 20, 21, 22, 23, 5, 24], np.uint8)]
    for n in (6, 9, 12, 15, 20, 25):
        h = synth.emit_homolog(rng, p)
        at = int(rng.integers(0, len(h) - n))
        ts.append(synth.plant(rng, 60 + 7 * n, [h[at:at + n]]))
    h = synth.emit_homolog(rng, p)
    ts.append(synth.plant(rng, 150, [h[20:33], h[200:214]]))
    return ts + [np.zeros(0, np.uint8)]


@pytest.mark.parametrize("m", [513, 700, 1024, 1025, 1400, 1536, 1537])
def test_bounds_read_off_searches(engine, monkeypatch, m):
    monkeypatch.setattr(model, "VIT16_WIDTHS", model.VIT16_WIDTHS + (1024, 1536))
    rng = np.random.default_rng(600 + m)
    p = synth.sample_profile(rng, m, f"w{m}")
    targets = _targets(rng, p)
    lens = np.array([len(t) for t in targets])
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]])
    o = O.Oracle(text=synth.profile_text(p))
    a = o.arrays(0)
    bound = np.array([model.vit_bound(a["msc"], a["t"], m, t) for t in targets], np.float32)
    real = lens > 0
    assert np.isnan(bound[~real]).all() and (m > 1536 or np.isfinite(bound[real]).all())
    if m <= 1536:
        exact = np.array([o.viterbi(0, t) for t in targets], np.float32)
        assert np.all(bound[real] >= exact[real])
        stat = np.array([(b - np.float32(o.bias(0, t))) / LN2 for b, t in zip(bound[real], np.array(targets, object)[real])])
        assert np.abs(stat).max() < 128
        mu = float(np.floor(stat.min()))
    else:
        stat, mu = np.zeros(1), -8.0
    p.stats = (-8.0, mu, -4.0, LAM)
    ps = engine.load_text(synth.profile_text(p))
    ts = engine.targets_digital(np.concatenate(targets), offs, lens)

    def passing(threshold):
        f2 = O.gumbel_surv(threshold, mu, LAM)
        cfg = sxhmm.SearchConfig(sxhmm.Cutoff.evalue(10.0, 10.0), sxhmm.PipelineConfig(f1=1.0, f2=f2)).to_c()
        engine.search(ps, ts, cfg)
        vp = engine.stats()["vprescreen"]
        assert vp["pairs_in"] == (real.sum() if m <= 1536 else 0)
        return vp["pairs_out"]

    if m > 1536:
        assert passing(0.0) == 0
        return
    checked = 0
    for s in stat:
        f2 = O.gumbel_surv(float(s), mu, LAM)
        if not 0.9e-5 < f2 < 1.1e-5 and (np.abs(stat - s) < 3 * STEP).sum() == 1:  # F2 does not filter by 1e-5
            above = (stat > s + 2 * STEP).sum()
            assert passing(s + SLACK - STEP) == above + 1, s
            assert passing(s + SLACK + STEP) == above, s
            checked += 1
    assert checked >= len(stat) - 4
