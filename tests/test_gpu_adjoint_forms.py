"""The adjoint's team widths and odd targets: M at the edges of one warp and of
several, targets of one residue, with '*' and degenerate codes, empty ones, and
enough pairs for several parts.  Gradients and lnZ against the oracle's FP64
expected counts: within 1e-3 absolute and relative (f32 sums over the rows), lnZ
within 1e-5 relative."""
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


def _case(m, extra=0):
    rng = np.random.default_rng(300 + m)
    p = synth.sample_profile(rng, m, f"adj{m}")
    hom = synth.emit_homolog(rng, p)
    targets = [synth.background_seq(rng, n) for n in (1, 2, 40)]
    targets += [synth.plant(rng, len(hom) + 20, [hom]), np.zeros(0, np.uint8),
                np.array([24, 3, 24, 24, 20, 21, 22, 23, 5, 24], np.uint8)]
    targets += [synth.background_seq(rng, 5 + q % 7) for q in range(extra)]
    return synth.profile_text(p), targets


@pytest.mark.parametrize("m,extra", [(1, 0), (3, 0), (127, 0), (128, 0), (129, 0), (256, 1100), (257, 0), (513, 0),
                                     (1200, 0), (2048, 0)])
def test_gradients_against_fp64(engine, m, extra):
    text, targets = _case(m, extra)
    lens = np.array([len(t) for t in targets])
    ps = engine.load_text(text)
    ts = engine.targets_digital(np.concatenate(targets), np.concatenate([[0], np.cumsum(lens)[:-1]]), lens)
    lnz, d_msc, d_isc, d_tr = engine.posterior_grad(ps, ts, np.zeros(len(targets), np.int32), np.arange(len(targets)), m)
    o = O.Oracle(text=text)
    for i, t in enumerate(targets):
        if len(t) == 0:
            assert lnz[i] == -np.inf and not d_msc[i].any() and not d_isc[i].any() and not d_tr[i].any()
            continue
        if i > 40 and i % 97:
            continue
        want = o.expected_counts_f64(0, t)
        assert abs(lnz[i] - want["lnz"]) <= 1e-5 * max(1.0, abs(want["lnz"]))
        for got, ref in ((d_msc[i], want["d_msc"]), (d_isc[i], want["d_isc"]), (d_tr[i][:7], want["d_t"]),
                         (d_tr[i][7], want["d_tbm"])):
            assert np.all(np.abs(got - ref) <= 1e-3 + 1e-3 * np.abs(ref)), (i, np.abs(got - ref).max())
