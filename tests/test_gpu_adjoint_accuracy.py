"""The adjoint's counts to the accuracy its arithmetic has.  A count is a sum of
non-negative products whose f32 roundings (2^-24 each, of either sign) add up as
a walk: a row passes some 40 of them on to the next, scale factors and rounded
parameters included, so L rows leave about sqrt(40 (L + 1)) 2^-24; eight times
that is allowed, and 1e-6 of a count for what underflows.  A contribution lost
anywhere (an edge column, a segment's first row, a warp's neighbour) shows from
a few hundred-thousandths of a count on."""
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


@pytest.mark.parametrize("m", [1, 31, 100, 128, 129, 256, 300, 513, 1200])
def test_counts_to_rounding(engine, m):
    rng = np.random.default_rng(7000 + m)
    p = synth.sample_profile(rng, m, f"acc{m}")
    homs = [synth.emit_homolog(rng, p) for _ in range(3)]
    targets = [synth.background_seq(rng, n) for n in (1, 2, 3, 50, 400)]
    targets += [homs[0], synth.plant(rng, len(homs[1]) + 120, homs[1:2]),
                synth.plant(rng, sum(map(len, homs)) + 40, homs),
                np.array([24, 3, 24, 24, 20, 21, 22, 23, 5, 24], np.uint8)]
    lens = np.array([len(t) for t in targets])
    text = synth.profile_text(p)
    ps = engine.load_text(text)
    ts = engine.targets_digital(np.concatenate(targets), np.concatenate([[0], np.cumsum(lens)[:-1]]), lens)
    lnz, d_msc, d_isc, d_tr = engine.posterior_grad(ps, ts, np.zeros(len(targets), np.int32), np.arange(len(targets)), m)
    o = O.Oracle(text=text)
    for i, t in enumerate(targets):
        want = o.expected_counts_f64(0, t)
        rel = 8 * 2.0 ** -24 * np.sqrt(40.0 * (len(t) + 1))
        assert abs(lnz[i] - want["lnz"]) <= rel
        for got, ref in ((d_msc[i], want["d_msc"]), (d_isc[i], want["d_isc"]), (d_tr[i][:7], want["d_t"]),
                         (d_tr[i][7], want["d_tbm"])):
            err = np.abs(got - ref)
            assert np.all(err <= 1e-6 + rel * np.abs(ref)), (i, len(t), err.max())
