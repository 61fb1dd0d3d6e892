"""The Forward pre-screen (csrc/forward_scan.cuh) at the edges of its teams:
one warp of four or eight columns a thread, and two to eight warps.  Its
estimate stays within the stated bound of the exact score, the oracle's
arithmetic: (L + 1)(2M + 6 ceil(M / 32) + 64) 2^-24 in the logarithm, plus the
f32 roundings of the two scores and of their logarithms (of values down to the
smallest f32, |ln| < 104): 2^-22 max(104, |score|)."""
import math

import numpy as np
import pytest

import sxhmm
from sxhmm import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 128, 129, 256, 257, 384, 385, 512, 513, 768, 769, 1024, 1025, 1537, 2048])
def test_estimate_within_its_bound(m):
    rng = np.random.default_rng(900 + m)
    profs = [synth.sample_profile(rng, m, f"f{m}"), synth.sample_profile(rng, m, f"g{m}")]
    if m > 2:  # D runs over every warp of the team
        profs[1].t[1:m, 5:7] = [0.0005, 0.9995]
        profs[1].t[1:m, 0:3] = [0.6, 0.1, 0.3]
    hom = synth.emit_homolog(rng, profs[0])
    targets = [synth.background_seq(rng, n) for n in (1, 2, 33, 150)]
    targets += [synth.plant(rng, len(hom) + 40, [hom]), np.array([24, 3, 24, 20, 21, 23, 5, 24], np.uint8)]
    lens = np.array([len(x) for x in targets], np.int32)
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.int64)
    e = sxhmm.Engine()
    try:
        ps = e.load_text("".join(synth.profile_text(p) for p in profs))
        ts = e.targets_digital(np.concatenate(targets), offs, lens)
        pp = np.repeat(np.arange(2, dtype=np.int32), len(targets))
        pt = np.tile(np.arange(len(targets), dtype=np.int32), 2)
        scan = e.score_prescreens(ps, ts, pp, pt)["fwd_scan"].astype(np.float64)
        exact = e.score_pairs(ps, ts, pp, pt, stages=("forward",))["forward"].astype(np.float64)
    finally:
        e.close()
    for q in range(len(pp)):
        if not math.isfinite(exact[q]):
            assert scan[q] == exact[q]
            continue
        bound = (int(lens[pt[q]]) + 1) * (2 * m + 6 * ((m + 31) // 32) + 64) * 2.0 ** -24
        assert abs(scan[q] - exact[q]) <= bound + 2.0 ** -22 * max(104.0, abs(exact[q]))
