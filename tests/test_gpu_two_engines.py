"""Two engines on one device, driven by two threads: one kernel serves several
widths of a profile with different amounts of shared memory, and neither
engine's launches may depend on the other's."""
import threading

import numpy as np
import pytest

import sxhmm
from sxhmm import synth

pytestmark = pytest.mark.gpu

CALLS = 3000


def test_widths_of_one_kernel_side_by_side():
    rng = np.random.default_rng(8)
    engines = [sxhmm.Engine(), sxhmm.Engine()]
    errors, got = [], [[], []]
    start = threading.Barrier(2)

    def drive(side, e, m):
        p = e.load_text(synth.profile_text(synth.sample_profile(np.random.default_rng(m), m, f"w{m}")))
        t = e.targets_digital(seq, offs, lens)
        start.wait()
        try:
            for _ in range(CALLS):
                s = e.score_pairs(p, t, [0, 0], [0, 1], stages=("viterbi", "forward"))
                got[side].append((s["viterbi"].tobytes(), s["forward"].tobytes()))
        except Exception as x:  # noqa: BLE001 -- reported by the test's own thread
            errors.append((m, len(got[side]), str(x)))

    targets = [synth.background_seq(rng, n) for n in (1, 2)]
    lens = np.array([len(x) for x in targets])
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]])
    seq = np.concatenate(targets)
    # 3,072 and 4,096 columns: 108 and 144 KB in the row passes, 96 and 128 KB in Viterbi
    threads = [threading.Thread(target=drive, args=(q, engines[q], m)) for q, m in enumerate((2100, 4000))]
    for x in threads:
        x.start()
    for x in threads:
        x.join()
    for e in engines:
        e.close()
    assert not errors
    assert all(len(g) == CALLS and len(set(g)) == 1 for g in got)
