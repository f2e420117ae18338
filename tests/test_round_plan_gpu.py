"""The round plan at the sizes where its tiles can go wrong."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _steps(p):
    """Candidates decided after each round, to the end of the job."""
    at = [0]
    while not p.done():
        p.run(max_rounds=1)
        at.append(p.stats(0).attempts)
    return at


def test_a_last_round_of_whole_waves_tests_every_candidate(ug):
    """A universe alone in its batch whose last round has exactly two tiles per SM, the last
    of them not full: every candidate is tested (many still survive there), and none is
    taken for a survivor that was one in an earlier round."""
    import torch

    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    kw = dict(dim=3, T=40, zgrid=1, excl=1, seed=5, round_size=65536, surv_cap=8192)
    lack = (0, 31, 62, 63, 95, 127)
    with ug.Packer([ug.Universe(attempts=4_000_000, **kw)], precision=ug.PREC_MIXED, rounds_per_sync=1) as p:
        at = [0]
        while len(at) < 3 or at[-1] - at[-2] != 65536 or at[-2] - at[-3] != 65536:
            p.run(max_rounds=1)
            at.append(p.stats(0).attempts)
            assert not p.done()
    last = 2 * nsm * 128
    with ug.Packer([ug.Universe(attempts=at[-1] + last, **kw)], precision=ug.PREC_FP64) as p:
        p.run()
        ref = p.accepted(0)[0]
    assert (ref >= at[-1] + last - 128).sum() > 0  # the last tile holds accepted candidates
    for n in lack:
        with ug.Packer([ug.Universe(attempts=at[-1] + last - n, **kw)], precision=ug.PREC_MIXED,
                       rounds_per_sync=1) as p:
            assert at[-1] in _steps(p)[-2:]  # the last round starts there
            idx = p.accepted(0)[0]
        assert np.array_equal(idx, ref[ref < at[-1] + last - n]), n


def test_windows_count_the_round_that_ran_out_of_slots(ug):
    """A round cut short for lack of slots (the host then grows the buffers) counts in the
    windows like any other: the stop does not depend on the buffers' first size.  The
    threshold is just below the rate of the first window, so one admission lost from it
    would stop the run there; the window after it has lost the first, crowded bucket."""
    kw = dict(dim=3, T=64, zgrid=1, excl=1, seed=2, round_size=65536)
    window = 20_000_000
    n = ug.pack(ug.Universe(attempts=window, **kw), precision=ug.PREC_MIXED, slot_hint=300_000)[0].n
    for hint in (300_000, 1):
        u = ug.Universe(attempts=3 * window, accept_rate=(n - 1) / window, **kw)
        s = ug.pack(u, precision=ug.PREC_MIXED, slot_hint=hint)[0]
        assert s.attempts == window + window // 32, hint
