"""Room for restored universes: in a batch whose own budget is smaller than the state's, and
again and again into one universe."""

import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
def test_a_state_runs_on_to_its_own_budget(ug, mode):
    """The hash grid and the points grow with the admissions of the restored run."""
    kw = dict(dim=3, T=32, zgrid=1, excl=1, seed=6, round_size=4096, group_mode=mode)
    big = ug.Universe(attempts=150_000, sub_attempts=60_000 * mode, **kw)
    small = ug.Universe(attempts=3000, sub_attempts=1000 * mode, **kw)
    with ug.Packer([big], precision=ug.PREC_MIXED, rounds_per_sync=1) as p:
        p.run(max_rounds=2)
        ck = p.checkpoint(0)
        p.run()
        full, (idx, gid) = p.stats(0), p.accepted(0)
    with ug.Packer([small], precision=ug.PREC_MIXED, force_hash=True) as p:
        p.restore(0, ck).run()
        st, (a, g) = p.stats(0), p.accepted(0)
        assert np.array_equal(a, idx) and np.array_equal(g, gid)
        assert (st.n, st.attempts, st.filled) == (full.n, full.attempts, full.filled)


def test_restoring_again_keeps_no_more_memory(ug):
    import torch

    u = ug.Universe(dim=3, T=48, zgrid=1, excl=1, seed=9, attempts=12_000)
    cks = []
    with ug.Packer([dataclasses.replace(u, round_size=1024)], rounds_per_sync=1) as p:
        while not p.done():
            p.run(max_rounds=2)
            cks.append(p.checkpoint(0))
    assert len(cks) > 3 and cks[-1]["idx"].size > 2 * cks[0]["idx"].size
    with ug.Packer([u], force_hash=True) as p:
        free = []
        for ck in cks:
            p.restore(0, ck)
            free.append(torch.cuda.mem_get_info()[0])
        assert min(free) == free[0]  # all that the universe can reach had its place before
        p.run()
        assert p.stats(0).attempts == u.attempts
