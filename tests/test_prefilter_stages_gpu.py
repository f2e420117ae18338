"""The prefilter's epilogue stages at the edges of their widths: timestep counts around the
operand padding, fewer columns than a stage takes, two passes, and live rows from a full
tile down to none, in every dimension, exclusion and group mode (decisions are exact, so the
accepted sets equal the oracle's)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,T,att,mode,euclid", [
    (1, 4, 700, 0, 0), (1, 33, 5000, 0, 0), (2, 4, 129, 0, 0), (2, 9, 6000, 0, 0), (2, 17, 8000, 2, 0),
    (2, 31, 9000, 1, 0), (2, 40, 20000, 0, 1), (2, 129, 12000, 2, 0), (2, 255, 5000, 0, 0),
    (3, 5, 2000, 0, 0), (3, 16, 9000, 0, 0), (3, 33, 20000, 0, 0), (3, 47, 12000, 2, 1),
    (3, 170, 2500, 0, 0), (3, 171, 2500, 0, 0), (3, 256, 700, 0, 1),
])
@pytest.mark.parametrize("hashed", [False, True])
def test_stage_edges(ug, oracle, dim, T, att, mode, euclid, hashed):
    u = ug.Universe(dim=dim, T=T, zgrid=1, excl=1, seed=7 * T + dim, attempts=att, group_mode=mode, euclid=euclid,
                    sub_attempts=att if mode == 1 else 0, round_size=2048)
    m = oracle.Model(dim=dim, T=T, zgrid=1, excl=1, seed=u.seed, euclid=euclid)
    ref = oracle.pack(m, att, group_mode=mode, sub_attempts=u.sub_attempts)
    with ug.Packer([u], precision=ug.PREC_MIXED, force_hash=hashed) as p:
        p.run()
        idx, gid = p.accepted(0)
    assert np.array_equal(idx, ref.acc_idx)
    if mode:
        assert np.array_equal(gid, ref.gid)
