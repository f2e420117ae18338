"""The survivor product at the edges of its tiles (16 rows of (survivor, axis) x 32
timesteps, steps of eight terms): trajectories against the oracle's."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12  # FP64: the two libms' logarithms and sines, fused against separate products


@pytest.mark.parametrize("dim,T,att", [(1, 4, 40), (1, 33, 300), (2, 5, 9), (2, 8, 500), (2, 31, 17), (2, 65, 700),
                                       (3, 7, 200), (3, 32, 6), (3, 97, 900), (3, 255, 40), (3, 256, 11)])
def test_trajectories_equal_the_oracle(ug, oracle, dim, T, att):
    m = oracle.Model(dim=dim, T=T, zgrid=1, excl=1, seed=T + dim)
    u = ug.Universe(dim=dim, T=T, zgrid=1, excl=1, seed=T + dim, attempts=att, round_size=1024)
    with ug.Packer([u]) as p:
        p.run()
        idx, pos = p.accepted(0)[0], p.positions(0)
    assert len(idx) > 0
    for k in range(0, len(idx), max(1, len(idx) // 12)):
        d = np.abs(pos[k] - oracle.positions(m, int(idx[k])))
        assert np.minimum(d, 2 - d).max() < TOL
