"""The FP64 form's test (32 candidates per CTA) at its edges: remainders of a tile, fewest
and most timesteps and terms, both streams, every exclusion and group mode, the crossing
rule; alone and for the universes that a mixed batch leaves to it."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,T,terms,rng,att,mode,kw", [
    (1, 4, 0, 0, 33, 0, {}), (1, 33, 0, 0, 900, 0, {}), (1, 40, 0, 0, 3000, 0, dict(cross1d=1)),
    (1, 24, 0, 1, 1500, 2, dict(cross1d=1)), (2, 4, 2, 1, 100, 0, {}), (2, 15, 0, 0, 31, 0, {}),
    (2, 17, 9, 1, 4001, 0, {}), (2, 33, 0, 1, 5000, 1, {}), (2, 64, 0, 0, 9000, 2, {}),
    (2, 120, 2, 1, 3000, 0, {}), (2, 256, 0, 1, 260, 0, {}), (3, 8, 0, 0, 2000, 0, dict(euclid=1)),
    (3, 31, 5, 1, 2500, 0, dict(pin_sin1=1)), (3, 49, 0, 0, 3000, 2, {}), (3, 256, 0, 0, 97, 0, {}),
])
@pytest.mark.parametrize("mixed", [False, True])
def test_accepted_sets_equal_the_oracle(ug, oracle, dim, T, terms, rng, att, mode, kw, mixed):
    if mixed and rng == 0 and not (kw.get("cross1d") and mode):
        pytest.skip("the tensor-core test takes this universe")
    conv = 1 - rng
    u = ug.Universe(dim=dim, T=T, terms=terms, rng=rng, zgrid=conv, excl=conv, seed=5 * T + dim, attempts=att,
                    group_mode=mode, sub_attempts=att if mode == 1 else 0, round_size=1024, **kw)
    m = oracle.Model(dim=dim, T=T, terms=terms, rng=rng, zgrid=conv, excl=conv, seed=u.seed, euclid=u.euclid,
                     cross1d=u.cross1d, pin=u.pin_sin1)
    ref = oracle.pack(m, att, group_mode=mode, sub_attempts=u.sub_attempts)
    us = [u] if not mixed else [ug.Universe(dim=2, T=20, zgrid=1, excl=1, seed=1, attempts=3000, round_size=1024), u]
    with ug.Packer(us, precision=int(mixed)) as p:
        p.run()
        idx, gid = p.accepted(len(us) - 1)
    assert np.array_equal(idx, ref.acc_idx)
    if mode:
        assert np.array_equal(gid, ref.gid)
