"""The prefilter on every kind of tile that the round plan makes -- full ones (up to 128 live
rows: the epilogue's narrowest stages), ones of 64 candidates, and full ones with a last
wave of 64 or 32 -- against the FP64 form, which shares none of its kernels.  Small rounds
of a universe alone take tiles of 32 only."""

import functools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ATTEMPTS = 3_000_000  # sparse packings resolve fewer candidates a round


def _tiles(plan):
    """Tiles of 128 in a round: below half the SMs' number a lone universe's are cut to 64;
    up to that number they stay; beyond it a last wave of up to half (a quarter) of the SMs
    is cut to 64 (32)."""
    import torch

    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    return {"full": nsm - 20, "64": nsm // 2 - 10, "full+64": nsm + nsm // 3, "full+32": nsm + 12}[plan]


@functools.cache
def _fp64_form(dim, T, mode, euclid):
    import ugb200 as ug

    with ug.Packer([_universe(ug, dim, T, mode, euclid, 65536)], precision=ug.PREC_FP64) as p:
        p.run()
        return p.accepted(0)


def _universe(ug, dim, T, mode, euclid, rs):
    return ug.Universe(dim=dim, T=T, zgrid=1, excl=1, seed=3 * T + dim, attempts=ATTEMPTS, group_mode=mode,
                       euclid=euclid, sub_attempts=20_000 if mode == 1 else 0, round_size=rs, surv_cap=8192)


@pytest.mark.parametrize("dim,T,mode,euclid", [
    (1, 4, 0, 0), (1, 33, 0, 0), (2, 4, 0, 0), (2, 9, 0, 0), (2, 17, 0, 0), (2, 31, 1, 0), (2, 40, 0, 1),
    (2, 65, 2, 0), (2, 129, 2, 0), (2, 255, 0, 0), (2, 256, 2, 0), (3, 5, 0, 0), (3, 16, 0, 0), (3, 33, 0, 0), (3, 47, 2, 1),
    (3, 128, 0, 0), (3, 170, 0, 0),
    (3, 171, 0, 0), (3, 193, 0, 1), (3, 176, 2, 0),  # two passes of the columns
])
@pytest.mark.parametrize("plan", ["full", "64", "full+64", "full+32"])
def test_tiles_of_every_kind(ug, dim, T, mode, euclid, plan):
    rs = 128 * _tiles(plan)
    ref, rgid = _fp64_form(dim, T, mode, euclid)
    with ug.Packer([_universe(ug, dim, T, mode, euclid, rs)], precision=ug.PREC_MIXED, rounds_per_sync=1) as p:
        at = [0]
        while not p.done():
            p.run(max_rounds=1)
            at.append(p.stats(0).attempts)
        idx, gid = p.accepted(0)
    assert (np.diff(at) == rs).sum() > 1  # rounds of that plan were among them
    assert np.array_equal(idx, ref)
    if mode:
        assert np.array_equal(gid, rgid)


def test_waits_after_one_that_gave_up_do_not_wait(ug):
    """A stuck pipeline is reported after one wait's limit, however many waits follow."""
    import ctypes as C
    import time

    from ugb200 import _lib

    st, took = C.c_int32(-1), []
    for _ in range(2):  # the first call may load the kernel
        t0 = time.perf_counter()
        assert _lib.load().ug_selftest_bounded_wait(200_000_000, C.byref(st)) == 0
        took.append(time.perf_counter() - t0)
        assert st.value == _lib.UG_ETIMEDOUT
    assert 0.2 <= took[1] < 0.4  # the kernel makes sixteen waits
