"""Read-backs of one batch: from several threads, and again and again."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def packed(ug):
    with ug.Packer([ug.Universe(dim=3, T=48, zgrid=1, excl=1, seed=s, attempts=40_000, round_size=4096)
                    for s in (1, 2)]) as p:
        p.run()
        yield p


def test_threads_read_one_batch(packed):
    want = [(packed.params(u), packed.positions(u)) for u in range(2)]
    bad = []

    def read(u):
        for _ in range(20):
            par, pos = packed.params(u), packed.positions(u)
            if not (np.array_equal(pos, want[u][1]) and all(np.array_equal(par[k], want[u][0][k]) for k in par)):
                bad.append(u)

    threads = [threading.Thread(target=read, args=(k % 2,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_reading_in_turn_allocates_nothing_after_the_first_pass(packed):
    import torch

    free = []
    for _ in range(4):
        for read in (packed.params, packed.positions):
            read(0)
            free.append(torch.cuda.mem_get_info()[0])
    assert len(set(free[2:])) == 1
