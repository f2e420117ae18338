"""The knot stream where a few-term list names a frequency twice: 64 redraws do not always
find a free one when nearly all of them are taken (terms = T - 1)."""

import math
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


@pytest.mark.parametrize("precision", [0, 1])
def test_accepted_sets_equal_the_oracle(ug, oracle, precision):
    u = ug.Universe(dim=2, T=120, terms=119, rng=1, seed=4, attempts=3000, round_size=1024)
    ref = oracle.pack(oracle.Model(dim=2, T=120, terms=119, rng=1, seed=4), 3000)
    with ug.Packer([u], precision=precision) as p:
        p.run()
        assert np.array_equal(p.accepted(0)[0], ref.acc_idx)


def test_a_repeated_frequency_adds_up_in_term_order(ug):
    """Stored trajectories, bit for bit: the coefficients of a frequency add up term by term
    (the sine's by a fused multiply-add, the cosine's product rounded first), then the sum
    over ascending frequencies, a fused multiply-add each."""
    import torch

    T, terms = 64, 63
    u = ug.Universe(dim=2, T=T, terms=terms, rng=1, seed=11, attempts=60000, round_size=1024)
    with ug.Packer([u]) as p:
        p.run()
        par, pos = p.params(0), p.positions(0)
    f = torch.from_numpy(par["f"]).cuda()
    cf, sf = f.cos().cpu().numpy(), f.sin().cpu().numpy()
    z = [(i + 1) * math.pi / (T + 1) for i in range(T)]
    rows = 0
    for i, ax in np.ndindex(*par["a2"].shape):
        even = [b for b in par["b"][i, ax] if b % 2 == 0]
        if len(set(even)) == len(even):
            continue
        rows += 1
        al, bt = [0.0] * (T + 1), [0.0] * (T + 1)
        for j in range(terms - 1):
            b, a = int(par["b"][i, ax, j]), par["a"][i, ax, j]
            if b % 2:
                al[b] += a
            else:
                al[b], bt[b] = _fma(a, cf[i, ax, j], al[b]), bt[b] + a * sf[i, ax, j]
        for t in range(T):
            acc = 0.0
            for b in range(2, T + 1):
                acc = _fma(al[b], math.sin(b * z[t]), acc)
                if b % 2 == 0:
                    acc = _fma(bt[b], math.cos(b * z[t]) - 1.0, acc)
            x = _fma(acc, 1.0 / math.sin(z[t]), par["a2"][i, ax])
            assert pos[i, ax, t] == x - 2.0 * math.floor((x + 1.0) * 0.5), (i, ax, t)
    assert rows > 20
