"""Frame kernels at the edges of their tiles: the rewind grid's product (64 rows of (path,
axis) x 72 rewind rows, chunks of 8 frequencies), the warp-wide crossing search and the
three-steps-a-pass refinement, against the same search in numpy."""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# float32 records: an offset is evaluated here at the recorded (rounded) z_emit, so it is
# off by the offset's slope (below 100 on these windows) times half an ulp of z (6e-8 z)
TOL = 2e-5


def _dump(n, nw, bmax, seed):
    r = np.random.default_rng(seed)
    b = np.stack([np.stack([np.sort(r.choice(np.arange(2, bmax + 1), nw, replace=False))
                            for _ in range(2)]) for _ in range(n)]).astype(float)
    w = r.dirichlet(np.ones(nw), (n, 2))
    a = w / b * r.choice([-1.0, 1.0], (n, 2, nw))
    f = np.where(b % 2 == 0, r.uniform(0, math.pi, b.shape), 0.0)
    return r.uniform(-1, 1, (n, 2)), a, b, f


def _x(a2, a, b, f, z):
    """Comoving positions [n][2] + shape of z."""
    s = a2[..., None] * np.sin(z)
    for j in range(a.shape[-1]):
        s = s + a[..., j, None] * (np.sin(b[..., j, None] * z + f[..., j, None]) - np.sin(f[..., j, None]))
    return s / np.sin(z)


def _reach(z, z_obs, bmax):
    b = np.arange(2, bmax + 1)[:, None]
    da = (np.cos(b * z) - 1) / (b * np.sin(z)) - (np.cos(b * z_obs) - 1) / (b * np.sin(z_obs))
    db = np.sin(b * z) / (b * np.sin(z)) - np.sin(b * z_obs) / (b * np.sin(z_obs))
    return np.where(b % 2 == 0, np.hypot(da, db), np.abs(db)).max(0)


@pytest.mark.parametrize("n,nw,bmax,front", [
    (1, 1, 2, "fit"), (31, 6, 7, "speed"), (32, 7, 8, "fit"), (33, 8, 9, "fit"), (65, 23, 24, "fit"),
    (7, 14, 15, "budget"),
    (5, 255, 256, "budget"),   # 513 rewind rows: a last column tile of 9
    (40, 1, 64, "fit"),        # few terms: summed directly
])
def test_hits_are_the_crossings_of_the_rewind_grid(ug, n, nw, bmax, front):
    from ugb200.frames import bake

    a2, a, b, f = _dump(n, nw, bmax, 100 * n + nw)
    at, K, z_min, z_obs = (0.13, -0.29), 2, 0.05 * math.pi, 0.4 * math.pi
    bk = bake(a2, a, b, f, observers=[("point", *at)], from_pi=0.4, to_pi=0.4, frames=1, zmin_pi=0.05,
              front=front, metric="square", speed=0.33, wraps=K)
    h = bk.hits[0][0]
    top = int(max(2, b.max()))
    i = np.arange(421 if front != "budget" else min(4000, max(420, 2 * top)) + 1)
    eta = lambda z: np.log(np.tan(z / 2))  # noqa: E731
    if front == "budget":
        z = z_obs - (z_obs - z_min) * i / i[-1]
        chi = _reach(z, z_obs, top)
    else:
        speed = 0.33 if front == "speed" else -1 / eta(z_min)
        chi = speed * (eta(z_obs) - eta(z_min)) * i / i[-1]
        z = 2 * np.arctan(np.exp(eta(z_obs) - chi / speed))
    x = _x(a2, a, b, f, z)
    want = np.zeros(n, int)
    for nx in range(-K, K + 1):
        for ny in range(-K, K + 1):
            dmin = max(0.0, 2.0 * max(abs(nx), abs(ny)) - 4.0)
            if dmin >= chi.max():
                continue
            i0 = 1 if front == "budget" else max(1, math.ceil(dmin * i[-1] / chi.max()))
            g = np.abs(x + np.array([2 * nx - at[0], 2 * ny - at[1]])[:, None]).max(1) - chi
            want += ((g[:, i0 - 1:-1] < 0) != (g[:, i0:] < 0)).sum(1)
    assert np.array_equal(np.bincount(h["src"], minlength=n), want)
    # each hit is an image of its source at its emission, on the front
    d = _x(a2[h["src"]], a[h["src"]], b[h["src"]], f[h["src"]], h["z_emit"].astype(float)[:, None, None])[..., 0] - at
    off = np.stack([h["dx"], h["dy"]], 1) - d
    assert np.abs(off - 2 * np.round(off / 2)).max() < TOL
    np.testing.assert_allclose(np.maximum(np.abs(h["dx"]), np.abs(h["dy"])), h["chi"], atol=TOL)


@pytest.mark.parametrize("dim,T,pin", [(1, 4, 0), (2, 31, 1), (3, 33, 0), (2, 64, 0), (1, 255, 0), (2, 256, 0)])
def test_dumped_parameters_equal_the_oracle(ug, oracle, dim, T, pin):
    """The warp-per-axis parameter dump at odd and even bands, smallest and largest."""
    u = ug.Universe(dim=dim, T=T, zgrid=1, excl=1, pin_sin1=pin, seed=T, attempts=2000, round_size=1024)
    m = oracle.Model(dim=dim, T=T, zgrid=1, excl=1, pin=pin, seed=T)
    with ug.Packer([u]) as p:
        p.run()
        idx, par = p.accepted(0)[0], p.params(0)
    for k in range(0, len(idx), max(1, len(idx) // 9)):
        c = oracle.candidate(m, int(idx[k]))
        assert np.array_equal(par["b"][k], c["b"])
        for q in ("a", "f", "a2"):  # an ulp of the two libms' logarithms
            np.testing.assert_allclose(par[q][k], c[q], rtol=1e-14, atol=1e-300)


@pytest.mark.parametrize("hits", [True, False])
def test_more_hits_than_the_first_room(ug, hits):
    """Paths that waver about the observer cross the young front some twenty times each: more
    hits than the room first made for them; the same as those of the paths in small groups."""
    from ugb200.frames import bake

    n, part = 6000, 1000
    r = np.random.default_rng(8)
    b = np.full((n, 2, 1), 100.0)
    a = np.full((n, 2, 1), 0.3)
    f = r.uniform(0, math.pi, (n, 2, 1))
    a2 = np.array([0.13, -0.29]) + 0.3 * np.sin(f[..., 0]) / math.sin(0.3 * math.pi) + r.uniform(-0.05, 0.05, (n, 2))
    kw = dict(observers=[("point", 0.13, -0.29)], from_pi=0.35, to_pi=0.45, frames=2, zmin_pi=0.05, front="fit",
              metric="square", density_bins=32, hits=hits)
    whole = bake(a2, a, b, f, **kw)
    parts = [bake(a2[k:k + part], a[k:k + part], b[k:k + part], f[k:k + part], **kw) for k in range(0, n, part)]
    assert whole.counts.min() > 1 << 17 and max(p.counts.max() for p in parts) < 1 << 16
    assert np.array_equal(whole.counts, sum(p.counts for p in parts))
    assert np.array_equal(whole.density, sum(p.density for p in parts))
    if hits:
        for fi in range(2):
            h = whole.hits[fi][0]
            want = np.concatenate([p.hits[fi][0] for p in parts])
            want["src"] += np.repeat(np.arange(0, n, part), [len(p.hits[fi][0]) for p in parts]).astype(np.uint32)
            key = ("src", "chi", "dx", "dy", "z_emit")
            assert np.array_equal(np.sort(h, order=key), np.sort(want, order=key))


@pytest.mark.parametrize("n,K,speed,metric", [
    (1, 16, 14.0, "square"), (3, 15, 11.0, "square"), (2, 36, 25.0, "square"), (2, 40, 0.33, "square"),
    (2, 17, 9.0, "euclid"), (5, 3, 2.0, "euclid"), (40, 2, 0.4, "euclid"),
])
def test_hits_over_many_images(ug, n, K, speed, metric):
    """Images beyond 32 a side, and more of them than the front reaches."""
    from ugb200.frames import bake

    a2, a, b, f = _dump(n, 6, 8, 7 * n + K)
    at, z_min, z_obs = (0.13, -0.29), 0.05 * math.pi, 0.4 * math.pi
    bk = bake(a2, a, b, f, observers=[("point", *at)], from_pi=0.4, to_pi=0.4, zmin_pi=0.05, front="speed",
              metric=metric, speed=speed, wraps=K)
    eta = lambda z: np.log(np.tan(z / 2))  # noqa: E731
    chi = speed * (eta(z_obs) - eta(z_min)) * np.arange(421) / 420
    x = _x(a2, a, b, f, 2 * np.arctan(np.exp(eta(z_obs) - chi / speed)))
    want = np.zeros(n, int)
    for nx in range(-K, K + 1):
        for ny in range(-K, K + 1):
            dmin = max(0.0, 2.0 * max(abs(nx), abs(ny)) - 4.0)
            if dmin >= chi[-1]:
                continue
            i0 = max(1, math.ceil(dmin * 420 / chi[-1]))
            d = x + np.array([2 * nx - at[0], 2 * ny - at[1]])[:, None]
            g = (np.abs(d).max(1) if metric == "square" else np.hypot(d[:, 0], d[:, 1])) - chi
            want += ((g[:, i0 - 1:-1] < 0) != (g[:, i0:] < 0)).sum(1)
    assert np.array_equal(np.bincount(bk.hits[0][0]["src"], minlength=n), want)


def test_images_out_of_reach_cost_nothing(ug):
    """One path, a front of radius one and 301 images a side: milliseconds (a thread per image
    took 3, a warp that walked them all 840)."""
    import time

    from ugb200.frames import bake

    took = []
    for _ in range(4):
        t0 = time.perf_counter()
        bake(*_dump(1, 6, 8, 1), observers=[("point", 0.13, -0.29)], from_pi=0.3, to_pi=0.4, frames=4,
             zmin_pi=0.05, front="fit", metric="square", wraps=150, hits=False)
        took.append(time.perf_counter() - t0)
    assert min(took) < 0.1


def test_a_frequency_listed_many_times_adds_up_the_same_way(ug):
    """Coefficients of repeated frequencies, within a warp's 32 terms and across them: the
    hits of a dump equal those of the dump with each frequency's terms added up, and two
    bakes are equal bit for bit."""
    from ugb200.frames import bake

    n, nw = 64, 70
    r = np.random.default_rng(12)
    b = r.integers(2, 34, (n, 2, nw)).astype(float)
    a = r.dirichlet(np.ones(nw), (n, 2)) / b * r.choice([-1.0, 1.0], (n, 2, nw))
    f = np.where(b % 2 == 0, r.uniform(0, math.pi, b.shape), 0.0)
    a2 = r.uniform(-1, 1, (n, 2))
    c = np.zeros((n, 2, 34), complex)
    for j in range(nw):
        np.add.at(c, (*np.indices((n, 2)), b[..., j].astype(int)), a[..., j] * np.exp(1j * f[..., j]))
    sums = np.broadcast_to(np.arange(2.0, 34.0), (n, 2, 32))
    kw = dict(observers=[("point", 0.1, 0.2)], from_pi=0.4, to_pi=0.4, zmin_pi=0.05, front="fit", metric="square")
    one, two = (bake(a2, a, b, f, **kw).hits[0][0] for _ in range(2))
    key = ("src", "chi", "dx", "dy", "z_emit")
    assert len(one) > n // 2 and np.array_equal(np.sort(one, order=key), np.sort(two, order=key))
    ref = bake(a2, np.abs(c[..., 2:]), sums, np.angle(c[..., 2:]), **kw).hits[0][0]
    assert np.array_equal(np.bincount(one["src"], minlength=n), np.bincount(ref["src"], minlength=n))
    x, y = np.sort(one, order=("src", "chi")), np.sort(ref, order=("src", "chi"))
    for k in ("dx", "dy", "chi", "z_emit"):
        np.testing.assert_allclose(x[k], y[k], atol=TOL)
