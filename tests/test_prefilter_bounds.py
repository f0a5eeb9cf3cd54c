"""Both thresholds of the quantized distance, as strictly as the kernels use them
(a candidate passes when its sum is below q_thr, and is counted without an exact test
when it is below q_in), in numpy: mtlphys_b200/csrc/engine.cpp set_prefilter,
pbf_device.cuh quantize, pbf_items.cuh count_neighbors_item."""
import math

import numpy as np
import pytest

from test_prefilter import dp4a_square, prefilter, words

F = np.float32
GEOMETRIES = [(0.1, 0.1), (0.1, 0.05), (0.1, 0.17), (0.1, 0.4), (0.03, 0.1)]


def inner(h, cs, lo, hi, units, lim):
    """q_in, and how far outside its cell a particle may be for it to hold."""
    u = cs / units
    fuzz = 0.02 + 4.0 * (max(abs(lo), abs(hi)) + 2.0 * lim) * 2.0 ** -23 / u
    r = h / u * (1.0 - 1e-5) - 2.3453 - 1.7321 * fuzz
    return (math.floor(r * r) - 2 if r > 0.0 else -1), 0.4 * u


def sums(ca, la, cb, lb, units, inv):
    return dp4a_square((words(ca, la, units, inv, 0.5) - words(cb, lb, units, inv, 0.0)) & 0xFFFFFFFF)


@pytest.mark.parametrize("h, cs", GEOMETRIES + [(0.25, 0.01)])
@pytest.mark.parametrize("origin", [0.0, -3.0, 700.0])
def test_pairs_within_h_are_below_the_outer_threshold(h, cs, origin):
    h, cs = float(F(h)), float(F(cs))
    pf = prefilter(h, cs, origin, origin + 40 * cs)
    if pf is None:
        return
    units, inv, thr, _ = pf
    rng = np.random.default_rng(2)
    n = 300_000
    a = rng.uniform(0, 40 * cs, (n, 3))
    step = rng.normal(size=(n, 3)) * rng.choice([0.0, 1.0], (n, 3), p=[0.2, 0.8])  # axes and planes among them
    step *= h * rng.choice([0.5, 0.999, 0.999999], (n, 1)) / np.maximum(np.linalg.norm(step, axis=1, keepdims=True), 1e-9)
    a, b = (a + origin).astype(F), (a + step + origin).astype(F)

    def anchored(p):
        c = np.floor((p.astype(np.float64) - origin) / cs).astype(np.int64) + rng.integers(-2, 3, p.shape)
        return c, (p - (F(origin) + c.astype(F) * F(cs)).astype(F)).astype(F)

    near = np.linalg.norm(a.astype(np.float64) - b.astype(np.float64), axis=1) < h
    s = sums(*anchored(a), *anchored(b), units, inv)
    assert near.sum() > n // 2 and (s[near] < thr).all()


@pytest.mark.parametrize("h, cs", GEOMETRIES)
@pytest.mark.parametrize("origin", [0.0, -3.0, 700.0])
def test_candidates_below_the_inner_threshold_are_within_h(h, cs, origin):
    """Any two particles of a 27-cell stencil, each inside its cell or q_slack outside:
    up to two cells apart, where byte differences wrap."""
    h, cs = float(F(h)), float(F(cs))
    pf = prefilter(h, cs, origin, origin + 300 * cs)
    if pf is None:
        return
    units, inv, _, lim = pf
    q_in, slack = inner(h, cs, origin, origin + 300 * cs, units, lim)
    rng = np.random.default_rng(3)
    n = 400_000
    ca = rng.integers(2, 298, (n, 3))
    cb = ca + rng.integers(-1, 2, (n, 3))

    def inside(c):  # uniform, with many at the walls of the cell
        at = rng.uniform(-slack, cs + slack, c.shape)
        wall = rng.random(c.shape) < 0.4
        at[wall] = rng.choice([-slack, 0.0, cs, cs + slack], wall.sum())
        corner = (F(origin) + c.astype(F) * F(cs)).astype(F)
        p = (corner.astype(np.float64) + at).astype(F)
        return p, (p - corner).astype(F)

    pa, la = inside(ca)
    pb, lb = inside(cb)
    counted = sums(ca, la, cb, lb, units, inv) < q_in
    far = np.linalg.norm(pa.astype(np.float64) - pb.astype(np.float64), axis=1) >= h
    assert not (counted & far).any()
    if q_in > 0 and h >= cs:
        assert counted.sum() > 100  # and the test is not empty
