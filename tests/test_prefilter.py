"""The byte-quantized distance prefilter of the lambda passes admits every
pair within h: a restatement in numpy of its arithmetic
(mtlphys_b200/csrc/engine.cpp set_prefilter, pbf_device.cuh quantize) against
exact distances, and on the GPU the neighbour counts and positions of steps
whose geometry strains it against the FP64 oracle."""
import math

import numpy as np
import pytest

from mtlphys_b200 import Engine, _abi
from parity import assert_equal_u32, assert_positions, position_tolerance

F = np.float32


def prefilter(h, cs, lo, hi):
    """(steps per cell, steps per metre, threshold, reach) or None when switched off."""
    units = math.floor(min(123.0 * cs / h, 252.0 / (2.0 + h / cs)))
    if units < 1:
        return None
    u = cs / units
    lim = 32768.0 * u
    most = max(abs(lo), abs(hi)) + 2.0 * lim
    fuzz = 0.02 + 4.0 * most * 2.0 ** -23 / u
    r = h / u * (1.0 + 1e-5) + 2.3453 + 1.7321 * fuzz
    if h / u + 1.5 + fuzz > 127.0 or fuzz > 1.0:
        return None
    return units, F(units / cs), math.floor(r * r) + 2, lim


def words(cell, l, units, inv, bias):
    q = [cell[:, a] * units + np.floor(l[:, a] * inv + F(bias if a else 0.0)).astype(np.int64) for a in range(3)]
    return (q[0] & 255) | ((q[1] & 255) << 8) | ((q[2] & 255) << 16)


def dp4a_square(d):
    b = np.stack([((d >> (8 * k)) & 255) for k in range(4)])
    b = np.where(b > 127, b - 256, b)
    return (b * b).sum(0)


@pytest.mark.parametrize("h, cs", [(0.1, 0.1), (0.1, 0.05), (0.1, 0.17), (0.1, 0.4), (0.03, 0.1), (0.25, 0.01)])
@pytest.mark.parametrize("origin", [0.0, -3.0, 700.0])
def test_no_pair_within_h_is_refused(h, cs, origin):
    h, cs = float(F(h)), float(F(cs))
    pf = prefilter(h, cs, origin, origin + 40 * cs)
    if pf is None:
        assert abs(origin) * 2.0 ** -21 > cs / 128  # coordinates too coarse for the steps
        return
    units, inv, thr, lim = pf
    rng = np.random.default_rng(1)
    n = 200_000
    a = rng.uniform(0, 40 * cs, (n, 3))
    step = rng.normal(size=(n, 3))
    step *= (h * rng.choice([0.2, 0.9, 0.999, 0.999999], (n, 1))) / np.linalg.norm(step, axis=1, keepdims=True)
    a, b = (a + origin).astype(F), (a + step + origin).astype(F)

    def anchored(p):  # hash cells up to 2 cells away from where the particle is now
        c = np.floor((p.astype(np.float64) - origin) / cs).astype(np.int64) + rng.integers(-2, 3, p.shape)
        corner = (F(origin) + c.astype(F) * F(cs)).astype(F)
        return c, (p - corner).astype(F)

    ca, la = anchored(a)
    cb, lb = anchored(b)
    near = np.linalg.norm(a.astype(np.float64) - b.astype(np.float64), axis=1) < h
    d = (words(ca, la, units, inv, 0.5) - words(cb, lb, units, inv, 0.0)) & 0xFFFFFFFF
    assert near.sum() > n // 4 and np.abs(la).max() < lim
    assert (dp4a_square(d)[near] <= thr).all()


@pytest.mark.gpu
@pytest.mark.parametrize("ratio, origin, check_positions", [
    (1.0, 0.0, True), (0.5, -1.0, True), (1.7, 0.0, True), (4.0, 0.0, True), (0.1, 0.0, True), (1.0, 700.0, False),
    (0.008, 0.0, False)])  # the last: cells far smaller than h, prefilter off
def test_counts_and_positions_match_the_oracle(cuda, ratio, origin, check_positions):
    from oracle import oracle as O

    h = 0.1
    rng = np.random.default_rng(5)
    n = 3001
    side = 0.9 if ratio >= 0.1 else 0.25
    pos = np.ones((n, 4), F)
    pos[:, :3] = rng.uniform(0.02, side, (n, 3)) + origin
    pos[:40, :3] = rng.uniform(-3.0, 3.0, (40, 3)) + origin          # outside the box
    pos[40:60, :3] = origin + 400.0 + rng.uniform(0, 0.1, (20, 3))   # far outside, close together
    pos[60:80, :3] = origin - 1e5 + rng.uniform(0, 0.1, (20, 3))
    vel = np.zeros((n, 4), F)
    vel[:, :3] = rng.normal(0, 0.3, (n, 3))
    p = _abi.default_params()
    box = 1.0 if ratio >= 0.1 else 0.25
    p.set(h=h, cell_size=h * ratio, bounds_min=(origin,) * 3, bounds_max=(origin + box,) * 3, solver_iterations=3)
    dt = 1.0 / 240.0
    e = Engine(0)
    try:
        e.set_params(p)
        e.reset(n, _abi.MP_SCENE_CUBE_DROP)
        e.set_positions(pos)
        e.set_velocities(vel)
        e.step(dt)
        assert e.check_errors() == 0
        got = {"pos": e.positions(), "counts": e.neighbor_counts(), "index": e.sorted_index()}
    finally:
        e.close()
    o = O.step(p, dt, pos, vel)
    assert_equal_u32(got["index"], o["sorted_index"], "sortedIndex")
    assert_equal_u32(got["counts"], o["neighbor_counts"], "neighbor counts")
    if check_positions:
        assert_positions(got["pos"], o["pos"], position_tolerance(p, dt, pos, vel))


@pytest.mark.gpu
@pytest.mark.parametrize("ratio, strays", [(1.0, 0), (1.0, 30), (0.5, 0), (1.7, 3), (4.0, 0)])
def test_spatial_hash_counts_match_the_oracle(cuda, ratio, strays):
    """buildSpatialHash's neighbour counts with every particle inside its cell
    (decided by the quantized distance but for a shell) and with some outside the
    grid, whose quantized offsets can wrap; rows of hundreds of candidates."""
    from oracle import oracle as O

    rng = np.random.default_rng(8)
    n = 6001
    pos = np.ones((n, 4), F)
    pos[:, :3] = rng.uniform(0.0, 1.0, (n, 3))
    pos[:900, :3] = 0.5 + rng.normal(0, 0.02, (900, 3))
    pos[900:1000, :3] = rng.choice([0.0, 1.0], (100, 3))  # on the walls
    if strays:
        pos[-strays:, :3] = rng.uniform(-0.8, 1.8, (strays, 3))
        pos[-1, 0] = np.nan
    p = _abi.default_params()
    p.set(cell_size=0.1 * ratio, bounds_min=(0.0,) * 3, bounds_max=(1.0,) * 3)
    e = Engine(0)
    try:
        e.set_params(p)
        e.reset(n, _abi.MP_SCENE_CUBE_DROP)
        e.set_positions(pos)
        e.build_spatial_hash()
        got = e.neighbor_counts()
        e.error_bits()
    finally:
        e.close()
    assert_equal_u32(got, O.build_spatial_hash(p, pos)[3], "neighbor counts")
