"""The extended solve's push factor at the ends of its fast range: pairs whose
squared distance, root or quotient is where a short square root and division
could round differently (coincident, denormal and tiny separations, roots
whose significand is all ones, distances next to the minimum distance), and
rows of candidates of every parity and length.  Compared bit for bit with the
oracle."""
import numpy as np
import pytest

from tests.helpers import assert_frame_equal

pytestmark = pytest.mark.gpu


def _separations(min_distance, rng):
    """x and y separations of pairs, as float32."""
    m = np.float32(min_distance)
    ones = [np.nextafter(np.float32(2.0 ** k), np.float32(0)) for k in range(-52, 1)]
    edge = [m, np.nextafter(m, np.float32(0)), np.nextafter(m, np.float32(9)), m / 2]
    tiny = [0.0, 1e-45, 1e-38, 1e-30, 2.0 ** -30, 2.0 ** -31, np.nextafter(np.float32(2.0 ** -30), np.float32(0))]
    x = np.array(ones + edge + tiny, np.float32)
    pairs = [(a, 0.0) for a in x] + [(0.0, a) for a in x]
    log = np.exp(rng.uniform(np.log(1e-7), np.log(min_distance), (100, 2)))
    return np.concatenate([np.array(pairs, np.float32), log.astype(np.float32)])


@pytest.mark.parametrize("min_distance", [1.0, 0.37, 2.5, 2.0 ** -22])
def test_push_of_one_pair(W, O, min_distance):
    # one pair per world, next to the origin, where float32 holds its separation
    sep = _separations(min_distance, np.random.default_rng(3))
    cfg = W.WrachConfig(cell_size=1, mode=1, iterations=2, gravity=0.0, min_distance=min_distance,
                        capacity=4)
    dims = (6.0, 6.0)
    ph = O.Physics(1, 2, 0.0, min_distance, 1.0, 9)
    w = O.world(dims[0], dims[1], 1)
    vel = np.zeros((2, 2), np.float32)
    with W.Simulation(cfg, worlds=[dims] * len(sep)) as sim:
        for k, d in enumerate(sep):
            sim.set_particles(np.array([(0, 0), d], np.float32), vel, world=k)
        sim.step(1)
        for k, d in enumerate(sep):
            pos = np.array([(0, 0), d], np.float32)
            ref = O.step(w, ph, *O.pack(w, pos, vel, 4), 1)[:3]
            assert_frame_equal(sim.read_frame(world=k), ref, "separation %r" % (d,))


@pytest.mark.parametrize("cap,cell_size", [(1, 1), (9, 1), (10, 2), (11, 2), (16, 2)])
def test_rows_of_every_length(W, O, cap, cell_size):
    # 0 .. cap + 2 particles per cell, so that rows start at odd and even
    # places and have every length up to 3 * cap, at both ends of the table too
    rng = np.random.default_rng(cap)
    gx, gy = 23, 19
    counts = rng.integers(0, cap + 3, gx * gy)
    counts[:3] = counts[-3:] = cap + 2
    cell = np.repeat(np.arange(gx * gy), counts)
    pos = (np.stack([cell % gx, cell // gx], 1) + rng.uniform(0.01, 0.99, (len(cell), 2))) * cell_size
    pos = pos.astype(np.float32)
    vel = rng.normal(0, 0.5, pos.shape).astype(np.float32)
    dims = (float(gx * cell_size) - 0.5, float(gy * cell_size) - 0.5)
    cfg = W.WrachConfig(dimensions=dims, cell_size=cell_size, mode=1, iterations=4, gravity=0.1,
                        cell_capacity=cap, capacity=len(pos))
    ph = O.Physics(1, 4, 0.1, 1.0, 1.0, cap)
    w = O.world(dims[0], dims[1], cell_size)
    with W.Simulation(cfg) as sim:
        sim.set_particles(pos, vel)
        ref = O.pack(w, pos, vel, len(pos))
        for frame in range(3):
            sim.step(1)
            ref = O.step(w, ph, ref[0], ref[1], ref[2], 1)[:3]
            assert_frame_equal(sim.read_frame(), ref, "frame %d" % frame)


@pytest.mark.parametrize("many", [-1, 0, 1])
@pytest.mark.parametrize("cap", [1, 9, 10])
def test_both_sides_of_the_few_particles_rule(W, O, cap, many):
    """Up to 256 particles per SM the solve kernels keep more loads and pushes
    in flight: rows of every parity and length, below, at and past that count."""
    import torch
    rng = np.random.default_rng(100 * cap)
    few = 256 * torch.cuda.get_device_properties(0).multi_processor_count
    n = few + many if many >= 0 else few // 8 + 1
    gx, gy = 211, 197
    pos = np.empty((0, 2))
    while len(pos) < n:
        counts = rng.integers(0, cap + 3, gx * gy)
        cell = np.repeat(np.arange(gx * gy), counts)
        more = np.stack([cell % gx, cell // gx], 1) + rng.uniform(0.01, 0.99, (len(cell), 2))
        pos = np.concatenate([pos, more])
    pos = pos[:n].astype(np.float32)
    vel = rng.normal(0, 0.5, pos.shape).astype(np.float32)
    dims = (gx - 0.5, gy - 0.5)
    cfg = W.WrachConfig(dimensions=dims, cell_size=1, mode=1, iterations=4, gravity=0.1,
                        cell_capacity=cap, capacity=n)
    ph = O.Physics(1, 4, 0.1, 1.0, 1.0, cap)
    w = O.world(dims[0], dims[1], 1)
    with W.Simulation(cfg) as sim:
        sim.set_particles(pos, vel)
        ref = O.pack(w, pos, vel, n)
        for frame in range(3):
            sim.step(1)
            ref = O.step(w, ph, ref[0], ref[1], ref[2], 1)[:3]
            assert_frame_equal(sim.read_frame(), ref, "frame %d" % frame)


@pytest.mark.parametrize("filler", [0, 60_000])
def test_push_of_one_pair_among_many(W, O, filler):
    # the same separations, with and without a full world that takes the
    # launches past the few-particles rule
    sep = _separations(1.0, np.random.default_rng(5))
    cfg = W.WrachConfig(cell_size=1, mode=1, iterations=3, gravity=0.0, capacity=max(filler, 4))
    dims = (6.0, 6.0)
    ph = O.Physics(1, 3, 0.0, 1.0, 1.0, 9)
    w = O.world(dims[0], dims[1], 1)
    vel = np.zeros((2, 2), np.float32)
    rng = np.random.default_rng(9)
    with W.Simulation(cfg, worlds=[dims] * len(sep) + [(300.0, 300.0)]) as sim:
        for k, d in enumerate(sep):
            sim.set_particles(np.array([(0, 0), d], np.float32), vel, world=k)
        sim.set_particles(rng.uniform(0, 300, (filler, 2)).astype(np.float32),
                          np.zeros((filler, 2), np.float32), world=len(sep))
        sim.step(1)
        for k, d in enumerate(sep):
            pos = np.array([(0, 0), d], np.float32)
            ref = O.step(w, ph, *O.pack(w, pos, vel, cfg.capacity), 1)[:3]
            assert_frame_equal(sim.read_frame(world=k), ref, "separation %r" % (d,))


@pytest.mark.parametrize("cap", [11, 16])
def test_rows_around_32_marks(W, O, cap):
    """Where rows may hold more than 32 marks, a warp whose rows do not takes
    the 32-bit walk: rows of 28 to 36 candidates at odd and even starts, in
    warps of their own and mixed with longer and shorter ones."""
    rng = np.random.default_rng(cap)
    gx, gy = 160, 24
    counts = np.zeros((gy, gx), np.int64)
    for y in range(0, gy, 3):
        # runs of 16 cells whose rows hold `rows` candidates, then empty cells
        for k, rows in enumerate(rng.permutation(np.arange(28, 37))[:8]):
            three = np.array([rows // 3, rows // 3, rows - 2 * (rows // 3)]).clip(0, cap)
            counts[y, 20 * k:20 * k + 15] = np.tile(three, 5)
            counts[y, 20 * k + 15:20 * k + 18] = rng.integers(0, cap + 3, 3)
    counts = counts.ravel()
    cell = np.repeat(np.arange(gx * gy), counts)
    pos = (np.stack([cell % gx, cell // gx], 1) + rng.uniform(0.01, 0.99, (len(cell), 2))) * 2
    pos = pos.astype(np.float32)
    vel = rng.normal(0, 0.5, pos.shape).astype(np.float32)
    dims = (gx * 2 - 0.5, gy * 2 - 0.5)
    cfg = W.WrachConfig(dimensions=dims, cell_size=2, mode=1, iterations=3, gravity=0.1,
                        cell_capacity=cap, capacity=len(pos))
    ph = O.Physics(1, 3, 0.1, 1.0, 1.0, cap)
    w = O.world(dims[0], dims[1], 2)
    with W.Simulation(cfg) as sim:
        sim.set_particles(pos, vel)
        ref = O.pack(w, pos, vel, len(pos))
        for frame in range(3):
            sim.step(1)
            ref = O.step(w, ph, ref[0], ref[1], ref[2], 1)[:3]
            assert_frame_equal(sim.read_frame(), ref, "frame %d" % frame)


def test_the_short_push_factor_everywhere(W):
    """Root and factor of every binary32 squared distance that the short code
    serves, against the general square root and division: the distances of the
    other tests, powers of two and their neighbours, significands of all ones,
    both ends of the range, and random ones over it."""
    rng = np.random.default_rng(17)
    two = np.float32(2.0) ** np.arange(-20, 21, dtype=np.float32)
    near = np.concatenate([np.nextafter(two[1:], np.float32(0)), np.nextafter(two[:-1], np.float32(4e9))])
    rand = np.exp2(rng.uniform(-20, 20, 180)).astype(np.float32)
    with W.Simulation(W.WrachConfig(dimensions=(4.0, 4.0), cell_size=1, mode=1, capacity=4)) as sim:
        for d in np.concatenate([[1.0, 0.37, 2.5, 0.1, 0.9], two, near, rand]).astype(np.float32):
            compared, wrong = sim.selftest_push(float(d))
            # all from 2^-60 to the distance's square but roots of all ones
            binades = 60 + 2 * np.log2(float(d))
            assert compared > 0.99 * (binades - 1) * 2 ** 23 and wrong == 0, (float(d), compared, wrong)
        for d in (2.0 ** -21, 2.0 ** 21):
            assert sim.selftest_push(d) == (0, 0)
        with pytest.raises(W.WrachError):
            sim.selftest_push(0.0)
