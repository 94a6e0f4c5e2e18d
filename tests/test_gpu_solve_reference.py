"""The reference-physics solve's warps: cells that straddle a warp's particles,
cells up to and past the capacity at every place of a warp, and the pair
sweep's order, bit for bit against the oracle."""
import numpy as np
import pytest

from tests.helpers import assert_frame_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [1, 2, 9, 16])
@pytest.mark.parametrize("n", [1, 31, 33, 2500])
@pytest.mark.parametrize("block", [0, 96])
def test_cells_across_warps(W, O, cap, n, block):
    # runs of cells with 1 .. cap + 3 particles and now and then a hundred,
    # close enough together that every pair of a sweep pushes
    rng = np.random.default_rng(cap * 100 + n)
    counts = rng.integers(1, cap + 4, n)
    counts[rng.random(n) < 0.02] = 100
    cell = np.repeat(np.arange(n), counts)[:n]
    gx, gy = 40, 1 + n // 40
    pos = np.stack([cell % gx, cell // gx], 1) * 3 + rng.uniform(0.3, 2.7, (n, 2))
    pos, vel = pos.astype(np.float32), rng.normal(0, 0.6, (n, 2)).astype(np.float32)
    order = rng.permutation(n)
    pos, vel = pos[order], vel[order]
    dims = (3.0 * gx - 1, 3.0 * gy - 1)
    cfg = W.WrachConfig(dimensions=dims, cell_size=3, mode=0, cell_capacity=cap, capacity=n,
                        solve_block=block)
    w, ph = O.world(dims[0], dims[1], 3), O.Physics(0, 1, 0.0, 1.0, 1.0, cap)
    with W.Simulation(cfg) as sim:
        sim.set_particles(pos, vel)
        ref = O.pack(w, pos, vel, n)
        for frame in range(4):
            sim.step(1)
            ref = O.step(w, ph, ref[0], ref[1], ref[2], 1)[:3]
            assert_frame_equal(sim.read_frame(), ref, "frame %d" % frame)


@pytest.mark.parametrize("zeros", [(-0.0, -0.0), (0.0, -0.0), (-0.0, 0.0), (0.0, 0.0)])
@pytest.mark.parametrize("axis", [0, 1])
def test_signed_zeros(W, O, zeros, axis):
    """Coordinates that are equal zeros: a push leaves the first -0 and turns
    the second into +0, and a velocity of -0 carries the sign to the output."""
    pos = np.zeros((4, 2), np.float32)
    pos[:2, axis], pos[:2, 1 - axis] = zeros, (1.0, 1.25)
    pos[2:, axis], pos[2:, 1 - axis] = zeros, (7.0, 7.0)  # coincident
    vel = np.full((4, 2), -0.0, np.float32)
    w, ph = O.world(12.0, 12.0, 3), O.Physics(0, 1, 0.0, 1.0, 1.0, 9)
    with W.Simulation(W.WrachConfig(dimensions=(12.0, 12.0), cell_size=3, mode=0, capacity=8)) as sim:
        sim.set_particles(pos, vel)
        ref = O.pack(w, pos, vel, 8)
        for frame in range(2):
            sim.step(1)
            ref = O.step(w, ph, ref[0], ref[1], ref[2], 1)[:3]
            assert_frame_equal(sim.read_frame(), ref, "frame %d" % frame)
