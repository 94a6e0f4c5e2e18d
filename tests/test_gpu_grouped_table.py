"""Grids of more than 16M cells, whose cell table is one record per group of
8 cells: sizes at the edges of groups and of the scan's tiles, cells past the
capacity and past 64 particles in the first, the last and inner groups, in both
physics modes, bit for bit against the oracle."""
import numpy as np
import pytest

from tests.helpers import assert_frame_equal

pytestmark = pytest.mark.gpu


# cells: a multiple of the scan's 2048, of a group's 8, and of neither
@pytest.mark.parametrize("gx,gy", [(4096, 4098), (4104, 4101), (4099, 4101)])
@pytest.mark.parametrize("mode", [0, 1])
def test_grouped_table(W, O, gx, gy, mode):
    rng = np.random.default_rng(gx + mode)
    dims = (gx - 0.5, gy - 0.5)
    # scattered particles, piles of 3 to 200 in single cells (the corners' and
    # next to them among them), and runs of neighbouring full cells
    spots = np.array([(0, 0), (gx - 1, gy - 1), (gx - 2, gy - 1), (gx - 9, gy - 1), (7, 0), (8, 0)]
                     + [(rng.integers(gx), rng.integers(gy)) for _ in range(60)])
    counts = rng.choice([3, 9, 10, 31, 32, 40, 64, 65, 200], len(spots))
    counts[:6] = [40, 200, 9, 10, 65, 32]
    piles = np.repeat(spots, counts, axis=0) + rng.uniform(0.05, 0.45, (counts.sum(), 2))
    run = np.stack([100 + np.arange(300) // 4, np.full(300, 77)], 1) + rng.uniform(0, 0.9, (300, 2))
    pos = np.concatenate([rng.uniform((0, 0), dims, (20_000, 2)), piles, run])
    pos = np.minimum(pos, np.array(dims)).astype(np.float32)
    vel = rng.normal(0, 0.5, pos.shape).astype(np.float32)
    n = len(pos)
    cfg = W.WrachConfig(dimensions=dims, cell_size=1, mode=mode, iterations=3,
                        gravity=0.1 if mode else 0.0, capacity=n)
    w = O.world(dims[0], dims[1], 1)
    ph = O.Physics(mode, 3 if mode else 1, 0.1 if mode else 0.0, 1.0, 1.0, 9)
    with W.Simulation(cfg) as sim:
        assert sim.cells() == gx * gy > 1 << 24
        sim.set_particles(pos, vel)
        ref = O.pack(w, pos, vel, n)
        assert_frame_equal(sim.read_frame(), ref, "upload")
        for frame in range(3):
            sim.step(1)
            ref = O.step(w, ph, ref[0], ref[1], ref[2], 1)[:3]
            assert_frame_equal(sim.read_frame(), ref, "frame %d" % frame)
        # more particles than the frame holds: refused, the frame as it was
        with pytest.raises(W.CapacityError):
            sim.add_particles(pos[:5], vel[:5])
        assert_frame_equal(sim.read_frame(), ref, "after a refused upload")
        sim.step(1)
        ref = O.step(w, ph, ref[0], ref[1], ref[2], 1)[:3]
        assert_frame_equal(sim.read_frame(), ref, "a frame after a refused upload")
