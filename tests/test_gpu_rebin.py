"""The three paths of the counting-sort rebin, bit for bit against the oracle's
stable counting sort: cells of up to 64 particles (ranked per slot), larger
cells (sorted in shared memory), and cells beyond 2048 particles (sorted in
global memory by one block).  Uploads and frames both go through the rebin."""
import numpy as np
import pytest

from tests.helpers import assert_frame_equal, make_sim, oracle_physics

pytestmark = pytest.mark.gpu


def _clustered(seed, dims, clusters, background):
    """`clusters`: [(cell x, cell y, count)], each cluster inside one cell of
    size 1; plus `background` particles spread over the box."""
    rng = np.random.default_rng(seed)
    parts = [rng.uniform((0, 0), dims, size=(background, 2))]
    for cx, cy, m in clusters:
        parts.append(np.column_stack([cx + rng.uniform(0.05, 0.95, m), cy + rng.uniform(0.05, 0.95, m)]))
    pos = np.concatenate(parts).astype(np.float32)
    order = rng.permutation(len(pos))  # uploads arrive in any order
    pos = pos[order]
    vel = rng.normal(0, 0.4, size=pos.shape).astype(np.float32)
    return pos, vel


def _run(W, O, dims, pos, vel, mode, frames, gravity=0.0):
    sim = make_sim(W, dims, 1, mode, 4, gravity, capacity=len(pos) + 16)
    try:
        w = O.world(dims[0], dims[1], 1)
        ph = oracle_physics(O, mode, 4, gravity)
        sim.add_particles(pos, vel)
        ref = O.pack(w, pos, vel, capacity=sim.capacity())
        assert_frame_equal(sim.read_frame(), ref, "upload")
        for f in range(frames):
            sim.step(1)
            ref = O.step(w, ph, ref[0], ref[1], ref[2], 1)[:3]
            assert_frame_equal(sim.read_frame(), ref, "frame %d" % (f + 1))
        return sim.stats()
    finally:
        sim.close()


@pytest.mark.parametrize("mode", [0, 1])
def test_large_cells(W, O, mode):
    dims = (64.0, 48.0)
    pos, vel = _clustered(1, dims, [(10, 10, 2048), (20, 20, 700), (30, 30, 65), (40, 12, 64),
                                    (5, 40, 33)], 2500)
    st = _run(W, O, dims, pos, vel, mode, 4, gravity=0.1 if mode else 0.0)
    assert st["huge_cells"] == 0


def test_cell_beyond_the_shared_memory_sort(W, O):
    dims = (32.0, 24.0)
    pos, vel = _clustered(2, dims, [(8, 8, 9000), (12, 12, 2049), (16, 16, 100)], 800)
    st = _run(W, O, dims, pos, vel, 1, 2, gravity=0.1)
    assert st["huge_cells"] >= 1


def test_floor_pile(W, O):
    # the shape a long run of the extended physics reaches: most particles in
    # the bottom row of cells, a few hundred per cell
    rng = np.random.default_rng(3)
    dims = (200.0, 60.0)
    n = 60000
    pos = np.column_stack([rng.uniform(0, 200.0, n), rng.uniform(0, 0.999, n) ** 3]).astype(np.float32)
    pos = np.concatenate([pos, rng.uniform((0, 1), dims, size=(3000, 2)).astype(np.float32)])
    vel = rng.normal(0, 0.3, size=pos.shape).astype(np.float32)
    st = _run(W, O, dims, pos, vel, 1, 3, gravity=0.1)
    assert st["huge_cells"] == 0


@pytest.mark.parametrize("count", [65, 255, 256, 257, 513, 2048])
@pytest.mark.parametrize("pages", [2, 3, 31, 32, 33, 60])
def test_large_cell_sources_over_pages(W, O, count, pages):
    # the sources of one large cell spread over `pages` runs of 1024 indices
    # (up to 32 of them are ranked by a bitmap, more are sorted), at both ends
    # and in the middle of each, and a second large cell after it
    rng = np.random.default_rng(count + pages)
    n = pages * 1024
    pos = np.column_stack([rng.uniform(8, 60, n), rng.uniform(8, 40, n)]).astype(np.float32)
    per = np.full(pages, count // pages)
    per[: count % pages] += 1
    for p, m in enumerate(per):
        ends = [0, 1023, 31, 32]
        pick = np.concatenate([ends, rng.permutation(np.setdiff1d(np.arange(1024), ends))])[:m]
        pos[p * 1024 + pick] = np.column_stack([rng.uniform(3, 3.9, m), rng.uniform(2, 2.9, m)])
    free = np.nonzero(pos[:, 0] >= 8)[0]
    free = free[:90]
    pos[free] = np.column_stack([rng.uniform(5, 5.9, len(free)), rng.uniform(2, 2.9, len(free))])
    vel = rng.normal(0, 0.2, pos.shape).astype(np.float32)
    st = _run(W, O, (64.0, 48.0), pos, vel, 1, 2, gravity=0.1)
    assert st["huge_cells"] == 0


def test_profiled_frames_match_graph_frames(W, O):
    # a profiled frame runs its launches one at a time on the frame's stream
    # (the large cells' sort included); graph frames run that sort on a
    # second stream beside the small cells' pass.  Both match the oracle.
    dims = (64.0, 48.0)
    pos, vel = _clustered(4, dims, [(10, 10, 300), (20, 20, 65), (30, 30, 64)], 2500)
    sim = make_sim(W, dims, 1, 1, 4, 0.1, capacity=len(pos) + 16)
    try:
        w = O.world(dims[0], dims[1], 1)
        ph = oracle_physics(O, 1, 4, 0.1)
        sim.add_particles(pos, vel)
        ref = O.pack(w, pos, vel, capacity=sim.capacity())
        for f in range(6):
            if f % 2 == 0:
                ms = sim.profile_frame()
                assert len(ms) == 8  # four Jacobi passes, four rebin launches
                assert all(m >= 0.0 for m in ms)
            else:
                sim.step(1)
            ref = O.step(w, ph, ref[0], ref[1], ref[2], 1)[:3]
            assert_frame_equal(sim.read_frame(), ref, "frame %d" % (f + 1))
    finally:
        sim.close()


@pytest.mark.parametrize("dims", [(31.5, 63.5), (32.5, 63.5), (40.0, 30.0)])
@pytest.mark.parametrize("add", [False, True])
def test_an_upload_past_the_capacity_places_nothing(W, O, dims, add):
    """One world's place steps do not wait for the host to know the count (the
    scan writes it; at a tile's edge, one cell row past it and inside one):
    a count that just fits is placed, one more leaves frame, cell table and
    counters as they are, large cells or not."""
    pos, vel = _clustered(5, dims, [(3, 4, 63), (9, 9, 64), (9, 10, 65), (20, 20, 700)], 900)
    n = len(pos)
    more = np.full((1, 2), 20.5, np.float32)
    sim = make_sim(W, dims, 1, 1, 4, 0.1, capacity=n)
    try:
        w, ph = O.world(dims[0], dims[1], 1), oracle_physics(O, 1, 4, 0.1)
        sim.set_particles(pos, vel)
        ref = O.pack(w, pos, vel, capacity=n)
        assert_frame_equal(sim.read_frame(), ref, "a count that just fits")
        sim.step(1)
        ref = O.step(w, ph, ref[0], ref[1], ref[2], 1)[:3]
        with pytest.raises(W.WrachError):
            if add:
                sim.add_particles(more, more * 0)
            else:
                sim.set_particles(np.concatenate([pos, more]), np.concatenate([vel, more * 0]))
        assert_frame_equal(sim.read_frame(), ref, "refused")
        sim.step(2)
        ref = O.step(w, ph, ref[0], ref[1], ref[2], 2)[:3]
        assert_frame_equal(sim.read_frame(), ref, "two frames later")
    finally:
        sim.close()


@pytest.mark.parametrize("gx,gy", [(1, 3), (11, 93), (32, 32), (25, 41), (13, 79), (23, 89), (32, 64),
                                   (683, 3), (37, 83), (1024, 3), (439, 7), (4096, 1), (17, 241)])
@pytest.mark.parametrize("mode", [0, 1])
def test_cells_at_the_edges_of_half_tiles(W, O, gx, gy, mode):
    """The scan's threads take four cells of either half of a 2048-cell tile:
    grids whose last cells are just before, at and past a half's and a tile's
    end, with counts above the capacity and above 64 in the last cells."""
    rng = np.random.default_rng(gx * gy)
    dims = (gx - 0.5, gy - 0.5)
    piles = [(gx - 1, gy - 1, 70), (max(gx - 2, 0), gy - 1, 11), (0, 0, 66), (gx // 2, gy // 2, 9)]
    parts = [rng.uniform((0, 0), dims, size=(3 * gx * gy // 4 + 5, 2))]
    for cx, cy, m in piles:
        parts.append(np.column_stack([cx + rng.uniform(0.02, 0.45, m), cy + rng.uniform(0.02, 0.45, m)]))
    pos = rng.permutation(np.concatenate(parts)).astype(np.float32)
    vel = rng.normal(0, 0.4, size=pos.shape).astype(np.float32)
    _run(W, O, dims, pos, vel, mode, 3, 0.1 if mode else 0.0)
