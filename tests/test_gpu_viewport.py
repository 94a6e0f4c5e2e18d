"""Viewport streaming with write-back to the store, bit for bit against the
oracle's rules: the frame is packed from the store's particles inside the
viewport (create_packed_data), a write-back makes the store its particles
outside the viewport followed by the frame, and moving the viewport writes
back and re-packs under the new anchor (walls included)."""
import numpy as np
import pytest

from tests.helpers import assert_frame_equal, make_sim, oracle_physics, same_bits

pytestmark = pytest.mark.gpu


def _field(seed, n, lo, hi):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(lo, hi, size=(n, 2)).astype(np.float32)
    vel = rng.normal(0, 0.6, size=(n, 2)).astype(np.float32)
    return pos, vel


def _store_equal(sim, ref, what, world=0):
    gp, gv = sim.store(world)
    rp, rv = ref
    assert len(gp) == len(rp), what + ": store size %d vs %d" % (len(gp), len(rp))
    assert same_bits(gp, rp) and same_bits(gv, rv), what + ": store contents"


@pytest.mark.parametrize("mode", [0, 1])
def test_write_back_and_moving_viewport(W, O, mode):
    dims, cs = (64.0, 48.0), 1
    pos, vel = _field(1, 5000, (-40.0, -30.0), (104.0, 78.0))
    sim = make_sim(W, dims, cs, mode, 4, 0.1 if mode else 0.0, capacity=8000)
    try:
        ph = oracle_physics(O, mode, 4, 0.1 if mode else 0.0)
        w = O.world(dims[0], dims[1], cs)
        sim.add_particles(pos, vel)
        store = (pos, vel)
        _store_equal(sim, store, "after add")
        frame = O.pack(w, pos, vel, capacity=sim.capacity())
        assert_frame_equal(sim.read_frame(), frame, "upload")
        sim.step(5)
        frame = O.step(w, ph, frame[0], frame[1], frame[2], 5)[:3]
        assert_frame_equal(sim.read_frame(), frame, "5 frames")
        # write-back alone leaves the frame as it is
        sim.write_back()
        store = O.write_back(w, store[0], store[1], frame[1], frame[2])
        _store_equal(sim, store, "write-back")
        assert_frame_equal(sim.read_frame(), frame, "frame after write-back")
        for anchor in [(10.5, -7.25), (-31.0, 20.0), (0.0, 0.0)]:
            sim.set_viewport(anchor)
            store = O.write_back(w, store[0], store[1], frame[1], frame[2])
            w = O.world(dims[0], dims[1], cs, anchor=anchor)
            _store_equal(sim, store, "store at %s" % (anchor,))
            frame = O.pack(w, store[0], store[1], capacity=sim.capacity())
            assert_frame_equal(sim.read_frame(), frame, "frame at %s" % (anchor,))
            s = sim.settings()
            assert (s.view_anchor[0], s.view_anchor[1]) == anchor
            sim.step(4)
            frame = O.step(w, ph, frame[0], frame[1], frame[2], 4)[:3]
            assert_frame_equal(sim.read_frame(), frame, "4 frames at %s" % (anchor,))
    finally:
        sim.close()


def test_moving_one_world_of_a_batch(W, O):
    dims = [(40.0, 30.0), (50.0, 20.0), (30.0, 30.0)]
    cfg = W.WrachConfig(cell_size=1, mode=1, iterations=4, gravity=0.1, capacity=4000)
    fields = [_field(10 + k, 1500, (-20.0, -20.0), (d[0] + 20.0, d[1] + 20.0)) for k, d in enumerate(dims)]
    with W.Simulation(cfg, worlds=dims) as sim:
        for k, (p, v) in enumerate(fields):
            sim.set_particles(p, v, world=k)
        sim.step(3)
        before = [sim.read_frame(world=k) for k in (0, 2)]
        sim.set_viewport((7.0, -5.0), world=1)
        ph = O.extended_physics(4, 0.1)
        w1 = O.world(dims[1][0], dims[1][1], 1)
        f1 = O.pack(w1, fields[1][0], fields[1][1], capacity=sim.capacity(1))
        f1 = O.step(w1, ph, f1[0], f1[1], f1[2], 3)[:3]
        store = O.write_back(w1, fields[1][0], fields[1][1], f1[1], f1[2])
        _store_equal(sim, store, "world 1 store", world=1)
        w1 = O.world(dims[1][0], dims[1][1], 1, anchor=(7.0, -5.0))
        assert_frame_equal(sim.read_frame(world=1), O.pack(w1, store[0], store[1], capacity=sim.capacity(1)),
                           "world 1 frame")
        for k, b in zip((0, 2), before):
            a = sim.read_frame(world=k)
            assert np.array_equal(a[2], b[2]) and same_bits(a[0], b[0]) and same_bits(a[1], b[1])


def test_a_move_that_changes_the_grid_is_refused(W):
    # 10 px wide with 3 px cells: anchored at 0 the grid is 4 cells wide, at
    # 2.5 it is 5
    sim = make_sim(W, (10.0, 9.0), 3, capacity=100)
    try:
        sim.add_particles(np.array([[1.0, 1.0]], np.float32), np.zeros((1, 2), np.float32))
        with pytest.raises(W.WrachError):
            sim.set_viewport((2.5, 0.0))
        assert tuple(sim.settings().view_anchor) == (0.0, 0.0)
        sim.set_viewport((3.0, 0.0))  # a whole cell: the grid keeps its size
        assert tuple(sim.settings().view_anchor) == (3.0, 0.0)
    finally:
        sim.close()


@pytest.mark.parametrize("n", [0, 1, 31, 33, 1023, 1024, 1025, 2049])
@pytest.mark.parametrize("outside", ["none", "all", "mixed", "last"])
def test_write_back_at_tile_edges(W, O, n, outside):
    """The store's rebuild moves 1024 items a block by a bit an item: its
    edges, with no item, every item, some or the last one outside."""
    dims = (16.0, 9.0)
    pos, vel = _field(n, n, (0.0, 0.0), (15.9, 8.9))
    out = {"none": np.zeros(n, bool), "all": np.ones(n, bool),
           "mixed": np.arange(n) % 7 < 3, "last": np.arange(n) == n - 1}[outside]
    pos[out] += np.float32([32.0, 0.0])
    sim = make_sim(W, dims, 1, 1, 2, 0.1, capacity=max(n, 1))
    try:
        w, ph = O.world(dims[0], dims[1], 1), oracle_physics(O, 1, 2, 0.1)
        sim.set_particles(pos, vel)
        frame = O.pack(w, pos, vel, capacity=sim.capacity())
        sim.step(1)
        frame = O.step(w, ph, frame[0], frame[1], frame[2], 1)[:3]
        sim.write_back()
        _store_equal(sim, O.write_back(w, pos, vel, frame[1], frame[2]), "n %d %s" % (n, outside))
        assert_frame_equal(sim.read_frame(), frame, "the frame stays")
    finally:
        sim.close()


@pytest.mark.parametrize("worlds", [1, 3])
@pytest.mark.parametrize("add", [False, True])
@pytest.mark.parametrize("why", ["capacity", 1, 2, 3, 7])
def test_a_refused_upload_leaves_the_store(W, O, worlds, add, why):
    """More particles than the frame takes, or (a number) that allocation of a
    growth failing: frame and store stay as they are, and what follows works
    from them."""
    dims, cap, at = (40.0, 30.0), 800, worlds - 1
    pos, vel = _field(21, 1000, (0.0, 0.0), (39.9, 29.9))
    pos[700:] += np.float32([64.0, 0.0])  # outside the viewport
    if why == "capacity":
        more = _field(22, 900, (0.0, 0.0), (39.9, 29.9))
    else:
        more = _field(22, 20000, (100.0, 0.0), (140.0, 29.9))
    cfg = W.WrachConfig(dimensions=dims, cell_size=1, mode=1, iterations=2, gravity=0.1, capacity=cap)
    w, ph = O.world(dims[0], dims[1], 1), O.extended_physics(2, 0.1)
    with W.Simulation(cfg, worlds=[dims] * worlds if worlds > 1 else None) as sim:
        for k in range(worlds):
            sim.set_particles(pos, vel, world=k)
        sim.step(2)
        frame = O.step(w, ph, *O.pack(w, pos, vel, cap), 2)[:3]
        with pytest.raises(W.WrachError) as e:
            if why != "capacity":
                sim.selftest_alloc(why)
            (sim.add_particles if add else sim.set_particles)(*more, world=at)
        sim.selftest_alloc(0)
        assert e.value.code == (2 if why == "capacity" else 4)
        _store_equal(sim, (pos, vel), "after the refusal", world=at)
        assert_frame_equal(sim.read_frame(world=at), frame, "after the refusal")
        extra = _field(23, 20, (0.0, 0.0), (39.9, 29.9))
        sim.add_particles(*extra, world=at)
        store = np.concatenate([pos, extra[0]]), np.concatenate([vel, extra[1]])
        _store_equal(sim, store, "a further upload", world=at)
        frame = O.pack(w, *store, cap)
        assert_frame_equal(sim.read_frame(world=at), frame, "a further upload")
        sim.step(1)
        frame = O.step(w, ph, *frame, 1)[:3]
        sim.set_viewport((64.0, 0.0), world=at)
        store = O.write_back(w, store[0], store[1], frame[1], frame[2])
        w = O.world(dims[0], dims[1], 1, anchor=(64.0, 0.0))
        _store_equal(sim, store, "a move", world=at)
        assert_frame_equal(sim.read_frame(world=at), O.pack(w, *store, cap), "a move")
        sim.set_particles(*extra, world=at)
        _store_equal(sim, extra, "a replacing upload", world=at)


@pytest.mark.parametrize("worlds", [1, 2])
def test_replacing_uploads_of_every_size(W, O, worlds):
    # from none to more and back: a replacing upload's particles are staged, and
    # its buffers and the store's change places
    dims = (40.0, 30.0)
    cfg = W.WrachConfig(dimensions=dims, cell_size=1, mode=1, iterations=2, gravity=0.1, capacity=3000)
    w, ph = O.world(dims[0], dims[1], 1), O.extended_physics(2, 0.1)
    with W.Simulation(cfg, worlds=[dims] * worlds if worlds > 1 else None) as sim:
        for k, n in enumerate([0, 5, 0, 900, 2900, 1, 2900, 0, 30]):
            pos, vel = _field(40 + k, n, (-10.0, 0.0), (39.9, 29.9))
            sim.set_particles(pos, vel, world=worlds - 1)
            _store_equal(sim, (pos, vel), "%d particles" % n, world=worlds - 1)
            ref = O.pack(w, pos, vel, 3000)
            assert_frame_equal(sim.read_frame(world=worlds - 1), ref, "%d particles" % n)
            sim.step(2)
            assert_frame_equal(sim.read_frame(world=worlds - 1), O.step(w, ph, *ref, 2)[:3], "frames of %d" % n)


@pytest.mark.parametrize("worlds", [1, 3])
@pytest.mark.parametrize("mode", [0, 1])
def test_a_refused_move_leaves_the_viewport(W, O, worlds, mode):
    """A move to where the store holds more particles than the frame takes, and
    one that each of its allocations fails in turn: settings, frame, the next
    steps' walls and the store stay, and the moves after it start from them."""
    dims, cap, at, K = (40.0, 30.0), 800, worlds - 1, 4 if mode else 1
    pos, vel = _field(31, 1700, (0.0, 0.0), (39.9, 29.9))
    pos[700:1600] += np.float32([64.0, 0.0])  # too many there
    pos[1600:] += np.float32([128.0, 0.0])
    cfg = W.WrachConfig(dimensions=dims, cell_size=1, mode=mode, iterations=K, gravity=0.1 if mode else 0.0,
                        capacity=cap)
    w, ph = O.world(dims[0], dims[1], 1), oracle_physics(O, mode, K, 0.1 if mode else 0.0)
    store = pos, vel
    with W.Simulation(cfg, worlds=[dims] * worlds if worlds > 1 else None) as sim:
        for k in range(worlds):
            sim.set_particles(pos, vel, world=k)
        sim.step(3)
        frame = O.step(w, ph, *O.pack(w, pos, vel, cap), 3)[:3]

        def unmoved(what):
            nonlocal frame
            assert tuple(sim.settings(at).view_anchor) == (0.0, 0.0), what
            _store_equal(sim, store, what, world=at)
            assert_frame_equal(sim.read_frame(world=at), frame, what)
            sim.step(2)
            frame = O.step(w, ph, *frame, 2)[:3]
            assert_frame_equal(sim.read_frame(world=at), frame, what + ", two frames later")

        with pytest.raises(W.CapacityError):
            sim.set_viewport((64.0, 0.0), world=at)
        unmoved("after the refusal")
        sim.write_back(world=at)
        store = O.write_back(w, store[0], store[1], frame[1], frame[2])
        _store_equal(sim, store, "write-back", world=at)
        grown = np.concatenate([store[0], pos[700:] + np.float32([96.0, 0.0])])
        store = grown, np.concatenate([store[1], vel[700:]])
        sim.set_particles(*store, world=at)
        frame = O.pack(w, *store, cap)
        nth = 1
        while True:
            sim.selftest_alloc(nth)
            try:
                sim.set_viewport((128.0, 0.0), world=at)
                break
            except W.WrachError as e:
                assert e.code == W._lib.WRACH_ERR_OUT_OF_MEMORY and nth < 12
                unmoved("allocation %d" % nth)
            nth += 1
        sim.selftest_alloc(0)
        for anchor in [(128.0, 0.0), (0.0, 0.0)]:
            if anchor[0] == 0.0:
                sim.set_viewport(anchor, world=at)
            store = O.write_back(w, store[0], store[1], frame[1], frame[2])
            w = O.world(dims[0], dims[1], 1, anchor=anchor)
            frame = O.pack(w, *store, cap)
            _store_equal(sim, store, "moved to %s" % (anchor,), world=at)
            assert_frame_equal(sim.read_frame(world=at), frame, "moved to %s" % (anchor,))
            sim.step(2)
            frame = O.step(w, ph, *frame, 2)[:3]
            assert_frame_equal(sim.read_frame(world=at), frame, "two frames at %s" % (anchor,))


@pytest.mark.parametrize("surrogate", [False, True])
def test_a_batch_moves_between_captured_frames(W, O, surrogate):
    """A batch keeps its captured frames over a move (they read the worlds'
    settings from the device): the frames after it have the new walls."""
    dims = [(40.0, 30.0), (50.0, 20.0)]
    cfg = W.WrachConfig(cell_size=1, mode=1, iterations=4, gravity=0.1, capacity=2000)
    fields = [_field(70 + k, 1200, (2.0, 2.0), (d[0] - 8.0, d[1] - 8.0)) for k, d in enumerate(dims)]
    ph = O.extended_physics(4, 0.1)
    worlds = [O.world(d[0], d[1], 1) for d in dims]
    ref = [O.pack(w, p, v, 2000) for w, (p, v) in zip(worlds, fields)]
    with W.Simulation(cfg, worlds=dims) as sim:
        for k, (p, v) in enumerate(fields):
            sim.set_particles(p, v, world=k)
        if surrogate:
            sim.surrogate_init(0, 1)
        # an impossible bound on the overlap: every surrogate frame falls back
        step = (lambda n: sim.surrogate_step(n, max_penetration=-1e9)) if surrogate else sim.step
        for anchor in [(1.0, 1.0), (0.0, 0.0)]:
            step(6)
            ref = [O.step(w, ph, *r, 6)[:3] for w, r in zip(worlds, ref)]
            sim.set_viewport(anchor, world=1)
            store = O.write_back(worlds[1], *fields[1], ref[1][1], ref[1][2])
            fields[1] = store
            worlds[1] = O.world(dims[1][0], dims[1][1], 1, anchor=anchor)
            ref[1] = O.pack(worlds[1], *store, 2000)
            for frames in (1, 5):
                step(frames)
                ref = [O.step(w, ph, *r, frames)[:3] for w, r in zip(worlds, ref)]
                for k in (0, 1):
                    assert_frame_equal(sim.read_frame(world=k), ref[k], "world %d at %s" % (k, anchor))
