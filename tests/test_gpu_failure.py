"""Failure detection without a GPU fault: a bounded device wait on a word
that nothing sets gives up after its limit and reports it, and the context
keeps working (the next frames match the oracle bit for bit).  Failures of
the host side (bad arguments, capacity) are the errors tested elsewhere."""
import numpy as np
import pytest

from tests.helpers import assert_frame_equal, make_sim, oracle_physics

pytestmark = pytest.mark.gpu


def test_bounded_wait_gives_up_and_the_context_stays_usable(W, O):
    dims = (50.0, 40.0)
    rng = np.random.default_rng(7)
    pos = rng.uniform((0, 0), dims, size=(1500, 2)).astype(np.float32)
    vel = rng.normal(0, 0.5, size=pos.shape).astype(np.float32)
    sim = make_sim(W, dims, 1, 1, 4, 0.1, capacity=3000)
    try:
        sim.add_particles(pos, vel)
        timed_out, waited = sim.selftest_wait(2000)
        assert timed_out and 2000 <= waited < 1_000_000
        assert sim.flags() == 0  # the probe leaves the sticky flags alone
        with pytest.raises(W.WrachError):
            sim.selftest_wait(2_000_000)  # above the 1 s cap
        w = O.world(*dims, 1)
        ref = O.pack(w, pos, vel, capacity=sim.capacity())
        sim.step(3)
        ref = O.step(w, oracle_physics(O, 1, 4, 0.1), ref[0], ref[1], ref[2], 3)[:3]
        assert_frame_equal(sim.read_frame(), ref, "frames after the probe")
    finally:
        sim.close()


@pytest.mark.parametrize("worlds", [1, 3])
@pytest.mark.parametrize("nth", range(1, 12))
def test_a_failed_growth_leaves_the_context_usable(W, O, worlds, nth):
    """An upload that has to grow the store, the staging buffers and the sort's
    scratch, with each of those allocations failing in turn (on the host): it
    reports that memory is out, and the frame goes on, through the captured
    frames, profiled ones and further uploads."""
    rng = np.random.default_rng(nth)
    dims, n = (40.0, 30.0), 500
    pos = rng.uniform((0, 0), dims, (n, 2)).astype(np.float32)
    vel = rng.normal(0, 0.5, pos.shape).astype(np.float32)
    far = rng.uniform(100, 200, (9000, 2)).astype(np.float32)
    more = rng.uniform((0, 0), dims, (10, 2)).astype(np.float32)
    cfg = W.WrachConfig(dimensions=dims, cell_size=1, mode=1, iterations=4, gravity=0.1, capacity=600)
    w, ph, at = O.world(dims[0], dims[1], 1), O.extended_physics(4, 0.1), worlds - 1
    with W.Simulation(cfg, worlds=[dims] * worlds if worlds > 1 else None) as sim:
        for k in range(worlds):
            sim.set_particles(pos, vel, world=k)
        sim.step(4)
        ref = O.step(w, ph, *O.pack(w, pos, vel, 600), 4)[:3]
        sim.selftest_alloc(nth)
        try:
            sim.add_particles(far, far * 0, world=at)
            assert nth > 10  # two of the store, two staging buffers, six of the sort
            ref = O.pack(w, pos, vel, 600)  # an upload packs the frame from the store
        except W.WrachError as e:
            assert e.code == W._lib.WRACH_ERR_OUT_OF_MEMORY and nth <= 10
        sim.selftest_alloc(0)
        assert_frame_equal(sim.read_frame(world=at), ref, "after the upload")
        for frame in range(4):
            if frame == 1:
                sim.profile_frame()
            else:
                sim.step(1)
            ref = O.step(w, ph, ref[0], ref[1], ref[2], 1)[:3]
            assert_frame_equal(sim.read_frame(world=at), ref, "frame %d" % frame)
        assert len(sim.read_keys(world=at)) == n
        sim.add_particles(more, more * 0, world=at)
        both = np.concatenate([pos, more]), np.concatenate([vel, more * 0])
        ref = O.pack(w, *both, 600)
        assert_frame_equal(sim.read_frame(world=at), ref, "a further upload")
        sim.step(3)
        assert_frame_equal(sim.read_frame(world=at), O.step(w, ph, *ref, 3)[:3], "and its frames")
