"""Readback into the caller's arrays: one launch writes those in pinned memory,
copies serve the others.  Whatever mix of pinned, pageable, missing and
unaligned arrays a caller passes, it holds the same bytes, and what lies past
the frame's particles stays as it was."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sim(W, worlds):
    r = np.random.default_rng(3)
    sim = W.Simulation(W.WrachConfig(dimensions=worlds[0], cell_size=2, mode=1, iterations=2,
                                     gravity=0.1, capacity=3000),
                       worlds=None if len(worlds) == 1 else worlds)
    for w, d in enumerate(worlds):
        n = 0 if w == 2 else 1201 + 700 * w
        sim.set_particles(r.uniform((0, 0), d, (n, 2)).astype(np.float32),
                          r.normal(0, 1, (n, 2)).astype(np.float32), world=w)
    sim.step(2)
    return sim


def _words(torch, count, pinned, skip):
    """`count` words of a sentinel, `skip` words into their allocation."""
    t = torch.full((count + skip,), 0x5A5A5A5A, dtype=torch.int32, pin_memory=pinned)
    return t.numpy()[skip:].view(np.uint32)


@pytest.mark.parametrize("worlds", [[(97.0, 61.0)], [(64.0, 33.0), (31.0, 130.0), (5.0, 5.0)]])
@pytest.mark.parametrize("kinds", ["ppp", "hhh", "php", "hhp", "pph", "p-p", "--p", "p--", "-hp", "pp-"])
@pytest.mark.parametrize("skip", [0, 1])
def test_every_mix_of_arrays_reads_the_same(W, worlds, kinds, skip):
    torch = pytest.importorskip("torch")
    sim = _sim(W, worlds)
    try:
        for w in range(len(worlds)):
            cap, cells = sim.capacity(w), sim.cells(w)
            n = int(sim.settings(w).particles_in_frame_count)
            # the frame as separate copies give it: one array a call
            want = [np.zeros(2 * cap, np.uint32), np.zeros(2 * cap, np.uint32),
                    np.zeros(cells + 2, np.uint32)]
            for k in range(3):
                args = [want[j].ctypes.data_as(ctypes.c_void_p) if j == k else None for j in range(3)]
                sim._check(_read(sim, w, args, cap))
            assert want[2][0] == 0 and want[2][-1] == n
            out = [None if c == "-" else _words(torch, len(want[k]), c == "p", skip)
                   for k, c in enumerate(kinds)]
            args = [None if a is None else a.ctypes.data_as(ctypes.c_void_p) for a in out]
            sim._check(_read(sim, w, args, cap))
            for k, a in enumerate(out):
                if a is None:
                    continue
                used = len(a) if k == 2 else 2 * n
                np.testing.assert_array_equal(a[:used], want[k][:used])
                assert (a[used:] == 0x5A5A5A5A).all()
    finally:
        sim.close()


def _read(sim, world, args, cap):
    f, u = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_uint32)
    p, v, i = args
    return sim._L.wrach_read(sim._ctx, world, p and ctypes.cast(p, f), v and ctypes.cast(v, f),
                             i and ctypes.cast(i, u), cap)
