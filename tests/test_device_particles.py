"""Particles read into and set from device buffers.

A read into device buffers replays the last step straight into them: large SRD boxes in
two passes (a map by particle id, then a gather), the others by scattered rows; later
reads of the same state copy it.  Each must return what the host getters return, bit for
bit: on both sides of the size rule, in crowded boxes whose cells overflow their buckets
and hold more than 4n (those particles lie in no slot), after single steps and graph
replays, and after sets of positions or velocities alone.
"""
from __future__ import annotations

import numpy as np
import pytest

from cudampcd_gb300 import capi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

BOXES = {
    "small": dict(L=(12, 10, 14), periodic=(1, 1, 0), n=10, drag=1e-3, seed=1),
    "extended": dict(L=(12, 10, 14), periodic=(1, 1, 0), n=10, algorithm=1, seed=2),
    "gathered_n5": dict(L=(66, 60, 50), periodic=(1, 1, 1), n=5, seed=3),        # batches of 16 cells
    "gathered_n10": dict(L=(50, 49, 42), periodic=(1, 1, 0), n=10, drag=1e-3, seed=4),   # of 8
    "gathered_n40": dict(L=(30, 31, 30), periodic=(1, 1, 0), n=40, seed=5),      # of 4
    "ensemble": dict(boxes=[dict(L=(8, 8, 20), periodic=(1, 1, 0), n=10, seed=6), dict(L=(6, 5, 9), n=5, seed=7)]),
}


def _read(h):
    out = [torch.full((h.N, 3), float("nan"), device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    h.get_particles_device(*(t.data_ptr() for t in out))
    return [t.cpu().numpy() for t in out]


@pytest.mark.parametrize("crowded", [False, True])
@pytest.mark.parametrize("name", list(BOXES))
def test_device_reads_match_host_reads(name, crowded):
    a, b = capi.Handle(**BOXES[name]), capi.Handle(**BOXES[name])
    try:
        if crowded:
            pos, vel = a.positions(), a.velocities()
            third = slice(0, a.N // 3)
            pos[third] = pos[third] * np.float32(0.1)   # a third of the particles in a thousandth of the box
            for h in (a, b):
                h.set_particles(pos, vel)
        for steps in (1, 7):
            a.step(steps)
            b.step(steps)
            p, v = _read(a)
            assert np.array_equal(p, b.positions()) and np.array_equal(v, b.velocities())
            p, v = _read(a)   # again: kept and copied
            assert np.array_equal(p, b.positions()) and np.array_equal(v, b.velocities())
        v = torch.from_numpy(b.velocities()[::-1].copy()).cuda()
        torch.cuda.synchronize()
        a.set_particles_device(0, v.data_ptr())
        b.set_velocities(v.cpu().numpy())
        a.step(2)
        b.step(2)
        p, v = _read(a)
        assert np.array_equal(p, b.positions()) and np.array_equal(v, b.velocities())
        assert a.counters()[1] == 0
    finally:
        a.close()
        b.close()
