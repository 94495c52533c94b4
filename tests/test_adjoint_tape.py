"""The adjoint's tape against the trajectory it records.

A forward records the tape of its steps as it runs where it fits, each step folding
the sample of the one before; the tape's lab cells, counts and collision cells must be
those of the states that plain steps reach, for one step, two, odd counts and intervals
that do not divide them, in boxes of each batch size and on the tile kernel.
"""
from __future__ import annotations

import numpy as np
import pytest

from cudampcd_gb300 import capi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

BOUNCE = 0x80000000
NONE = 0xFFFFFFFF


@pytest.mark.parametrize("steps,every", [(1, 1), (2, 5), (3, 2), (7, 3), (13, 20)])
@pytest.mark.parametrize("n", [5, 10, 70])
def test_tape_matches_the_trajectory(n, steps, every):
    """n = 70 runs on the tile kernel, which folds each sample at once."""
    L = (6, 5, 9)
    a, b = (capi.Handle(L=L, periodic=(1, 1, 0), n=n, dt=0.05, drag=0.01, seed=9) for _ in range(2))
    try:
        pos, vel = b.positions(), b.velocities()
        for h in (a, b):
            h.set_step(4)
            h.set_particles(pos, vel)
        profile = torch.empty(L[2], dtype=torch.float32, device="cuda")
        a.profile_forward(steps, every, profile.data_ptr())
        key, lab, ncell, count, _ = a.profile_tape(steps)
        u = np.zeros(L[2])
        for t in range(steps):
            b.step(1)
            x, v = b.positions().astype(np.float64), b.velocities()
            c = np.floor(x + np.array(L) / 2.0).astype(np.int64) % np.array(L)
            cell = c[:, 2] + L[2] * (c[:, 0] + L[0] * c[:, 1])
            assert np.array_equal(lab[t] & np.uint32(~BOUNCE & 0xFFFFFFFF), cell)
            assert np.array_equal(count[t], np.bincount(cell, minlength=a.C))
            collided = key[t] != NONE
            inside = np.bincount(key[t][collided], minlength=a.C)
            assert np.all(inside <= ncell[t]) and np.all((ncell[t] > 0) >= (inside > 0))
            sums = np.bincount(cell, weights=v[:, 0], minlength=a.C) / np.maximum(count[t], 1)
            u += sums.reshape(L[1], L[0], L[2]).mean((0, 1)) / steps
        # FP32 cell sums of about n velocities of order 1: n 2^-24 a cell, averaged over the layer
        assert np.abs(profile.cpu().numpy() - u).max() <= n * 2.0 ** -24
    finally:
        a.close()
        b.close()
