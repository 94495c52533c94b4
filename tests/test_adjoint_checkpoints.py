"""The adjoint of a forward that keeps checkpoints instead of its tape.

MPCD_GB_TAPE_BYTES = 0, read when a handle is created, sends every forward there (without it
a tape of up to 4 GiB is kept).  The backward then recomputes the forward segment by
segment and carries the adjoint velocities from one segment to the one before it.  The
tape must be the kept one, word for word, so that the two gradients are those of the same
map; their sums over cells do not depend on the order of arrival, so that they are the same bits, the
drag gradient to FP64 rounding.
"""
from __future__ import annotations

import numpy as np
import pytest

from cudampcd_gb300 import capi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

BOUNCE = 0x80000000
NONE = 0xFFFFFFFF
LIMIT = "MPCD_GB_TAPE_BYTES"


def _pair(monkeypatch, **box):
    kept = capi.Handle(**box)
    monkeypatch.setenv(LIMIT, "0")
    segments = capi.Handle(**box)
    monkeypatch.delenv(LIMIT)
    return kept, segments


def _start(h, pos, vel, step=4):
    h.set_step(step)
    h.set_particles(pos, vel)


@pytest.mark.parametrize("steps,every", [(1, 1), (3, 1), (7, 3), (8, 4), (13, 20), (13, 5)])
@pytest.mark.parametrize("n", [5, 10, 70])
def test_checkpoints_give_the_gradients_of_the_kept_tape(monkeypatch, n, steps, every):
    """Segments of one step, that divide the steps, that do not, and a single one."""
    L = (6, 5, 9)
    kept, segments = _pair(monkeypatch, L=L, periodic=(1, 1, 0), n=n, dt=0.05, drag=0.01, seed=9)
    try:
        pos, vel = kept.positions(), kept.velocities()
        dU = torch.linspace(-1.0, 2.0, L[2], device="cuda")
        got = []
        for h in (kept, segments):
            _start(h, pos, vel)
            profile, dv = torch.empty(L[2], device="cuda"), torch.empty((h.N, 3), device="cuda")
            torch.cuda.synchronize()
            h.profile_forward(steps, every, profile.data_ptr())
            assert h.step_index == 4 + steps
            drag = h.profile_backward(dU.data_ptr(), dv.data_ptr())
            got.append((profile.cpu().numpy(), dv.cpu().numpy(), drag, h.profile_tape(steps)))
        a, b = got
        for x, y in zip(a[3], b[3]):
            assert np.array_equal(x, y)
        # FP32 cell sums of about n velocities of order 1, in any order
        assert np.abs(a[0] - b[0]).max() <= n * 2.0 ** -24
        assert np.array_equal(a[1], b[1])
        assert abs(a[2] - b[2]) <= 1e-12 * abs(a[2])
    finally:
        kept.close()
        segments.close()


@pytest.mark.parametrize("limit", [None, "0"])
@pytest.mark.parametrize("n", [5, 10])
def test_collision_cells_are_those_of_the_shifted_grid(monkeypatch, n, limit):
    """The cell of a particle's collision, from the state before the step: streamed (bounced
    at a wall), shifted by the step's grid shift and wrapped; alone without ghosts, none."""
    if limit is not None:
        monkeypatch.setenv(LIMIT, limit)
    L, dt, steps = (6, 5, 9), 0.05, 7
    a, b = (capi.Handle(L=L, periodic=(1, 1, 0), n=n, dt=dt, drag=0.01, seed=9) for _ in range(2))
    try:
        pos, vel = b.positions(), b.velocities()
        for h in (a, b):
            _start(h, pos, vel)
        profile = torch.empty(L[2], device="cuda")
        a.profile_forward(steps, 3, profile.data_ptr())
        key, _, ncell, _, _ = a.profile_tape(steps)
        size = np.array(L, np.float64)
        for t in range(steps):
            x, v = b.positions().astype(np.float64), b.velocities().astype(np.float64)
            wall = size[2] / 2.0 - 1.0
            nz = x[:, 2] + v[:, 2] * dt
            out = np.abs(nz) > wall
            left = np.where(out, (np.sign(nz) * wall - x[:, 2]) / np.where(out, v[:, 2], 1.0), dt)
            x = x + v * left[:, None] - v * (dt - left)[:, None]
            y = x + np.array(b.shift(b.step_index), np.float64) + size / 2.0
            y -= np.floor(y / size) * size
            cell = np.floor(y).astype(np.int64)
            cell = cell[:, 2] + L[2] * (cell[:, 0] + L[0] * cell[:, 1])
            # a particle within FP32 rounding of a cell face may be on either side
            clear = (np.abs(y - np.round(y)) > 1e-5).all(1)
            n_c = ncell[t][cell]
            expected = np.where(n_c > 0, cell, NONE)
            assert clear.mean() > 0.99
            assert np.array_equal(key[t][clear].astype(np.int64), expected[clear])
            b.step(1)
    finally:
        a.close()
        b.close()
