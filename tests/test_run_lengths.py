"""Run lengths of the SRD step kernel.

A warp of the run kernel sweeps a run of up to 32 consecutive cells; the engine
chooses the length from the cells of the box and the warps of the GPU.  The length
is a work decomposition only: SRD cell sums are exact, so the states must be
bit-identical for every length (MPCD_GB_RUN_CELLS, read when a handle is created,
forces one): a single cell, odd lengths that end inside a batch of cells and inside
a column, one more and one less than a batch, and the longest.
"""
from __future__ import annotations

import os

import numpy as np
import pytest

from cudampcd_gb300 import capi

pytestmark = pytest.mark.gpu

BOXES = {
    "n5": dict(L=(7, 9, 13), periodic=(1, 1, 1), n=5, seed=3),              # batches of 16 cells
    "n10": dict(L=(6, 5, 11), periodic=(1, 1, 0), n=10, drag=1e-3, seed=4),   # of 8
    "n20": dict(L=(5, 7, 9), periodic=(1, 1, 0), n=20, drag=1e-3, seed=5),    # of 4
    "ensemble": dict(boxes=[dict(L=(8, 5, 20), periodic=(1, 1, 0), n=5, seed=11),
                            dict(L=(5, 8, 21), periodic=(1, 1, 0), n=10, seed=12),
                            dict(L=(4, 4, 23), periodic=(1, 1, 0), n=20, seed=13)]),
}


def _states(box, cells, monkeypatch):
    if cells:
        monkeypatch.setenv("MPCD_GB_RUN_CELLS", str(cells))
    else:
        monkeypatch.delenv("MPCD_GB_RUN_CELLS", raising=False)
    h = capi.Handle(**box)
    try:
        h.step(1)
        h.step_and_sample(13)   # single steps and graph replays
        return h.positions(), h.velocities(), h.sample_mean()[0]
    finally:
        h.close()


@pytest.mark.parametrize("cells", [1, 3, 7, 9, 22, 32])
@pytest.mark.parametrize("name", list(BOXES))
def test_run_length_changes_nothing(name, cells, monkeypatch):
    base = _states(BOXES[name], 0, monkeypatch)
    other = _states(BOXES[name], cells, monkeypatch)
    for a, b in zip(base, other):
        assert np.array_equal(a, b)
