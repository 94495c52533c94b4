"""The run kernels against the tile kernel.

Production steps (Philox draws) and their replays run on ext_run_kernel (extended
collision, n <= 36) and srd_run_kernel (n <= 64), with the wall-pressure estimator too;
MPCD_GB_TILE_KERNEL=1, read when a handle is created, keeps a handle on the tile kernel.
Both walk a cell's participants in particle-id order with the same partial sums
(extended) or sum exactly (SRD), so the states must be bit-identical: at the densities
where an extended run is 24, 16, 8 or fewer cells (n = 1 .. 36; 37 is the tile kernel's on
both sides), with runs that end inside a column and rounds of fewer than 8 cells, and
with particles crowded so that a run's entries do not fit the warp's buffer (the run is
swept in parts) and cells hold more than their bucket's depth and more than 4n.
"""
from __future__ import annotations

import numpy as np
import pytest

from cudampcd_gb300 import capi

pytestmark = pytest.mark.gpu


def _pair(monkeypatch, **kw):
    run = capi.Handle(**kw)
    monkeypatch.setenv("MPCD_GB_TILE_KERNEL", "1")
    tile = capi.Handle(**kw)
    monkeypatch.delenv("MPCD_GB_TILE_KERNEL")
    return run, tile


def _same(a, b, what):
    assert np.array_equal(a.positions(), b.positions()), f"positions {what}"
    assert np.array_equal(a.velocities(), b.velocities()), f"velocities {what}"


def _advance(a, b, what):
    for h in (a, b):
        h.step(1)
    _same(a, b, f"{what}, one step")
    for h in (a, b):
        h.step_and_sample(8)   # a graph replay and single steps
    _same(a, b, f"{what}, sampled steps")
    (da, va), (db, vb) = a.sample_mean(), b.sample_mean()
    assert np.array_equal(da, db)
    assert np.abs(va - vb).max() <= 1e-5   # FP32 atomic sums in storage order
    assert a.counters() == b.counters()


@pytest.mark.parametrize("n", [1, 2, 5, 6, 7, 13, 20, 36, 37])
def test_run_kernel_matches_tile_kernel(n, monkeypatch):
    a, b = _pair(monkeypatch, L=(7, 5, 11), periodic=(1, 1, 0), n=n, dt=0.05, drag=1e-3, algorithm=1, seed=20 + n)
    try:
        _advance(a, b, f"n={n}")
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("n", [2, 10, 36])
def test_crowded_runs_are_swept_in_parts(n, monkeypatch):
    a, b = _pair(monkeypatch, L=(6, 7, 13), periodic=(1, 1, 0), n=n, dt=0.05, algorithm=1, seed=40 + n)
    rng = np.random.default_rng(n)
    pos = np.empty((a.N, 3), np.float32)
    half = a.N // 2   # half of the particles in a 3 x 3 x 2 corner at the wall, the others anywhere
    pos[:half] = np.array([-3.0, -3.5, -5.5]) + rng.random((half, 3)) * np.array([3.0, 3.0, 2.0])
    pos[half:] = (rng.random((a.N - half, 3)) - 0.5) * np.array([6.0, 7.0, 11.0])
    vel = rng.normal(size=(a.N, 3)).astype(np.float32)
    order = rng.permutation(a.N)   # ids in no spatial order
    try:
        for h in (a, b):
            h.set_particles(pos[order], vel)
        assert a.layout()[3].max() > 4 * n
        _advance(a, b, f"crowded n={n}")
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("algorithm", [0, 1])
@pytest.mark.parametrize("n", [5, 10, 20])
def test_pressure_matches_tile_kernel(algorithm, n, monkeypatch):
    """The estimator's impulses: FP64 per thread here, FP32 per thread in the tile kernel
    (each partial within steps * 2^-24 of its size, over impulses that add up)."""
    a, b = _pair(monkeypatch, L=(9, 8, 7), periodic=(1, 1, 0), n=n, dt=0.05, drag=1e-3, algorithm=algorithm, seed=n)
    try:
        for h in (a, b):
            h.wall_pressure(restart=True)
        _advance(a, b, "with the estimator")
        pa, pb = a.wall_pressure(), b.wall_pressure()
        assert pa[2] == pb[2] == 9
        assert np.allclose(pa[:2], pb[:2], rtol=1e-5, atol=0)
    finally:
        a.close()
        b.close()
