"""Extended ensembles on the run kernel.

The run kernel takes an extended ensemble when no box is denser than 36 particles a cell:
its runs come from the host's table, and a warp changes its box and grid shifts between
runs.  Every box must evolve as a handle of its own, bit for bit: single steps, step graphs,
reads between them, samples, and a box crowded past its buckets and past 4n in a cell.
"""
from __future__ import annotations

import numpy as np
import pytest

from cudampcd_gb300 import capi

pytestmark = pytest.mark.gpu

BOXES = [
    dict(L=(8, 8, 22), periodic=(1, 1, 0), n=5, drag=1e-3, seed=11),
    dict(L=(13, 7, 30), periodic=(1, 1, 0), n=10, drag=1e-4, seed=12),
    dict(L=(8, 16, 20), periodic=(1, 1, 0), n=20, drag=1e-2, seed=13),
    dict(L=(6, 5, 7), periodic=(1, 1, 1), n=8, drag=0.0, seed=14),
    dict(L=(3, 4, 5), periodic=(1, 1, 0), n=1, drag=0.0, dt=0.1, seed=15),
    dict(L=(8, 8, 12), periodic=(1, 1, 0), n=36, drag=2e-3, temperature=0.5, seed=16),
]


def _check(ens, singles):
    pe, ve = ens.positions(), ens.velocities()
    for r, h in enumerate(singles):
        p0, n, _, _ = ens.box_range(r)
        assert np.array_equal(pe[p0:p0 + n], h.positions()), f"positions of box {r}"
        assert np.array_equal(ve[p0:p0 + n], h.velocities()), f"velocities of box {r}"


@pytest.mark.parametrize("crowded", [False, True])
@pytest.mark.parametrize("boxes", [BOXES, BOXES[::-1], BOXES[5:] + BOXES[4:5]], ids=["mixed", "reversed", "extremes"])
def test_boxes_of_an_extended_ensemble_evolve_as_single_handles(boxes, crowded):
    boxes = [dict(b, algorithm=1) for b in boxes]
    ens, singles = capi.Handle(boxes=boxes), [capi.Handle(**b) for b in boxes]
    try:
        if crowded:   # a third of every box in a thousandth of it
            pos, vel = [], []
            for h in singles:
                p, v = h.positions(), h.velocities()
                p[:h.N // 3] *= np.float32(0.1)
                h.set_particles(p, v)
                pos.append(p)
                vel.append(v)
            ens.set_particles(np.concatenate(pos), np.concatenate(vel))
        for steps in (1, 1, 7, 12):
            for h in (ens, *singles):
                h.step(steps)
            _check(ens, singles)
        for h in (ens, *singles):
            h.step_and_sample(9)
        density, velocity = ens.sample_mean()
        for r, (box, h) in enumerate(zip(boxes, singles)):
            _, _, c0, nc = ens.box_range(r)
            d, v = h.sample_mean()
            assert np.array_equal(density[c0:c0 + nc], d), f"density of box {r}"
            # FP32 sums of a cell's velocities in any order, 9 of them over 8
            assert np.abs(velocity[c0:c0 + nc] - v).max() <= 4 * box["n"] * 2.0 ** -22, f"velocity of box {r}"
        _check(ens, singles)
        assert ens.counters()[1] == 0
    finally:
        ens.close()
        for h in singles:
            h.close()
