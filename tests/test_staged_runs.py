"""Staged runs of the SRD ensembles.

An ensemble's run kernel copies the particles of the batches ahead into a ring of 160
per warp (densities up to 32; denser ensembles read them from global memory, as a single
box does).  The ring, its wrap and the batches that wait for room change nothing: every
box must evolve bit-identically to a single-box handle, at the densities of each batch
size and at the two sides of the rule, with runs of odd length, with crowded cells (4n
of a cell collide, the largest a ring must hold beside an unfinished pass) and with
empty ones.
"""
from __future__ import annotations

import numpy as np
import pytest

from cudampcd_gb300 import capi

pytestmark = pytest.mark.gpu

MIXES = {
    "n1_n6": [dict(n=1, L=(5, 7, 9)), dict(n=6, L=(6, 5, 13))],
    "n7_n12": [dict(n=7, L=(7, 4, 11)), dict(n=12, L=(5, 5, 10))],
    "n13_n32": [dict(n=13, L=(5, 4, 9)), dict(n=32, L=(4, 5, 8))],
    "n20_n33": [dict(n=20, L=(4, 5, 8)), dict(n=33, L=(4, 4, 7))],
}


@pytest.mark.parametrize("crowded", [False, True])
@pytest.mark.parametrize("name", list(MIXES))
def test_ensemble_boxes_match_single_handles(name, crowded):
    boxes = [dict(b, periodic=(1, 1, r), dt=0.05, drag=1e-3, seed=70 + r) for r, b in enumerate(MIXES[name])]
    ens = capi.Handle(boxes=boxes)
    singles = [capi.Handle(**b) for b in boxes]
    try:
        if crowded:
            rng = np.random.default_rng(5)
            states = []
            for b, h in zip(boxes, singles):
                L = np.array(b["L"], np.float64)
                pos = (rng.random((h.N, 3)) - 0.5) * (L - [0, 0, 2])
                half = h.N // 2   # half of them in two layers, within four columns
                pos[:half] = -L / 2 + [0, 0, 1] + rng.random((half, 3)) * [2, 2, 2]
                states.append((pos.astype(np.float32), rng.normal(size=(h.N, 3)).astype(np.float32)))
                h.set_particles(*states[-1])
            ens.set_particles(*(np.concatenate(x) for x in zip(*states)))
        for steps in (1, 7):
            for h in [ens] + singles:
                h.step(steps)
            p, v = ens.positions(), ens.velocities()
            for r, h in enumerate(singles):
                first, N, _, _ = ens.box_range(r)
                assert np.array_equal(p[first:first + N], h.positions()), (r, steps)
                assert np.array_equal(v[first:first + N], h.velocities()), (r, steps)
        assert ens.counters()[1] == 0
    finally:
        ens.close()
        for h in singles:
            h.close()
