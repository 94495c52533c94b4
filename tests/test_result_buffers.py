"""Result arrays whose memory later reads may reuse.

A read takes the memory of an earlier result once nothing refers to it; a result that is
still referred to, itself or through a view, must keep its values, and one that outlives
its simulation must too.
"""
from __future__ import annotations

import gc

import numpy as np
import pytest

import cudampcd_gb300 as pympcd
from cudampcd_gb300 import capi

pytestmark = pytest.mark.gpu


def _simulation():
    p = pympcd.Params()
    p.n = 10
    p.periodicity = (1, 1, 0)
    p.volume_size = (8, 8, 10)
    p.seed = 4
    return pympcd.Simulation(p, "cuda")


@pytest.mark.parametrize("kind", ["simulation", "handle"])
def test_results_keep_their_values(kind):
    s = _simulation() if kind == "simulation" else capi.Handle(L=(8, 8, 12), periodic=(1, 1, 0), n=10, seed=4)

    def fields():
        s.step_and_sample(3)
        return s.get_mean_fields() if kind == "simulation" else s.sample_mean()

    kept, copies, views = [], [], []
    for k in range(8):
        d, v = fields()
        if k % 2:   # every other result is kept: whole, or only a view of it
            copies.append((d.copy(), v[..., 1].copy()))
            kept.append(d)
            views.append(v[..., 1])
        del d, v
        gc.collect()
    del s
    gc.collect()
    for (d, v), a, b in zip(copies, kept, views):
        assert np.array_equal(d, a) and np.array_equal(v, b)
    assert len({a.__array_interface__["data"][0] for a in kept}) == len(kept)
