"""The handle's sample after a forward profile.

A forward leaves the sample sums of its steps with the handle: the mean fields are those of
as many sampled steps, and further sampled steps continue the average, whether the forward
kept its tape or checkpoints, on a fresh handle and after other sampling.
"""
from __future__ import annotations

import numpy as np
import pytest

from cudampcd_gb300 import capi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("before", [0, 5])
@pytest.mark.parametrize("after", [0, 4])
@pytest.mark.parametrize("limit", [None, "0"], ids=["tape", "checkpoints"])
def test_fields_after_a_forward_are_those_of_its_steps(monkeypatch, limit, before, after):
    if limit is not None:
        monkeypatch.setenv("MPCD_GB_TAPE_BYTES", limit)
    n, steps = 10, 7
    box = dict(L=(6, 5, 9), periodic=(1, 1, 0), n=n, drag=0.01, seed=9)
    a, b = capi.Handle(**box), capi.Handle(**box)
    try:
        if before:
            for h in (a, b):
                h.step_and_sample(before)
                h.sample_mean()
        profile = torch.empty(9, device="cuda")
        a.profile_forward(steps, 3, profile.data_ptr())
        b.step_and_sample(steps)
        if after:
            for h in (a, b):
                h.step_and_sample(after)
        (d0, v0), (d1, v1) = a.sample_mean(), b.sample_mean()
        assert np.array_equal(d0, d1)
        # FP32 sums of a cell's velocities, of order 1 and at most 4n of them, in any order
        assert np.abs(v0 - v1).max() <= 4 * n * 2.0 ** -22
        assert np.array_equal(a.positions(), b.positions())
    finally:
        a.close()
        b.close()
