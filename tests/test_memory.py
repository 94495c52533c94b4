"""A handle asks for no more memory than there is.

Buckets are deeper than they need be, and a forward profile keeps its tape, where memory is
plentiful; where it is not, a handle that fits with the shallow buckets is still created, and
behaves as any other.
"""
from __future__ import annotations

import numpy as np
import pytest

from cudampcd_gb300 import capi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MIB = 1 << 20


def _free():
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("L", [(64, 64, 64), (110, 100, 60)], ids=["0.8 GB", "2 GB"])
def test_a_handle_that_fits_with_shallow_buckets_is_created(monkeypatch, L):
    """n = 20: 40 slots a cell, 48 where there is room.  The box of under 1 GiB of buckets finds
    out when an allocation fails, the larger one asks first."""
    box = dict(L=L, periodic=(1, 1, 1), n=20, seed=3)
    cells = L[0] * L[1] * L[2]
    roomy = capi.Handle(**box)
    roomy.step(3)
    expected = roomy.positions()
    roomy.close()
    monkeypatch.setenv("MPCD_GB_BUCKET_DEPTH", "40")
    before = _free()
    shallow = capi.Handle(**box)
    need = before - _free()
    shallow.close()
    monkeypatch.delenv("MPCD_GB_BUCKET_DEPTH")
    spare = (8 * 64 * cells) // 2   # half of what the deeper buckets take beyond that
    assert spare > 32 * MIB
    hold = torch.empty(_free() - need - spare, dtype=torch.uint8, device="cuda")
    try:
        h = capi.Handle(**box)
        try:
            h.step(3)
            assert np.array_equal(h.positions(), expected)
            assert h.counters()[1] == 0
        finally:
            h.close()
    finally:
        del hold
        torch.cuda.empty_cache()


def test_a_forward_leaves_memory_that_is_short(monkeypatch):
    """With 6 GB left a tape of 2.3 GB is not kept; the forward is the same."""
    box = dict(L=(64, 64, 34), periodic=(1, 1, 0), n=10, drag=1e-3, seed=5)
    profiles, taken = [], []
    for short in (False, True):
        h = capi.Handle(**box)
        hold = torch.empty(max(0, _free() - 6000 * MIB) if short else 0, dtype=torch.uint8, device="cuda")
        try:
            profile = torch.empty(34, device="cuda")
            before = torch.cuda.mem_get_info()[0]
            h.profile_forward(200, 20, profile.data_ptr())
            taken.append(before - torch.cuda.mem_get_info()[0])
            profiles.append(profile.cpu().numpy())
        finally:
            h.close()
            del hold
            torch.cuda.empty_cache()
    assert taken[0] > 2000 * MIB > 1000 * MIB > taken[1]
    assert np.abs(profiles[0] - profiles[1]).max() <= 10 * 2.0 ** -24
