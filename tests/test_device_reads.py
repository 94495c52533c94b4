"""Device reads: what a caller gets when a step failed, and reads mixed with partial writes."""
from __future__ import annotations

import numpy as np
import pytest

from cudampcd_gb300 import capi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_nothing_is_written_after_a_failed_step(monkeypatch):
    """A step that runs out of extension slots leaves its error with the handle: a read into
    device buffers raises it, as a host read does, and the buffers stay as they were."""
    monkeypatch.setenv("MPCD_GB_BUCKET_DEPTH", "5")
    h = capi.Handle(L=(120, 100, 22), periodic=(1, 1, 0), n=20, seed=21)
    try:
        with pytest.raises(capi.GbError, match="extension"):
            h.step(1)
        out = [torch.full((h.N, 3), 7.0, device="cuda") for _ in range(2)]
        torch.cuda.synchronize()
        with pytest.raises(capi.GbError, match="extension"):
            h.get_particles_device(*(t.data_ptr() for t in out))
        assert all(bool((t == 7.0).all()) for t in out)
        with pytest.raises(capi.GbError, match="extension"):
            h.positions()
    finally:
        h.close()
