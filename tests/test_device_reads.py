"""Device reads: what a caller gets when a step failed, and reads mixed with partial writes."""
from __future__ import annotations

import contextlib
import ctypes

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


BOXES = {
    "small": dict(L=(12, 10, 14), periodic=(1, 1, 0), n=10, drag=1e-3, seed=1),
    "extended": dict(L=(12, 10, 14), periodic=(1, 1, 0), n=10, algorithm=1, seed=2),
    "gathered": dict(L=(66, 60, 50), periodic=(1, 1, 1), n=5, seed=3),
    "extended_large": dict(L=(60, 60, 50), periodic=(1, 1, 1), n=5, algorithm=1, seed=4),
    "sparse_large": dict(L=(110, 100, 90), periodic=(1, 1, 1), n=1, seed=5),   # more cells than the gather's scratch holds
    "tile_kernel": dict(L=(8, 7, 9), periodic=(1, 1, 0), n=70, seed=6),
    "ensemble": dict(boxes=[dict(L=(8, 8, 20), periodic=(1, 1, 0), n=10, seed=6), dict(L=(6, 5, 9), n=5, seed=7)]),
}


def _sweeps(call):
    """Kernels that sweep the cells in `call`."""
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    names = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    return sum("run_kernel" in n or "::step_kernel" in n for n in names)


@pytest.mark.parametrize("name", list(BOXES))
def test_one_replay_serves_a_read_and_the_write_that_follows(name):
    """Programs that read all particles and set velocities only, or change the body force, or read
    on the host: an exchange after the first sweeps the cells for its step and once more."""
    h, r = capi.Handle(**BOXES[name]), capi.Handle(**BOXES[name])
    try:
        pos, vel = (torch.empty((h.N, 3), device="cuda") for _ in range(2))
        torch.cuda.synchronize()

        start = r.positions(), r.velocities()

        def exchange(k):
            h.step(1)
            h.get_particles_device(pos.data_ptr(), vel.data_ptr())
            if k % 3 == 0:
                back = vel.flip(0).contiguous()
                torch.cuda.synchronize()
                h.set_particles_device(0, back.data_ptr())
            elif k % 3 == 1:
                h.set_drag(0.01 * k)
            else:
                h.velocities()

        for _ in range(2):   # (a process's first profile may miss kernels)
            _sweeps(lambda: torch.ones(8, device="cuda").sum())
        exchange(0)
        sweeps = [_sweeps(lambda: exchange(k)) for k in (1, 2, 3)]
        step = max(_sweeps(lambda: r.step(1)) for _ in range(3))   # an ensemble's may be several launches
        if step == 0:
            pytest.skip("the profiler records no kernels here")
        assert max(sweeps) <= 2 * step   # (a profile may miss a kernel)
        r.set_step(0)
        r.set_particles(*start)
        for k in range(4):   # the same program with host reads and writes
            r.step(1)
            v = r.velocities()
            if k % 3 == 0:
                r.set_velocities(v[::-1].copy())
            elif k % 3 == 1:
                r.set_drag(0.01 * k)
        assert np.array_equal(h.positions(), r.positions()) and np.array_equal(h.velocities(), r.velocities())
    finally:
        h.close()
        r.close()


@pytest.mark.parametrize("name", list(BOXES))
def test_reads_follow_what_the_program_does_with_the_state(name):
    """Exchanges of everything, then partial ones, then everything again: each read is the
    host's, whichever way it takes."""
    h, r = capi.Handle(**BOXES[name]), capi.Handle(**BOXES[name])
    try:
        pos, vel = (torch.empty((h.N, 3), device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        for k, partial in enumerate([False, False, True, True, False, False, True]):
            h.step(1 + k % 2)
            r.step(1 + k % 2)
            h.get_particles_device(pos.data_ptr(), vel.data_ptr())
            p, v = r.positions(), r.velocities()
            assert np.array_equal(pos.cpu().numpy(), p) and np.array_equal(vel.cpu().numpy(), v)
            pos.fill_(float("nan"))   # the caller's buffers are the caller's again
            v = v[::-1].copy()
            back_p, back_v = torch.from_numpy(p).cuda(), torch.from_numpy(v).cuda()
            torch.cuda.synchronize()
            h.set_particles_device(0 if partial else back_p.data_ptr(), back_v.data_ptr())
            r.set_velocities(v) if partial else r.set_particles(p, v)
        assert np.array_equal(h.positions(), r.positions()) and np.array_equal(h.velocities(), r.velocities())
    finally:
        h.close()
        r.close()


def test_a_read_into_overlapping_buffers_leaves_the_state():
    h, r = capi.Handle(**BOXES["small"]), capi.Handle(**BOXES["small"])
    try:
        both = torch.empty((h.N, 3), device="cuda")
        torch.cuda.synchronize()
        for x in (h, r):
            x.step(2)
        h.get_particles_device(both.data_ptr(), both.data_ptr())
        assert np.array_equal(h.positions(), r.positions()) and np.array_equal(h.velocities(), r.velocities())
    finally:
        h.close()
        r.close()


@contextlib.contextmanager
def _managed(n):
    """n floats of managed memory (which is not the GPU's own), by pointer and as an array."""
    cu, at = ctypes.CDLL("libcuda.so.1"), ctypes.c_uint64()
    assert cu.cuMemAllocManaged(ctypes.byref(at), ctypes.c_size_t(4 * n), 1) == 0
    try:
        yield at.value, np.ctypeslib.as_array((ctypes.c_float * n).from_address(at.value))
    finally:
        assert cu.cuMemFree_v2(at) == 0


@pytest.mark.parametrize("name", ["small", "extended", "gathered"])
def test_buffers_that_are_not_the_gpus_own_are_copied(name):
    """Only memory of the handle's GPU is read and written by kernels."""
    h, r = capi.Handle(**BOXES[name]), capi.Handle(**BOXES[name])
    torch.zeros(1, device="cuda")   # a current context for the allocations
    try:
        with _managed(3 * h.N) as (dp, p), _managed(3 * h.N) as (dv, v):
            for k in range(4):
                h.step(1)
                r.step(1)
                h.get_particles_device(dp, dv)
                torch.cuda.synchronize()
                assert np.array_equal(p.reshape(-1, 3), r.positions()) and np.array_equal(v.reshape(-1, 3), r.velocities())
                v[:] = v.reshape(-1, 3)[::-1].ravel().copy()
                h.set_particles_device(dp if k % 2 else 0, dv)
                r.set_velocities(v.reshape(-1, 3).copy())
        assert np.array_equal(h.positions(), r.positions()) and np.array_equal(h.velocities(), r.velocities())
    finally:
        h.close()
        r.close()
