"""The gradients of the 64 x 64 x 32 (+2 walls) channel, n = 10, 200 steps: how far they are from
64 bits, and how far the drag gradient depends on the order in which sums arrive.

The reference is the reverse sweep in float64 over the events of the forward's tape, with the
rotation axes drawn again from the documented counters.
"""
from __future__ import annotations

import math

import pytest

from cudampcd_gb300 import capi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

L, N_CELL, DT, SEED, S = (64, 64, 34), 10, 0.02, 5, 200
BOUNCE, NONE = 0x80000000, 0xFFFFFFFF
ALPHA = 2.0 * math.pi / 3.0


def _axes(step):
    """Axes of all cells by storage index, float64 (Philox4x32-10, counter {cell, step, 2, 0}, key = seed)."""
    low = 0xFFFFFFFF
    s = torch.arange(L[0] * L[1] * L[2], device="cuda")
    z, col = s % L[2], s // L[2]
    c = [(col % L[0]) + L[0] * ((col // L[0]) + L[1] * z), torch.full_like(s, step), torch.full_like(s, 2), torch.zeros_like(s)]
    k0, k1 = SEED & low, SEED >> 32
    for _ in range(10):
        p0, p1 = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
        c = [(p1 >> 32 & low) ^ c[1] ^ k0, p1 & low, (p0 >> 32 & low) ^ c[3] ^ k1, p0 & low]
        k0, k1 = k0 + 0x9E3779B9 & low, k1 + 0xBB67AE85 & low
    u = [(w >> 8).double() * 2.0 ** -24 for w in c[:2]]
    z = 1.0 - 2.0 * u[0]
    rho = (1.0 - z * z).clamp(min=0.0).sqrt()
    return torch.stack((rho * torch.cos(2 * math.pi * u[1]), rho * torch.sin(2 * math.pi * u[1]), z), 1)


def _reference(tape, dU, step0):
    key, lab, ncell, cnt, b0 = (torch.from_numpy(a.view("int32")).cuda() for a in tape)
    C = L[0] * L[1] * L[2]
    w = 1.0 / (S * L[0] * L[1])
    lam, drag = torch.zeros((key.shape[1], 3), dtype=torch.float64, device="cuda"), 0.0
    layer = torch.arange(C, device="cuda") % L[2]
    for t in reversed(range(S)):
        k, l = key[t].long() & 0xFFFFFFFF, lab[t].long() & 0xFFFFFFFF
        term = dU.double()[layer] * w / cnt[t].clamp(min=1)
        mu = torch.where((l & BOUNCE != 0)[:, None], -lam, lam)
        mu[:, 0] += term[l & ~BOUNCE]
        who = torch.nonzero(k != NONE)[:, 0]
        cell, m = k[who], mu[who]
        drag += m[:, 0].sum().item()
        mean = torch.zeros((C, 3), dtype=torch.float64, device="cuda").index_add(0, cell, m) / ncell[t].clamp(min=1)[:, None]
        axis, s = _axes(step0 + t)[cell], mean[cell]
        r = m - s
        par = axis * (r * axis).sum(1, keepdim=True)
        lam = mu
        lam[who] = s + par + math.cos(ALPHA) * (r - par) - math.sin(ALPHA) * torch.cross(r, axis, dim=1)
    return torch.where((b0.long() & BOUNCE != 0)[:, None], -lam, lam), drag * DT


def test_channel_gradients_against_64_bits_and_from_run_to_run():
    h = capi.Handle(L=L, periodic=(1, 1, 0), n=N_CELL, dt=DT, drag=1e-3, seed=SEED)
    try:
        step0 = h.step_index
        profile, z = torch.empty(L[2], device="cuda"), torch.arange(L[2], device="cuda")
        h.profile_forward(S, 20, profile.data_ptr())
        dU = (1e-3 * (z - L[2] / 2.0 + 0.5) ** 2 / 256.0 - 2e-3).float()   # as of a loss against a parabola
        dv = torch.empty((h.N, 3), device="cuda")
        torch.cuda.synchronize()
        drags = [h.profile_backward(dU.data_ptr(), dv.data_ptr()) for _ in range(8)]
        ref_v, ref_g = _reference(h.profile_tape(S), dU, step0)
        err_v = ((dv.double() - ref_v).norm() / ref_v.norm()).item()
        err_g = abs(drags[0] - ref_g) / abs(ref_g)
        spread = (max(drags) - min(drags)) / abs(ref_g)
        print(f"velocity gradient {err_v:.2e}, drag gradient {err_g:.2e} from 64 bits; from run to run {spread:.2e}")
        # a step's rotation and mean are right to about 2^-23 of their size
        assert err_v < S * 2.0 ** -23 and err_g < S * 2.0 ** -23
        # the sums over cells do not depend on the order of arrival (the drag gradient's standard
        # deviation was 9e-10 of its value when they did)
        assert spread < 1e-9
    finally:
        h.close()
