"""Sub-steps of lattices whose sizes the oracle cannot hold, at the sides where
the offsets change: 512^3 (32-bit byte offsets, whole rows per block) and 814^3
(86 GB; a plane of 4.3 GB, past the byte offsets that 812^3 still has).

One sub-step of the whole lattice is set against slabs of two planes and their
ghosts at both ends and in the middle.  A slab draws the whole lattice's noise
but has small planes and its own kernels: 32-bit byte offsets at both sides, one
charge face per launch.  Two ghost planes hold what a sub-step of its own planes
can depend on (an odd pass on the even one, a second charge face on the first),
so the slab needs no exchange and its planes agree to the last bit.

At 512^3 the charge step is also compared as a whole with one face per launch
(LGV_CHARGE_FUSED=0), and measurements on both sides of the largest side of the
one-pass form (512) are compared with sums by torch."""
import ctypes as C
import math

import numpy as np
import pytest

from lgvtest import GpuLattice

pytestmark = pytest.mark.gpu

IDEAL, HB, CHARGE, EM = 3, 4, 5, 6
COEF = dict(mass0=-4.813, lam=10.0, H=0.003, chi=5.0, gamma=1.0, diffusion=1.0 / 3.0, seed=4242)


def device_state(g, torch):
    u = torch.empty((g.N, g.N, g.N, 10), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    g.L.check(g.lib.lgv_get_state_device(g.h, C.c_void_p(u.data_ptr())), "get_state_device")
    g.L.check(g.lib.lgv_synchronize(g.h), "synchronize")
    return u


def started(lgv, N):
    g = GpuLattice(lgv, N, **COEF)
    g.initialize(1, 0.4)
    g.initialize(2)
    return g


class NoExchange:
    def exchange(self, slab, comps):
        pass


@pytest.mark.parametrize("N", [512, 814])
def test_substeps_equal_small_slabs(lgv, N):
    import torch

    from langevina_b200 import slab as S

    ends = (0, N // 4 * 2, N - 2)
    g = started(lgv, N)
    for ev, dt, gauss in ((IDEAL, 0.04, 0), (HB, 0.03, 0), (HB, 0.03, 1), (CHARGE, 0.1, 0), (EM, 0.02, 0)):
        u = device_state(g, torch)
        boxes = [u[[(k0 - 2 + q) % N for q in range(6)]].cpu().numpy() for k0 in ends]
        del u
        ctr = g.counter()
        if ev == HB:
            g.L.check(g.lib.lgv_set_hb_proposal(g.h, gauss), "proposal")
        g.step(ev, dt)
        u = device_state(g, torch)
        got = [u[k0:k0 + 2].cpu().numpy() for k0 in ends]
        del u
        for k0, box, whole in zip(ends, boxes, got):
            s = S.SlabLattice(N, k0, 2, NoExchange(), **COEF)
            try:
                s.L = g.L
                g.L.check(s.lib.lgv_set_state(s.h, g.L.ptr(box)), "set_state")
                if ev == HB:
                    g.L.check(s.lib.lgv_set_hb_proposal(s.h, gauss), "proposal")
                s.set_counter(ctr)
                s.step(ev, dt)
                mine = s.get_interior()
            finally:
                s.close()
            changed = slice(0, 4) if ev in (HB, EM) else slice(4, 10) if ev == CHARGE else slice(0, 10)
            assert not np.array_equal(whole[..., changed], box[2:4][..., changed])
            assert np.array_equal(mine, whole), (ev, gauss, k0, np.abs(mine - whole).max())
    g.close()
    torch.cuda.empty_cache()


def test_charge_step_equals_one_face_per_launch_at_512(lgv, monkeypatch):
    import torch

    out = []
    for fused in ("1", "0"):
        monkeypatch.setenv("LGV_CHARGE_FUSED", fused)
        g = started(lgv, 512)
        g.step(CHARGE, 0.1, nsteps=2)
        out.append(device_state(g, torch))
        g.close()
    assert torch.equal(*out)
    v = out[0][..., 4:].sum(dim=(0, 1, 2)).abs().max().item()  # the zero modes that initialisation took out
    assert v < 1e-6
    del out
    torch.cuda.empty_cache()


@pytest.mark.parametrize("N", [512, 514])
def test_measurement_around_the_one_pass_bound(lgv, N):
    """A wall is a mean over N^2 sites.  The two-pass form adds them in two chains of N terms, the other sums here in
    shorter pieces: (2 N + 64) 2^-53 times the mean of |obs| bounds both, the modes by a further log2 N steps."""
    import torch

    g = started(lgv, N)
    g.step(HB, 0.05, nsteps=2)
    u = device_state(g, torch)
    m = g.measure()
    g.close()
    rel = (2 * N + 64) * 2.0 ** -53
    f = u.permute(3, 0, 1, 2)
    p2 = f[:4].square().sum(0)
    sigma = p2.sqrt()
    rows = [(m.wall, l, f[l]) for l in range(10)] + [(m.wall, 10, p2), (m.wall_phase, 0, sigma),
                                                     (m.wall_phase, 1, f[0] / sigma), (m.wall_phase, 13, p2)]
    for where, row, x in rows:
        for axis, dims in enumerate(((0, 1), (0, 2), (1, 2))):
            want, scale = x.mean(dim=dims), x.abs().mean(dim=dims)
            d = (torch.from_numpy(where[axis][row]).cuda() - want).abs()
            assert bool((d <= rel * scale).all()), (row, axis, (d / scale).max().item() / rel)
        if where is m.wall:
            assert abs(m.OAverage[row] - x.mean().item()) <= rel * x.abs().mean().item()
    for axis in range(3):
        w = m.wall[axis]
        want = np.fft.rfft(w, axis=-1) / N
        got = m.wall_k[axis][..., 0] + 1j * m.wall_k[axis][..., 1]
        assert np.all(np.abs(got - want) <= (2 * math.isqrt(N) * 8 + 64) * 2.0 ** -52 * np.abs(w).mean(-1, keepdims=True))
    del u, f, p2, sigma
    torch.cuda.empty_cache()
