"""PME with more particles than 2^31 / 32: at order 6, 32 threads spread each particle.  All but two are neutral
and without LJ; the two charges, one in the first cell and one at the very end of the cell order, feel
the reciprocal forces of the two alone, bit for bit (integer spreading, the same transforms)."""
import ctypes as C

import numpy as np
import pytest
import torch

import sc2019_md_gb300 as m

pytestmark = pytest.mark.gpu

L, NC = 2000.0, 200


def _force(ctx, pos, q):
    n = pos.shape[1]
    out = [torch.zeros(n, device="cuda") for _ in range(3)]
    args = [C.c_void_p(a.data_ptr()) for a in (pos[0], pos[1], pos[2], q)]
    m._check(m.lib().mdrl_force_eval_device(ctx._h, n, *args, None, *(C.c_void_p(a.data_ptr()) for a in out), None, None))
    return out


def test_charges_past_the_thread_limit():
    free, _ = torch.cuda.mem_get_info()
    if free < 40 << 30:
        pytest.skip("needs 40 GB of device memory")
    n = (1 << 26) + 64
    g = torch.Generator(device="cuda").manual_seed(1)
    pos = torch.rand((3, n), generator=g, device="cuda").mul_(L).clamp_(max=float(np.nextafter(np.float32(L), np.float32(0))))
    top = float(np.nextafter(np.float32(L), np.float32(0)))
    pos[:, 0] = 1.25                                    # the first cell
    pos[:, -1] = top                                    # the last cell
    q = torch.zeros(n, device="cuda")
    q[0], q[-1] = 1.0, -1.0
    p = m.default_params(box=[L] * 3, ncell=[NC] * 3, cutoff=9.5, sigma=[1.0], epsilon=[0.0], mass=[1.0], coulomb_k=332.0)
    pme = dict(order=6, grid=(64, 64, 64), beta=0.3)
    with m.Context(p) as ctx:
        ctx.set_pme(**pme)
        F = _force(ctx, pos, q)
        got = [[float(v[0]), float(v[-1])] for v in F]
        two = torch.stack([pos[:, 0], pos[:, -1]], 1).contiguous()
    del pos, F
    with m.Context(p) as ctx:
        ctx.set_pme(**pme)
        F = _force(ctx, two, torch.tensor([1.0, -1.0], device="cuda"))
        want = [[float(v[0]), float(v[1])] for v in F]
    assert np.abs(want).max() > 0
    assert got == want
