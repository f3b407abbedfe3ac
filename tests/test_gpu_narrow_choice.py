"""The two runs that tests/test_gpu_narrow.py compares take different kernels, and the narrow one's
scratch is sized by the system."""
import numpy as np
import pytest
import torch

import sc2019_md_gb300 as m
from test_gpu_narrow import BOX, DT, RC, arrays  # noqa: F401

pytestmark = pytest.mark.gpu


def _context():
    return m.Context(m.default_params(box=BOX, cutoff=RC, ntypes=3, sigma=[1.2, 1.5, 1.8], epsilon=[0.05, 0.1, 0.2],
                                      mass=[12.0, 14.0, 16.0], coulomb_k=332.06371, dt_fs=DT))


def test_each_run_takes_its_kernel(arrays):  # noqa: F811
    pos, vel, q, ty, nb = arrays
    for n, want in ((nb, "narrow"), (len(pos), "cta")):
        with _context() as ctx:
            ctx.set_state(pos[:n, 0], pos[:n, 1], pos[:n, 2], vel[:n], q[:n], ty[:n])
            assert ctx.kernels()["step"] == want
            ctx.step(1)
            assert ctx.kernels()["step"] == want
            ctx.set_tile(1, 1, 1)
            assert ctx.kernels()["step"] == "warp"


def test_scratch_of_a_small_system():
    """Two contexts of 27 cells: the second set_state takes scratch for its 378 units (9 MB), not for every
    warp that fits on the GPU (60 MB), and gives it back when its state has no use for it."""
    rng = np.random.default_rng(3)
    g = np.stack(np.meshgrid(*[np.arange(9)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = ((g + 0.5 + rng.uniform(-0.2, 0.2, g.shape)) * (37.5 / 9)).astype(np.float32)     # 27 per cell
    more = np.concatenate([pos, rng.uniform(0.5, 12.0, (120, 3)).astype(np.float32)])       # one cell above 96
    kw = dict(box=[37.5] * 3, cutoff=RC, sigma=[0.2], epsilon=[0.01], mass=[12.0])
    with m.Context(m.default_params(**kw)) as a, m.Context(m.default_params(**kw)) as b:
        a.set_state(*(np.ascontiguousarray(more[:, k]) for k in range(3)))                  # sizes the buffers
        b.set_state(*(np.ascontiguousarray(more[:, k]) for k in range(3)))
        a.set_state(*(np.ascontiguousarray(pos[:, k]) for k in range(3)))
        free0 = torch.cuda.mem_get_info()[0]
        b.set_state(*(np.ascontiguousarray(pos[:, k]) for k in range(3)))
        assert a.kernels()["step"] == b.kernels()["step"] == "narrow"
        assert 0 <= free0 - torch.cuda.mem_get_info()[0] < 16 << 20
        b.set_state(*(np.ascontiguousarray(more[:, k]) for k in range(3)))
        assert b.kernels()["step"] == "cta"
        assert torch.cuda.mem_get_info()[0] >= free0
