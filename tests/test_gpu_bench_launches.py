"""The launches that the bench counts per step are those of the step's graph: small systems bin in one
launch only when their cells allow it too (dense cells and many cells take the general path)."""
import numpy as np
import pytest

import sc2019_md_gb300 as m

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,ncell,want", [(1728, 36.0, 4, 3), (4000, 36.0, 4, 7), (4000, 150.0, 17, 7), (5000, 60.0, 7, 7)])
def test_launches_of_a_step(n, L, ncell, want):
    rng = np.random.default_rng(n)
    k = int(np.ceil(n ** (1 / 3)))
    site = rng.permutation(k ** 3)[:n]
    pos = ((np.stack([site // (k * k), (site // k) % k, site % k], 1) + 0.5) * (L / k)).astype(np.float32)
    with m.Context(m.default_params(box=[L] * 3, ncell=[ncell] * 3, cutoff=8.0, sigma=[1.0], epsilon=[0.1], mass=[40.0])) as ctx:
        ctx.set_state(*(np.ascontiguousarray(pos[:, d]) for d in range(3)))
        ctx.step(2)
        assert ctx.kernels()["step_launches"] == want
        import bench
        leg = bench.md_leg(m, ctx, 1, 0, lambda: None)
        assert leg["step_launches"] == want
