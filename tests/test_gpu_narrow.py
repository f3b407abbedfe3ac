"""Dynamics that runs the default tile's units one warp each (no cell above 96 particles at set_state,
2,646 units: more than one for each resident warp) against the CTA kernel: the same forces and velocities
bit for bit.  The second run holds a crowded cell beyond everyone's reach, so it takes the CTA kernel.
The step moves the particles into cells from empty to 300: on both sides of a tile, of the shared
accumulators (96) and of a chunk (256)."""
import numpy as np
import pytest

import sc2019_md_gb300 as m

pytestmark = pytest.mark.gpu
BOX, RC, DT = (37.5, 37.5, 262.5), 12.0, 2.0


def _grid(rng, lo, hi, n, jitter):
    """n points of a jittered grid over the box [lo, hi), at least (1 - 2 jitter) of a spacing apart."""
    lo, hi = np.asarray(lo, float), np.asarray(hi, float)
    h = (np.prod(hi - lo) / n) ** (1 / 3)
    while True:
        k = np.floor((hi - lo) / h).astype(int)
        if np.prod(k) >= n:
            break
        h *= 0.98
    g = np.stack(np.meshgrid(*(np.arange(v) for v in k), indexing="ij"), -1).reshape(-1, 3)
    g = g[np.sort(rng.permutation(len(g))[:n])]
    return (lo + (g + 0.5 + rng.uniform(-jitter, jitter, (n, 3))) * h).astype(np.float32)


@pytest.fixture(scope="module")
def arrays():
    rng = np.random.default_rng(12)
    e = 12.5
    parts = [_grid(rng, (0, 0, 0), (37.5, 37.5, 3 * e), 900, 0.2)]         # 33 per cell, across the x and y faces
    disp = [np.zeros((900, 3))]
    # a cell, its particles, and the cells that they come from in shares
    for cell, k, homes in (((0, 0, 3), 300, [(0, 0, 3), (0, 0, 5), (0, 0, 6), (0, 0, 7)]),
                           ((0, 0, 4), 257, [(0, 0, 4), (1, 0, 5), (1, 0, 6), (1, 0, 7)]),
                           ((1, 0, 3), 97, [(1, 0, 3), (2, 0, 5)]), ((2, 1, 3), 96, [(2, 1, 3)]),
                           ((1, 2, 3), 32, [(1, 2, 3)]), ((1, 1, 3), 1, [(1, 1, 3)]), ((2, 2, 4), 64, [(2, 2, 4)])):
        lo = np.asarray(cell) * e
        parts.append(_grid(rng, lo + 0.2, lo + e - 0.2, k, 0.2))
        disp.append((np.asarray(cell) - np.asarray(homes)[np.arange(k) % len(homes)]) * e)
    base, disp = np.concatenate(parts), np.concatenate(disp)
    far = _grid(rng, (12.7, 12.7, 112.7), (24.8, 24.8, 124.8), 110, 0.2)
    pos = np.concatenate([base - disp, far]).astype(np.float32)
    vel = np.concatenate([disp / DT, np.zeros_like(far)]).astype(np.float32)
    return (pos, vel, rng.choice([-0.42, 0.42], len(pos)).astype(np.float32),
            rng.integers(0, 3, len(pos)).astype(np.int32), len(base))


def _occupancy(p):
    c = np.floor(p / 12.5).astype(int)
    return np.bincount((c[:, 0] * 3 + c[:, 1]) * 21 + c[:, 2], minlength=189)


@pytest.mark.parametrize("order", [0, 1, 2, 3])
@pytest.mark.parametrize("arith,exact,ke", [(m.ARITH_FMA, True, 332.06371), (m.ARITH_FMA, False, 332.06371),
                                            (m.ARITH_SEPARATE, False, 332.06371), (m.ARITH_FMA, True, 0.0)])
@pytest.mark.parametrize("energy", [0, m.FLAG_ENERGY])
def test_forces_equal_the_cta_kernel(arrays, order, arith, exact, ke, energy):
    pos, vel, q, ty, nb = arrays
    assert _occupancy(pos[:nb]).max() <= 96 < _occupancy(pos).max()
    tab = dict(table_order=order) if order else dict(eval=m.EVAL_DIRECT)
    flags = energy | (m.FLAG_EXACT_DIFF if exact else 0)
    out = []
    for n in (nb, len(pos)):
        with m.Context(m.default_params(box=BOX, cutoff=RC, ntypes=3, sigma=[1.2, 1.5, 1.8], epsilon=[0.05, 0.1, 0.2],
                                        mass=[12.0, 14.0, 16.0], coulomb_k=ke, dt_fs=DT, **tab, table_bins=256,
                                        arith=arith, flags=flags)) as ctx:
            ctx.set_state(pos[:n, 0], pos[:n, 1], pos[:n, 2], vel[:n], q[:n], ty[:n])
            st = ctx.step(1)
            out.append([a[:nb].view(np.uint32) for a in ctx.state()])
            assert st["max_cell_occupancy"] == 300
    for a, b in zip(*out):
        assert np.array_equal(a, b)
