"""Systems binned by one CTA (at most 4,096 particles and 4,096 cells) at its edges: the thread count,
the limits on both sides (the next size takes the general path), empty cells, one cell that holds
everything.  Partner counts and forces against the oracle; a trajectory equals that of the same
system with particles appended far away that push it over the limit (the general path)."""
import numpy as np
import pytest

import sc2019_md_gb300 as m
from sc2019_md_gb300 import systems
from helpers import liquid_argon, oracle_from_ctx

pytestmark = pytest.mark.gpu

SUM_TOL = 2e-6
FIX_ABS = 64 * 2.0 ** -24


@pytest.mark.parametrize("n,L,rc", [(1, 37.5, 12.0), (1023, 37.5, 12.0), (1025, 37.5, 12.0), (4096, 42.3, 12.0),
                                    (4097, 42.3, 12.0), (3000, 64.2, 4.0), (3000, 68.4, 4.0)])
@pytest.mark.parametrize("tile", [None, (4, 6, 0)])
def test_evaluation(n, L, rc, tile):
    s = systems.small_ljc(n, L, rc, seed=n)
    with m.Context(s.params(table_bins=256, flags=m.FLAG_ENERGY)) as ctx:
        if tile:
            ctx.set_tile(*tile)
        F, st, cnt = ctx.force(s.pos[:, 0], s.pos[:, 1], s.pos[:, 2], s.q, s.type, counts=True)
        o = oracle_from_ctx(ctx, s)
    Fo, Fabs, cnto, sto = o.force_cells()
    assert np.array_equal(cnt, cnto) and st["pairs"] == sto["pairs"]
    assert st["max_cell_occupancy"] == np.bincount(o_cells(s)).max()
    assert (np.abs(F - Fo) <= SUM_TOL * Fabs + FIX_ABS).all()


def o_cells(s):
    e = np.float32(np.float64(np.float32(s.box[0])) / s.ncell[0])
    c = np.minimum((s.pos / e).astype(int), s.ncell[0] - 1)
    return (c[:, 0] * s.ncell[1] + c[:, 1]) * s.ncell[2] + c[:, 2]


def test_everything_in_one_cell():
    rng = np.random.default_rng(2)
    pos = (rng.random((700, 3)) * 8.0 + 1.0).astype(np.float32)
    with m.Context(m.default_params(box=(36.0,) * 3, cutoff=12.0)) as ctx:
        _, st, cnt = ctx.force(pos[:, 0], pos[:, 1], pos[:, 2], counts=True)
    r2 = ((pos[:, None].astype(np.float64) - pos[None]) ** 2).sum(-1)
    assert st["max_cell_occupancy"] == 700
    assert abs(st["pairs"] - ((r2 > 0) & (r2 <= 144.0)).sum() // 2) <= 2     # FP32 at the cutoff


@pytest.mark.parametrize("integrator", [m.INT_VELOCITY_VERLET, m.INT_EULER])
@pytest.mark.parametrize("accum", [m.ACC_FIXED64, m.ACC_KAHAN])
def test_trajectory_equals_the_general_path(integrator, accum):
    """Resting atoms beyond everyone's reach (9 A apart, cutoff 8.5) take the same number of steps in the
    second run; the liquid's own atoms do not feel them, so its trajectory is the same bit for bit."""
    s = liquid_argon()
    n = 4097 - s.n
    layers = -(-n // 16)
    box = (36.0, 36.0, 60.0 + 9.0 * layers)                # the liquid, then sparse layers along z
    g = np.arange(4) * 9.0 + 4.5
    ext = np.stack(np.meshgrid(g, g, 50.0 + 9.0 * np.arange(layers), indexing="ij"), -1).reshape(-1, 3)
    ext = ext[:n].astype(np.float32)
    out = []
    for extra in (ext[:0], ext):
        pos = np.concatenate([s.pos, extra])
        vel = np.concatenate([s.vel, np.zeros_like(extra)])
        with m.Context(m.default_params(box=box, cutoff=8.5, integrator=integrator, accum=accum, flags=m.FLAG_ENERGY)) as ctx:
            ctx.set_state(pos[:, 0], pos[:, 1], pos[:, 2], vel)
            ctx.step(12)
            out.append([a[: s.n] for a in ctx.state()])
    for a, b in zip(*out):
        if accum == m.ACC_FIXED64:
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        else:
            assert np.abs(a - b).max() <= 1e-4 * max(1.0, np.abs(b).max())
