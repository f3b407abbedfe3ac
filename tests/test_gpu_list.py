"""The list force kernel of force evaluations at the sizes where it can go wrong: empty and ragged
cells, tiles and groups with remainders, lists longer than one, every tile size (grids below 400, below
2,000 and above 2,000 cells), fine and whole items, 3 cells per axis (every column wraps).

Partner counts and pair totals equal the oracle's; forces within SUM_TOL of sum |f_ij| plus 64
fixed-point quanta (k flushes per particle round to 0.29 sqrt(k) quanta rms, 5 for the largest k here);
the result does not depend on the split nor on what else the launch holds, bit for bit.
"""
import numpy as np
import pytest

import sc2019_md_gb300 as m
from sc2019_md_gb300 import systems
from helpers import oracle_from_ctx

pytestmark = pytest.mark.gpu

SUM_TOL = 2e-6
FIX_ABS = 64 * 2.0 ** -24


def _force(sysm, tile=None, **kw):
    with m.Context(sysm.params(**kw)) as ctx:
        if tile is not None:
            ctx.set_tile(*tile)
        F, st, cnt = ctx.force(sysm.pos[:, 0], sysm.pos[:, 1], sysm.pos[:, 2], sysm.q, sysm.type, counts=True)
        return F, st, cnt, oracle_from_ctx(ctx, sysm)


@pytest.mark.parametrize("n,L,rc,dmin", [(1, 37.5, 12.0, 1.0), (97, 30.3, 10.0, 1.0), (3501, 30.3, 10.0, 1.0),
                                         (9003, 30.3, 10.0, 0.6), (2603, 80.4, 10.0, 1.0), (30001, 80.4, 10.0, 1.0),
                                         (9001, 52.3, 4.0, 1.0), (20002, 52.3, 4.0, 1.0)])
@pytest.mark.parametrize("order,exact", [(1, False), (2, True)])
def test_list_kernel_sizes(n, L, rc, dmin, order, exact):
    sysm = systems.small_ljc(n, L, rc, seed=n, dmin=dmin)
    kw = dict(table_bins=256, table_order=order, flags=m.FLAG_ENERGY | (m.FLAG_EXACT_DIFF if exact else 0))
    F, st, cnt, o = _force(sysm, **kw)
    Fo, Fabs, cnto, sto = o.force_cells()
    assert np.array_equal(cnt, cnto)
    assert st["pairs"] == sto["pairs"]
    assert (np.abs(F - Fo) <= SUM_TOL * Fabs + FIX_ABS).all()
    for key in ("e_lj", "e_coul", "virial"):
        assert abs(st[key] - sto[key]) <= 1e-5 * max(abs(sto[key]), 1.0), (key, st[key], sto[key])
    for G in (1, 3):
        F2, st2, cnt2, _ = _force(sysm, tile=(1, G, 1), **kw)
        assert np.array_equal(F.view(np.uint32), F2.view(np.uint32)) and np.array_equal(cnt, cnt2)
        assert st2["pairs"] == st["pairs"]


def test_fine_and_whole_items_agree():
    """A replica alone (few items: fine ones) and among copies (whole items), without energies too."""
    reps = [systems.replica(3300 + k, k) for k in range(8)]
    pos, vel, q, t, spec = systems.concat(reps)
    p = reps[0].params(table_bins=256)
    with m.Batch(p, spec) as b:
        F, _, _ = b.force(pos[:, 0], pos[:, 1], pos[:, 2], q, t)
        offs = b.offsets
    for k, s in enumerate(reps):
        with m.Context(s.params(table_bins=256)) as ctx:
            F1, _, _ = ctx.force(s.pos[:, 0], s.pos[:, 1], s.pos[:, 2], s.q, s.type)
        assert np.array_equal(F[offs[k]:offs[k + 1]].view(np.uint32), F1.view(np.uint32)), k
