"""Force evaluations of unevenly filled boxes: droplets in mostly empty cells, one system and batches, and
slabs of them.  Counts and forces against the oracle, and the list kernel's time against the CTA kernel's,
whose work is split by pairs of cells (the list kernel's items must follow the cells' real occupancy)."""
import dataclasses

import numpy as np
import pytest

import sc2019_md_gb300 as m
from sc2019_md_gb300 import systems
from helpers import oracle_from_ctx

pytestmark = pytest.mark.gpu

SUM_TOL = 2e-6
FIX_ABS = 64 * 2.0 ** -24


def droplet(n, L, edge, seed, at=None, rest=0):
    """n particles on a jittered lattice of a cube of `edge` in a box of L, `rest` more spread over the box."""
    rng = np.random.default_rng(seed)
    k = int(np.ceil(n ** (1 / 3)))
    site = rng.permutation(k ** 3)[:n]
    ijk = np.stack([site // (k * k), (site // k) % k, site % k], 1)
    lo = np.full(3, (L - edge) / 2) if at is None else np.asarray(at)
    pos = lo + (ijk + 0.5 + rng.uniform(-0.2, 0.2, (n, 3))) * (edge / k)
    pos = np.concatenate([pos, rng.uniform(0, L, (rest, 3))]) % L
    pos = pos.astype(np.float32)
    pos[pos >= np.float32(L)] = 0.0
    base = systems.small_ljc(64, 37.5, 12.0, seed=seed)
    nc = int(L // 10.0)
    q = rng.choice([-0.42, 0.42], len(pos)).astype(np.float32)
    return dataclasses.replace(base, box=(L,) * 3, cutoff=10.0, ncell=(nc,) * 3, pos=pos, vel=np.zeros_like(pos), q=q,
                               type=rng.integers(0, 4, len(pos)).astype(np.int32))


@pytest.mark.parametrize("n,L,edge,at,rest", [(3000, 62.0, 14.0, None, 0), (3000, 62.0, 14.0, (55.0, 55.0, 55.0), 200),
                                              (4000, 101.0, 14.0, None, 50), (4000, 101.0, 14.0, (95.0, 3.0, 95.0), 0),
                                              (900, 151.0, 9.0, (70.5, 70.5, 70.5), 1000), (2500, 151.0, 12.0, (145.0,) * 3, 0)])
@pytest.mark.parametrize("order,exact", [(1, False), (2, True)])
def test_droplets(n, L, edge, at, rest, order, exact):
    s = droplet(n, L, edge, n, at, rest)
    x, y, z = (np.ascontiguousarray(s.pos[:, k]) for k in range(3))
    with m.Context(s.params(table_bins=256, table_order=order, flags=m.FLAG_EXACT_DIFF if exact else 0)) as ctx:
        F, st, cnt = ctx.force(x, y, z, s.q, s.type, counts=True)
        o = oracle_from_ctx(ctx, s)
        Ff, _ = ctx.force_fixed(x, y, z, s.q, s.type)
        nx = s.ncell[0]
        parts = [ctx.force_fixed(x, y, z, s.q, s.type, home=(a, b)) for a, b in ((0, nx // 2), (nx // 2, nx // 2), (nx // 2, nx))]
    Fo, Fabs, cnto, sto = o.force_cells()
    assert np.array_equal(cnt, cnto) and st["pairs"] == sto["pairs"]
    assert (np.abs(F - Fo) <= SUM_TOL * Fabs + FIX_ABS).all()
    assert np.array_equal(sum(p[0] for p in parts), Ff)
    assert sum(p[1]["pairs"] for p in parts) == st["pairs"] and parts[1][1]["pairs"] == 0


@pytest.mark.parametrize("energy", [0, m.FLAG_ENERGY])
def test_batches_of_droplets(energy):
    """Uneven replicas of all three paths beside each other: each as a batch of its own, and the replicas'
    totals add up."""
    reps = [droplet(n, L, e, k, at) for k, (n, L, e, at) in enumerate([
        (2500, 62.0, 13.0, None), (700, 151.0, 9.0, (145.0,) * 3), (600, 25.0, 8.0, (20.0,) * 3), (300, 15.0, 6.0, None),
        (1500, 101.0, 13.0, None), (40, 33.0, 6.0, None), (1200, 27.0, 11.0, None)])]
    pos, q, t = (np.concatenate([getattr(s, a) for s in reps]) for a in ("pos", "q", "type"))
    spec = [(s.n, s.box) for s in reps]
    p = reps[0].params(flags=energy)
    with m.Batch(p, spec) as b:
        assert len(set(b.layout()["path"])) == 3
        F, st, cnt = b.force(pos[:, 0], pos[:, 1], pos[:, 2], q, t, counts=True)
        rs, offs = b.replica_stats(), b.offsets
    assert sum(r["pairs"] for r in rs) == st["pairs"]
    for k, s in enumerate(reps):
        with m.Batch(p, spec[k:k + 1]) as b:
            F1, st1, cnt1 = b.force(s.pos[:, 0], s.pos[:, 1], s.pos[:, 2], s.q, s.type, counts=True)
        sl = slice(offs[k], offs[k + 1])
        assert np.array_equal(F[sl].view(np.uint32), F1.view(np.uint32)) and np.array_equal(cnt[sl], cnt1)
        assert rs[k]["pairs"] == st1["pairs"]
        if energy:
            for key in ("e_lj", "e_coul", "virial"):
                assert abs(rs[k][key] - st1[key]) <= 1e-12 * max(abs(st1[key]), 1.0)


@pytest.mark.parametrize("n,L,edge", [(13000, 200.0, 30.0), (27000, 200.0, 30.0)])
def test_dense_droplets_are_not_slower_than_by_cell_pairs(n, L, edge):
    s = droplet(n, L, edge, 1)
    x, y, z = (np.ascontiguousarray(s.pos[:, k]) for k in range(3))
    ms = {}
    with m.Context(s.params(table_bins=256, sigma=(m.C.c_double * 16)(*[0.5] * 16))) as ctx:
        for tile in (None, (4, 6, 0)):
            if tile:
                ctx.set_tile(*tile)
            ctx.force(x, y, z, s.q, s.type)
            ms[tile] = sorted(ctx.force(x, y, z, s.q, s.type)[1]["force_ms"] for _ in range(7))[3]
    assert ms[None] <= ms[(4, 6, 0)], ms
