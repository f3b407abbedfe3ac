"""Replicas with two cells on an axis and many on others (minimum images): every pair once, whatever the
window around a cell covers (whole axes, wrapped and unwrapped cells, cells exactly rc wide), and no
slower than the explicit pairs of cells.  Counts and forces against the oracle's all-image evaluation."""
import dataclasses

import numpy as np
import pytest

import sc2019_md_gb300 as m
from sc2019_md_gb300 import systems
from helpers import oracle_from_ctx

pytestmark = pytest.mark.gpu

SUM_TOL = 2e-6
FIX_ABS = 64 * 2.0 ** -24
RC = 4.0


def thin(cells, edge, n, seed):
    rng = np.random.default_rng(seed)
    box = tuple(float(np.float32(c * edge)) for c in cells)
    k = np.maximum(1, np.ceil(np.asarray(box) / (np.prod(box) / n) ** (1 / 3)).astype(int))
    site = rng.permutation(int(k.prod()))[:n]
    ijk = np.stack([site // (k[1] * k[2]), (site // k[2]) % k[1], site % k[2]], 1)
    pos = ((ijk + 0.5 + rng.uniform(-0.3, 0.3, (n, 3))) * (np.asarray(box) / k)).astype(np.float32)
    L = np.asarray(box, np.float32)
    pos = np.clip(pos, 0, np.nextafter(L, np.float32(0)))
    base = systems.small_ljc(64, 37.5, 12.0, seed=seed)
    nc = tuple(int(np.floor(np.float64(np.float32(b)) / RC)) for b in box)
    return dataclasses.replace(base, box=box, cutoff=RC, ncell=nc, pos=pos, vel=np.zeros_like(pos),
                               q=rng.choice([-0.42, 0.42], n).astype(np.float32), type=rng.integers(0, 4, n).astype(np.int32))


SHAPES = [((2, 2, 2), 4.2, 300), ((2, 2, 3), 4.1, 350), ((2, 3, 4), 4.3, 700), ((4, 2, 3), 4.2, 700), ((2, 5, 6), 4.1, 1500),
          ((6, 5, 2), 4.1, 1500), ((5, 2, 7), 4.4, 1700), ((2, 2, 16), 4.2, 1600), ((16, 2, 2), 4.2, 1600), ((2, 16, 2), 4.2, 1600),
          ((2, 9, 10), 4.05, 2500), ((2, 4, 6), 4.0, 1000), ((5, 2, 2), 4.01, 400), ((3, 2, 2), 5.9, 500)]


@pytest.mark.parametrize("tile", [None, (1, 3, 1)])
def test_thin_replicas(tile):
    # boxes of exactly 4 rc need (2 rc)(1 + 2^-10): those axes have edges just above 4.0
    reps = [thin(c, e if e > 4.0 else 4.0 * (1 + 1.5 / 1024), n, k) for k, (c, e, n) in enumerate(SHAPES)]
    reps.append(thin((8, 2, 8), 4.004, 1800, 99))
    wide = dataclasses.replace(thin((6, 2, 5), 4.2, 900, 100))           # edges of exactly rc along x
    L = 24.0
    wide = dataclasses.replace(wide, box=(L, *wide.box[1:]), ncell=(6, *wide.ncell[1:]),
                               pos=np.column_stack([wide.pos[:, 0] * np.float32(L / wide.box[0] * 0.9999), wide.pos[:, 1:]]).astype(np.float32))
    reps.append(wide)
    pos, vel, q, t, spec = systems.concat(reps)
    p = reps[0].params(table_bins=256, flags=m.FLAG_ENERGY)
    with m.Batch(p, spec) as b:
        if tile:
            b.set_tile(*tile)
        assert set(b.layout()["path"]) == {m.PATH_MIN_IMAGE}
        F, st, cnt = b.force(pos[:, 0], pos[:, 1], pos[:, 2], q, t, counts=True)
        rs, offs = b.replica_stats(), b.offsets
    assert st["pairs"] == sum(r["pairs"] for r in rs)
    for r, s in enumerate(reps):
        with m.Context(s.params(table_bins=256)) as ctx:
            o = oracle_from_ctx(ctx, s)
        _, F32, Fabs, cnto, sto = o.force_allimage()
        sl = slice(offs[r], offs[r + 1])
        assert rs[r]["pairs"] == sto["pairs"], (r, s.ncell)
        assert np.array_equal(cnt[sl], cnto), (r, s.ncell)
        assert (np.abs(F[sl] - F32) <= SUM_TOL * Fabs + FIX_ABS).all(), (r, s.ncell)


@pytest.mark.parametrize("cells", [(2, 40, 40), (2, 2, 400)])
def test_thin_replicas_are_not_slower_than_pairs_of_cells(cells):
    n = int(np.prod(cells)) * 27
    s = dataclasses.replace(thin(cells, 4.2, n, 1), sigma=[0.5] * 4)
    ms = {}
    with m.Batch(s.params(table_bins=256), [(n, s.box)]) as b:
        for tile in (None, (4, 6, 0)):
            if tile:
                b.set_tile(*tile)
            ms[tile] = sorted(b.force(s.pos[:, 0], s.pos[:, 1], s.pos[:, 2], s.q, s.type)[1]["force_ms"] for _ in range(7))[3]
    assert ms[None] <= ms[(4, 6, 0)], ms


def test_overflowing_cell_of_a_thin_replica():
    """70,000 particles in one cell: reported, in bounded time, and the batch then evaluates correctly."""
    rng = np.random.default_rng(2)
    box = (8.4, 8.4, 42.0)
    crowd = rng.uniform(0.1, 4.0, (70000, 3))
    pos = np.concatenate([crowd, rng.uniform(0, 1, (500, 3)) * np.asarray(box)]).astype(np.float32)
    s = thin((2, 2, 10), 4.2, 400, 3)
    p = s.params(table_bins=256)
    z = np.zeros(len(pos), np.float32)
    with m.Batch(p, [(len(pos), box)]) as b:
        with pytest.raises(m.MdrlError) as e:
            b.force(pos[:, 0], pos[:, 1], pos[:, 2], z, np.zeros(len(pos), np.int32))
        assert e.value.status == 2
