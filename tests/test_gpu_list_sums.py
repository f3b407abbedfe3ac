"""Partial sums of the list kernel: what is added in FP32, and what in exact integers or with compensation.

Each case plants terms that cancel where the sums have to keep a small one beside them."""
import itertools

import numpy as np
import pytest

import sc2019_md_gb300 as m

pytestmark = pytest.mark.gpu

L, RC, EDGE = 62.5, 12.0, 12.5


def _hilbert(pos, cell):
    """Index along the 24-bit Hilbert curve of the in-cell order (Skilling's transform)."""
    loc = (pos.astype(np.float64) - np.asarray(cell) * EDGE) * (256.0 / EDGE)
    x = np.clip(loc.astype(int), 0, 255).T.copy()
    bit = 128
    while bit > 1:
        low = bit - 1
        for k in range(3):
            hi = (x[k] & bit) != 0
            t = np.where(hi, 0, (x[0] ^ x[k]) & low)
            x[0] ^= np.where(hi, low, t)
            x[k] ^= t
        bit >>= 1
    x[1] ^= x[0]
    x[2] ^= x[1]
    t = np.zeros_like(x[0])
    bit = 128
    while bit > 1:
        t ^= np.where(x[2] & bit, bit - 1, 0)
        bit >>= 1
    x ^= t
    h = np.zeros_like(x[0])
    for b in range(7, -1, -1):
        for k in range(3):
            h = (h << 1) | ((x[k] >> b) & 1)
    return h


def _params(**kw):
    return m.default_params(**{**dict(box=[L] * 3, cutoff=RC, ntypes=3, sigma=[1.0] * 3, epsilon=[0.0] * 3, mass=[1.0] * 3,
                                      table_bins=256), **kw})


def test_forces_of_different_lists_add_exactly():
    """An atom with two neighbours whose y forces cancel exactly, 1e5 kcal/mol/A each, in different cells, and
    between them in the cell order more than 512 atoms without forces, a weak neighbour, and 512 more: the
    three are in different lists, and the weak one's force comes out as if the strong ones were not there."""
    rng = np.random.default_rng(1)
    i = np.array([24.5, 24.5, 13.0])
    lo = np.array([2, 2, 0]) * EDGE
    f = lo + rng.uniform(0.05, EDGE - 0.05, (6000, 3))
    f = f[np.linalg.norm(f - i, axis=1) < RC - 0.5].astype(np.float32)
    f = f[np.argsort(_hilbert(f, (2, 2, 0)), kind="stable")]
    near = np.linalg.norm(f - i, axis=1) < 7.0
    at = [k for k in np.flatnonzero(near) if 600 < k < len(f) - 600]
    c = at[len(at) // 2]
    pos = np.concatenate([[i, [25.5, 23.5, 13.0], [25.5, 25.5, 13.0]], f]).astype(np.float32)
    t = np.ones(len(pos), np.int32)
    t[:3] = 0
    t[3 + c] = 2
    coef = np.zeros((3, 3, 4))
    coef[0, 0, 0] = 1.28e7                     # 2^-7 of it at r2 = 2: 1e5 per component
    r2 = float(((f[c] - i) ** 2).sum())
    coef[0, 2, 0] = coef[2, 0, 0] = 1.234567 * r2 ** 7
    keep = np.arange(len(pos)) > 2
    keep[0] = True
    with m.Context(_params()) as ctx:
        ctx.set_pair_coefficients(coef)
        assert ctx.kernels()["eval"] == "list"
        F, st = ctx.force_fixed(*(np.ascontiguousarray(pos[:, k]) for k in range(3)), type=t)
        W, _ = ctx.force_fixed(*(np.ascontiguousarray(pos[keep, k]) for k in range(3)), type=t[keep])
    assert abs(F[1, 1]) > 9e4 * 2 ** 24 and abs(F[2, 1]) > 9e4 * 2 ** 24
    assert abs(W[0, 1]) > 0.1 * 2 ** 24
    assert F[0, 1] == W[0, 1] and F[0, 2] == W[0, 2]


def _planted(types, at, order=1, a12=(), a14=()):
    pos = np.array([[24.0, 18.0, 18.0]] + at, np.float32)
    coef = np.zeros((4, 4, 4))
    for k, (e, f) in enumerate(zip(a12, a14)):
        coef[0, k + 1, 0] = coef[k + 1, 0, 0] = f
        coef[0, k + 1, 2] = coef[k + 1, 0, 2] = e
    with m.Context(_params(ntypes=4, sigma=[1.0] * 4, epsilon=[0.0] * 4, mass=[1.0] * 4, flags=m.FLAG_ENERGY,
                           table_order=order)) as ctx:
        ctx.set_pair_coefficients(coef)
        assert ctx.kernels()["eval"] == "list"
        return ctx.force(*(np.ascontiguousarray(pos[:, k]) for k in range(3)), type=np.array([0] + types, np.int32))[1]


@pytest.mark.parametrize("order", [1, 2, 3])
def test_energies_that_cancel_across_lanes(order):
    """Two pair energies (and virials) of 6,400 and -6,400 and one of 8e-5 in one list, in every order: the small
    one is what is left.  Lanes hold one pair each; the sums over lanes keep 2^-46 of the largest term:
    1e-9 here."""
    at = [[26.0, 19.0, 18.0], [26.0, 17.0, 18.0], [26.0, 18.0, 19.0]]
    e, f = (1.0e8, -1.0e8, 1.2345), (1.0e8, -1.0e8, 1.2345)
    want = _planted([3], at[2:], order, e, f)
    assert want["e_lj"] > 5e-5
    for types in itertools.permutations([1, 2, 3]):
        got = _planted(list(types), at, order, e, f)
        assert got["pairs"] == 6
        assert abs(got["e_lj"] - want["e_lj"]) < 1e-9
        assert abs(got["virial"] - want["virial"]) < 1e-9


def test_infinite_energies_stay_infinite():
    """A pair energy that overflows FP32 while its force is finite: the total is infinite, not NaN."""
    st = _planted([1], [[24.5, 18.0, 18.0]], 1, (3.0e38,), (1.0,))
    assert st["e_lj"] == np.inf and np.isfinite(st["virial"])
    st = _planted([1, 2], [[24.5, 18.0, 18.0], [26.0, 17.0, 18.0]], 1, (-3.0e38, 1.0), (1.0, 1.0))
    assert st["e_lj"] == -np.inf and np.isfinite(st["virial"])


@pytest.mark.parametrize("each,ok", [(1.0e11, True), (4.0e11, False)])
def test_sums_beyond_the_fixed_point_range_are_reported(each, ok):
    """Two forces that the accumulators hold and whose sum (8e11 kcal/mol/A) they do not, in one list."""
    pos = np.array([[24.0, 18.0, 18.0], [26.0, 19.0, 18.0], [26.0, 17.0, 18.0]], np.float32)
    coef = np.zeros((3, 3, 4))
    coef[0, 1, 0] = coef[1, 0, 0] = each / 2.0 * 5.0 ** 7
    with m.Context(_params()) as ctx:
        ctx.set_pair_coefficients(coef)
        call = lambda: ctx.force(*(np.ascontiguousarray(pos[:, k]) for k in range(3)), type=np.array([0, 1, 1], np.int32))  # noqa: E731
        if ok:
            assert abs(call()[0][0, 0] + 2 * each) < 1e-2 * each
        else:
            with pytest.raises(m.MdrlError) as e:
                call()
            assert e.value.status == 3
