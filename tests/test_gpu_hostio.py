"""Host arrays read and written in place: any address (elements that are not aligned go through copies),
nothing outside the arrays, and pages nobody has touched before; results equal those of ordinary
arrays bit for bit."""
import ctypes as C
import mmap

import numpy as np
import pytest

import sc2019_md_gb300 as m
from sc2019_md_gb300 import systems

pytestmark = pytest.mark.gpu

GUARD = 64


class Buf:
    """An array of n items of `size` bytes, `shift` bytes into fresh pages, with guard bytes around it."""

    def __init__(self, n, size, shift, src=None):
        self.len = n * size
        self.map = mmap.mmap(-1, self.len + 2 * GUARD + 64)
        self.at = GUARD + shift
        self.guards = [slice(0, self.at), slice(self.at + self.len, len(self.map))]
        self.addr = C.addressof(C.c_char.from_buffer(self.map, self.at))
        if src is not None:
            self.map[self.at:self.at + self.len] = np.ascontiguousarray(src).tobytes()

    def get(self, dtype):
        assert all(set(self.map[g]) <= {0} for g in self.guards)
        return np.frombuffer(self.map[self.at:self.at + self.len], dtype)


def _call(fn, *args):
    conv = [C.cast(a.addr, t) if isinstance(a, Buf) else a for a, t in zip(args, fn.argtypes)]
    s = fn(*conv)
    assert s == 0, m.lib().mdrl_last_error()


@pytest.mark.parametrize("shift", [0, 4, 1])
@pytest.mark.parametrize("n", [1728, 40001])
def test_any_address(shift, n):
    s = systems.small_ljc(n, 36.1 if n < 5000 else 74.0, 12.0, seed=n)
    cols = [np.ascontiguousarray(s.pos[:, k]) for k in range(3)]
    with m.Context(s.params(table_bins=256)) as ctx:
        F, st, cnt = ctx.force(*cols, s.q, s.type, counts=True)
        Ff, _ = ctx.force_fixed(*cols, s.q, s.type)
        ctx.set_state(*cols, s.vel, s.q, s.type)
        frame = ctx.state()
        ins = [Buf(n, 4, shift, a) for a in (*cols, s.q, s.type)]
        out = [Buf(n, 4, shift) for _ in range(4)]
        _call(m.lib().mdrl_force_eval, ctx._h, n, *ins, *out, C.byref(m.Stats()))
        for k in range(3):
            assert np.array_equal(out[k].get(np.uint32), F[:, k].copy().view(np.uint32))
        assert np.array_equal(out[3].get(np.int32), cnt)
        fix = Buf(3 * n, 8, shift)
        _call(m.lib().mdrl_force_eval_fixed, ctx._h, n, *ins, 0, s.ncell[0], fix, C.byref(m.Stats()))
        assert np.array_equal(fix.get(np.int64).reshape(3, n).T, Ff)
        vel = [Buf(n, 4, shift, s.vel[:, k]) for k in range(3)]
        _call(m.lib().mdrl_set_state, ctx._h, n, *ins[:3], *vel, *ins[3:])
        out = [Buf(n, 4, shift) for _ in range(9)]
        _call(m.lib().mdrl_get_state, ctx._h, *out)
        for k in range(9):
            assert np.array_equal(out[k].get(np.uint32), frame[k // 3][:, k % 3].copy().view(np.uint32))


@pytest.mark.parametrize("shift", [0, 8, 4, 1])
def test_pair_eval_any_address(shift):
    rng = np.random.default_rng(5)
    n = 1001
    ref, nbr = (rng.uniform(0, 25.5, (n, 4)).astype(np.float32) for _ in range(2))
    t = np.zeros(n, np.int32)
    with m.Context(m.default_params(coulomb_k=332.0637)) as ctx:
        want = ctx.pair_eval(ref, nbr, t, t)
        ins = [Buf(n, 16, shift, ref), Buf(n, 16, shift, nbr), Buf(n, 4, shift, t), Buf(n, 4, shift, t)]
        out = [Buf(n, 16, shift), Buf(n, 8, shift)]
        _call(m.lib().mdrl_pair_eval, ctx._h, n, *ins, *out)
    for b, w in zip(out, want):
        assert np.array_equal(b.get(np.uint32), w.view(np.uint32).reshape(-1))


def test_large_fresh_frame():
    """Frames above the size from which threads populate the pages."""
    reps = [systems.replica(4000, k) for k in range(12)]
    pos, vel, q, t, spec = systems.concat(reps)
    grow = 10                                            # 480,000 atoms: 17 MB of frame
    spec = spec * grow
    pos, vel, q, t = (np.concatenate([a] * grow) for a in (pos, vel, q, t))
    with m.Batch(reps[0].params(), spec) as b:
        b.set_state(pos[:, 0], pos[:, 1], pos[:, 2], vel, q, t)
        x, v, F = b.state()
        out = [Buf(b.n, 4, 0) for _ in range(9)]
        _call(m.lib().mdrl_batch_get_state, b._h, *out)
    assert np.array_equal(x, pos)
    for k in range(9):
        assert np.array_equal(out[k].get(np.uint32), (x, v, F)[k // 3][:, k % 3].copy().view(np.uint32))
