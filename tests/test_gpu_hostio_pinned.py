"""Page-locked arrays at any byte address: where the elements are not aligned they go through copies, as
pageable ones do; results equal those of ordinary arrays bit for bit, and nothing outside the arrays
changes."""
import ctypes as C

import numpy as np
import pytest
import torch

import sc2019_md_gb300 as m
from sc2019_md_gb300 import systems

pytestmark = pytest.mark.gpu

GUARD = 64


class Pinned:
    """n items of `size` bytes, `shift` bytes from an aligned page-locked address, between guard bytes."""

    def __init__(self, n, size, shift, src=None):
        self.buf = torch.zeros(n * size + 2 * GUARD + 64, dtype=torch.uint8).pin_memory()
        base = -self.buf.data_ptr() % 64
        self.at, self.len = base + GUARD + shift, n * size
        self.addr = self.buf.data_ptr() + self.at
        if src is not None:
            raw = np.frombuffer(np.ascontiguousarray(src).tobytes(), np.uint8).copy()
            self.buf[self.at:self.at + self.len] = torch.from_numpy(raw)

    def get(self, dtype):
        b = self.buf.numpy()
        assert not b[:self.at].any() and not b[self.at + self.len:].any()
        return np.frombuffer(b[self.at:self.at + self.len].tobytes(), dtype)


def _call(fn, *args):
    conv = [C.cast(a.addr, t) if isinstance(a, Pinned) else a for a, t in zip(args, fn.argtypes)]
    s = fn(*conv)
    assert s == 0, m.lib().mdrl_last_error()


@pytest.mark.parametrize("shift", [0, 1, 2, 4])
@pytest.mark.parametrize("n", [1728, 20001])
def test_any_address(shift, n):
    s = systems.small_ljc(n, 36.1 if n < 5000 else 60.0, 12.0, seed=n)
    cols = [np.ascontiguousarray(s.pos[:, k]) for k in range(3)]
    L = m.lib()
    with m.Context(s.params(table_bins=256)) as ctx:
        F, st, cnt = ctx.force(*cols, s.q, s.type, counts=True)
        Ff, _ = ctx.force_fixed(*cols, s.q, s.type)
        cell, _, order = ctx.bin(*cols)
        ctx.set_state(*cols, s.vel, s.q, s.type)
        frame = ctx.state()
        ins = [Pinned(n, 4, shift, a) for a in (*cols, s.q, s.type)]
        out = [Pinned(n, 4, shift) for _ in range(4)]
        _call(L.mdrl_force_eval, ctx._h, n, *ins, *out, C.byref(m.Stats()))
        for k in range(3):
            assert np.array_equal(out[k].get(np.uint32), F[:, k].copy().view(np.uint32))
        assert np.array_equal(out[3].get(np.int32), cnt)
        fix = Pinned(3 * n, 8, shift)
        _call(L.mdrl_force_eval_fixed, ctx._h, n, *ins, 0, s.ncell[0], fix, C.byref(m.Stats()))
        assert np.array_equal(fix.get(np.int64).reshape(3, n).T, Ff)
        out = [Pinned(n, 4, shift) for _ in range(2)]
        _call(L.mdrl_bin, ctx._h, n, *ins[:3], out[0], None, out[1])
        assert np.array_equal(out[0].get(np.int32), cell) and np.array_equal(out[1].get(np.int32), order)
        vel = [Pinned(n, 4, shift, s.vel[:, k]) for k in range(3)]
        _call(L.mdrl_set_state, ctx._h, n, *ins[:3], *vel, *ins[3:])
        out = [Pinned(n, 4, shift) for _ in range(9)]
        _call(L.mdrl_get_state, ctx._h, *out)
        for k in range(9):
            assert np.array_equal(out[k].get(np.uint32), frame[k // 3][:, k % 3].copy().view(np.uint32))


@pytest.mark.parametrize("shift", [0, 8, 4, 2, 1])
def test_pair_eval_any_address(shift):
    rng = np.random.default_rng(6)
    n = 1001
    ref, nbr = (rng.uniform(0, 25.5, (n, 4)).astype(np.float32) for _ in range(2))
    t = np.zeros(n, np.int32)
    with m.Context(m.default_params(coulomb_k=332.0637)) as ctx:
        want = ctx.pair_eval(ref, nbr, t, t)
        ins = [Pinned(n, 16, shift, ref), Pinned(n, 16, shift, nbr), Pinned(n, 4, shift, t), Pinned(n, 4, shift, t)]
        out = [Pinned(n, 16, shift), Pinned(n, 8, shift)]
        _call(m.lib().mdrl_pair_eval, ctx._h, n, *ins, *out)
    for b, w in zip(out, want):
        assert np.array_equal(b.get(np.uint32), w.view(np.uint32).reshape(-1))


@pytest.mark.parametrize("shift", [0, 1, 4])
def test_batch_any_address(shift):
    reps = [systems.replica(v, r) for r, v in enumerate((600, 2500, 6000))]
    pos, vel, q, t, spec = systems.concat(reps)
    cols = [np.ascontiguousarray(pos[:, k]) for k in range(3)]
    n = len(pos)
    L = m.lib()
    with m.Batch(reps[0].params(), spec) as b:
        F, _, _ = b.force(*cols, q, t)
        b.set_state(*cols, vel, q, t)
        frame = b.state()
        ins = [Pinned(n, 4, shift, a) for a in (*cols, q, t)]
        out = [Pinned(n, 4, shift) for _ in range(3)]
        _call(L.mdrl_batch_force_eval, b._h, *ins, *out, None, C.byref(m.Stats()))
        for k in range(3):
            assert np.array_equal(out[k].get(np.uint32), F[:, k].copy().view(np.uint32))
        v = [Pinned(n, 4, shift, vel[:, k]) for k in range(3)]
        _call(L.mdrl_batch_set_state, b._h, *ins[:3], *v, *ins[3:])
        out = [Pinned(n, 4, shift) for _ in range(9)]
        _call(L.mdrl_batch_get_state, b._h, *out)
        for k in range(9):
            assert np.array_equal(out[k].get(np.uint32), frame[k // 3][:, k % 3].copy().view(np.uint32))
