"""A refused evaluation or binning has used the state's buffers: steps after it are refused (a binning by
index leaves counts that a step would index with), and a new set_state gives what a fresh context gives."""
import numpy as np
import pytest

import sc2019_md_gb300 as m
from sc2019_md_gb300 import systems

pytestmark = pytest.mark.gpu


def _bad(x, where):
    x = x.copy()
    x[where] = -1.0
    return x


@pytest.mark.parametrize("n,L", [(1800, 37.5), (9000, 50.0)])       # the one-CTA binning and the general one
@pytest.mark.parametrize("entry", ["bin", "force", "force_fixed", "set_state"])
def test_step_after_a_refused_call(n, L, entry):
    s = systems.small_ljc(n, L, 12.0, seed=n)
    x, y, z = (np.ascontiguousarray(s.pos[:, k]) for k in range(3))
    with m.Context(s.params()) as ref:
        ref.set_state(x, y, z, s.vel, s.q, s.type)
        ref.step(3)
        want = ref.state()
    with m.Context(s.params()) as ctx:
        ctx.set_state(x, y, z, s.vel, s.q, s.type)
        ctx.step(1)
        call = {"bin": lambda v: ctx.bin(v, y, z), "force": lambda v: ctx.force(v, y, z, s.q, s.type),
                "force_fixed": lambda v: ctx.force_fixed(v, y, z, s.q, s.type),
                "set_state": lambda v: ctx.set_state(v, y, z, s.vel, s.q, s.type)}[entry]
        with pytest.raises(m.MdrlError) as e:
            call(_bad(x, n // 2))
        assert e.value.status == 1
        for fn in (lambda: ctx.step(2), ctx.state, ctx.time_force):
            with pytest.raises(m.MdrlError) as e:
                fn()
            assert e.value.status == 6
        ctx.set_state(x, y, z, s.vel, s.q, s.type)
        ctx.step(3)
        got = ctx.state()
    for a, b in zip(want, got):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_batch_after_a_refused_evaluation():
    reps = [systems.replica(v, r) for r, v in enumerate((600, 2500, 6000))]
    pos, vel, q, t, spec = systems.concat(reps)
    x, y, z = (np.ascontiguousarray(pos[:, k]) for k in range(3))
    with m.Batch(reps[0].params(), spec) as b:
        b.set_state(x, y, z, vel, q, t)
        with pytest.raises(m.MdrlError):
            b.force(_bad(x, 700), y, z, q, t)
        for fn in (lambda: b.step(1), b.replica_stats, b.state):
            with pytest.raises(m.MdrlError) as e:
                fn()
            assert e.value.status == 6
        b.set_state(x, y, z, vel, q, t)
        st = b.step(2)
        assert sum(r["pairs"] for r in b.replica_stats()) == st["pairs"]
