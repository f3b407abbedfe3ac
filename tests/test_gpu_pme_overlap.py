"""The reciprocal part runs on a stream of its own beside the pair kernel: dynamics give the same bits
run after run, and a call that fails between the two parts (a host-side injected error, during the
graph's capture too) leaves a context that gives them again."""
import os

import numpy as np
import pytest

import sc2019_md_gb300 as m
from sc2019_md_gb300 import systems

pytestmark = pytest.mark.gpu


def _start(ctx, s, vel):
    ctx.set_state(s.pos[:, 0], s.pos[:, 1], s.pos[:, 2], vel, s.q, s.type)


def _run(ctx, s, vel, steps):
    _start(ctx, s, vel)
    st = ctx.step(steps)
    return [np.asarray(a).copy() for a in ctx.state()], st["pairs"]


def _arm(spec):
    """Read when a context is created; counts from the return of mdrl_create."""
    os.environ["MDRL_FAULT"] = spec
    try:
        with m.Context(m.default_params()):
            pass
    finally:
        del os.environ["MDRL_FAULT"]


@pytest.mark.parametrize("energy", [0, m.FLAG_ENERGY])
@pytest.mark.parametrize("call", ["cudaGetLastError@1", "cudaGetLastError@2", "cudaGetLastError@3", "cudaGetLastError@4",
                                  "cudaStreamWaitEvent@2"])
def test_failed_step_then_the_same_bits(call, energy):
    s = systems.small_ljc(5000, 54.0, 12.0, seed=7, ntypes=2, dmin=2.2)
    vel = np.zeros_like(s.pos)
    with m.Context(s.params(flags=energy)) as ctx:
        ctx.set_pme()
        want, pairs = _run(ctx, s, vel, 4)
    with m.Context(s.params(flags=energy)) as ctx:
        ctx.set_pme()
        _start(ctx, s, vel)
        _arm(call)
        with pytest.raises(m.MdrlError) as e:
            ctx.step(4)
        assert "injected" in str(e.value)
        got, pairs2 = _run(ctx, s, vel, 4)
    assert pairs == pairs2
    for a, b in zip(want, got):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
