"""Arrays of a call that share storage: inputs are read before results are written over them, and of results
that share storage the later argument's stay, as if every array were copied by itself in order."""
import numpy as np
import pytest

import sc2019_md_gb300 as m
from sc2019_md_gb300 import systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 4001, 300001])
def test_pair_eval(n):
    rng = np.random.default_rng(n)
    ref, nbr = (rng.uniform(0, 25.5, (n, 4)).astype(np.float32) for _ in range(2))
    tr, tn = (rng.integers(0, 3, n).astype(np.int32) for _ in range(2))
    L = m.lib()
    with m.Context(m.default_params(coulomb_k=332.0, ntypes=3, sigma=[2.0, 3.0, 3.5], epsilon=[0.1, 0.2, 0.3],
                                    mass=[1.0] * 3)) as ctx:
        out, aux = ctx.pair_eval(ref, nbr, tr, tn)
        # the types in the results' storage (at its end and, shifted, at its start), then in aux's
        buf, two = np.zeros(4 * n, np.float32), np.zeros(2 * n, np.float32)
        buf[3 * n:].view(np.int32)[:] = tr
        buf[:n].view(np.int32)[:] = tn
        m._check(L.mdrl_pair_eval(ctx._h, n, m._fp(ref), m._fp(nbr), m._ip(buf[3 * n:].view(np.int32)),
                                  m._ip(buf[:n].view(np.int32)), m._fp(buf), m._fp(two)))
        assert np.array_equal(buf.view(np.uint32), out.reshape(-1).view(np.uint32))
        two[n:].view(np.int32)[:] = tr
        m._check(L.mdrl_pair_eval(ctx._h, n, m._fp(ref), m._fp(nbr), m._ip(two[n:].view(np.int32)), m._ip(tn), m._fp(buf),
                                  m._fp(two)))
        assert np.array_equal(two.view(np.uint32), aux.reshape(-1).view(np.uint32))
        # positions under the results
        pos = ref.copy()
        m._check(L.mdrl_pair_eval(ctx._h, n, m._fp(pos), m._fp(nbr), m._ip(tr), m._ip(tn), m._fp(pos), None))
        assert np.array_equal(pos.view(np.uint32), out.view(np.uint32))
        # aux over the second half of out: the later argument's values stay
        m._check(L.mdrl_pair_eval(ctx._h, n, m._fp(ref), m._fp(nbr), m._ip(tr), m._ip(tn), m._fp(buf), m._fp(buf[2 * n:])))
        assert np.array_equal(buf[2 * n:].view(np.uint32), aux.reshape(-1).view(np.uint32))
        assert np.array_equal(buf[:2 * n].view(np.uint32), out.reshape(-1)[:2 * n].view(np.uint32))


@pytest.mark.parametrize("n,L", [(1728, 36.1), (20001, 60.0)])
def test_results_that_share_storage(n, L):
    s = systems.small_ljc(n, L, 12.0, seed=n)
    x, y, z = (np.ascontiguousarray(s.pos[:, k]) for k in range(3))
    lib = m.lib()
    with m.Context(s.params()) as ctx:
        F, _, _ = ctx.force(x, y, z, s.q, s.type)
        one, both = np.zeros(n, np.float32), np.zeros(n + 1, np.float32)
        # fz one element into fy
        m._check(lib.mdrl_force_eval(ctx._h, n, m._fp(x), m._fp(y), m._fp(z), m._fp(s.q), m._ip(s.type), m._fp(one),
                                     m._fp(both[:n]), m._fp(both[1:]), None, None))
        assert np.array_equal(one.view(np.uint32), F[:, 0].copy().view(np.uint32))
        assert np.array_equal(both[1:].view(np.uint32), F[:, 2].copy().view(np.uint32))
        assert both[0].view(np.uint32) == F[0, 1].view(np.uint32)
        # forces over the positions
        a = [v.copy() for v in (x, y, z)]
        m._check(lib.mdrl_force_eval(ctx._h, n, *map(m._fp, a), m._fp(s.q), m._ip(s.type), *map(m._fp, a), None, None))
        assert all(np.array_equal(a[k].view(np.uint32), F[:, k].copy().view(np.uint32)) for k in range(3))
        ctx.set_state(x, y, z, s.vel, s.q, s.type)
        want = ctx.state()
        both = np.zeros(n + 1, np.float32)
        m._check(lib.mdrl_get_state(ctx._h, m._fp(both[:n]), m._fp(both[1:]), m._fp(one), *[None] * 6))
        assert np.array_equal(both[1:], want[0][:, 1]) and both[0] == want[0][0, 0] and np.array_equal(one, want[0][:, 2])
