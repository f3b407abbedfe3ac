"""Steps run in graphs of two and an odd one of one: any split of a number of steps over calls gives the
same bits, from either buffer slot, and after calls that drop the graphs."""
import numpy as np
import pytest

import sc2019_md_gb300 as m
from helpers import liquid_argon

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [None, (1, 1, 1)])
@pytest.mark.parametrize("integrator", [m.INT_VELOCITY_VERLET, m.INT_EULER])
def test_any_split_gives_the_same_bits(tile, integrator):
    s = liquid_argon()
    out = []
    for split in ([7], [1] * 7, [2, 2, 3], [3, 4], [1, 5, 0, 1]):
        with m.Context(m.default_params(box=s.box, cutoff=8.5, integrator=integrator, flags=m.FLAG_ENERGY)) as ctx:
            if tile:
                ctx.set_tile(*tile)
            ctx.set_state(s.pos[:, 0], s.pos[:, 1], s.pos[:, 2], s.vel)
            total = 0
            for k in split:
                st = ctx.step(k)
                total += st["pairs_total"] if k else 0
                if k == 3:
                    ctx.set_tile(*((4, 2, 0) if not tile else (1, 2, 1)))       # drops the graphs
                    ctx.set_tile(*((4, 6, 0) if not tile else tile))
            out.append((total, [a.view(np.uint32) for a in ctx.state()]))
    for total, arrays in out[1:]:
        assert total == out[0][0]
        for a, b in zip(out[0][1], arrays):
            assert np.array_equal(a, b)
