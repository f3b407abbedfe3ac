"""The C model's run on the GPU, bit for bit against the oracle's restatement, at the sizes where the
one-launch-per-iteration kernel can go wrong: one particle, chunk edges (128 particles tested at a
time), and a box so dense that a particle's pairs fill the compacted list (512) several times."""
import numpy as np
import pytest

import oracle
import sc2019_md_gb300 as m

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,box,cutoff", [(1, 24.0, 8.0), (2, 24.0, 8.0), (127, 24.0, 8.0), (128, 12.0, 5.9),
                                          (129, 24.0, 8.0), (513, 6.0, 3.0), (1900, 9.0, 9.0)])
def test_cmodel_bits(n, box, cutoff):
    rng = np.random.default_rng(n)
    k = int(np.ceil(n ** (1 / 3)))
    g = (np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] + 0.5) * (box / k)
    pos = np.mod(g + rng.uniform(-0.1, 0.1, (n, 3)) * box / k, box).astype(np.float32)
    pos[pos >= np.float32(box)] = 0.0
    vel = rng.uniform(-1e11, 1e11, (n, 3)).astype(np.float32)
    p, v, e, cnt = m.cmodel_run(pos, vel, 7, box=box, cutoff=cutoff, counts=True)
    po, vo, eo, cnto = oracle.cmodel_run(pos, vel, 7, box=box, cutoff=cutoff)
    for a, b in ((p, po), (v, vo), (e, eo)):
        assert np.array_equal(np.asarray(a, np.float32).view(np.uint32), np.asarray(b, np.float32).reshape(a.shape).view(np.uint32))
    assert np.array_equal(cnt, cnto)
