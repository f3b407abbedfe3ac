"""A batch's evaluation runs the replicas that need every image beside the others: alternating
evaluations of two configurations, and one after an injected failure between the launches, give the
bits of a fresh batch, with and without energies and partner counts."""
import os

import numpy as np
import pytest

import sc2019_md_gb300 as m
from sc2019_md_gb300 import systems

pytestmark = pytest.mark.gpu

SIZES = (520, 700, 1100, 2300, 3600, 4100)        # every image, cell pairs, half shell


def _arm(spec):
    os.environ["MDRL_FAULT"] = spec
    try:
        with m.Context(m.default_params()):
            pass
    finally:
        del os.environ["MDRL_FAULT"]


@pytest.mark.parametrize("energy", [0, m.FLAG_ENERGY])
@pytest.mark.parametrize("counts", [False, True])
def test_evaluations_do_not_run_into_each_other(energy, counts):
    reps = [systems.replica(n, r) for r, n in enumerate(SIZES)]
    args = []
    for turn in (0, 1):
        pos = np.concatenate([np.mod(s.pos + np.float32(1.7 * turn), np.float32(s.box[0])).astype(np.float32) for s in reps])
        args.append((np.ascontiguousarray(pos[:, 0]), np.ascontiguousarray(pos[:, 1]), np.ascontiguousarray(pos[:, 2]),
                     np.concatenate([s.q for s in reps]), np.concatenate([s.type for s in reps])))
    p = reps[0].params(flags=energy)
    shapes = [(s.n, s.box) for s in reps]

    def evaluate(b, a):
        F, st, cnt = b.force(*a, counts=counts)
        return F.view(np.uint32), st["pairs"], None if cnt is None else np.asarray(cnt).copy()

    want = []
    for a in args:
        with m.Batch(p, shapes) as b:
            want.append(evaluate(b, a))
    with m.Batch(p, shapes) as b:
        for k in range(12):
            if k == 6:
                _arm("cudaStreamWaitEvent(b->side")
                with pytest.raises(m.MdrlError):
                    b.force(*args[1], counts=counts)
            got = evaluate(b, args[k % 2])
            assert np.array_equal(got[0], want[k % 2][0]) and got[1] == want[k % 2][1]
            if counts:
                assert np.array_equal(got[2], want[k % 2][2])
