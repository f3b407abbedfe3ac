"""Evaluations after tuning take the kernel of an untuned context, whatever tile the tuner chose for
dynamics; a tile that the caller sets is taken.  The tuner's choice is planted through its cache file."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import sc2019_md_gb300 as m
from sc2019_md_gb300 import systems

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

CODE = """
import sys
import numpy as np
sys.path.insert(0, {root!r})
import sc2019_md_gb300 as m
from sc2019_md_gb300 import systems
s = systems.small_ljc(2500, 37.5, 12.0, seed=31)
a = [np.ascontiguousarray(s.pos[:, k]) for k in range(3)]
with m.Context(s.params()) as ctx:
    F0 = ctx.force(*a, s.q, s.type)[0]
    assert ctx.kernels()["eval"] == "list"
    ctx.set_state(*a, s.vel, s.q, s.type)
    ctx.autotune()
    print(ctx.tile())
    assert ctx.kernels()["eval"] == "list"
    F1 = ctx.force(*a, s.q, s.type)[0]
    assert np.array_equal(F0.view(np.uint32), F1.view(np.uint32))
"""


def test_evaluation_after_a_tuner_that_chose_a_cta_tile(tmp_path):
    cache = tmp_path / "tiles"
    env = dict(os.environ, MDRL_TUNE_CACHE=str(cache))
    run = lambda: subprocess.run([sys.executable, "-c", CODE.format(root=str(ROOT))], env=env, capture_output=True,  # noqa: E731
                                 text=True, timeout=300)
    r = run()
    assert r.returncode == 0, r.stderr
    key = cache.read_text().split()[0]
    cache.write_text(f"{key} 4 6 0 0.01\n")
    r = run()
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip() == "(4, 6, 0)"


def test_caller_tiles_and_the_tuner():
    s = systems.small_ljc(2500, 37.5, 12.0, seed=31)
    a = [np.ascontiguousarray(s.pos[:, k]) for k in range(3)]
    with m.Context(s.params()) as ctx:
        for tile, want in (((4, 6, 0), "cta"), ((8, 4, 1), "cta"), ((1, 2, 1), "list")):
            ctx.set_tile(*tile)
            assert ctx.kernels()["eval"] == want
        ctx.set_state(*a, s.vel, s.q, s.type)
        assert ctx.kernels()["step_launches"] == 0
        ctx.step(3)
        assert ctx.kernels()["step_launches"] > 0
        ctx.set_tile(4, 6, 0)
        ctx.autotune(retime=True)
        assert ctx.kernels()["eval"] == "list"
    with m.Context(s.params(accum=m.ACC_FP32_ATOMIC)) as ctx:
        assert ctx.kernels()["eval"] == "cta"
