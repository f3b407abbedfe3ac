"""A call that takes the caller's arrays returns with nothing in flight, whatever its status: the GPU
reads and writes pageable arrays in place, so the caller must be able to free them at once.  The arrays
here outlive the calls; what is checked is that the streams are idle when an error comes back."""
import os

import numpy as np
import pytest
import torch

import sc2019_md_gb300 as m

pytestmark = pytest.mark.gpu

N, L = 400_000, 160.0
CALLS = ("cudaMemcpyAsync", "cudaStreamSynchronize", "cudaMemsetAsync", "cudaEventRecord", "cudaGetLastError",
         "cudaStreamWaitEvent", "cudaOccupancy", "cudaFuncSetAttribute", "cudaMemcpy(")


def _arm(spec):
    os.environ["MDRL_FAULT"] = spec
    try:
        with m.Context(m.default_params()):
            pass
    finally:
        del os.environ["MDRL_FAULT"]


@pytest.fixture(scope="module")
def arrays():
    rng = np.random.default_rng(3)
    k = int(round(N ** (1 / 3))) + 1
    site = np.sort(rng.permutation(k ** 3)[:N])
    ijk = np.stack([site // (k * k), (site // k) % k, site % k], 1)
    pos = ((ijk + 0.5 + rng.uniform(-0.2, 0.2, (N, 3))) * (L / k)).astype(np.float32)
    return [np.ascontiguousarray(pos[:, d]) for d in range(3)] + [np.zeros(N, np.float32), np.zeros(N, np.int32)]


def _params(**kw):
    return m.default_params(**{**dict(box=[L] * 3, cutoff=10.0, sigma=[1.5], epsilon=[0.1], mass=[40.0], coulomb_k=332.0), **kw})


def _every_failure(fn, pending):
    """fn with each of the failing calls in turn, until a run in which the fault finds no call left."""
    hits = 0
    for call in CALLS:
        for k in range(1, 40):
            _arm(f"{call}@{k}")
            try:
                fn()
            except m.MdrlError as e:
                assert "injected" in str(e)
                assert not pending(), (call, k)
                hits += 1
            else:
                break
    _arm("none")                     # what is left of the last count must not reach a later call
    assert hits >= 2


def test_refused_call_enqueues_nothing(arrays):
    """Fewer particles than the bonded terms name: refused before any kernel reads the arrays."""
    x, y, z, q, t = arrays
    bonds = (np.array([[0, N]], np.int32), np.array([[1.0, 1.5]]))
    with m.Context(_params()) as ctx:
        ctx.force(x, y, z, q, t)
        ctx.set_bonded(bonds=bonds)
        for _ in range(5):
            with pytest.raises(m.MdrlError) as e:
                ctx.force(x, y, z, q, t)
            assert e.value.status == 1 and not ctx.pending()


@pytest.mark.parametrize("pme", [False, True])
@pytest.mark.parametrize("entry", ["force", "force_pinned", "force_device", "force_fixed", "set_state", "get_state", "bin",
                                   "pair_eval"])
def test_errors_leave_nothing_in_flight(arrays, entry, pme):
    x, y, z, q, t = arrays
    with m.Context(_params(flags=m.FLAG_ENERGY)) as ctx:
        if pme:
            ctx.set_pme()
        ctx.set_state(x, y, z, None, q, t)
        if entry == "force_device":
            d = [torch.as_tensor(a, device="cuda") for a in (x, y, z)]
            out = [torch.zeros(N, device="cuda") for _ in range(3)]

            def fn():
                import ctypes as C
                m._check(m.lib().mdrl_force_eval_device(ctx._h, N, *(C.c_void_p(a.data_ptr()) for a in d), None, None,
                                                        *(C.c_void_p(a.data_ptr()) for a in out), None, None))
        elif entry == "force_pinned":
            pin = [torch.as_tensor(a).pin_memory().numpy() for a in (x, y, z, q)]
            out = [torch.zeros(N).pin_memory().numpy() for _ in range(3)]

            def fn():
                m._check(m.lib().mdrl_force_eval(ctx._h, N, *(m._fp(a) for a in pin), None, *(m._fp(a) for a in out),
                                                 None, None))
        else:
            four = np.stack([x, y, z, q], 1)
            state = [np.zeros(N, np.float32) for _ in range(9)]
            fn = {"force": lambda: ctx.force(x, y, z, q, t, counts=True), "force_fixed": lambda: ctx.force_fixed(x, y, z, q, t),
                  "set_state": lambda: ctx.set_state(x, y, z, None, q, t),
                  "get_state": lambda: m._check(m.lib().mdrl_get_state(ctx._h, *(m._fp(a) for a in state))),
                  "bin": lambda: ctx.bin(x, y, z), "pair_eval": lambda: ctx.pair_eval(four, four, t, t)}[entry]
        _every_failure(fn, ctx.pending)
        fn()


@pytest.mark.parametrize("entry", ["force", "set_state", "state"])
def test_batch_errors_leave_nothing_in_flight(entry):
    from sc2019_md_gb300 import systems
    reps = [systems.replica(n, r) for r, n in enumerate((520, 700, 1100, 2300, 3600, 20000))]
    pos, vel, q, t, spec = systems.concat(reps)
    with m.Batch(reps[0].params(flags=m.FLAG_ENERGY), spec) as b:
        b.set_state(pos[:, 0], pos[:, 1], pos[:, 2], vel, q, t)
        fn = {"force": lambda: b.force(pos[:, 0], pos[:, 1], pos[:, 2], q, t),
              "set_state": lambda: b.set_state(pos[:, 0], pos[:, 1], pos[:, 2], vel, q, t), "state": b.state}[entry]
        _every_failure(fn, b.pending)
        fn()
