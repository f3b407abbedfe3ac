"""The work that a user of this package has it do, as cases that can be timed and compared.

Sizes are those of the package's own workloads, tests and bench: the C model's 500 atoms, the
10,000-pair plugin stream, the 1,728-atom cube, the DHFR-sized 23,558 atoms with bonded terms, the
92,224-atom and 1,048,576-atom LJ + Coulomb systems and the 512-replica batch, with ragged ones
between them.  Positions are a jittered lattice (a random subset of its sites in random order), so
that a system of any size has a known smallest separation and is made in milliseconds.  Force
evaluations take the violent 1.0 A separations of those workloads; dynamics starts from states that
an integrator can follow (a liquid), since a truncated trajectory of an exploding one says nothing.

A drawn case is one of the same kinds with its size, box shape, table order, bins, options and
side of the host link drawn over the ranges that the listed ones span.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import sc2019_md_gb300 as m

KE = 332.0637
AMU = 4.184e-4            # (kcal/mol/A)/amu -> A/fs^2
KB = 0.0019872041


# ---- the cases -------------------------------------------------------------------------------

def listed():
    return [
        # the drop-in of the C model's entry point at its own size: 500 atoms, 100 iterations
        dict(name="cmodel-500", kind="cmodel", n=500, iters=100),
        # the per-pair plugin on a stream of the golden vectors' length, their arithmetic
        dict(name="pairs-10k", kind="pairs", n=10000, order=1, bins=256, sep=True, coul=False),
        # the smallest force call: the 1,728-atom cube, host arrays in and out, every default
        dict(name="force-1728-host", kind="force", n=1728, lx=25.5, ly=25.5, lz=25.5, rc=8.5, ntypes=1, coul=False,
             order=1, bins=256, exact=False, sep=False, energy=False, device=False, warp=0, sep0=1.0),
        # a ragged system with energies, virial and partner counts, third-order tables
        dict(name="force-31007-energy", kind="force", n=31007, lx=61.3, ly=72.9, lz=69.4, rc=10.0, ntypes=3, coul=True,
             order=3, bins=128, exact=False, sep=False, energy=True, device=False, warp=0, sep0=1.0),
        # the headline system in the reference's own datapath, host arrays, default tile
        dict(name="force-92k-host", kind="force", n=92224, lx=108.86, ly=108.86, lz=77.76, rc=12.0, ntypes=4, coul=True,
             order=1, bins=1024, exact=False, sep=False, energy=False, device=False, warp=0, sep0=1.0),
        # the same system at 1e-5 force error (exact difference, second order), device arrays, pinned tile
        dict(name="force-92k-device", kind="force", n=92224, lx=108.86, ly=108.86, lz=77.76, rc=12.0, ntypes=4, coul=True,
             order=2, bins=512, exact=True, sep=False, energy=False, device=True, warp=1, sep0=1.0),
        # the large single system: 16 types, device arrays
        dict(name="force-1m-device", kind="force", n=1048576, lx=224.0, ly=224.0, lz=224.0, rc=10.0, ntypes=16, coul=True,
             order=2, bins=512, exact=True, sep=False, energy=False, device=True, warp=1, sep0=1.0),
        # small dynamics with energies every step: liquid argon, 20 steps, then a trajectory frame
        dict(name="md-argon-1728", kind="md", n=1728, lx=36.0, ly=36.0, lz=36.0, rc=8.5, order=1, bins=256, exact=False,
             energy=True, warp=0, pme=0, steps=20),
        # a molecular topology: bonds, angles and dihedrals on 23,558 beads (the DHFR set's size)
        dict(name="md-chains-23558", kind="chains", n=23558, rc=9.0, order=1, bins=512, energy=False, warp=0, steps=10),
        # dynamics with full electrostatics on the headline box: smooth PME, pinned tile
        dict(name="md-pme-92k", kind="md", n=92224, lx=108.86, ly=108.86, lz=77.76, rc=12.0, order=2, bins=512, exact=True,
             energy=False, warp=1, pme=4, steps=10),
        # an ensemble: 64 replicas of uneven size, one force evaluation of all from host arrays
        dict(name="batch-force-64", kind="batch", nrep=64, lo=500, hi=20000, rc=10.0, order=1, bins=512, warp=0, steps=0),
        # the large ensemble: 512 replicas of liquid argon, 25 steps, then every replica's frame
        dict(name="batch-step-512", kind="batch", nrep=512, lo=500, hi=20000, rc=10.0, order=1, bins=512, warp=1, steps=25),
    ]


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, n, rc, density):
    """Edges of a box of n particles at `density`, of uneven shape, each at least 3 cutoffs."""
    L = (n / density) ** (1.0 / 3.0)
    while True:
        a, b = rng.uniform(0.85, 1.2), rng.uniform(0.85, 1.2)
        e = [L * a, L * b, L / (a * b)]
        if min(e) > 3.0 * rc + 0.02:
            return [round(v, 2) for v in e]
        if L < 3.3 * rc:
            return [round(max(L, 3.0 * rc + 0.05), 2)] * 3


def draw(rng):
    kind = rng.choice(["force", "force", "force", "md", "md", "chains", "batch", "pairs", "cmodel"])
    if kind == "cmodel":
        return dict(kind="cmodel", n=_logu(rng, 100, 800), iters=_logu(rng, 20, 120))
    if kind == "pairs":
        return dict(kind="pairs", n=_logu(rng, 1000, 300000), order=rng.choice([0, 1, 2, 3]), bins=rng.choice([256, 512]),
                    sep=rng.random() < 0.5, coul=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind="batch", nrep=_logu(rng, 8, 200), lo=500, hi=rng.choice([4000, 20000]), rc=10.0, order=rng.choice([1, 2]),
                    bins=rng.choice([256, 512]), warp=rng.choice([0, 1]), steps=rng.choice([0, 0, 5, 12]))
    if kind == "chains":
        return dict(kind="chains", n=_logu(rng, 3000, 60000), rc=9.0, order=rng.choice([1, 2]), bins=512,
                    energy=rng.random() < 0.3, warp=rng.choice([0, 1]), steps=rng.randint(2, 12))
    if kind == "md":
        pme = rng.choice([0, 4, 6])
        rc = round(rng.uniform(8.0, 12.0), 1)
        n = _logu(rng, max(4000, int(0.11 * (3.0 * rc) ** 3)) if pme else 1500, 100000)
        dens = 0.1 if pme else 1728 / 36.0 ** 3
        if not pme:
            rc = min(rc, round((n / dens) ** (1 / 3) / 3.05, 1))
        e = _box(rng, n, rc, dens)
        return dict(kind="md", n=n, lx=e[0], ly=e[1], lz=e[2], rc=rc, order=rng.choice([1, 2]), bins=rng.choice([256, 512]),
                    exact=rng.random() < 0.5, energy=rng.random() < 0.4, warp=rng.choice([0, 1]), pme=pme, steps=rng.randint(2, 15))
    rc = round(rng.uniform(8.0, 12.5), 1)
    n = _logu(rng, max(1700, int(0.105 * (3.0 * rc + 0.1) ** 3)), 1000000)
    e = _box(rng, n, rc, 0.1)
    exact = rng.random() < 0.5
    return dict(kind="force", n=n, lx=e[0], ly=e[1], lz=e[2], rc=rc, ntypes=rng.choice([1, 2, 4, 16]), coul=rng.random() < 0.8,
                order=rng.choice([0, 1, 1, 2, 2, 3]), bins=rng.choice([128, 256, 512, 1024]), exact=exact,
                sep=not exact and rng.random() < 0.2, energy=rng.random() < 0.3, device=rng.random() < 0.5,
                warp=rng.choice([0, 0, 1, 2]), sep0=1.0)


# ---- inputs ----------------------------------------------------------------------------------

def _lattice(n, box, rng, sep=None, jitter=None):
    """(n, 3) float32 positions in [0, box): random sites of a lattice of at least n, each moved by
    up to `jitter` A per axis (or as far as keeps every pair `sep` apart along its axis)."""
    box = np.asarray(box, np.float64)
    a = (box.prod() / n) ** (1.0 / 3.0)
    k = np.maximum(1, np.floor(box / a).astype(int))
    while k.prod() < n:
        k[np.argmax(box / k)] += 1
    step = box / k
    j = np.maximum(0.0, (step - sep) / 2) if sep is not None else np.full(3, jitter)
    site = rng.permutation(int(k.prod()))[:n]
    ijk = np.stack([site // (k[1] * k[2]), (site // k[2]) % k[1], site % k[2]], 1)
    pos = (ijk + 0.5) * step + rng.uniform(-1.0, 1.0, (n, 3)) * j
    out = pos.astype(np.float32)
    L = box.astype(np.float32)
    return np.clip(out, 0.0, np.nextafter(L, np.float32(0)))


def _maxwell(mass, temp, rng):
    v = rng.standard_normal((len(mass), 3)) * np.sqrt(KB * temp * AMU / mass)[:, None]
    return (v - (mass[:, None] * v).sum(0) / mass.sum()).astype(np.float32)


def _box32(case):
    return tuple(float(np.float32(case[k])) for k in ("lx", "ly", "lz"))


def _charges(n, rng, amp=0.42):
    q = np.full(n, amp)
    q[: n // 2] = -amp
    if n % 2:
        q[-1] = 0.0
    rng.shuffle(q)
    return q.astype(np.float32)


def _chains(n, rng, length=30, bond=1.53, angle=math.radians(111.0)):
    """Zig-zag chains (trans) laid side by side: positions, box, terms.  The last one is shorter."""
    rise, side = bond * math.sin(angle / 2), bond * math.cos(angle / 2)
    nch = -(-n // length)
    layers = max(1, round((nch * 16.0 * (length * rise + 2.0)) ** (1 / 3) / (length * rise + 2.0)))
    k = math.ceil(math.sqrt(nch / layers))
    box = (float(np.float32(k * 4.0)), float(np.float32(k * 4.0)), float(np.float32(layers * (length * rise + 2.0))))
    c, s = np.divmod(np.arange(n), length)
    lay, r = np.divmod(c, k * k)
    pos = np.stack([(r // k) * 4.0 + 1.0 + side * (s % 2), (r % k) * 4.0 + 1.0, lay * (length * rise + 2.0) + 1.0 + s * rise], 1)
    pos += rng.uniform(-0.03, 0.03, pos.shape)
    idx = np.arange(n)
    run = lambda w: idx[: n - w + 1][(idx[: n - w + 1] % length) <= length - w]  # noqa: E731
    b, a, d = run(2), run(3), run(4)
    terms = {"bonds": (np.stack([b, b + 1], 1), np.tile([300.0, bond], (len(b), 1))),
             "angles": (np.stack([a, a + 1, a + 2], 1), np.tile([60.0, angle, 0.0, 0.0], (len(a), 1))),
             "dihedrals": (np.stack([d, d + 1, d + 2, d + 3], 1), np.tile([1.4, 3.0, 0.0], (len(d), 1)))}
    L = np.asarray(box, np.float32)
    return np.clip(pos.astype(np.float32), 0.0, np.nextafter(L, np.float32(0))), box, terms


def _system(case, seed):
    """Everything the case's inputs are, as plain numpy and numbers (also what exact() starts from)."""
    rng = np.random.default_rng([int(seed), 20191117])
    k, n = case["kind"], case.get("n")
    if k == "cmodel":
        pos = _lattice(-(-n // 2), (24.0, 24.0, 24.0), rng, jitter=0.2)      # dimers, 0.36 to 0.46 A
        u = rng.standard_normal((n // 2, 3))
        u *= rng.uniform(0.36, 0.46, (n // 2, 1)) / np.linalg.norm(u, axis=1, keepdims=True)
        pos = np.concatenate([pos, np.clip(pos[: n // 2] + u, 0.0, 23.999)]).astype(np.float32)
        return dict(pos=pos, vel=np.zeros_like(pos))
    if k == "pairs":
        box = (64.0, 64.0, 64.0)
        ref = np.zeros((n, 4), np.float32)
        nbr = np.zeros((n, 4), np.float32)
        ref[:, :3] = rng.random((n, 3)) * 64.0
        r = 1.0 + 11.0 * rng.random(n) ** 0.5                    # some beyond the cutoff of 10
        u = rng.standard_normal((n, 3))
        nbr[:, :3] = np.mod(ref[:, :3] + u / np.linalg.norm(u, axis=1, keepdims=True) * r[:, None], 64.0)
        nbr[:, :3] = np.clip(nbr[:, :3], 0, np.nextafter(np.float32(64), np.float32(0)))
        ref[:, 3], nbr[:, 3] = _charges(n, rng), _charges(n, rng)
        return dict(box=box, ref=ref, nbr=nbr, tr=rng.integers(0, 4, n).astype(np.int32),
                    tn=rng.integers(0, 4, n).astype(np.int32), sigma=[2.0, 2.6, 3.2, 3.8], eps=[0.02, 0.08, 0.14, 0.20],
                    mass=[12.011, 14.007, 15.999, 39.95], ke=KE if case["coul"] else 0.0, rc=10.0)
    if k == "batch":
        # which sizes is part of the case; steps run on liquid argon, evaluations on the dense charged replicas
        u = np.random.default_rng(case["nrep"]).uniform(math.log(case["lo"]), math.log(case["hi"]), case["nrep"])
        sizes = [int(v) for v in np.exp(u).round()]
        md = case["steps"] > 0
        boxes = [(float(np.float32((v / (1728 / 36.0 ** 3 if md else 0.1)) ** (1 / 3))),) * 3 for v in sizes]
        pos = np.concatenate([_lattice(v, b, rng, jitter=0.25) for v, b in zip(sizes, boxes)])
        q = None if md else np.concatenate([_charges(v, rng) for v in sizes])
        t = np.zeros(len(pos), np.int32)
        return dict(sizes=sizes, boxes=boxes, pos=pos, q=q, type=t, sigma=[3.4], eps=[0.238], mass=[39.95], ke=0.0 if md else KE,
                    rc=case["rc"], min_log2=0, vel=_maxwell(np.full(len(pos), 39.95), 120.0, rng))
    if k == "chains":
        pos, box, terms = _chains(n, rng)
        return dict(pos=pos, box=box, q=None, type=np.zeros(n, np.int32), sigma=[1.0], eps=[0.05], mass=[14.0], ke=0.0,
                    rc=case["rc"], min_log2=-2, vel=_maxwell(np.full(n, 14.0), 300.0, rng), terms=terms)
    box = _box32(case)
    if k == "md":
        if case["pme"]:     # a molten salt of four kinds
            sig, eps, mass = [1.8, 1.9, 2.0, 2.1], [0.05, 0.08, 0.11, 0.14], [12.011, 14.007, 15.999, 39.95]
            t = rng.integers(0, 4, n).astype(np.int32)
            return dict(pos=_lattice(n, box, rng, jitter=0.05), box=box, q=_charges(n, rng), type=t, sigma=sig, eps=eps, mass=mass,
                        ke=KE, rc=case["rc"], min_log2=0, vel=_maxwell(np.asarray(mass)[t], 300.0, rng))
        return dict(pos=_lattice(n, box, rng, jitter=0.05), box=box, q=None, type=np.zeros(n, np.int32), sigma=[3.4], eps=[0.238],
                    mass=[39.95], ke=0.0, rc=case["rc"], min_log2=-2, vel=_maxwell(np.full(n, 39.95), 120.0, rng))
    T = case["ntypes"]
    sig = [3.4] if T == 1 else [float(v) for v in np.linspace(2.0 if T <= 4 else 2.5, 3.8, T)]
    eps = [0.238] if T == 1 else [float(v) for v in np.linspace(0.02 if T <= 4 else 0.05, 0.2, T)]
    q = _charges(n, rng) if case["coul"] else None
    return dict(pos=_lattice(n, box, rng, sep=case["sep0"]), box=box, q=q, type=rng.integers(0, T, n).astype(np.int32),
                sigma=sig, eps=eps, mass=[20.0 + k for k in range(T)], ke=KE if case["coul"] else 0.0, rc=case["rc"], min_log2=0)


def _pme(case):
    """Splitting and grid: erfc(beta rc) = 1e-5, about 1 A, sizes that factor into 2, 3, 5 and 7."""
    grid = []
    for a in ("lx", "ly", "lz"):
        k = max(16, math.ceil(case[a]))
        while 210 ** 12 % k:
            k += 1
        grid.append(k)
    return 3.1234 / case["rc"], grid


def _params(case, s):
    order = case["order"]
    kw = dict(cutoff=s["rc"], ntypes=len(s["sigma"]), sigma=s["sigma"], epsilon=s["eps"], mass=s["mass"], coulomb_k=s["ke"],
              table_order=order or 1, table_bins=case["bins"], table_min_log2=s.get("min_log2", -2), dt_fs=2.0,
              eval=m.EVAL_TABLE if order else m.EVAL_DIRECT,
              arith=m.ARITH_SEPARATE if case.get("sep") else m.ARITH_FMA,
              flags=(m.FLAG_ENERGY if case.get("energy") else 0) | (m.FLAG_EXACT_DIFF if case.get("exact") else 0))
    if "box" in s:
        kw["box"] = s["box"]
    return m.default_params(**kw)


class State:
    pass


def prepare(case, seed):
    s = _system(case, seed)
    st = State()
    st.case, st.s = case, s
    k = case["kind"]
    if k == "cmodel":
        return st
    if k == "batch":
        st.b = m.Batch(_params(case, s), list(zip(s["sizes"], s["boxes"])))
        st.args = [np.ascontiguousarray(s["pos"][:, d]) for d in range(3)]
        if case["warp"]:
            st.b.set_tile(1, case["warp"], 1)
        if case["steps"]:
            st.b.set_state(*st.args, s["vel"], s["q"], s["type"])
        return st
    st.ctx = m.Context(_params(case, s))
    if k == "pairs":
        return st
    if case["warp"]:
        st.ctx.set_tile(1, case["warp"], 1)
    st.args = [np.ascontiguousarray(s["pos"][:, d]) for d in range(3)]
    if k in ("md", "chains"):
        if case.get("pme"):
            beta, grid = _pme(case)
            st.ctx.set_pme(True, beta=beta, grid=grid, order=case["pme"])
        if k == "chains":
            st.ctx.set_bonded(**s["terms"])
        st.ctx.set_state(*st.args, s["vel"], s["q"], s["type"])
        return st
    if case["device"]:
        dev = lambda a: None if a is None else torch.as_tensor(a, device="cuda")  # noqa: E731
        st.dev = [dev(a) for a in st.args] + [dev(s["q"]), dev(s["type"])]
        st.out = [torch.empty(case["n"], device="cuda") for _ in range(3)]
        st.cnt = torch.empty(case["n"], dtype=torch.int32, device="cuda") if case["energy"] else None
    return st


def _energies(case, r, kinetic):
    out = {"pairs": int(r["pairs"])}
    if case.get("energy"):
        out["e_lj"], out["virial"] = float(r["e_lj"]), float(r["virial"])
        if kinetic:
            out["kinetic"] = float(r["kinetic"])
    return out


def run(st):
    case, s = st.case, st.s
    k = case["kind"]
    if k == "cmodel":
        pos, vel, energy, _ = m.cmodel_run(s["pos"], s["vel"], case["iters"])
        return {"pos": pos, "vel": vel, "energy": energy}
    if k == "pairs":
        out, aux = st.ctx.pair_eval(s["ref"], s["nbr"], s["tr"], s["tn"])
        return {"force": out, "aux": aux}
    if k == "batch":
        if case["steps"] == 0:
            F, r, _ = st.b.force(*st.args, s["q"], s["type"])
            return {"force": F, "pairs": int(r["pairs"])}
        r = st.b.step(case["steps"])
        x, v, F = st.b.state()
        return {"pos": x, "vel": v, "force": F, "pairs": int(r["pairs"])}
    if k in ("md", "chains"):
        r = st.ctx.step(case["steps"])
        x, v, F = st.ctx.state()
        return {"pos": x, "vel": v, "force": F, **_energies(case, r, True)}
    if case["device"]:
        stats = m.Stats()
        ptr = [None if t is None else t.data_ptr() for t in st.dev + st.out + [st.cnt]]
        status = m.lib().mdrl_force_eval_device(st.ctx._h, case["n"], *ptr, C.byref(stats))
        if status != 0:
            raise m.MdrlError(status, m.lib().mdrl_last_error().decode())
        out = {"fx": st.out[0], "fy": st.out[1], "fz": st.out[2], **_energies(case, stats.as_dict(), False)}
        if case["energy"]:
            out["counts"] = st.cnt
        return out
    F, r, cnt = st.ctx.force(*st.args, s["q"], s["type"], counts=case["energy"])
    out = {"force": F, **_energies(case, r, False)}
    if case["energy"]:
        out["counts"] = cnt
    return out


def work(case):
    """Inputs read once and results written once; flops: 28 of an in-cutoff pair (difference and
    square 8, tables 6, combination and components 8, accumulation 6) on every pair once."""
    k = case["kind"]
    if k == "cmodel":
        n = case["n"]
        return {"bytes": 48.0 * n, "flops": 9.0 * n * (n - 1) * case["iters"]}
    if k == "pairs":
        return {"bytes": (32 + 8 + 16 + 8) * case["n"], "flops": 22.0 * case["n"]}
    if k == "batch":
        n = case["nrep"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        pairs = n * (0.037 if case["steps"] else 0.1) * 4.0 / 3.0 * math.pi * case["rc"] ** 3 / 2
        steps = max(1, case["steps"])
        return {"bytes": n * 4.0 * (8 if case["steps"] == 0 else 2 * 6 + 1 + 3), "flops": 28.0 * pairs * steps}
    n, rc = case["n"], case["rc"]
    steps = case.get("steps", 1)
    vol = case["lx"] * case["ly"] * case["lz"] if "lx" in case else n * 22.0
    pairs = n * (n / vol) * 4.0 / 3.0 * math.pi * rc ** 3 / 2
    flops = 28.0 * pairs * steps
    if case.get("pme"):
        g = _pme(case)[1]
        pts = g[0] * g[1] * g[2]
        flops += steps * (n * case["pme"] ** 3 * 8.0 + 5.0 * pts * math.log2(pts))
    if k == "chains":
        flops += steps * 3.0 * 100.0 * n
    return {"bytes": n * 4.0 * (8 if k == "force" else 2 * 6 + 2 + 3), "flops": flops}


# ---- the same in 64 bits, from plain torch ------------------------------------------------------

def _pair_terms(r2, A, B, qq, beta):
    """fscal (force = fscal d) and LJ energy of pairs at r2: 12A r^-14 - 6B r^-8 + qq (...)."""
    i2 = 1.0 / r2
    i6 = i2 * i2 * i2
    fs = (12.0 * A * i6 - 6.0 * B) * i6 * i2
    if qq is not None:
        r = torch.sqrt(r2)
        if beta:
            fs = fs + qq * (torch.erfc(beta * r) / r + 2.0 * beta / math.sqrt(math.pi) * torch.exp(-(beta * r) ** 2)) * i2
        else:
            fs = fs + qq * i2 / r
    return fs, (A * i6 - B) * i6


def _lj(s, dev):
    sg, ep = torch.tensor(s["sigma"], dtype=torch.float64, device=dev), torch.tensor(s["eps"], dtype=torch.float64, device=dev)
    sig, e = 0.5 * (sg[:, None] + sg[None]), torch.sqrt(ep[:, None] * ep[None])
    return 4 * e * sig ** 12, 4 * e * sig ** 6


def _forces64(pos, box, s, q, t, beta=0.0):
    """(forces, LJ energy, virial, partner counts) of every periodic pair within the cutoff."""
    dev, n = pos.device, len(pos)
    L = torch.tensor(box, dtype=torch.float64, device=dev)
    rc2 = float(np.float32(s["rc"])) ** 2
    TA, TB = _lj(s, dev)
    one = TA.numel() == 1
    F = torch.zeros(n, 3, dtype=torch.float64, device=dev)
    e = torch.zeros((), dtype=torch.float64, device=dev)
    w = torch.zeros((), dtype=torch.float64, device=dev)
    cnt = torch.zeros(n, dtype=torch.int32, device=dev)

    def block(i, j, shift):
        """i (C, I), j (C, J) indices (-1: none); shift (C, 3) is added to the j's."""
        nonlocal e, w
        pi, pj = pos[i.clamp(min=0)], pos[j.clamp(min=0)] + shift[:, None]
        d = pi[:, :, None] - pj[:, None]
        r2 = (d * d).sum(-1)
        ok = (r2 > 0) & (r2 <= rc2) & (i >= 0)[:, :, None] & (j >= 0)[:, None]
        r2 = torch.where(ok, r2, torch.ones_like(r2))
        if one:
            A, B = TA[0, 0], TB[0, 0]
        else:
            ti, tj = t[i.clamp(min=0)][:, :, None], t[j.clamp(min=0)][:, None]
            A, B = TA[ti, tj], TB[ti, tj]
        qq = None if q is None or not s["ke"] else s["ke"] * q[i.clamp(min=0)][:, :, None] * q[j.clamp(min=0)][:, None]
        fs, el = _pair_terms(r2, A, B, qq, beta)
        zero = torch.zeros((), dtype=torch.float64, device=dev)
        fs = torch.where(ok, fs, zero)
        e = e + 0.5 * torch.where(ok, el, zero).sum()
        w = w + 0.5 * (fs * r2).sum()
        f = (fs[..., None] * d).sum(2)
        at = i >= 0
        F.index_add_(0, i[at], f[at])
        cnt.index_add_(0, i[at], ok.sum(2, dtype=torch.int32)[at])

    nc = [int(b // s["rc"]) for b in box]
    if min(nc) < 3:
        everyone = torch.arange(n, device=dev)[None]
        for a in range(-1, 2):
            for b in range(-1, 2):
                for c in range(-1, 2):
                    block(everyone, everyone, torch.tensor([[a, b, c]], dtype=torch.float64, device=dev) * L)
        return F, e, w, cnt
    ncd = torch.tensor(nc, device=dev)
    c3 = torch.minimum((pos / (L / ncd)).floor().long().clamp(min=0), ncd - 1)
    cell = (c3[:, 0] * nc[1] + c3[:, 1]) * nc[2] + c3[:, 2]
    tot = nc[0] * nc[1] * nc[2]
    order = torch.argsort(cell)
    count = torch.bincount(cell, minlength=tot)
    M = int(count.max())
    rank = torch.arange(n, device=dev) - torch.cumsum(count, 0)[cell[order]] + count[cell[order]]
    slots = torch.full((tot, M), -1, dtype=torch.long, device=dev)
    slots[cell[order], rank] = order
    ids = torch.arange(tot, device=dev)
    h = torch.stack([ids // (nc[1] * nc[2]), (ids // nc[2]) % nc[1], ids % nc[2]], 1)
    per = max(1, int(3e7) // (M * M))
    for dx in range(-1, 2):
        for dy in range(-1, 2):
            for dz in range(-1, 2):
                to = h + torch.tensor([dx, dy, dz], device=dev)
                img = torch.div(to, ncd, rounding_mode="floor")
                to = to - img * ncd
                nb = (to[:, 0] * nc[1] + to[:, 1]) * nc[2] + to[:, 2]
                for a in range(0, tot, per):
                    block(slots[a:a + per], slots[nb[a:a + per]], img[a:a + per].double() * L)
    return F, e, w, cnt


def _recip64(pos, box, q, ke, beta, grid, order):
    """Reciprocal-space forces of smooth PME (cardinal B-splines), by differentiating the energy."""
    dev = pos.device
    x = pos.clone().requires_grad_(True)
    L = torch.tensor(box, dtype=torch.float64, device=dev)
    K = torch.tensor(grid, device=dev)
    u = x / L * K
    base = u.detach().floor()
    th = []
    for a in range(3):
        wt = [u[:, a] - base[:, a] + j for j in range(order)]        # arguments of M_order
        v = [1.0 - (z - 1.0).abs() if j < 2 else torch.zeros_like(z) for j, z in enumerate(wt)]
        for o in range(3, order + 1):
            v = [(wt[j] * v[j] + ((o - wt[j]) * v[j - 1] if j else 0.0)) / (o - 1) for j in range(order)]
        th.append(torch.stack(v, 1))
    k = torch.arange(order, device=dev)
    idx = [torch.remainder(base[:, a].long()[:, None] - k, grid[a]) for a in range(3)]
    flat = (idx[0][:, :, None, None] * grid[1] + idx[1][:, None, :, None]) * grid[2] + idx[2][:, None, None, :]
    val = q[:, None, None, None] * th[0][:, :, None, None] * th[1][:, None, :, None] * th[2][:, None, None, :]
    Q = torch.zeros(grid[0] * grid[1] * grid[2], dtype=torch.float64, device=dev).index_add(0, flat.reshape(-1), val.reshape(-1))
    X = torch.fft.fftn(Q.reshape(grid))
    knots = {4: [1 / 6, 4 / 6, 1 / 6], 6: [1 / 120, 26 / 120, 66 / 120, 26 / 120, 1 / 120]}[order]   # M_p at 1 .. p-1
    m2 = torch.zeros((), dtype=torch.float64, device=dev)
    b2 = torch.ones((), dtype=torch.float64, device=dev)
    for a in range(3):
        mm = torch.fft.fftfreq(grid[a], 1.0 / grid[a], dtype=torch.float64, device=dev)
        ph = 2.0 * math.pi * mm / grid[a]
        re = sum(c * torch.cos(ph * j) for j, c in enumerate(knots))
        im = sum(c * torch.sin(ph * j) for j, c in enumerate(knots))
        shape = [1, 1, 1]
        shape[a] = grid[a]
        b2 = b2 * (1.0 / (re * re + im * im)).reshape(shape)
        m2 = m2 + ((mm / box[a]) ** 2).reshape(shape)
    G = torch.where(m2 > 0, ke * torch.exp(-math.pi ** 2 * m2 / beta ** 2) / (math.pi * box[0] * box[1] * box[2] * m2.clamp(min=1e-30)) * b2,
                    torch.zeros((), dtype=torch.float64, device=dev))
    E = 0.5 * (G * (X.real ** 2 + X.imag ** 2)).sum()
    return -torch.autograd.grad(E, x)[0]


def _bonded64(pos, box, terms):
    """Forces of the bonded terms, by differentiating their energy."""
    dev = pos.device
    L = torch.tensor(box, dtype=torch.float64, device=dev)
    x = pos.clone().requires_grad_(True)
    t = {k: (torch.as_tensor(a, device=dev), torch.as_tensor(p, dtype=torch.float64, device=dev)) for k, (a, p) in terms.items()}
    vec = lambda a, b: (x[a] - x[b]) - torch.round((x[a] - x[b]).detach() / L) * L  # noqa: E731
    (b, bp), (a, ap), (d, dp) = t["bonds"], t["angles"], t["dihedrals"]
    E = (bp[:, 0] * (vec(b[:, 0], b[:, 1]).norm(dim=1) - bp[:, 1]) ** 2).sum()
    if len(a):
        u, v = vec(a[:, 0], a[:, 1]), vec(a[:, 2], a[:, 1])
        th = torch.atan2(torch.linalg.cross(u, v).norm(dim=1), (u * v).sum(1))
        E = E + (ap[:, 0] * (th - ap[:, 1]) ** 2).sum()
    if len(d):
        f, g, h = vec(d[:, 0], d[:, 1]), vec(d[:, 1], d[:, 2]), vec(d[:, 3], d[:, 2])
        A, B = torch.linalg.cross(f, g), torch.linalg.cross(h, g)
        phi = torch.atan2((torch.linalg.cross(B, A) * g).sum(1) / g.norm(dim=1), (A * B).sum(1))
        E = E + (dp[:, 0] * (1.0 + torch.cos(dp[:, 1] * phi + dp[:, 2]))).sum()
    return -torch.autograd.grad(E, x)[0]


def _md64(pos, vel, box, s, q, t, steps, dt, extra, beta=0.0):
    """Velocity Verlet; returns positions, velocities, forces and the last evaluation's sums."""
    dev = pos.device
    L = torch.tensor(box, dtype=torch.float64, device=dev)
    mass = torch.tensor(s["mass"], dtype=torch.float64, device=dev)[t][:, None]

    def force(x):
        F, e, w, c = _forces64(x, box, s, q, t, beta)
        return F + extra(x) if extra else F, e, w, c

    F = force(pos)[0]
    for _ in range(steps):
        vel = vel + F * (0.5 * dt * AMU) / mass
        pos = torch.remainder(pos + vel * dt, L)
        F, e, w, c = force(pos)
        vel = vel + F * (0.5 * dt * AMU) / mass
    kin = 0.5 * (mass * vel * vel).sum() / AMU
    return pos, vel, F, e, w, kin


def exact(case, seed):
    s = _system(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    up = lambda a, dt=torch.float64: None if a is None else torch.as_tensor(a, device=dev).to(dt)  # noqa: E731
    k = case["kind"]
    if k == "cmodel":
        pos, vel = up(s["pos"]), up(s["vel"])
        eps, sig = 1.995996 * 1.995996, 0.1675 * 2
        mass, dt, energy = 39.95 / 6.022e23 / 1000, 2e-15, []
        for _ in range(case["iters"]):
            d = pos[:, None] - pos[None]
            d = d - 24.0 * torch.round(d / 24.0)
            r2 = (d * d).sum(-1)
            ok = (r2 > 0) & (r2 <= 64.0)
            i2 = torch.where(ok, 1.0 / torch.where(ok, r2, torch.ones_like(r2)), torch.zeros_like(r2))
            f = 48 * eps * sig ** 12 * i2 ** 7 - 24 * eps * sig ** 6 * i2 ** 4
            energy.append([0.5 * (4 * eps * sig ** 12 * i2 ** 6 - 4 * eps * sig ** 6 * i2 ** 3).sum(), None])
            vel = vel + (f[..., None] * d).sum(1) / mass * dt
            energy[-1][1] = 0.5 * mass * (vel * vel).sum()
            pos = torch.remainder(pos + vel * dt, 24.0)
        return {"pos": pos, "vel": vel, "energy": torch.tensor([[float(a), float(b)] for a, b in energy], dtype=torch.float64)}
    if k == "pairs":
        a, b = up(s["ref"]), up(s["nbr"])
        L = 64.0
        d = a[:, :3] - b[:, :3]
        d = d - L * torch.round(d / L)
        r2 = (d * d).sum(1)
        TA, TB = _lj(s, dev)
        tr, tn = up(s["tr"], torch.long), up(s["tn"], torch.long)
        ok = (r2 > 0) & (r2 <= 100.0)
        fs, _ = _pair_terms(torch.where(ok, r2, torch.ones_like(r2)), TA[tr, tn], TB[tr, tn], s["ke"] * a[:, 3] * b[:, 3] if s["ke"] else None, 0.0)
        fs = torch.where(ok, fs, torch.zeros_like(fs))
        return {"force": torch.cat([fs[:, None] * d, torch.zeros_like(fs)[:, None]], 1), "aux": torch.stack([r2, fs], 1)}
    t, q = up(s["type"], torch.long), up(s["q"])
    if k == "batch":
        if case["nrep"] * case["steps"] > 250:
            return None                       # minutes of small kernels
        out, at = [], 0
        for n, box in zip(s["sizes"], s["boxes"]):
            sl = slice(at, at + n)
            at += n
            x, v = up(s["pos"][sl]), up(s["vel"][sl])
            if case["steps"]:
                out.append(_md64(x, v, box, s, None, t[sl], case["steps"], 2.0, None)[:3])
            else:
                out.append((_forces64(x, box, s, q[sl], t[sl])[0],))
        cat = [torch.cat([o[j] for o in out]) for j in range(len(out[0]))]
        return {"force": cat[0], "pairs": None} if not case["steps"] else {"pos": cat[0], "vel": cat[1], "force": cat[2], "pairs": None}
    pos = up(s["pos"])
    if k in ("md", "chains"):
        beta, extra = 0.0, None
        if case.get("pme"):
            beta, grid = _pme(case)
            extra = lambda x: _recip64(x, s["box"], q, s["ke"], beta, grid, case["pme"])  # noqa: E731
        if k == "chains":
            extra = lambda x: _bonded64(x, s["box"], s["terms"])  # noqa: E731
        x, v, F, e, w, kin = _md64(pos, up(s["vel"]), s["box"], s, q, t, case["steps"], 2.0, extra, beta)
        out = {"pos": x, "vel": v, "force": F, "pairs": None}
        if case["energy"]:
            out |= {"e_lj": e, "kinetic": kin, "virial": None if case.get("pme") else w}
        return out
    F, e, w, cnt = _forces64(pos, s["box"], s, q, t)
    out = {"pairs": None}
    out |= {"fx": F[:, 0], "fy": F[:, 1], "fz": F[:, 2]} if case["device"] else {"force": F}
    if case["energy"]:
        out |= {"e_lj": e, "virial": w, "counts": None}
    return out
