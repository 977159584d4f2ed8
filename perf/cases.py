"""The work whose speed is tracked: what a program that uses this package has it do, through the public entry points,
at the sizes of the package's own workloads.

Kinds of cases
  debris  World: compound debris scenes with host-owned state. A pass writes the bodies (pinned host arrays), takes
          `steps` steps and reads the bodies back, as a host engine does that keeps the state (a roll-out of 1 to 8
          steps from a given state, the range of a served request).
  bricks  the same on the 5-storey frame with loose single bricks: the smallest world.
  pool    ScenePool: resident worlds of 1,000 to 100,000 bodies, one tick of the request loop: the state of the
          worlds that have a request is written, they take one step together, their state is read.
  solve   World.structure_solve: external loads and zero potentials written, the load path solved, potentials read.
  tick    the solve tick of the request loop: loads added to some structures of the lattice, at most 128 sweeps.
  frame   one frame of a standing structure with resting debris that has been woken, damage on, in the frame order:
          step, rebuild, connectivity, loads, load-path frame, the pieces' fields, connectivity.
  boxes   BoxWorld: piles of boxes that have landed (no sleep); a pass takes `steps` steps and reads the state. A
          world without sleep stays busy, so a pass may go on from the last one's state.
  sat     the batched narrow phase on host arrays (boxes, or convex cells of the hull library).

Only potentials of a fully bearing structure have a value in exact(): they solve a linear system by sweeps that are
plain arithmetic. Trajectories do not: which pairs touch, the order of impulses and which clamp holds are decisions
on rounded values that 64 bits decide otherwise after a few steps, and a SAT's axis and clipped points likewise.
"""
from __future__ import annotations

import math
from types import SimpleNamespace as State

import numpy as np
import torch

import shatterforge_b200 as sf
from shatterforge_b200 import boxes as X
from shatterforge_b200 import hulls
from shatterforge_b200 import scenes as S
from shatterforge_b200 import serving

DT = 1.0 / 60.0
ITERATIONS = 8


def listed():
    return [
        # the smallest world there is: one step of 1,024 bricks landing beside the frame; all latency
        dict(name="bricks_1024_step", kind="bricks", bodies=1024, age=85, steps=1, removed=True),
        # the mix's median scene, a request of 8 steps while it lands
        dict(name="debris_one_scene", kind="debris", scenes=1, lo=3623, hi=3623, p_geom=0.3, spacing=2.5, age=60,
             steps=8, reduce=0, warm=0),
        # the 256-scene mix in free fall (few contacts: the broadphase and the pose passes)
        dict(name="debris_mix_fall", kind="debris", scenes=256, lo=500, hi=20000, p_geom=0.3, spacing=2.5, age=5,
             steps=4, reduce=0, warm=0),
        # the same at its contact peak (the manifolds, the colouring and the solve)
        dict(name="debris_mix_peak", kind="debris", scenes=256, lo=500, hi=20000, p_geom=0.3, spacing=2.5, age=110,
             steps=4, reduce=0, warm=0),
        # large compound bodies (50 bricks on average, up to 256) with contact reduction and warm start
        dict(name="debris_large_bodies", kind="debris", scenes=1, lo=2000, hi=2000, p_geom=0.02, spacing=5.0,
             age=90, steps=2, reduce=1, warm=1),
        # the request loop's step tick on worlds of 1k-100k bodies, half of them with a request
        dict(name="pool_tick", kind="pool", slots=24, lo=1000, hi=100000, age=40),
        # a small building designed to the tolerance the package's workloads use
        dict(name="solve_frame5", kind="solve", structures=0, layout=0, lo=0, hi=0, tol=1e-6, max_sweeps=50000),
        # 37 buildings at once, to the same tolerance
        dict(name="solve_lattice", kind="solve", structures=37, layout=2, lo=1000, hi=40000, tol=1e-6, max_sweeps=60000),
        # a whole frame of the 5-storey building and its debris, damage on
        dict(name="frame_5_storeys", kind="frame", bodies=1024),
        # the throughput pile: one large scene (one cluster)
        dict(name="boxes_pile_20000", kind="boxes", scenes=1, boxes=20000, substeps=12, cells=False, age=90, steps=2),
        # many small piles: one block a scene
        dict(name="boxes_148_piles", kind="boxes", scenes=148, boxes=2000, substeps=12, cells=False, age=90, steps=2),
        # the narrow phase alone, on a caller's arrays
        dict(name="sat_cells", kind="sat", cells=True, pairs=200000),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bricks", "debris", "debris", "debris", "pool", "solve", "tick", "frame", "boxes", "sat"])
    if kind == "bricks":
        return dict(kind=kind, bodies=_log_uniform(rng, 64, 4000), age=rng.randint(60, 120), steps=rng.randint(1, 8),
                    removed=rng.random() < 0.5)
    if kind == "debris":
        n = _log_uniform(rng, 1, 256)
        large = n <= 4 and rng.random() < 0.5
        lo, hi = sorted((_log_uniform(rng, 300, 4000), _log_uniform(rng, 500, 20000)))
        if large:
            lo, hi = sorted((rng.randint(100, 600), rng.randint(100, 600)))
        opt = int(rng.random() < 0.3)
        return dict(kind=kind, scenes=n, lo=lo, hi=hi, p_geom=0.02 if large else 0.3, spacing=5.0 if large else 2.5,
                    age=rng.randint(3, 110), steps=rng.randint(1, 4 if n > 16 else 8), reduce=opt, warm=opt)
    if kind == "pool":
        return dict(kind=kind, slots=rng.randint(2, 24), lo=1000, hi=_log_uniform(rng, 2000, 100000), age=rng.randint(5, 80))
    if kind == "solve":
        if rng.random() < 0.3:
            return dict(kind=kind, structures=0, layout=0, lo=0, hi=0, tol=rng.choice([1e-4, 1e-5, 1e-6]), max_sweeps=50000)
        return dict(kind=kind, structures=_log_uniform(rng, 1, 37), layout=rng.randint(1, 1000), lo=1000,
                    hi=_log_uniform(rng, 3000, 40000), tol=rng.choice([1e-4, 1e-5, 1e-6]), max_sweeps=_log_uniform(rng, 1000, 60000))
    if kind == "tick":
        return dict(kind=kind, structures=37, layout=rng.randint(1, 1000), lo=1000, hi=40000,
                    requests=rng.randint(1, 37), max_sweeps=rng.randint(16, 128))
    if kind == "frame":
        return dict(kind=kind, bodies=_log_uniform(rng, 50, 2000))
    if kind == "boxes":
        n = _log_uniform(rng, 1, 148)
        return dict(kind=kind, scenes=n, boxes=_log_uniform(rng, 20, 20000 if n == 1 else 2000), substeps=rng.choice([4, 12]),
                    cells=rng.random() < 0.2, age=rng.randint(40, 100), steps=rng.randint(1, 2))
    return dict(kind=kind, cells=rng.random() < 0.5, pairs=_log_uniform(rng, 1000, 200000))


# ---------------------------------------------------------------- what a program has in hand before the call
def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=torch.cuda.is_available()).numpy()


def _host_state(n):
    return _pinned((n, 13), torch.float32), _pinned((n,), torch.float32), _pinned((n,), torch.uint8)


def _world_state(w):
    """The world's bodies in pinned host arrays, and a second set to read results into."""
    src, out = _host_state(w.info.n_bodies), _host_state(w.info.n_bodies)
    w.bodies(out=src)
    return src, out


def _debris_scenes(case, seed):
    """Scenes of the debris mix's body counts (log-uniform in lo..hi, the same for every seed), their bodies from the seed."""
    n = case["slots"] if case["kind"] == "pool" else case["scenes"]
    spread = np.random.default_rng(3).uniform(math.log(case["lo"]), math.log(case["hi"]), n)
    counts = [max(1, int(round(c))) for c in np.exp(spread)]
    lib = S.ClusterLibrary(seed ^ 0x2545F491)
    return [S.debris_scene(c, seed * 1000003 + k, lib=lib, p_geom=case.get("p_geom", 0.3), spacing=case.get("spacing", 2.5))
            for k, c in enumerate(counts)]


def _lattice(case):
    """The lattice's buildings stand; what changes from seed to seed is what they carry."""
    return S.structure_lattice(seed=case["layout"], n_struct=case["structures"], lo=case["lo"], hi=case["hi"],
                               total=378000.0 * case["hi"] / 40000.0)


def _unit_quaternions(rng, n):
    q = rng.normal(size=(n, 4))
    return q / np.linalg.norm(q, axis=1, keepdims=True)


def _frame5(seed):
    sc, removed = S.frame5_structure(seed + 1)
    return sc.without_static(removed)


def _loads(n, seed):
    """External loads of up to one brick's weight, on one brick in four."""
    rng = np.random.default_rng(seed)
    return np.where(rng.random(n) < 0.25, rng.uniform(0.0, 300.0, n), 0.0).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    st = State(kind=kind, case=case)
    if kind in ("bricks", "debris"):
        if kind == "bricks":
            sc = S.frame5_debris_scene(seed + 1, n_debris=case["bodies"], removed=case["removed"])
            st.world = sf.World(sc, iterations=ITERATIONS)
        else:
            st.world = sf.World(_debris_scenes(case, seed), iterations=ITERATIONS, pinch_kill=0, reduce=case["reduce"],
                                warm_start=case["warm"])
        st.world.step(DT, case["age"])
        st.src, st.out = _world_state(st.world)
    elif kind == "pool":
        scenes = _debris_scenes(case, seed)
        st.pool = serving.ScenePool([serving.slot_for(s) for s in scenes], iterations=ITERATIONS, pinch_kill=0)
        for k, s in enumerate(scenes):
            st.pool.load(k, s)
        st.pool.step(DT, case["age"])
        st.slots = list(range(0, case["slots"], 2))       # the worlds with a request
        st.src = {}
        for k in st.slots:
            st.src[k] = _host_state(scenes[k].n_bodies)
            for to, got in zip(st.src[k], st.pool.bodies(k)):
                to[...] = got
    elif kind in ("solve", "tick"):
        sc = _lattice(case) if case["structures"] else _frame5(seed)
        st.world = sf.World(sc)
        st.phi0 = np.zeros(sc.n_static, np.float32)
        st.ext = _loads(sc.n_static, seed)
        rng = np.random.default_rng(seed + 1)
        if kind == "tick":
            st.ids = sorted(int(k) for k in rng.choice(case["structures"], case["requests"], replace=False))
            mine = [np.nonzero(sc.static_sid == k)[0] for k in st.ids]
            st.load_brick = np.concatenate([rng.choice(m, 3) for m in mine]).astype(np.uint32)
            st.load_value = rng.uniform(50.0, 500.0, len(st.load_brick)).astype(np.float32)
    elif kind == "frame":
        sc = S.frame5_structure(seed + 1)[0]
        n = case["bodies"]
        sc.body_first, sc.body_brick_xyz, sc.body_brick_mat, sc.body_pose = S.loose_debris(
            n, seed + 101, box_lo=(8.0, 0.5, -6.0), box_hi=(20.0, 3.0, 6.0))
        st.world = w = sf.World(sc.contiguous(), iterations=ITERATIONS, detach_bodies=256, detach_bricks=4096, damage=1)
        st.ids = [0]
        w.structure_warm(0)
        st.frame = 0
        for _ in range(180):   # the warm-up sweeps done, the debris at rest
            _frame(st)
        state13, _, flags = w.bodies()
        alive = flags & 1
        state13[:, 7:] = 0.0
        st.src = (state13, np.zeros(len(flags), np.float32), alive)      # at rest, awake
        st.phi0, st.ext = w.phi(), w.ext()
    elif kind == "boxes":
        rng = np.random.default_rng(seed)
        scenes = []
        for _ in range(case["scenes"]):
            p = X.pile(case["boxes"])
            p[:, 0] += rng.uniform(-0.03, 0.03, len(p)).astype(np.float32)
            p[:, 2] += rng.uniform(-0.03, 0.03, len(p)).astype(np.float32)
            scenes.append(p)
        st.world = X.BoxWorld(scenes, X.box_params(allow_sleep=0, substeps=case["substeps"]))
        if case["cells"]:
            lib = hulls.library().packed()
            ids = rng.integers(1, len(lib), st.world.n).astype(np.uint32)
            ids[::5] = 0
            st.world.set_hulls(lib, ids)
        st.world.step(np.float32(DT), case["age"])
    elif kind == "sat":
        rng = np.random.default_rng(seed)
        n = case["pairs"]
        st.lib = hulls.library().packed() if case["cells"] else None
        pair = []
        for _ in range(2):
            x = np.zeros((n, 11 if case["cells"] else 10), np.float32)
            reach, h0, h1 = (0.45, 0.15, 0.5) if case["cells"] else (0.6, 0.1, 0.6)
            x[:, :3] = rng.uniform(-reach, reach, (n, 3))
            x[:, 3:7] = _unit_quaternions(rng, n)
            x[:, 7:10] = rng.uniform(h0, h1, (n, 3))
            if case["cells"]:
                x[:, 10] = rng.integers(0, len(st.lib), n)
            pair.append(x)
        st.a, st.b = pair
    else:
        raise ValueError(kind)
    return st


# ---------------------------------------------------------------- one pass
def _frame(st):
    w = st.world
    st.frame += 1
    w.step(DT)
    w.rebuild_bodies()
    w.connectivity()
    w.structure_loads(st.ids)
    fr = w.structure_frame(st.frame, st.ids, dt=DT)
    bf = w.bodies_frame(DT, fr.crushed)
    w.connectivity()
    return fr, bf


def run(st):
    kind, case = st.kind, st.case
    if kind in ("bricks", "debris"):
        st.world.set_bodies(*st.src)
        st.world.step(DT, case["steps"])
        return st.world.bodies(out=st.out)
    if kind == "pool":
        for k in st.slots:
            st.pool.write_bodies(k, *st.src[k])
        st.pool.step_slots(st.slots, DT, 1)
        return [st.pool.bodies(k) for k in st.slots]
    if kind == "solve":
        st.world.set_phi(st.phi0)
        st.world.set_ext(st.ext)
        st.world.structure_solve(-1, 1.7, case["tol"], case["max_sweeps"])
        sweeps, resid = st.world.solve_detail()
        return {"phi": st.world.phi64(), "sweeps": sweeps, "resid": resid}
    if kind == "tick":
        st.world.set_phi(st.phi0)
        st.world.set_ext(st.ext)
        serving.structure_add_loads(st.world, st.load_brick, st.load_value)
        serving.structure_solve_set(st.world, st.ids, 1.7, 1e-6, case["max_sweeps"])
        return {"phi": st.world.phi64()}
    if kind == "frame":
        st.world.set_bodies(*st.src)
        st.world.set_phi(st.phi0)
        st.world.set_ext(st.ext)
        fr, bf = _frame(st)
        return {"bodies": st.world.bodies(), "phi": st.world.phi64(), "ext": st.world.ext(),
                "joints": int(fr.joints), "sweeps": int(fr.sweeps)}
    if kind == "boxes":
        st.world.step(np.float32(DT), case["steps"])
        return st.world.state()
    if case["cells"]:
        return sf.collide_hulls(st.lib, st.a, st.b, margin=0.02)
    return sf.collide_boxes(st.a, st.b, margin=0.02)


# ---------------------------------------------------------------- what a pass cannot do without
BODY_STATE, BODY_FIXED, BRICK = 57, 52, 21      # bytes: pose, velocities, timer, flags / mass, inertia / offset, id, material


def _mean_log_uniform(lo, hi):
    return lo if hi <= lo else (hi - lo) / math.log(hi / lo)


def _rigid_work(bodies, bricks, steps):
    # per step the state read and written once, the fixed data read once, and the host copies in and out once; per
    # substep a brick's 27 cells of neighbours and about one contact of 8 iterations
    return {"bytes": steps * (bodies * (2 * BODY_STATE + BODY_FIXED) + bricks * BRICK) + 2 * bodies * BODY_STATE,
            "flops": steps * 2.0 * bricks * (27 * 8 + ITERATIONS * 200)}


def work(case):
    kind = case["kind"]
    if kind == "bricks":
        return _rigid_work(case["bodies"], case["bodies"], case["steps"])
    if kind == "debris":
        n = case["scenes"] * _mean_log_uniform(case["lo"], case["hi"])
        return _rigid_work(n, n / case["p_geom"], case["steps"])
    if kind == "pool":
        n = (case["slots"] + 1) // 2 * _mean_log_uniform(case["lo"], case["hi"])
        return _rigid_work(n, n / 0.3, 1)
    if kind in ("solve", "tick"):
        # a brick's cell, material, neighbours, bonds, load and potential read once, its potential written; 16
        # operations a brick and sweep, the number of sweeps growing with the structure and the tolerance
        n = 3138 if not case["structures"] else 378000.0 * case["hi"] / 40000.0 * case["structures"] / 37.0
        if kind == "tick":
            n *= case["requests"] / 37.0
        sweeps = case["max_sweeps"] if kind == "tick" else min(case["max_sweeps"], 1500 if not case["structures"] else 10000)
        return {"bytes": n * 68.0, "flops": 16.0 * n * sweeps}
    if kind == "frame":
        n = 3150
        r = _rigid_work(case["bodies"], case["bodies"], 1)
        return {"bytes": r["bytes"] + n * 68.0 * 2, "flops": r["flops"] + 16.0 * n * 3}
    if kind == "boxes":
        n = case["scenes"] * case["boxes"]
        # state in and out once a step; about two manifolds of 4 points a box, twice a sub-step
        return {"bytes": n * 88.0 * 2 * case["steps"] + n * 88.0,
                "flops": case["steps"] * n * 2.0 * (2 * case["substeps"] * 900 + 6 * 400)}
    if case["cells"]:
        return {"bytes": case["pairs"] * (2 * 44 + 36 * 4 + 4.0), "flops": case["pairs"] * 40000.0}
    return {"bytes": case["pairs"] * (2 * 40 + 20 * 4 + 4.0), "flops": case["pairs"] * 3000.0}


# ---------------------------------------------------------------- the values in 64 bits
def exact(case, seed):
    if case["kind"] != "solve" or case["structures"]:
        return None
    sc = _frame5(seed)
    xyz, n = sc.static_xyz.astype(np.int64), sc.n_static
    key = {tuple(c): i for i, c in enumerate(xyz.tolist())}
    near = np.full((n, 6), n)
    for d, (dx, dy, dz) in enumerate(((1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1))):
        near[:, d] = [key.get((x + dx, y + dy, z + dz), n) for x, y, z in xyz.tolist()]
    # concrete throughout: a vertical link has conductance 1, a horizontal one 0.3, a footing 4; a brick weighs 300 and
    # carries its load
    side = float(np.float32(0.3))
    link = np.array([side, side, 1.0, 1.0, side, side])
    rhs = 300.0 + _loads(n, seed).astype(np.float64)
    total = (near < n) @ link + 4.0 * (xyz[:, 1] == 0)
    halves = []
    for parity in (0, 1):
        i = np.nonzero(xyz.sum(1) % 2 == parity)[0]
        halves.append((i, np.ascontiguousarray(near[i].T), rhs[i], total[i]))
    phi = np.zeros(n + 1)
    omega, sweeps, resid = float(np.float32(1.7)), 0, math.inf
    while sweeps < case["max_sweeps"] and resid >= float(np.float32(case["tol"])):
        most = 0.0
        for i, nb, r, k in halves:
            step = omega * ((r + link @ phi[nb]) / k - phi[i])
            phi[i] += step
            most = max(most, float(np.abs(step).max()))
        sweeps += 1
        resid = most / max(1.0, float(phi[:n].max()))
    return {"phi": phi[:n].copy(), "sweeps": None, "resid": None}
