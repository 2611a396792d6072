"""The work that programs have this library do, for timing: the cases and their ranges.

Every case goes through the public interface (oibvh_gb300.api, and the C ABI
where a program reads results into a buffer of its own). A pass is one unit of
a user's program: bodies move, their trees are refitted or rebuilt, the pairs
are detected, and the colliding triangle pairs are read back. The library
lists them in no particular order; a pass sorts them, as a contact solver
that has to repeat itself does, into a contact buffer of a fixed size (-1
past the last contact).

Kinds of passes:
  query    two deforming bodies: refit both, detect one pair
  rebuild  two bodies, one of them built anew every pass (topology-changing
           simulation; per-frame rebuilds instead of refits)
  scene    many bodies built anew in one scene build, then detected
  bodies   many rigid bodies, every pair tested: transform, refit, detect
  frame    a batch of mesh pairs as one captured frame
  serve    a burst of queries to the query server
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from oibvh_gb300 import _native, meshes, workloads
from oibvh_gb300.api import DeviceType, OibvhTree, Scene, Server

ENTRY, EXPAND = 4, 3  # what the reference's program passes to detectCollision


def listed():
    return [
        # Two small convex-ish props (320 triangles each) against each other every step of a
        # game or robotics loop: nothing but latency.
        {"name": "query_320", "kind": "query", "triangles": 320, "where": "host", "overlap": 0.1},
        # The reference's own program: two 20,480-triangle bodies, positions from the host,
        # refit and detect each frame.
        {"name": "query_20k", "kind": "query", "triangles": 20480, "where": "host", "overlap": 0.1},
        # The repository's deforming workload: two 1.31 M-triangle bodies that touch lightly,
        # positions written on the GPU by a simulation.
        {"name": "query_1310k", "kind": "query", "triangles": 1310720, "where": "device", "overlap": 0.01},
        # One pair of 131,072-triangle sheets, a tenth of them coplanar: cloth on cloth, where
        # the float test is not enough (FP64-filtered).
        {"name": "exact_131k", "kind": "query", "triangles": 131072, "where": "host", "overlap": 0.1, "exact": True, "lift": 0.0},
        # A small body whose topology changes, built anew each step.
        {"name": "rebuild_1k", "kind": "rebuild", "triangles": 1280, "bits": 30, "overlap": 0.1},
        # A fracturing or remeshed body of odd size, built anew each step.
        {"name": "rebuild_300k", "kind": "rebuild", "triangles": 300007, "bits": 30, "overlap": 0.1},
        # A level being loaded, or a whole remeshed scene: 64 pairs of 1k..1M triangles in one build.
        {"name": "scene_64", "kind": "scene", "pairs": 64, "bits": 30},
        # An N-body scene of 24 rigid props, all 276 pairs tested each step.
        {"name": "bodies_24", "kind": "bodies", "bodies": 24, "triangles": 5120, "spread": 2.2},
        # A batch of environments in reinforcement learning or sampling-based planning, captured
        # once and replayed, with the tuning as it comes.
        {"name": "frame_64", "kind": "frame", "pairs": 64, "tune": False, "exact": False},
        # The repository's batched benchmark: 512 pairs, 103 M triangles, autotuned once.
        {"name": "frame_512", "kind": "frame", "pairs": 512, "tune": True, "exact": False},
        # The repository's precision benchmark at a quarter of its pairs: sheets in one captured frame.
        {"name": "exact_frame_16", "kind": "frame", "pairs": 16, "tune": False, "exact": True},
        # A burst of queries from several clients at the query server.
        {"name": "serve_64", "kind": "serve", "burst": 64, "pool": 24},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "query", "rebuild", "rebuild", "scene", "bodies", "frame", "frame", "serve"])
    if kind == "query":
        exact = rng.random() < 0.25
        return {"kind": kind, "triangles": _log_uniform(rng, 200, 131072 if exact else 1310720),
                "where": rng.choice(["host", "device"]), "overlap": round(rng.uniform(0.01, 0.1), 3), "exact": exact,
                "lift": rng.choice([0.0, 5e-8]) if exact else 0.0}
    if kind == "rebuild":
        return {"kind": kind, "triangles": _log_uniform(rng, 200, 1000000), "bits": 63 if rng.random() < 0.25 else 30,
                "overlap": round(rng.uniform(0.01, 0.1), 3)}
    if kind == "scene":
        return {"kind": kind, "pairs": _log_uniform(rng, 2, 64), "bits": 63 if rng.random() < 0.25 else 30}
    if kind == "bodies":
        return {"kind": kind, "bodies": rng.randint(4, 32), "triangles": _log_uniform(rng, 100, 20000),
                "spread": round(rng.uniform(1.8, 3.0), 2)}
    if kind == "frame":
        exact = rng.random() < 0.3
        return {"kind": kind, "pairs": _log_uniform(rng, 2, 16 if exact else 512), "tune": rng.random() < 0.5, "exact": exact}
    return {"kind": kind, "burst": _log_uniform(rng, 8, 192), "pool": rng.randint(8, 32)}


# ------------------------------------------------------------------ inputs
_BASE = {}


def _ball(triangles, variant):
    """A noise-displaced unit icosphere cut off after `triangles` faces (all of it at 20 * 4^s)."""
    key = (triangles, variant)
    if key not in _BASE:
        s = max(0, math.ceil(math.log(triangles / 20.0, 4.0) - 1e-9))
        m = meshes.noise_displace(meshes.icosphere(s), 0.05, seed=100 + variant)
        if triangles < m.n_triangles:
            used, tri = np.unique(m.tri[:triangles], return_inverse=True)
            m = meshes.Mesh(m.xyz[used], tri.reshape(-1, 3).astype(np.uint32))
        _BASE[key] = m
    return _BASE[key]


def _rng(seed, salt):
    return np.random.Generator(np.random.PCG64([int(seed), salt]))


def _two_bodies(case, seed):
    """Meshes A and B of a two-body case, placed, with the seed's jitter."""
    rng = _rng(seed, 1)
    if case.get("exact"):
        n = max(10, int(round(math.sqrt(case["triangles"] / 2.0))))
        return _sheets(rng, n, case["overlap"], case["lift"])
    a, b = _ball(case["triangles"], 0), _ball(case["triangles"], 1)
    # A meets B with the first faces of both (a cut ball keeps those)
    ca, cb = _facing(a), _facing(b)
    d = workloads.distance_for_overlap(1.0, 1.0, case["overlap"])
    spin = meshes.random_rotation(rng)
    to_a, to_b = _turn(ca, (1.0, 0.0, 0.0)), _turn(cb, (-1.0, 0.0, 0.0))
    a = meshes.rigid_transform(a, spin @ to_a, (0.0, 0.0, 0.0))
    b = meshes.rigid_transform(b, spin @ to_b, spin @ np.array([d, 0.0, 0.0]))
    sigma = 1e-3 if case["triangles"] > 100000 else 2e-3
    return (meshes.Mesh(meshes.jitter(a.xyz, sigma, seed, 1), a.tri), meshes.Mesh(meshes.jitter(b.xyz, sigma, seed, 2), b.tri))


def _sheets(rng, n, overlap, lift):
    """Two sine sheets, `overlap` of their columns coplanar or `lift` apart."""
    return workloads.sheet_pair_meshes(n, float(rng.uniform(0.05, 0.5)), float(rng.uniform(0.0, 2.0 * math.pi)),
                                       float(rng.uniform(0.0, 2.0 * math.pi)), lift, overlap=overlap)


def _facing(m):
    """Direction of the middle of the faces a cut ball always has."""
    c = m.xyz[m.tri[: max(1, m.n_triangles // 2)].reshape(-1)].astype(np.float64).mean(0)
    n = float(np.sqrt((c * c).sum()))
    return c / n if n > 1e-3 else np.array([1.0, 0.0, 0.0])


def _turn(u, v):
    """A rotation that takes the unit vector u to v."""
    u, v = np.asarray(u, dtype=np.float64), np.asarray(v, dtype=np.float64)
    w, c = np.cross(u, v), float(u @ v)
    if c < -0.999999:
        w = np.cross(u, (0.0, 1.0, 0.0) if abs(u[1]) < 0.9 else (1.0, 0.0, 0.0))
        w = w / np.sqrt(w @ w)
        return 2.0 * np.outer(w, w) - np.eye(3)
    k = np.array([[0, -w[2], w[1]], [w[2], 0, -w[0]], [-w[1], w[0], 0]])
    return np.eye(3) + k + k @ k / (1.0 + c)


def _scene_of(trees, pairs=None, built=True):
    scene = Scene(0)
    for t in trees:
        if built:
            t.build()
        scene.addOibvhTree(t)
    if pairs is not None:
        scene.set_pairs(pairs)
    return scene


def _packed(mesh_list):
    return torch.from_numpy(np.concatenate([np.pad(m.xyz, ((0, 0), (0, 1))) for m in mesh_list], 0)).cuda()


def _room(case):
    """Entries of a program's contact buffer: about twice what such bodies come to."""
    kind = case["kind"]
    if kind == "serve":
        return 1000 * case["burst"] + 8192
    if kind == "bodies":
        return 1024 + 8 * case["bodies"] * int(math.sqrt(case["triangles"]))
    if kind in ("query", "rebuild"):
        return 1024 + (2 * case["triangles"] if case.get("exact") else 12 * int(math.sqrt(case["triangles"])))
    return 180000 * case["pairs"] if case.get("exact") else 16384 + 2500 * case["pairs"]


def _buffers(case):
    n = _room(case)
    if case["kind"] in ("scene", "frame") or case.get("exact"):
        return {"read": torch.empty((n, 4), dtype=torch.int32, pin_memory=True),
                "contacts": torch.empty(n, dtype=torch.int64, device="cuda")}
    return {"contacts": np.empty(n, dtype=np.int64)}


def prepare(case, seed):
    state = _prepare(case, seed)
    state.update(_buffers(case))
    return state


def _prepare(case, seed):
    kind = case["kind"]
    if kind in ("query", "rebuild"):
        a, b = _two_bodies(case, seed)
        trees = [OibvhTree(a), OibvhTree(b)]
        state = {"case": case, "trees": trees, "xyz": [a.xyz, b.xyz]}
        if kind == "rebuild":
            for t in trees:
                t.set_morton_bits(case["bits"])
        state["scene"] = _scene_of(trees)
        if case.get("exact"):
            state["scene"].set_precision(_native.PRECISION_FP64_FILTERED)
        if case.get("where") == "device":
            state["dev"] = [torch.from_numpy(a.xyz).cuda(), torch.from_numpy(b.xyz).cuda()]
        return state
    if kind == "bodies":
        rng = _rng(seed, 2)
        n = case["bodies"]
        ms = [_ball(max(20, int(case["triangles"] * rng.uniform(0.5, 1.0))), i % 4) for i in range(n)]
        side = case["spread"] * n ** (1.0 / 3.0) / 2.0
        mats = np.empty((n, 12), dtype=np.float32)
        for i in range(n):
            at = rng.uniform(-side, side, 3)
            mats[i] = np.concatenate([meshes.random_rotation(rng) * rng.uniform(0.7, 1.0), at[:, None]], 1).reshape(12)
        trees = [OibvhTree(m) for m in ms]
        scene = _scene_of(trees, built=False)
        scene.build()
        return {"case": case, "trees": trees, "scene": scene, "rest": _packed(ms),
                "h_mats": torch.from_numpy(mats).pin_memory(), "mats": torch.empty((n, 12), device="cuda")}
    if kind in ("scene", "frame"):
        exact = bool(case.get("exact"))
        if exact:
            w = workloads.sheets(case["pairs"], 256, seed=seed)
            ms, mats = w.meshes, np.tile(np.eye(3, 4, dtype=np.float32).reshape(12), (2 * case["pairs"], 1))
        else:
            w = workloads.batched(case["pairs"], seed=seed)
            ms, mats = w.rest, w.matrices(0)
        trees = [OibvhTree(m) for m in ms]
        for t in trees:
            t.set_morton_bits(case.get("bits", 30))
        scene = _scene_of(trees, w.pairs, built=False)
        scene.build()
        h_mats = torch.from_numpy(mats).pin_memory()
        state = {"case": case, "trees": trees, "scene": scene, "rest": _packed(ms), "h_mats": h_mats, "mats": h_mats.cuda()}
        scene.transform(state["rest"].data_ptr(), state["mats"].data_ptr())
        if kind == "frame":
            if exact:
                scene.set_precision(_native.PRECISION_FP64_FILTERED)
            scene.refit()
            if case["tune"]:
                scene.autotune(ENTRY, 3)
            scene.capture_frame(ENTRY, EXPAND, True, state["rest"].data_ptr(), state["mats"].data_ptr())
        return state
    rng = _rng(seed, 3)
    ms = [_ball(_spread(rng, 500, 200000), i % 3) for i in range(case["pool"])]
    trees = [OibvhTree(m) for m in ms]
    server = Server(memory_budget=2 << 30, max_batch=256, lanes=4)
    for t in trees:
        t.build()
        server.add_mesh(t)
    server.start()
    queries = []
    for _ in range(case["burst"]):
        a, b = (int(x) for x in rng.integers(0, case["pool"], 2))
        v = rng.standard_normal(3)
        t = v / math.sqrt(float(v @ v)) * rng.uniform(0.3, 1.8)
        queries.append((a, b, np.concatenate([meshes.random_rotation(rng), t[:, None]], 1).astype(np.float32)))
    return {"case": case, "trees": trees, "server": server, "queries": queries}


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# ------------------------------------------------------------------ passes
def _key(rec):
    """(bvhA, bvhB, triA, triB) in one number: bodies below 2^10, faces below 2^21."""
    return (((rec[:, 0] << 10 | rec[:, 1]) << 21 | rec[:, 2]) << 21) | rec[:, 3]


def _contacts(state):
    """The colliding pairs in the program's contact buffer, sorted."""
    keys = _key(state["scene"].int_tri_pairs(sort=False).astype(np.int64))
    keys.sort()
    out = state["contacts"]
    out[: keys.size] = keys
    out[keys.size :] = -1
    return out


def _contacts_on_gpu(state):
    """The same where there are too many for the host: read into pinned memory
    and sorted on the GPU, where the program goes on with them."""
    read, out = state["read"], state["contacts"]
    n = ctypes.c_uint64()
    _native.check(_native.lib().oibvh_scene_get_int_tri_pairs(
        state["scene"].handle, ctypes.cast(ctypes.c_void_p(read.data_ptr()), _native._u32p), read.shape[0], ctypes.byref(n)),
        "oibvh_scene_get_int_tri_pairs")
    found = int(n.value)
    if found > read.shape[0]:
        raise RuntimeError("the contact buffer is too small")
    out[:found] = torch.sort(_key(read[:found].cuda(non_blocking=True).long()))[0]
    out[found:] = -1
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "serve":
        return _serve(state)
    scene, trees = state["scene"], state["trees"]
    if kind == "query":
        if case["where"] == "host":
            for t, xyz in zip(trees, state["xyz"]):
                t.refit(xyz)
        else:
            for t, xyz in zip(trees, state["dev"]):
                t.set_positions_device(xyz.data_ptr())
            scene.refit()
        scene.detectCollision(DeviceType.GPU0, ENTRY, EXPAND)
        return [_contacts_on_gpu(state) if case.get("exact") else _contacts(state), scene.candidate_count()]
    if kind == "rebuild":
        trees[1].set_positions(state["xyz"][1])
        trees[1].build()
        scene.detectCollision(DeviceType.GPU0, ENTRY, EXPAND)
        return [_contacts(state), scene.candidate_count()]
    state["mats"].copy_(state["h_mats"], non_blocking=True)
    if kind == "frame":
        scene.launch_frame()
        scene.finish_frame()
        return [_contacts_on_gpu(state), scene.candidate_count()]
    scene.transform(state["rest"].data_ptr(), state["mats"].data_ptr())
    if kind == "scene":
        scene.build()
    else:
        scene.refit()
    scene.detectCollision(DeviceType.GPU0, ENTRY, EXPAND)
    if kind == "bodies":
        return [_contacts(state), scene.candidate_count()]
    return [_contacts_on_gpu(state), scene.candidate_count()]


def _serve(state):
    server = state["server"]
    tickets = [server.submit(a, b, m) for a, b, m in state["queries"]]
    got, counts = [], []
    n = ctypes.c_uint64()
    for t in tickets:
        found = int(server.wait(t)["n_pairs"])
        pairs = np.empty((max(found, 1), 2), dtype=np.uint32)
        _native.check(_native.lib().oibvh_server_get_pairs(
            server._h, t, pairs.ctypes.data_as(_native._u32p), found, ctypes.byref(n)), "oibvh_server_get_pairs")
        server.release(t)
        keys = pairs[:found].view(np.int64).reshape(-1)
        keys.sort()
        got.append(keys)
        counts.append(found)
    out, total = state["contacts"], sum(counts)
    out[:total] = np.concatenate(got)
    out[total:] = -1
    return [out, np.array(counts)]


# ------------------------------------------------------------------ what a pass cannot do without
_REFIT = 6 + 12 + 24       # per triangle: half a vertex and a face read, an internal node written
_BUILD = _REFIT + 16       # and the sorted face with its original index
_MOVE = 6 + 6              # half a vertex read and written


def work(case):
    kind = case["kind"]
    if kind == "query":
        t, per = 2 * case["triangles"], _REFIT
    elif kind == "rebuild":
        t, per = case["triangles"], _BUILD
    elif kind == "bodies":
        t, per = 0.75 * case["bodies"] * case["triangles"], _MOVE + _REFIT
    elif kind in ("scene", "frame"):
        mean = 131072 if case.get("exact") else 103e6 / 1024
        t, per = 2 * case["pairs"] * mean, _MOVE + (_BUILD if kind == "scene" else _REFIT)
    else:
        t, per = case["burst"] * 33000, _MOVE + _REFIT  # B of every query; sizes log-uniform over 500..200k
    # three minima and three maxima per merged node
    return {"bytes": float(t * per), "flops": float(6 * t)}


def exact(case, seed):
    return None  # every output is a whole number (face indices and counts): they stay equal
