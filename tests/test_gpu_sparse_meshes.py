"""Meshes with far more vertices than their faces use (a part of a shared vertex
buffer): the few CTAs of their faces do not also go through all the vertices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sparse(n_faces, n_verts, seed, size=0.1):
    """n_faces small triangles whose corners lie anywhere in a buffer of n_verts positions."""
    rng = np.random.default_rng(seed)
    xyz = rng.uniform(-1.0, 1.0, (n_verts, 3)).astype(np.float32)
    at = rng.choice(n_verts, 3 * n_faces, replace=False) if 3 * n_faces <= n_verts else rng.integers(0, n_verts, 3 * n_faces)
    tri = at.reshape(-1, 3).astype(np.uint32)
    if 3 * n_faces <= n_verts:
        c = rng.uniform(-1.0, 1.0, (n_faces, 1, 3))
        xyz[tri.reshape(-1)] = (c + rng.uniform(-size, size, (n_faces, 3, 3))).astype(np.float32).reshape(-1, 3)
    return xyz, tri


def _launches(fn):
    from oibvh_gb300 import _native as N

    a = N.lib().oibvh_get_launch_count()
    fn()
    return N.lib().oibvh_get_launch_count() - a


# one launch up to as many vertices as faces (or 1024), and 32,768 faces
@pytest.mark.parametrize("faces,verts,launches", [(300, 150, 1), (300, 1024, 1), (300, 1025, 2), (300, 200000, 2),
                                                  (5000, 5000, 1), (5000, 5001, 2), (32768, 32768, 1), (32769, 20000, 2)])
@pytest.mark.parametrize("where", ["host", "device"])
def test_refit_of_a_tree(gpu, faces, verts, launches, where):
    import torch

    from oibvh_gb300 import OibvhTree

    xyz, tri = _sparse(faces, verts, faces + verts)
    t = OibvhTree(xyz=xyz, tri=tri)
    t.build()
    f, _ = t.sorted_faces()
    for k in range(2):
        moved = (xyz + np.random.default_rng(k).normal(0, 0.1, xyz.shape)).astype(np.float32)
        d = torch.from_numpy(moved).cuda()
        n = _launches((lambda: t.refit(moved)) if where == "host" else (lambda: t.refit_device(d.data_ptr())))
        assert n == launches
        a = moved[f]
        got = t.aabb_tree()
        assert np.array_equal(got[-faces:], np.concatenate([a.min(1), a.max(1)], 1))
        assert np.array_equal(got[0], np.concatenate([a.reshape(-1, 3).min(0), a.reshape(-1, 3).max(0)]))
    t.refit()  # the positions now held
    assert np.array_equal(t.aabb_tree(), got)


@pytest.mark.parametrize("verts", [4096, 4097, 300000])
def test_a_large_frame_with_such_a_tree(gpu, verts):
    """2^20 faces and more, one tree of 300 over many vertices: moved in a launch of its own."""
    import torch

    from oibvh_gb300 import DeviceType, OibvhTree, Scene

    rng = np.random.default_rng(verts)
    n = (1 << 20) + 100
    c = rng.uniform(-1.0, 1.0, (n, 1, 3))
    big = ((c + rng.uniform(-0.004, 0.004, (n, 3, 3))).astype(np.float32).reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3))
    soups = [_sparse(300, verts, 1), big, _sparse(700, 3000, 2)]
    scenes = []
    for _ in range(2):
        sc = Scene()
        for x, t in soups:
            sc.addOibvhTree(OibvhTree(xyz=x, tri=t))
        sc.build()
        scenes.append(sc)
    a, b = scenes
    packed = torch.from_numpy(np.concatenate([np.pad(x, ((0, 0), (0, 1))) for x, _ in soups], 0)).cuda()
    mats = torch.from_numpy(np.tile(np.eye(3, 4, dtype=np.float32).reshape(12), (3, 1))).cuda()
    a.capture_frame(0, 1, True, packed.data_ptr(), mats.data_ptr())
    kernels = set()
    for k in range(2):
        mats.copy_(torch.from_numpy(np.tile(np.eye(3, 4, dtype=np.float32).reshape(12), (3, 1)) + rng.normal(0, 0.05, (3, 12)).astype(np.float32)))
        p = a.profile_frame()
        kernels.add(p["kernels"] - p["walk_rounds"])
        b.transform(packed.data_ptr(), mats.data_ptr())
        b.refit()
        b.detectCollision(DeviceType.GPU0, 0, 1)
        want = b.int_tri_pairs()
        assert want.shape[0] > 0 and np.array_equal(a.int_tri_pairs(), want)
        a.launch_frame()
        a.finish_frame()
        assert np.array_equal(a.int_tri_pairs(), want)
        for x, y in zip(a._trees, b._trees):
            assert np.array_equal(x.aabb_tree().view(np.uint32), y.aabb_tree().view(np.uint32))
    # [transform,] refit, counters, narrow phase, results
    assert kernels == {4 if verts <= 4096 else 5}


@pytest.mark.parametrize("verts", [900, 4097, 250000])
def test_server_batches_with_such_a_mesh(gpu, verts):
    from oibvh_gb300 import DeviceType, OibvhTree, Scene, Server

    soups = [_sparse(300, verts, 11, 0.2), _sparse(900, 2000, 12, 0.2), _sparse(5000, 15000, 13, 0.1)]
    trees = [OibvhTree(xyz=x, tri=t) for x, t in soups]
    for t in trees:
        t.build()
    server = Server(memory_budget=1 << 30, max_batch=16, lanes=2)
    ids = [server.add_mesh(t) for t in trees]
    server.start()
    rng = np.random.default_rng(verts)
    queries = [(a, b, np.eye(3, 4, dtype=np.float32) + rng.normal(0, 0.05, (3, 4)).astype(np.float32))
               for a in range(3) for b in range(3) for _ in range(3)]
    tickets = [server.submit(ids[a], ids[b], m) for a, b, m in queries]
    import torch

    for t, (a, b, m) in zip(tickets, queries):
        info = server.wait(t)
        got = server.pairs(t)
        server.release(t)
        sc = Scene()
        other = [OibvhTree(xyz=x, tri=f) for x, f in (soups[a], soups[b])]
        for o in other:
            sc.addOibvhTree(o)
        sc.build()
        packed = torch.from_numpy(np.concatenate([np.pad(x, ((0, 0), (0, 1))) for x in (soups[a][0], soups[b][0])], 0)).cuda()
        mats = torch.from_numpy(np.stack([np.eye(3, 4, dtype=np.float32).reshape(12), m.reshape(12)])).cuda()
        sc.transform(packed.data_ptr(), mats.data_ptr())
        sc.refit()
        sc.detectCollision(DeviceType.GPU0, 0, 1)
        assert np.array_equal(got, sc.int_tri_pairs()[:, 2:]) and int(info["n_pairs"]) == got.shape[0]
    server.close()
