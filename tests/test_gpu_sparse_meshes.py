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
