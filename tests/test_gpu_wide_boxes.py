"""Node boxes of builds with 63-bit keys, level by level over the faces in the
order that the build returns, on both sides of the builds in one launch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _levels(leaves):
    """Every level's boxes, root first: the union of two children, a lone last one's own box."""
    out = [leaves]
    while out[0].shape[0] > 1:
        below = out[0]
        e = below[: below.shape[0] // 2 * 2].reshape(-1, 2, 6)
        up = np.concatenate([e[:, :, :3].min(1), e[:, :, 3:].max(1)], 1)
        out.insert(0, np.concatenate([up, below[-1:]]) if below.shape[0] % 2 else up)
    return out


def _mesh(n, seed):
    rng = np.random.default_rng(seed)
    nv = max(3, n // 2 + 7)
    return rng.uniform(-1, 1, (nv, 3)).astype(np.float32), rng.integers(0, max(3, nv - 3), (n, 3)).astype(np.uint32)


def _check(t, xyz, tri):
    f, p = t.sorted_faces()
    assert np.array_equal(np.sort(p), np.arange(tri.shape[0])) and np.array_equal(f, tri[p])
    a = xyz[f]
    want = np.concatenate(_levels(np.concatenate([a.min(1), a.max(1)], 1)))
    assert np.array_equal(t.aabb_tree(), want)


@pytest.mark.parametrize("n", [1, 2, 3, 5, 1023, 1025, 4096, 4097, 8193, 70001])
def test_tree_build(gpu, n):
    from oibvh_gb300 import OibvhTree

    xyz, tri = _mesh(n, n)
    t = OibvhTree(xyz=xyz, tri=tri)
    t.set_morton_bits(63)
    for _ in range(2):
        t.build()
        _check(t, xyz, tri)


def test_scene_build(gpu):
    from oibvh_gb300 import OibvhTree, Scene

    meshes = [_mesh(n, 7 + n) for n in (1, 5000, 2, 4096, 300, 33000)]
    trees = [OibvhTree(xyz=x, tri=t) for x, t in meshes]
    sc = Scene()
    for t in trees:
        t.set_morton_bits(63)
        sc.addOibvhTree(t)
    sc.build()
    for t, (x, f) in zip(trees, meshes):
        _check(t, x, f)
