"""Tree and scene builds against the restated build (Morton order, faces, node
boxes bit for bit) at the sizes where the sort's and the renumbering's tiles
begin and end, in both key widths, with unused vertices and equal keys."""
import numpy as np
import pytest

from oracle.oracle import Port

pytestmark = pytest.mark.gpu


def _mesh(n, seed, kind):
    """n random triangles: a soup, an indexed mesh with unused vertices, or one with few distinct keys."""
    rng = np.random.default_rng(seed)
    if kind == "soup":
        xyz = rng.uniform(-1, 1, (3 * n, 3)).astype(np.float32)
        return xyz, rng.permutation(3 * n).astype(np.uint32).reshape(n, 3)
    nv = max(3, n // 2 + 7)
    xyz = rng.uniform(-1, 1, (nv, 3)).astype(np.float32)
    if kind == "equal":
        xyz = np.round(xyz)  # many equal Morton keys: the order is the faces' own
    tri = rng.integers(0, max(3, nv - 3), (n, 3)).astype(np.uint32)
    return xyz, tri


def _check(tree, xyz, tri, bits):
    f, p = tree.sorted_faces()
    assert np.array_equal(np.sort(p), np.arange(tri.shape[0]))
    assert np.array_equal(f, tri[p])  # the caller's numbering
    if bits == 30:
        aabbs, st, perm = Port.oibvh_build(xyz, tri)
        assert np.array_equal(p, perm) and np.array_equal(f, st)
        assert np.array_equal(tree.aabb_tree().view(np.uint32), aabbs.view(np.uint32))


def _order63(xyz, tri):
    """Stable order by the 63-bit key, in numpy with the build's float32 steps."""
    a = xyz[tri]
    mn, mx = a.min(1), a.max(1)
    c = ((mn + mx).astype(np.float32) * np.float32(0.5)).astype(np.float32)
    lo, hi = xyz.min(0), xyz.max(0)
    with np.errstate(invalid="ignore", divide="ignore"):
        u = ((c - lo).astype(np.float32) / (hi - lo).astype(np.float32)).astype(np.float32)
        q = np.clip(u * np.float32(2097152.0), np.float32(0), np.float32(2097151.0))
    q = np.nan_to_num(q, nan=0.0).astype(np.uint64)
    key = np.zeros(tri.shape[0], dtype=np.uint64)
    for b in range(21):
        for k in range(3):
            key |= ((q[:, k] >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b + 2 - k)
    return np.argsort(key, kind="stable")


SIZES = [1, 2, 3, 31, 255, 1023, 1024, 1025, 2049, 4095, 4096, 4097, 8191, 8193, 20000, 70001]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", ["soup", "unused", "equal"])
def test_tree_build(gpu, n, kind):
    from oibvh_gb300 import OibvhTree

    xyz, tri = _mesh(n, n, kind)
    t = OibvhTree(xyz=xyz, tri=tri)
    for _ in range(2):  # the second one starts from the first one's numbering
        t.build()
        _check(t, xyz, tri, 30)
    t.set_morton_bits(63)
    t.build()
    _check(t, xyz, tri, 63)
    assert np.array_equal(t.sorted_faces()[1], _order63(xyz, tri))


@pytest.mark.parametrize("sizes", [(1, 5000, 2, 4096, 300), (4097, 12289, 1, 64), tuple(range(1, 60, 3)), (33000, 90000)])
@pytest.mark.parametrize("bits", [30, 63])
def test_scene_build(gpu, sizes, bits):
    from oibvh_gb300 import OibvhTree, Scene

    meshes = [_mesh(n, 50 + n, ("soup", "unused", "equal")[i % 3]) for i, n in enumerate(sizes)]
    trees = [OibvhTree(xyz=x, tri=t) for x, t in meshes]
    sc = Scene()
    for t in trees:
        t.set_morton_bits(bits)
        sc.addOibvhTree(t)
    for _ in range(2):
        sc.build()
        for t, (x, f) in zip(trees, meshes):
            _check(t, x, f, bits)
            if bits == 63:
                assert np.array_equal(t.sorted_faces()[1], _order63(x, f))


@pytest.mark.parametrize("n", [1, 2, 5, 1023, 1024, 1025, 5000, 32767, 32768, 32769, 60000])
@pytest.mark.parametrize("where", ["host", "device"])
def test_refits_in_a_row(gpu, n, where):
    """Refits from the caller's positions (one launch up to 32,768 faces, two
    above) follow each other with nothing cleared in between."""
    import torch

    from oibvh_gb300 import OibvhTree

    xyz, tri = _mesh(n, 900 + n, "unused")
    t = OibvhTree(xyz=xyz, tri=tri)
    t.build()
    f, p = t.sorted_faces()
    rng = np.random.default_rng(n)
    for _ in range(4):
        moved = (xyz + rng.normal(0, 0.1, xyz.shape)).astype(np.float32)
        if where == "host":
            t.refit(moved)
        else:
            d = torch.from_numpy(moved).cuda()
            t.refit_device(d.data_ptr())
        a = moved[f]
        leaves = np.concatenate([a.min(1), a.max(1)], 1)
        got = t.aabb_tree()
        assert np.array_equal(got[-n:], leaves)
        assert np.array_equal(got[0], np.concatenate([leaves[:, :3].min(0), leaves[:, 3:].max(0)]))
        level = leaves  # every level: the union of its two children, a lone last one's own box
        while level.shape[0] > 1:
            odd = level[-1:] if level.shape[0] % 2 else level[:0]
            e = level[: level.shape[0] // 2 * 2].reshape(-1, 2, 6)
            level = np.concatenate([np.concatenate([e[:, :, :3].min(1), e[:, :, 3:].max(1)], 1), odd])
            at = got.shape[0] - n if level.shape[0] == (n + 1) // 2 else at
            at -= level.shape[0]
            assert np.array_equal(got[at : at + level.shape[0]], level)
    for _ in range(2):  # the positions now held, again
        t.refit()
        assert np.array_equal(t.aabb_tree(), got)


# the sort's tiles: 2048 faces up to half as many tiles of 4096 as there are SMs, then 4096
@pytest.mark.parametrize("n", [6143, 6145, 10240, 10241, 311296, 311297, 319488])
@pytest.mark.parametrize("kind", ["unused", "equal"])
def test_tree_build_sort_tiles(gpu, n, kind):
    from oibvh_gb300 import OibvhTree

    xyz, tri = _mesh(n, n, kind)
    t = OibvhTree(xyz=xyz, tri=tri)
    for bits in (30, 63):
        t.set_morton_bits(bits)
        t.build()
        _check(t, xyz, tri, bits)
    assert np.array_equal(t.sorted_faces()[1], _order63(xyz, tri))
