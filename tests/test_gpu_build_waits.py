"""A build whose waits run out: reported, the tree counts as not built and its
faces lead nowhere, and the next build starts from what was there before. (The
limit is set so low that a tile gives up at the first look that finds the tiles
before it unfinished, which some of hundreds always do.)"""
import numpy as np
import pytest

from oracle.oracle import Port

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _polls(gpu):
    from oibvh_gb300 import _native as N

    yield
    N.lib().oibvh_debug_set_build_polls(0xFFFFFFFF)


def _mesh(n, seed):
    rng = np.random.default_rng(seed)
    nv = n // 2 + 7
    return rng.uniform(-1, 1, (nv, 3)).astype(np.float32), rng.integers(0, nv - 3, (n, 3)).astype(np.uint32)


def _check(t, xyz, tri):
    aabbs, faces, perm = Port.oibvh_build(xyz, tri)
    f, p = t.sorted_faces()
    assert np.array_equal(p, perm) and np.array_equal(f, faces)
    assert np.array_equal(t.aabb_tree().view(np.uint32), aabbs.view(np.uint32))


def _gives_up(build):
    from oibvh_gb300 import _native as N

    N.lib().oibvh_debug_set_build_polls(0)
    with pytest.raises(N.OibvhError) as e:
        build()
    assert e.value.status == N.ERR_TIMEOUT
    N.lib().oibvh_debug_set_build_polls(0xFFFFFFFF)


def _state_error(call):
    from oibvh_gb300 import _native as N

    with pytest.raises(N.OibvhError) as e:
        call()
    assert e.value.status == N.ERR_STATE


@pytest.mark.parametrize("built_before", [False, True])
@pytest.mark.parametrize("bits", [30, 63])
def test_a_tree_build_that_gives_up(gpu, built_before, bits):
    from oibvh_gb300 import OibvhTree, Scene

    xyz, tri = _mesh(1200000, 1)
    t = OibvhTree(xyz=xyz, tri=tri)
    other = OibvhTree(xyz=xyz[:30], tri=np.arange(30, dtype=np.uint32).reshape(-1, 3))
    other.build()
    if built_before:
        t.build()
    t.set_morton_bits(bits)
    _gives_up(t.build)
    sc = Scene()
    sc.addOibvhTree(t)
    sc.addOibvhTree(other)
    for call in (t.refit, sc.refit, sc.detectCollision):
        _state_error(call)
    t.set_morton_bits(30)
    t.build()
    _check(t, xyz, tri)
    sc.detectCollision()


def test_a_scene_build_that_gives_up(gpu):
    from oibvh_gb300 import OibvhTree, Scene

    meshes = [_mesh(n, n) for n in (700000, 3000, 500000)]
    trees = [OibvhTree(xyz=x, tri=t) for x, t in meshes]
    trees[1].build()
    sc = Scene()
    for t in trees:
        sc.addOibvhTree(t)
    _gives_up(sc.build)
    for call in (trees[0].refit, trees[1].refit, sc.refit, sc.detectCollision):
        _state_error(call)
    sc.build()
    for t, (x, f) in zip(trees, meshes):
        _check(t, x, f)


def test_a_frame_whose_tree_was_lost(gpu):
    """A captured frame does not walk a tree that a build has given up."""
    from oibvh_gb300 import OibvhTree, Scene

    meshes = [_mesh(700000, 5), _mesh(2000, 6)]
    trees = [OibvhTree(xyz=x, tri=t) for x, t in meshes]
    sc = Scene()
    for t in trees:
        t.build()
        sc.addOibvhTree(t)
    sc.capture_frame(4, 3, True)
    sc.launch_frame()
    sc.finish_frame()
    n = sc.candidate_count()
    _gives_up(trees[0].build)
    _state_error(sc.launch_frame)
    trees[0].build()
    sc.launch_frame()
    sc.finish_frame()
    assert sc.candidate_count() == n
