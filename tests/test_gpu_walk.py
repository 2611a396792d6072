"""The traversal against the oracle at the sizes where its split changes: one
pair (its record in the kernel's arguments) and several, few and many start
tests, steps with at most 8 pairs and full ones, rings that overflow to the
next round's list, lists that are dealt out and lists that are claimed."""
import numpy as np
import pytest

from oracle.oracle import Port, sort_pairs

pytestmark = pytest.mark.gpu


def _soup(n, seed, size=0.4):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1.0, 1.0, (n, 1, 3))
    xyz = (c + rng.uniform(-size, size, (n, 3, 3))).astype(np.float32).reshape(-1, 3)
    return xyz, np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


def _scene(soups):
    from oibvh_gb300 import OibvhTree, Scene

    trees = [OibvhTree(xyz=x, tri=t) for x, t in soups]
    sc = Scene()
    for t in trees:
        t.build()
        sc.addOibvhTree(t)
    return sc


def _want(soups):
    port = Port()
    for x, t in soups:
        port.add_mesh(x, t)
    w, n = port.detect()
    return sort_pairs(w), n


# sizes at the edges of a step (8, 32), of a warp's start tests and of tree levels; the large
# ones overlap everywhere, so that rings overflow and lists are claimed
@pytest.mark.parametrize("sizes", [(1, 1), (1, 9), (8, 8), (9, 7), (31, 33), (32, 32), (255, 257), (1023, 1025),
                                   (4097, 700), (3, 64, 65), (500, 1, 90, 129, 2000)])
@pytest.mark.parametrize("start,ring", [(8, 64), (16, 128), (22, 512)])
def test_walk_equals_the_oracle(gpu, sizes, start, ring):
    from oibvh_gb300 import DeviceType

    soups = [_soup(n, 100 + i) for i, n in enumerate(sizes)]
    sc = _scene(soups)
    sc.set_tuning(start_pairs_log2=start, walk_front=ring)
    want, n = _want(soups)
    for entry in (0, 4, 30):
        sc.detectCollision(DeviceType.GPU0, entry, 1)
        assert np.array_equal(sc.int_tri_pairs(), want), entry
        assert sc.candidate_count() == n
    sc.broad(DeviceType.GPU0, 4, 3)  # the walk that only stores its candidates
    assert sc.candidate_count() == n and sc.candidates().shape[0] == n
    sc.narrow()
    assert np.array_equal(sc.int_tri_pairs(), want)


@pytest.mark.parametrize("front", [1, 8, 63, 4096])
def test_walk_lists_that_overflow_are_regrown(gpu, front):
    from oibvh_gb300 import DeviceType

    soups = [_soup(1500, 7), _soup(1700, 8)]
    sc = _scene(soups)
    sc.set_queue_capacity(front=front)
    sc.set_tuning(start_pairs_log2=8, walk_front=64)
    want, n = _want(soups)
    sc.detectCollision(DeviceType.GPU0, 0, 1)
    assert np.array_equal(sc.int_tri_pairs(), want) and sc.candidate_count() == n


@pytest.mark.parametrize("n_tri", [1, 2, 3, 4, 5, 8, 9, 16, 17, 33, 200])
def test_few_candidates_on_every_axis(gpu, n_tri):
    """A round's last candidates, tested by several lanes each: triangles whose
    float test turns on one axis or another (shared edges, coplanar, lifted)."""
    from oibvh_gb300 import DeviceType
    from oibvh_gb300.meshes import Mesh
    from tests_support import near_degenerate_pair

    a, b = near_degenerate_pair(70 + n_tri, n_tri)
    soups = [(a.xyz, a.tri), (b.xyz, b.tri)]
    soups.append(_soup(2 * n_tri, n_tri, 0.1))
    sc = _scene(soups)
    want, n = _want(soups)
    sc.detectCollision(DeviceType.GPU0, 4, 3)
    assert np.array_equal(sc.int_tri_pairs(), want) and sc.candidate_count() == n
    sc.set_pairs([(0, 1)])
    sc.detectCollision(DeviceType.GPU0, 4, 3)
    assert np.array_equal(sc.int_tri_pairs(), want[(want[:, 0] == 0) & (want[:, 1] == 1)])


@pytest.mark.parametrize("sizes", [(1, 9000), (2, 40000), (5, 33000), (16385, 16384), (70000, 300)])
def test_sparse_trees_two_levels_at_once(gpu, sizes):
    """Warps with a pair or two, down trees of different depths."""
    from oibvh_gb300 import DeviceType

    soups = [_soup(n, 40 + i, 0.02) for i, n in enumerate(sizes)]
    sc = _scene(soups)
    want, n = _want(soups)
    for start in (8, 16):
        sc.set_tuning(start_pairs_log2=start)
        sc.detectCollision(DeviceType.GPU0, 0, 1)
        assert np.array_equal(sc.int_tri_pairs(), want) and sc.candidate_count() == n
