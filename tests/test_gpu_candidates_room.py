"""Large float passes keep their candidates for a kernel of their own. Where
there is no room for them the walk tests them itself, and goes on doing so."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _hook_off(gpu):
    from oibvh_gb300 import _native as N

    N.lib().oibvh_debug_fail_alloc_after(-1)
    yield
    N.lib().oibvh_debug_fail_alloc_after(-1)


def _soup(n, seed, size, at=0.0):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1.0, 1.0, (n, 1, 3)) + at
    return (c + rng.uniform(-size, size, (n, 3, 3))).astype(np.float32).reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


def _trees(soups):
    from oibvh_gb300 import OibvhTree

    trees = [OibvhTree(xyz=x, tri=t) for x, t in soups]
    for t in trees:
        t.build()
    return trees


def _scene(trees, pairs=None):
    from oibvh_gb300 import Scene

    sc = Scene()
    for t in trees:
        sc.addOibvhTree(t)
    if pairs is not None:
        sc.set_pairs(pairs)
    return sc


def test_a_list_that_found_no_room_is_not_asked_for_again(gpu):
    from oibvh_gb300 import DeviceType
    from oibvh_gb300 import _native as N

    L = N.lib()
    trees = _trees([_soup(n, n, 0.008) for n in (400000, 350000, 300000)])
    whole = _scene(trees)
    whole.detectCollision(DeviceType.GPU0, 4, 3)
    want, n_cands = whole.int_tri_pairs(), whole.candidate_count()
    assert want.shape[0] > 0

    def attempts(fn):
        a0 = L.oibvh_debug_alloc_attempts()
        fn()
        return L.oibvh_debug_alloc_attempts() - a0

    def check(sc):
        assert np.array_equal(sc.int_tri_pairs(), want) and sc.candidate_count() == n_cands

    # each allocation of the first detect in turn: the candidates' is the one that it does without
    # (after that come detects that the hook does not reach)
    done = 0
    for k in range(40):
        sc = _scene(trees)
        L.oibvh_debug_fail_alloc_after(k)
        try:
            sc.detectCollision(DeviceType.GPU0, 4, 3)
        except N.OibvhError as e:
            assert e.status == N.ERR_OOM
            continue
        check(sc)
        for _ in range(2):  # whatever it asked for now would not be there
            L.oibvh_debug_fail_alloc_after(0)
            assert attempts(lambda: sc.detectCollision(DeviceType.GPU0, 4, 3)) == 0, k
            check(sc)
        L.oibvh_debug_fail_alloc_after(-1)
        sc.capture_frame(4, 3, True)
        sc.launch_frame()
        sc.finish_frame()
        check(sc)
        done += 1
        if done == 2:
            break
    assert done == 2


def test_more_candidates_than_a_list_can_hold(gpu):
    """2.15e9 pairs of overlapping boxes (none of them hits): past 2^31 - 1
    entries, where the walk has to test them itself."""
    from oibvh_gb300 import DeviceType

    n = 46400
    rng = np.random.default_rng(5)
    corner = np.array([[1.0, -0.5, -0.5], [-0.5, 1.0, -0.5], [-0.5, -0.5, 1.0]])

    def plates(s):
        lift = rng.uniform(0.0, 1e-3, (n, 1, 1)) + s
        return (corner + lift).astype(np.float32).reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)

    trees = _trees([plates(0.0), plates(0.01), _soup(1 << 20, 9, 0.001, at=50.0)])
    sc = _scene(trees, [(0, 1), (0, 2)])
    for _ in range(2):
        sc.detectCollision(DeviceType.GPU0, 4, 3)
        assert sc.candidate_count() == n * n and sc.getIntTriPairCount() == 0
