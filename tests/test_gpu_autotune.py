"""The setting that the autotuner returns is the one that it leaves the scene
with, so that it can be given to another scene."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _soup(n, seed, size):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1.0, 1.0, (n, 1, 3))
    return (c + rng.uniform(-size, size, (n, 3, 3))).astype(np.float32).reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("sizes", [(1, 1), (2000, 2500), (900, 1000, 1100), (400000, 350000, 300000)])
@pytest.mark.parametrize("precision", [0, 1])
def test_the_returned_setting_is_the_scenes(gpu, sizes, precision):
    from oibvh_gb300 import DeviceType, OibvhTree, Scene

    soups = [_soup(n, n + i, 0.01 if max(sizes) > 10000 else 0.1) for i, n in enumerate(sizes)]
    scenes = []
    for _ in range(2):
        sc = Scene()
        for x, t in soups:
            tree = OibvhTree(xyz=x, tri=t)
            tree.build()
            sc.addOibvhTree(tree)
        sc.set_precision(precision)
        scenes.append(sc)
    a, b = scenes
    b.detectCollision(DeviceType.GPU0, 0, 1)
    want, n = b.int_tri_pairs(), b.candidate_count()
    got = a.autotune(0, 1)
    assert got == a.tuning()
    b.set_tuning(**got)
    assert b.tuning() == got
    for sc in scenes:
        sc.detectCollision(DeviceType.GPU0, 0, 1)
        assert np.array_equal(sc.int_tri_pairs(), want) and sc.candidate_count() == n
