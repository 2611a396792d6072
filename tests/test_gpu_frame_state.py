"""What a captured frame reports and what it depends on: its statistics are a
direct detect's, and calls between frames do not reach into the next one."""
import numpy as np
import pytest

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
    return sc, trees


def test_frame_statistics_are_the_detects(gpu):
    """Lists between rounds of the size a direct detect of the same state has:
    which pairs share a warp depends on their order in the lists, so the sizes
    agree roughly (a factor of two), not exactly."""
    from oibvh_gb300 import DeviceType

    sc, _ = _scene([_soup(1500, 1), _soup(1700, 2)])
    sc.set_tuning(start_pairs_log2=8, walk_front=64)
    sc.detectCollision(DeviceType.GPU0, 0, 1)
    direct = sc.stats()
    assert direct["front_peak"] > 100 and direct["steps"] > 1
    sc.capture_frame(0, 1, True)
    sc.launch_frame()
    sc.finish_frame()
    frame = sc.stats()
    assert frame["candidates"] == direct["candidates"] and frame["hits"] == direct["hits"]
    assert direct["front_peak"] / 2 <= frame["front_peak"] <= 2 * direct["front_peak"]
    assert abs(frame["steps"] - direct["steps"]) <= 1


def test_frame_steps_of_a_single_round(gpu):
    from oibvh_gb300 import DeviceType

    sc, _ = _scene([_soup(1, 3), _soup(1, 4)])
    sc.detectCollision(DeviceType.GPU0, 0, 1)
    assert sc.stats()["steps"] == 1
    sc.capture_frame(0, 1, True)
    sc.launch_frame()
    sc.finish_frame()
    assert sc.stats()["steps"] == 1 and sc.stats()["front_peak"] == 0


def test_pairs_read_while_a_frame_runs_are_whole_records(gpu):
    """Between launch and finish the count is still the one before, and the
    records are read behind the frame's work: all of them are the new frame's."""
    import torch

    sc, trees = _scene([_soup(600, 5, 0.2), _soup(600, 6, 0.2)])
    sc.capture_frame(0, 1, True)

    def frame(seed):
        rng = np.random.default_rng(seed)
        for t in trees:
            t.set_positions(rng.permutation(_soup(600, seed, 0.2)[0].reshape(600, 9)).reshape(-1, 3))
            seed += 1
        sc.launch_frame()

    frame(10)
    sc.finish_frame()
    first = sc.int_tri_pairs()
    assert 0 < first.shape[0] <= 4096
    torch.cuda._sleep(20_000_000)  # (some 10 ms ahead of the frame on its stream)
    frame(20)
    seen = sc.int_tri_pairs()
    sc.finish_frame()
    second = sc.int_tri_pairs()
    assert seen.shape[0] == first.shape[0]
    got, new = {tuple(r) for r in seen}, {tuple(r) for r in second}
    assert new != {tuple(r) for r in first}
    assert len(got & new) == min(len(first), len(second))  # (records past the new count are left over)


@pytest.mark.parametrize("captured,between", [(0, 6), (6, 0), (0, 9), (9, 4)])
@pytest.mark.parametrize("call", ["detect", "broad"])
def test_a_detect_from_another_level_leaves_the_frame_alone(gpu, captured, between, call):
    from oibvh_gb300 import DeviceType

    soups = [_soup(n, 30 + n, 0.2) for n in (700, 900, 1100)]
    sc, _ = _scene(soups)
    sc.set_tuning(start_pairs_log2=8)
    sc.detectCollision(DeviceType.GPU0, captured, 1)
    want, n = sc.int_tri_pairs(), sc.candidate_count()
    sc.capture_frame(captured, 1, True)
    for _ in range(2):
        sc.launch_frame()
        sc.finish_frame()
        assert np.array_equal(sc.int_tri_pairs(), want) and sc.candidate_count() == n
        getattr(sc, "detectCollision" if call == "detect" else "broad")(DeviceType.GPU0, between, 1)
        assert sc.candidate_count() == n


@pytest.mark.parametrize("by", ["scene", "tree"])
@pytest.mark.parametrize("n", [300, 6000])
def test_a_build_between_frames_is_followed(gpu, by, n):
    """A build renumbers the vertices: the rest positions that a frame moves
    have to be in the new order."""
    import torch

    from oibvh_gb300 import DeviceType

    soups = [_soup(n, 50 + i, 0.1) for i in range(3)]
    packed = torch.from_numpy(np.concatenate([np.pad(x, ((0, 0), (0, 1))) for x, _ in soups], 0)).cuda()
    mats = torch.tensor(np.tile(np.eye(3, 4, dtype=np.float32).reshape(12), (3, 1))).cuda()
    sc, trees = _scene(soups)
    sc.capture_frame(0, 1, True, packed.data_ptr(), mats.data_ptr())
    other, _ = _scene(soups)
    rng = np.random.default_rng(n)
    for _ in range(2):
        # the order depends on the positions built from: others than at the capture
        moved = [rng.permutation(x.reshape(-1, 9)).reshape(-1, 3).copy() for x, _ in soups]
        for t, x in zip(trees, moved):
            t.set_positions(x)
        if by == "scene":
            sc.build()
        else:
            trees[1].build()
        mats.copy_(torch.from_numpy(rng.normal(0, 0.6, (3, 12)).astype(np.float32)))
        sc.launch_frame()
        sc.finish_frame()
        other.transform(packed.data_ptr(), mats.data_ptr())
        other.refit()
        other.detectCollision(DeviceType.GPU0, 0, 1)
        want = other.int_tri_pairs()
        assert want.shape[0] > 0 and np.array_equal(sc.int_tri_pairs(), want)
        assert sc.candidate_count() == other.candidate_count()


@pytest.mark.parametrize("sizes,precision", [((400000, 350000, 300000), 0), ((2000, 3000, 2500), 0), ((2000, 3000, 2500), 1)])
def test_captures_in_a_row_do_not_grow_the_queues(gpu, sizes, precision):
    """A frame that is captured again (here: because its tuning was set) has the
    headroom of its last capture; only a larger frame needs more."""
    import torch

    sc, _ = _scene([_soup(n, n, 0.01) for n in sizes])
    sc.set_precision(precision)

    def again():
        sc.set_tuning(descend_ratio=16)
        sc.launch_frame()
        sc.finish_frame()
        return sc.tuning()["front_capacity"], torch.cuda.mem_get_info()[0]

    sc.capture_frame(0, 1, True)
    front, free = again()
    for _ in range(6):
        f, now = again()
        assert f == front
        assert free - now < 32 << 20, (free, now)
