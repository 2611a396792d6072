"""Boxes that do not hold their children's: positions with NaN or infinity, and
positions set without a refit. Which leaf pairs are candidates then depends on
every box test on the way down, so the walk has to make each of them, however
its warps share the pairs out: the candidates equal those of a plain walk, level
by level, over the trees' own boxes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Tree:
    """Level-ordered boxes of a tree, as the library returns them."""

    def __init__(self, tree):
        self.box = tree.aabb_tree()
        self.n = tree.getPrimCount()
        self.L = int(np.ceil(np.log2(self.n))) if self.n > 1 else 0
        vl = (1 << self.L) - self.n
        self.count = [(1 << k) - (vl >> (self.L - k)) for k in range(self.L + 1)]
        self.off = np.concatenate([[0], np.cumsum(self.count)])

    def at(self, level, i):
        return self.box[self.off[level] + i]

    def down(self, level, i):
        return [(level + 1, c) for c in (2 * i, 2 * i + 1) if c < self.count[level + 1]]


def _overlap(a, b):
    return bool(np.all(a[:3] <= b[3:]) and np.all(a[3:] >= b[:3]))


def _size2(b):
    d = (b[3:] - b[:3]).astype(np.float32)
    return np.float32(np.float32(d[0] * d[0] + d[1] * d[1]) + d[2] * d[2])


def _walk(A, B, start, ratio=np.float32(16.0)):
    """Leaf indices of every leaf pair that the walk reaches."""
    la, lb = min(start, A.L), min(start, B.L)
    todo = [((la, i), (lb, j)) for i in range(A.count[la]) for j in range(B.count[lb])]
    out = []
    while todo:
        nxt = []
        for (a, b) in todo:
            ba, bb = A.at(*a), B.at(*b)
            if not _overlap(ba, bb):
                continue
            leaf_a, leaf_b = a[0] == A.L, b[0] == B.L
            if leaf_a and leaf_b:
                out.append((a[1], b[1]))
                continue
            sa, sb = _size2(ba), _size2(bb)
            only_a = not leaf_a and (leaf_b or sa > ratio * sb)
            only_b = not leaf_b and (leaf_a or (not only_a and sb > ratio * sa))
            for x in [a] if only_b else A.down(*a):
                for y in [b] if only_a else B.down(*b):
                    nxt.append((x, y))
        todo = nxt
    return sorted(out)


def _soup(n, seed, size, kind, part=0.03):
    rng = np.random.default_rng(seed)
    if n == 1:
        size, part = 0.9, 0.0  # (a lone triangle meets several others)
    c = rng.uniform(-1.0, 1.0, (n, 1, 3))
    xyz = (c + rng.uniform(-size, size, (n, 3, 3))).astype(np.float32).reshape(-1, 3)
    bad = rng.random(xyz.shape) < part
    if kind == "nan":
        xyz[bad] = np.nan
    elif kind == "inf":
        xyz[bad] = np.where(rng.random(xyz.shape) < 0.5, np.float32(np.inf), np.float32(-np.inf))[bad]
    return xyz, np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


def _start(na, nb, log2, entry=0):
    """The start level of a scene's only pair."""
    return max(entry, int(np.floor(log2 / 2.0)))


@pytest.mark.parametrize("sizes", [(1, 700), (300, 900), (1025, 640), (2000, 2100)])
@pytest.mark.parametrize("kind", ["nan", "inf", "moved"])
@pytest.mark.parametrize("log2", [8, 12])
def test_every_box_on_the_way_down_is_tested(gpu, sizes, kind, log2):
    from oibvh_gb300 import DeviceType, OibvhTree, Scene

    # sparse: warps hold a pair or two, and which ones is up to their sharing out
    size = 0.03 if max(sizes) > 1000 else 0.06
    soups = [_soup(n, 7 + i + n, size, kind) for i, n in enumerate(sizes)]
    trees = [OibvhTree(xyz=x, tri=t) for x, t in soups]
    sc = Scene()
    for t in trees:
        t.build()
        sc.addOibvhTree(t)
    if kind == "moved":  # the leaves follow the positions, the boxes above do not
        rng = np.random.default_rng(sum(sizes))
        for t, (x, _) in zip(trees, soups):
            t.set_positions((x + rng.normal(0, 0.05, x.shape)).astype(np.float32))
    sc.set_tuning(start_pairs_log2=log2)
    with np.errstate(invalid="ignore", over="ignore"):
        want = _walk(_Tree(trees[0]), _Tree(trees[1]), _start(*sizes, log2))
    assert want
    for _ in range(3):
        sc.broad(DeviceType.GPU0, 0, 1)
        got = sorted((int(a), int(b)) for _, _, a, b in sc.candidates())
        assert got == want
        sc.detectCollision(DeviceType.GPU0, 0, 1)
        assert sc.candidate_count() == len(want)
