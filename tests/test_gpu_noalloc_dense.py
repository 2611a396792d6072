"""The allocation-free detect with pairs that fill its lists: what its fixed
scratch has room for is found, the rest is refused. The sizes here are some way
inside the room that it has had (a soup of 8,000 triangles, or of 400,000 small
ones, was always too much)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _soup(n, seed, size):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1.0, 1.0, (n, 1, 3))
    return (c + rng.uniform(-size, size, (n, 3, 3))).astype(np.float32).reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


def _ball(triangles, seed):
    from oibvh_gb300 import meshes

    m = meshes.noise_displace(meshes.icosphere(int(np.ceil(np.log(triangles / 20.0) / np.log(4.0) - 1e-9))), 0.05, seed=seed)
    return m.xyz, m.tri[:triangles]


def _sheet(seed):
    from oibvh_gb300 import workloads

    m = workloads.sheet_pair_meshes(256, 0.2, 0.3, 0.3, 0.0, overlap=1.0)[seed]
    return m.xyz, m.tri


PAIRS = {
    "soup": lambda i: _soup(4000, i + 1, 0.4),
    "small_triangles": lambda i: _soup(60000, i + 1, 0.05),
    "touching": lambda i: _ball(327680, 100 + i),
    "coincident": lambda i: _ball(81920, 100),
    "sheets": _sheet,
}


def _detect(trees, level, cap):
    import torch

    from oibvh_gb300 import _native as N

    out = torch.empty((cap, 4), dtype=torch.int32, device="cuda")
    n = ctypes.c_uint32(0)
    torch.cuda.synchronize()
    st = N.lib().oibvh_pair_detect_noalloc(trees[0].handle, trees[1].handle, level, ctypes.c_void_p(out.data_ptr()), cap,
                                           ctypes.byref(n), None)
    return st, out[: min(cap, n.value)].cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("pair", sorted(PAIRS))
@pytest.mark.parametrize("level", [0, 4, 10])
def test_dense_pairs_fit(gpu, pair, level):
    from oibvh_gb300 import DeviceType, OibvhTree, Scene
    from oibvh_gb300 import _native as N

    trees = [OibvhTree(xyz=x, tri=t) for x, t in (PAIRS[pair](0), PAIRS[pair](1))]
    sc = Scene()
    for t in trees:
        t.build()
        sc.addOibvhTree(t)
    sc.detectCollision(DeviceType.GPU0, 4, 3)
    want = sc.int_tri_pairs()
    for _ in range(2):
        st, got = _detect(trees, level, want.shape[0] + 1000)
        assert st == 0, N.lib().oibvh_last_error().decode()
        got = got[np.lexsort((got[:, 3], got[:, 2], got[:, 1], got[:, 0]))]
        assert np.array_equal(got, want)


def test_pairs_past_the_scratch_are_refused(gpu):
    from oibvh_gb300 import OibvhTree
    from oibvh_gb300 import _native as N

    trees = [OibvhTree(xyz=x, tri=t) for x, t in (_soup(20000, 1, 0.4), _soup(20000, 2, 0.4))]
    for t in trees:
        t.build()
    assert _detect(trees, 4, 1 << 22)[0] == N.ERR_OVERFLOW
    small = [OibvhTree(xyz=x, tri=t) for x, t in (_soup(500, 1, 0.1), _soup(500, 2, 0.1))]
    for t in small:
        t.build()
    assert _detect(small, 4, 1 << 16)[0] == 0  # nothing of the refused call is left behind
