"""Detects beside other work: a kernel that holds most of the GPU for a while,
and other threads' detects, each on a scene and a stream of its own."""
import ctypes
import subprocess
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HOLD = r"""
#include <cuda_runtime.h>
// Holds its SM (its shared memory leaves no room for another CTA) for `ns` nanoseconds.
__global__ void k_hold(unsigned long long ns)
{
    extern __shared__ int room[];
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    for (unsigned i = 0; i < 100000000u; ++i) {
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        if (t - t0 >= ns) break;
        __nanosleep(1000);
    }
    if (threadIdx.x == 0) room[0] = 0;
}
extern "C" int hold(int ctas, unsigned long long ns, void* stream)
{
    const int bytes = 200 * 1024;
    cudaError_t e = cudaFuncSetAttribute(k_hold, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) k_hold<<<ctas, 32, bytes, (cudaStream_t)stream>>>(ns);
    return e == cudaSuccess ? (int)cudaGetLastError() : (int)e;
}
"""


def _soup(n, seed, size):
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


@pytest.fixture(scope="module")
def hold(gpu, tmp_path_factory):
    from oibvh_gb300 import build as B

    d = tmp_path_factory.mktemp("hold")
    (d / "hold.cu").write_text(HOLD)
    subprocess.check_call([B.nvcc_path(), *B.ARCH, "-shared", "-Xcompiler", "-fPIC", "-o", str(d / "hold.so"), str(d / "hold.cu")])
    f = ctypes.CDLL(str(d / "hold.so")).hold
    f.argtypes = [ctypes.c_int, ctypes.c_ulonglong, ctypes.c_void_p]
    return f


@pytest.mark.parametrize("what", ["detect", "precision", "frame", "noalloc"])
def test_a_detect_does_not_wait_for_another_streams_kernel(hold, what):
    import torch

    from oibvh_gb300 import DeviceType
    from oibvh_gb300 import _native as N

    sc = _scene([_soup(n, n, 0.05) for n in (3000, 4000, 5000)])
    if what == "precision":
        sc.set_precision(N.PRECISION_FP64_FILTERED)
    mine, other = torch.cuda.Stream(), torch.cuda.Stream()
    out = torch.empty((1 << 16, 4), dtype=torch.int32, device="cuda")
    n = ctypes.c_uint32(0)
    if what == "frame":
        sc.capture_frame(4, 3, True, stream=mine)

    def run():
        if what == "frame":
            sc.launch_frame(stream=mine)
            sc.finish_frame(stream=mine)
            return sc.getIntTriPairCount()
        if what == "noalloc":
            t = sc._trees
            assert N.lib().oibvh_pair_detect_noalloc(t[0].handle, t[1].handle, 4, ctypes.c_void_p(out.data_ptr()), out.shape[0],
                                                     ctypes.byref(n), ctypes.c_void_p(mine.cuda_stream)) == 0
            return int(n.value)
        sc.detectCollision(DeviceType.GPU0, 4, 3, stream=mine)
        return sc.getIntTriPairCount()

    want = run()  # (queues sized, nothing is allocated in what follows)
    assert run() == want > 0
    torch.cuda.synchronize()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    held = torch.cuda.Event()
    assert hold(2 * sms // 3, 100_000_000, other.cuda_stream) == 0
    held.record(other)
    got = run()
    waited = held.query()
    torch.cuda.synchronize()
    assert got == want
    assert not waited, "the detect came back after the other stream's kernel had ended"


@pytest.mark.parametrize("precision", [0, 1])
def test_detects_of_several_threads(gpu, precision):
    import torch

    from oibvh_gb300 import DeviceType

    def work(k, out):
        try:
            st = torch.cuda.Stream()
            sc = _scene([_soup(n, 10 * k + n, 0.06) for n in (900 + 300 * k, 2500, 700)])
            sc.set_precision(precision)
            sc.detectCollision(DeviceType.GPU0, 4, 3, stream=st)
            want, n = sc.int_tri_pairs(), sc.candidate_count()
            barrier.wait()
            for _ in range(40):
                sc.detectCollision(DeviceType.GPU0, 4, 3, stream=st)
                assert sc.candidate_count() == n and np.array_equal(sc.int_tri_pairs(), want)
            out[k] = (want.shape[0], n)
        except BaseException as e:  # noqa: BLE001
            barrier.abort()
            out[k] = e

    threads = 8
    barrier = threading.Barrier(threads)
    out = [None] * threads
    ts = [threading.Thread(target=work, args=(k, out)) for k in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for r in out:
        if isinstance(r, BaseException):
            raise r
        assert r[0] > 0 and r[1] >= r[0]


def _dense():
    """Two soups whose walk takes more rounds than are launched at first."""
    return [_soup(200000, 1, 0.02), _soup(200000, 2, 0.02)]


def test_walks_go_on_for_as_many_rounds_as_they_need(gpu):
    """A detect's, a frame's and a server batch's first launches cover the
    rounds of lighter work; the rest follows."""
    import torch

    from oibvh_gb300 import DeviceType, OibvhTree, Scene, Server

    soups = _dense()
    trees = [OibvhTree(xyz=x, tri=t) for x, t in soups]
    for t in trees:
        t.build()
    sc = Scene()
    for t in trees:
        sc.addOibvhTree(t)
    sc.detectCollision(DeviceType.GPU0, 4, 3)  # its queues grow
    want, n = sc.int_tri_pairs(), sc.candidate_count()
    assert sc.stats()["steps"] > 4 and want.shape[0] > 10000

    fresh = Scene()
    for t in trees:
        fresh.addOibvhTree(t)
    fresh.set_tuning(front_capacity=sc.tuning()["front_capacity"], hit_capacity=sc.tuning()["hit_capacity"])
    fresh.detectCollision(DeviceType.GPU0, 4, 3)
    assert fresh.stats()["retries"] == 0
    assert np.array_equal(fresh.int_tri_pairs(), want) and fresh.candidate_count() == n

    # a frame captured with the bodies apart
    packed = torch.from_numpy(np.concatenate([np.pad(x, ((0, 0), (0, 1))) for x, _ in soups], 0)).cuda()
    mats = np.tile(np.eye(3, 4, dtype=np.float32).reshape(12), (2, 1))
    mats[1, 3] = 100.0
    d_mats = torch.from_numpy(mats).cuda()
    fresh.capture_frame(4, 3, True, packed.data_ptr(), d_mats.data_ptr())
    fresh.launch_frame()
    fresh.finish_frame()
    assert fresh.candidate_count() == 0 and fresh.stats()["frame_redos"] == 0
    mats[1, 3] = 0.0
    d_mats.copy_(torch.from_numpy(mats))
    for _ in range(2):  # redone, then captured again
        fresh.launch_frame()
        fresh.finish_frame()
        assert np.array_equal(fresh.int_tri_pairs(), want) and fresh.candidate_count() == n

    server = Server(memory_budget=1 << 30, max_batch=16, lanes=2)
    ids = [server.add_mesh(t) for t in trees]
    server.set_queue_capacity(front=sc.tuning()["front_capacity"], hits=sc.tuning()["hit_capacity"])
    server.start()
    for b in (1, 3):
        tickets = [server.submit(ids[0], ids[1], np.eye(3, 4, dtype=np.float32)) for _ in range(b)]
        for t in tickets:
            assert int(server.wait(t)["n_pairs"]) == want.shape[0]
            assert np.array_equal(server.pairs(t), want[:, 2:])
            server.release(t)
    server.close()


def test_a_list_that_runs_over_in_the_last_round_is_measured(gpu):
    """Its size is known although no further round was launched: the queue is
    grown to it, not doubled until it fits."""
    from oibvh_gb300 import DeviceType

    near = _soup(3000, 5, 0.4)
    sc = _scene([near, _soup(3000, 6, 0.4)])
    apart = (near[0] + np.float32(50.0)).astype(np.float32)
    sc._trees[0].refit(apart)
    for _ in range(140):  # light detects: fewer and fewer rounds are launched
        sc.detectCollision(DeviceType.GPU0, 4, 3)
    assert sc.candidate_count() == 0
    sc.set_queue_capacity(front=16)
    sc._trees[0].refit(near[0])
    sc.detectCollision(DeviceType.GPU0, 4, 3)
    st = sc.stats()
    assert st["front_peak"] > 30000  # eleven doublings from 16
    assert st["retries"] <= 4
    want = _scene([near, _soup(3000, 6, 0.4)])
    want.detectCollision(DeviceType.GPU0, 4, 3)
    assert sc.candidate_count() == want.candidate_count() and np.array_equal(sc.int_tri_pairs(), want.int_tri_pairs())


@pytest.mark.parametrize("sizes,precision", [((420000, 400000, 300000), 0), ((200000, 200000), 1), ((3000, 2500, 2000), 1)])
def test_passes_with_a_narrow_phase_behind_them_run_again(gpu, sizes, precision):
    """After light passes too few rounds are launched for a heavy one: its
    narrow phase must not take what the walk has found so far for all of it."""
    from oibvh_gb300 import DeviceType

    near = [_soup(n, 60 + i, 0.01 if n > 10000 else 0.2) for i, n in enumerate(sizes)]
    scenes = [_scene(near) for _ in range(2)]
    for sc in scenes:
        sc.set_precision(precision)
    sc, other = scenes
    other.detectCollision(DeviceType.GPU0, 4, 3)
    want, n, steps = other.int_tri_pairs(), other.candidate_count(), other.stats()["steps"]
    assert want.shape[0] > 0 and steps > 2
    sc.set_tuning(front_capacity=other.tuning()["front_capacity"])
    for _ in range(2):
        for i, t in enumerate(sc._trees):
            t.refit((near[i][0] + np.float32(50.0 * i)).astype(np.float32))
        for _ in range(20):
            sc.detectCollision(DeviceType.GPU0, 4, 3)
            assert sc.candidate_count() == 0
        for i, t in enumerate(sc._trees):
            t.refit(near[i][0])
        for _ in range(2):
            sc.detectCollision(DeviceType.GPU0, 4, 3)
            assert sc.candidate_count() == n and np.array_equal(sc.int_tri_pairs(), want)
