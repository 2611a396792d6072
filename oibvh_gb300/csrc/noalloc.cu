// oibvh_pair_detect_noalloc: collision detection for one mesh pair that
// allocates no memory at all, neither on the device nor pinned on the host.
//
// Who needs it: callers that must not allocate while they run. A physics or
// robotics step with a hard frame budget cannot afford cudaMalloc, which may
// synchronise the whole device and take an unbounded time; an application
// whose device memory is owned by an outside pool allocator (all of it
// reserved up front) may not create allocations of its own.
// oibvh_scene_detect grows its queues on demand; this entry point instead
// runs the same traversal kernels over a fixed scratch area that lives in
// this file.
//
// The scratch is a file-scope __device__ array: every GPU that loads the
// library holds it (kNoAllocBytes, about 4 MB) until the process exits. Host
// code cannot use the array's name as a device address, so the first call on
// a device (with that device current) resolves the address with
// cudaGetSymbolAddress and caches it together with the id of the device's
// context; make that first call at start-up. A later call in a
// new context (after cudaDeviceReset) resolves it again. Every call shares
// the one array: the counters are cleared at the start of each call, and
// calls whose GPU work overlaps (several host threads, or several streams)
// race on it and must be serialised by the caller.
#include <cstring>
#include <mutex>
#include <string>

#include "../../include/oibvh_gb300.h"
#include "oibvh_common.cuh"
#include "oibvh_launch.h"

namespace oibvh {

// Fixed capacity of each of the two traversal work lists (BVTT node pairs).
constexpr uint32_t kNoAllocItems = 1u << 18;
// Rounds that go out before the host looks whether anything is left (most pairs take two to four).
constexpr uint32_t kNoAllocRounds = 3;
// Header: the counters, rounded up (the pair's record goes with the kernels' arguments).
constexpr size_t kNoAllocHeader = 4096;
constexpr size_t kNoAllocBytes = kNoAllocHeader + 2 * (size_t)kNoAllocItems * sizeof(uint64_t);

static_assert(kCountTotal * sizeof(uint32_t) <= kNoAllocHeader, "header fits");

__device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

// Defined in host.cu: the device view of a tree handle.
int tree_device_view(oibvh_tree_t t, TreeView* out, int* device, bool* built);
int noalloc_fail(int code, const std::string& msg);

namespace {

std::mutex g_scratch_mu;
unsigned char* g_scratch_addr[64] = {};
unsigned long long g_scratch_ctx[64] = {};  // id of the context the address belongs to

// Device address of g_noalloc_scratch on `dev` (the current device, its
// context already initialised by the caller).
int scratch_address(int dev, unsigned char** out)
{
    if (dev < 0 || dev >= 64) return noalloc_fail(OIBVH_ERR_UNSUPPORTED, "device index above 63");
    const unsigned long long ctx = current_context_id();
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_addr[dev] || ctx != g_scratch_ctx[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess)
            return noalloc_fail(OIBVH_ERR_CUDA, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
        g_scratch_addr[dev] = (unsigned char*)p;
        g_scratch_ctx[dev] = current_context_id();
    }
    *out = g_scratch_addr[dev];
    return OIBVH_OK;
}

#define NA_CUDA(expr)                                                                                   \
    do {                                                                                                \
        const cudaError_t _e = (expr);                                                                  \
        if (_e != cudaSuccess) return noalloc_fail(OIBVH_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(_e)); \
    } while (0)

}  // namespace

}  // namespace oibvh

using namespace oibvh;

extern "C" __attribute__((visibility("default"))) int oibvh_pair_detect_noalloc(
    oibvh_tree_t a, oibvh_tree_t b, uint32_t entry_level, uint32_t* d_out4, uint32_t out_cap, uint32_t* n_hits,
    void* stream)
{
    try {
        if (!a || !b || !n_hits) return noalloc_fail(OIBVH_ERR_ARG, "a, b or n_hits is NULL");
        if (out_cap && !d_out4) return noalloc_fail(OIBVH_ERR_ARG, "d_out4 is NULL");
        if (((uintptr_t)d_out4) % 16)
            return noalloc_fail(OIBVH_ERR_ARG, "d_out4 must be 16-byte aligned (the kernels store 16-byte records)");
        *n_hits = 0;
        TreeView trees[2] = {};
        PairView pair{};
        int dev_a = -1, dev_b = -1;
        bool built_a = false, built_b = false;
        int st = tree_device_view(a, &trees[0], &dev_a, &built_a);
        if (st == OIBVH_OK) st = tree_device_view(b, &trees[1], &dev_b, &built_b);
        if (st != OIBVH_OK) return st;
        if (!built_a || !built_b) return noalloc_fail(OIBVH_ERR_STATE, "both trees must be built");
        if (dev_a != dev_b) return noalloc_fail(OIBVH_ERR_ARG, "the trees live on different devices");
        int cur = -1;
        NA_CUDA(cudaGetDevice(&cur));
        if (cur != dev_a) NA_CUDA(cudaSetDevice(dev_a));
        struct Restore {
            int d, c;
            ~Restore()
            {
                if (d != c) cudaSetDevice(c);
            }
        } restore{dev_a, cur};

        unsigned char* base = nullptr;
        st = scratch_address(dev_a, &base);
        if (st != OIBVH_OK) return st;

        // start level: the entry level, deepened to a ~2^16-pair cross product (as oibvh_scene_detect)
        const TreeShape& A = trees[0].shape;
        const TreeShape& B = trees[1].shape;
        const uint32_t start = entry_level > 8u ? entry_level : 8u;
        pair.a = 0;
        pair.b = 1;
        pair.ta = trees[0];
        pair.tb = trees[1];
        pair.front_off = 0;
        pair.entry_a = start < A.L ? start : A.L;
        pair.entry_b = start < B.L ? start : B.L;
        pair.front_cnt_a = A.level_count(pair.entry_a);
        pair.front_cnt_b = B.level_count(pair.entry_b);
        const uint64_t total0 = (uint64_t)pair.front_cnt_a * pair.front_cnt_b;
        if (total0 > (uint64_t)64 * kNoAllocItems)
            return noalloc_fail(OIBVH_ERR_ARG, "entry level " + std::to_string(entry_level) + " starts from " +
                                                   std::to_string(total0) + " node pairs; the fixed scratch allows " +
                                                   std::to_string((uint64_t)64 * kNoAllocItems));

        cudaStream_t s = (cudaStream_t)stream;
        uint32_t* d_counts = (uint32_t*)base;
        DetectArgs args{};
        args.n_pairs = 1;
        args.one = pair;
        args.work[0] = (uint64_t*)(base + kNoAllocHeader);
        args.work[1] = args.work[0] + kNoAllocItems;
        args.work_cap = kNoAllocItems;
        args.hits = (uint4*)d_out4;
        args.hit_cap = out_cap;
        args.counts = d_counts;
        args.fuse_narrow = 1;
        int sms = 1, per_sm = walk_blocks_per_sm();
        NA_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev_a));
        args.grid = sms * per_sm;

        uint32_t counts[kCountHost];
        for (;;) {
            NA_CUDA(launch_begin(args, 0, s));
            for (uint32_t r = 0;; r += kNoAllocRounds) {
                NA_CUDA(launch_walk(args, (uint32_t)total0, r, r + kNoAllocRounds, true, s));
                NA_CUDA(cudaMemcpyAsync(counts, d_counts, sizeof(counts), cudaMemcpyDeviceToHost, s));
                NA_CUDA(cudaStreamSynchronize(s));
                if (counts[kCountFlags] || counts[kCountLeft] == 0) break;
            }
            // The lists cannot grow. Sharing the pairs out every few steps takes more of them than walking on
            // from where they are, so a pair whose lists ran over is walked again that way before it is refused.
            if (!(counts[kCountFlags] & kFlagFrontOverflow) || args.stay) break;
            args.stay = 1;
            args.start_steps = args.walk_steps = 0xffffffffu;
        }
        *n_hits = counts[kCountHits];
        if (counts[kCountFlags] & kFlagFrontOverflow)
            return noalloc_fail(OIBVH_ERR_OVERFLOW, "the pair needs more than " + std::to_string(kNoAllocItems) +
                                                        " queued node pairs, the fixed scratch; use oibvh_scene_detect");
        if (counts[kCountFlags] & kFlagHitOverflow)
            return noalloc_fail(OIBVH_ERR_OVERFLOW, "out_cap is too small: " + std::to_string(counts[kCountHits]) +
                                                        " colliding pairs (in *n_hits)");
        if (counts[kCountFlags]) return noalloc_fail(OIBVH_ERR_STATE, "unexpected device flag");
        return OIBVH_OK;
    } catch (...) {
        return noalloc_fail(OIBVH_ERR_CUDA, "unexpected C++ exception");
    }
}
