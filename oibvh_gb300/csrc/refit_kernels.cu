// Single-launch bottom-up construction / refit of oibvh trees.
//
// Reference: oibvh_tree_construction_kernel{,2} (src/cuda/oibvh.cu:80-219)
// launched once per level group by OibvhTree::build/refit
// (src/cuda/oibvhTree.cu:193-235,338-357) after calculate_aabb_kernel
// (src/cuda/oibvh.cu:24-40). Here one kernel does all of it, for any number
// of trees at once:
//   * a CTA owns 2^g consecutive Morton-ordered leaves (a level group of g
//     levels, g = 9, 10 or 11, chosen by the tuning; 2^g / 4 threads), four
//     per thread: it loads the four 16-byte face records and the twelve
//     vertices with independent loads, builds the leaf boxes in registers,
//     reduces two levels inside the thread, five across the warp (shuffles)
//     and g - 7 across the CTA (one box per warp through shared memory),
//     writing every internal node it produces;
//   * the CTA finishing last among a group of 2^g sibling subtree roots (one
//     atomic counter per group, threadfence-reduction pattern) loads the
//     group and climbs the next g levels the same way, up to the root.
// No CTA waits for another (no spin loop).
//
// Leaf boxes are not stored: a leaf's box is min/max of its three vertices
// and is recomputed where it is needed (broad-phase tests at the leaf level,
// oibvh_tree_get_aabbs), which removes half of the node writes per refit.
#include "oibvh_common.cuh"
#include "oibvh_launch.h"
#include "refit_device.cuh"

namespace oibvh {

// Level groups: a CTA reduces 2^kLog nodes by kLog levels (four nodes per
// thread), kLog = 9, 10 (default) or 11; the group depth is a tuning knob.
constexpr uint32_t kRefitLogDefault = 10;
constexpr int kStageCounters = 64;  // counters per climbing stage and tree (groups of the widest stage, kLog 9)

// `jobs` == nullptr: a single tree passed by value in `one`. kXyz: its positions
// are still the caller's, in `src`: the CTAs convert them (a slice of the
// vertices each) and take the leaves' corners from the source, so a small
// tree's refit is one launch (320 triangles: a refit and detect pass 62 to
// 55 us). Corners cost four loads so instead of one, which larger trees feel.
// kRest: the trees are moved first, by `mov`: the CTAs write the moved positions
// (a slice each) and move the leaves' corners themselves, so the positions are
// not read back and a launch is saved (12.9 M triangles: 38 us of transforms and
// 155 of refit become 174; 103 M: 314 and 1249 become 1456).
//
// What bounds it: the L1 (70 % busy with gathers and the nodes' 32-byte stores)
// and the chain of a CTA's few steps; DRAM is at 55 %. Measured against four
// leaves a thread, 12.9 M triangles at 160 us: two leaves a thread 184, eight 179;
// 32 neighbouring leaves per load 163; corners that siblings share loaded once 240.
enum RefitFrom { kOwn = 0, kXyz = 1, kRest = 2 };
template <int kLog, int kFrom>
__global__ void __launch_bounds__((1 << kLog) / 4, 1536 / ((1 << kLog) / 4))
    k_refit(const RefitJob* __restrict__ jobs, uint32_t n_jobs, const uint32_t* __restrict__ block_job,
            const RefitJob one, const RefitSource src, const RefitRest mov)
{
    constexpr uint32_t kRefitLog = kLog, kRefitChunk = 1u << kLog;
    __shared__ Box sm8[(1 << kLog) / 128];
    __shared__ uint32_t s_last;

    RefitJob job = one;
    uint32_t ji = 0;
    if (jobs != nullptr && block_job != nullptr) {
        ji = __ldg(block_job + blockIdx.x);
        job = jobs[ji];
    } else if (jobs != nullptr) {
        uint32_t lo = 0, hi = n_jobs - 1;
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if (jobs[mid].block_begin <= blockIdx.x) lo = mid;
            else hi = mid - 1;
        }
        ji = lo;
        job = jobs[lo];
    }
    const TreeShape S = job.shape;
    const uint32_t chunk = blockIdx.x - job.block_begin;
    if constexpr (kFrom == kXyz) {
        float4* pos = const_cast<float4*>(job.pos);
        for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < src.nV; v += gridDim.x * blockDim.x) {
            const float* p = src.xyz + 3 * (size_t)(src.vperm ? __ldg(src.vperm + v) : v);
            pos[v] = make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), 0.0f);
        }
    }
    const float4* corners = job.pos;
    float m[12] = {};
    bool moved = false;
    auto move = [&](const float4& p) { return rigid_move([&](int k) { return m[k]; }, p); };
    if constexpr (kFrom == kRest) {
        const BuildJob& b = mov.jobs[ji];
        const float4* rest = mov.rest ? mov.rest + b.vert_off : b.pos;
        float4* out = b.pos_out;
#pragma unroll
        for (int k = 0; k < 12; ++k) m[k] = __ldg(mov.mats + 12 * (size_t)ji + k);
        // (always so: a tree is refitted from the positions it is moved to. Without the test the compiler
        // spills 72 B a thread, not 52: 103 M triangles 1452 us, not 1426)
        moved = job.pos == out;
        if (moved) corners = rest;
        const uint32_t per = ((b.nV + job.n_blocks - 1) / job.n_blocks + 7u) & ~7u;
        const uint32_t end = min(b.nV, (chunk + 1) * per);
        for (uint32_t v = chunk * per + threadIdx.x; v < end; v += blockDim.x) out[v] = move(__ldg(rest + v));
    }
    if (S.L == 0) return;  // a single leaf: no internal node

    // ---- leaves: calculate_aabb_kernel (src/cuda/oibvh.cu:24-40), in registers ----
    const uint32_t leaf0 = (chunk << kRefitLog) + 4 * threadIdx.x;
    uint4 f[4];
    if (leaf0 + 3 < S.nT) {  // leaf0 is a multiple of 4: 64-byte aligned, two 256-bit loads
        load_face_pair(job.face + leaf0, f[0], f[1]);
        load_face_pair(job.face + leaf0 + 2, f[2], f[3]);
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) f[k] = (leaf0 + k < S.nT) ? __ldg(job.face + leaf0 + k) : make_uint4(0, 0, 0, 0);
    }
    Box v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if constexpr (kFrom == kXyz) {
            auto corner = [&](uint32_t i) {
                const float* p = src.xyz + 3 * (size_t)(src.vperm ? __ldg(src.vperm + i) : i);
                return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), 0.0f);
            };
            v[k] = box_of(corner(f[k].x), corner(f[k].y), corner(f[k].z));
        } else if constexpr (kFrom == kRest) {
            const float4 a = __ldg(corners + f[k].x), b = __ldg(corners + f[k].y), c = __ldg(corners + f[k].z);
            v[k] = moved ? box_of(move(a), move(b), move(c)) : box_of(a, b, c);
        } else {
            v[k] = leaf_box(job.pos, f[k]);
        }
    }

    uint32_t levels = min((uint32_t)kRefitLog, S.L);
    reduce_block<kLog>(v, S, job.box, S.L, chunk << kRefitLog, levels, sm8);
    uint32_t lvl = S.L - levels;
    if (lvl == 0) return;

    // ---- climb: the last CTA of each 1024-node group continues upward ----
    uint32_t idx = chunk;
    for (int stage = 0;; ++stage) {
        const uint32_t g = idx >> kRefitLog;
        const uint32_t gcnt = min(kRefitChunk, S.level_count(lvl) - (g << kRefitLog));
        if (threadIdx.x == 0) {
            __threadfence();
            // (wraps to 0 with the last arrival: nobody has to clear it for the next refit)
            const uint32_t old = atomicInc(job.counters + stage * kStageCounters + g, gcnt - 1);
            s_last = (old == gcnt - 1) ? 1u : 0u;
        }
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        const uint32_t base = g << kRefitLog;
        const uint32_t off = S.level_offset(lvl);
        const uint32_t cnt = S.level_count(lvl);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t j = base + 4 * threadIdx.x + k;
            v[k] = (j < cnt) ? load_node_cg(job.box + 2 * (size_t)(off + j)) : Box{0, 0, 0, 0, 0, 0};
        }
        levels = min((uint32_t)kRefitLog, lvl);
        reduce_block<kLog>(v, S, job.box, lvl, base, levels, sm8);
        lvl -= levels;
        if (lvl == 0) return;
        idx = g;
        __syncthreads();  // s_last and sm8 are reused by the next stage
    }
}

// Leaf boxes of one tree as float4 pairs (for oibvh_tree_get_aabbs).
__global__ void __launch_bounds__(256) k_leaf_boxes(const uint4* __restrict__ face, const float4* __restrict__ xyz,
                                                    uint32_t nT, float4* __restrict__ out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nT) return;
    const Box b = leaf_box(xyz, __ldg(face + i));
    out[2 * (size_t)i] = make_float4(b.nx, b.ny, b.nz, 0.0f);
    out[2 * (size_t)i + 1] = make_float4(b.xx, b.xy, b.xz, 0.0f);
}

uint32_t refit_blocks_for(uint32_t nT, uint32_t group_log2)
{
    const uint32_t g = group_log2 ? group_log2 : kRefitLogDefault;
    return (nT + (1u << g) - 1) >> g;
}
uint32_t refit_counters_per_tree() { return 4 * kStageCounters; }

// A tree of up to this many faces is refitted from the caller's positions in one
// launch, if it has no more vertices than faces (a closed mesh has half as many; or
// a thousand, which one CTA converts as fast as a launch starts). A CTA converts its
// share of the vertices, and there is one for 1024 faces only: 300 faces over 2948
// vertices took 19.4 us in one launch and 19.0 in two, over a million 1315 and 22;
// 4096 faces over 12,288 23.2 and 21.6, over 2050 19.0 (20.9 in two); 32,768 over
// 98,304 24.2 and 23.9, over 16,386 20.1 (22.8).
constexpr uint32_t kRefitXyzMax = 32768, kRefitXyzFew = 1024;
bool refit_takes_xyz(uint32_t nT, uint32_t nV)
{
    return nT <= kRefitXyzMax && nV <= (nT < kRefitXyzFew ? kRefitXyzFew : nT);
}

cudaError_t launch_refit_one(const RefitJob& job, const RefitSource& src, cudaStream_t s)
{
    note_launches(1);
    constexpr uint32_t kThreads = (1u << kRefitLogDefault) / 4;
    if (src.xyz) k_refit<kRefitLogDefault, kXyz><<<job.n_blocks, kThreads, 0, s>>>(nullptr, 1, nullptr, job, src, RefitRest{});
    else k_refit<kRefitLogDefault, kOwn><<<job.n_blocks, kThreads, 0, s>>>(nullptr, 1, nullptr, job, src, RefitRest{});
    return cudaGetLastError();
}

namespace {
template <int kFrom>
cudaError_t launch_many(const RefitJob* d_jobs, uint32_t n_jobs, uint32_t total_blocks, const uint32_t* block_job,
                        uint32_t group_log2, const RefitRest& rest, cudaStream_t s)
{
    if (n_jobs == 0 || total_blocks == 0) return cudaSuccess;
    const RefitJob none{};
    const RefitSource own{};
    note_launches(1);
    switch (group_log2 ? group_log2 : kRefitLogDefault) {
    case 9: k_refit<9, kFrom><<<total_blocks, 128, 0, s>>>(d_jobs, n_jobs, block_job, none, own, rest); break;
    case 10: k_refit<10, kFrom><<<total_blocks, 256, 0, s>>>(d_jobs, n_jobs, block_job, none, own, rest); break;
    case 11: k_refit<11, kFrom><<<total_blocks, 512, 0, s>>>(d_jobs, n_jobs, block_job, none, own, rest); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch_refit(const RefitJob* d_jobs, uint32_t n_jobs, uint32_t total_blocks, const uint32_t* block_job,
                         uint32_t group_log2, cudaStream_t s)
{
    return launch_many<kOwn>(d_jobs, n_jobs, total_blocks, block_job, group_log2, RefitRest{}, s);
}

// A captured frame of this many faces or more is moved by its refit; in smaller ones
// the launch saved is about 2 us, and a frame's profile keeps the two stages apart.
constexpr uint64_t kTransformRefitFaces = 1u << 20;
bool transform_refit_pays(uint64_t n_faces) { return n_faces >= kTransformRefitFaces; }
// A tree's vertices are moved by the CTAs of its faces, 1024 each: one with many more
// vertices than its faces can use would keep the others waiting (300 faces over a
// million vertices: over a millisecond), so that a frame or a server batch with such a
// tree is moved in a launch of its own.
bool transform_refit_takes(uint32_t nT, uint32_t nV) { return nV <= (nT < 1024u ? 4096u : 3u * nT); }

cudaError_t launch_transform_refit(const RefitJob* d_jobs, uint32_t n_jobs, uint32_t total_blocks,
                                   const uint32_t* block_job, uint32_t group_log2, const RefitRest& rest, cudaStream_t s)
{
    return launch_many<kRest>(d_jobs, n_jobs, total_blocks, block_job, group_log2, rest, s);
}

cudaError_t launch_leaf_boxes(const uint4* face, const float4* xyz, uint32_t nT, float4* out, cudaStream_t s)
{
    note_launches(1);
    k_leaf_boxes<<<(nT + 255) / 256, 256, 0, s>>>(face, xyz, nT, out);
    return cudaGetLastError();
}

} // namespace oibvh
