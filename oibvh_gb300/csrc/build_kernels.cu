// Build-time kernels: mesh bounds, Morton codes, their stable LSD radix sort,
// the sorted face records and the vertex renumbering, for any number of trees
// in one launch a stage; and the rigid transform of every tree's vertices in
// one launch.
//
// Reference: src/cuda/oibvh.cu:6-70 (strech_by_3, morton3D,
// calculate_aabb_and_morton_kernel) and src/cuda/oibvhTree.cu:253-299
// (mesh bounds from Mesh::m_aabb, two thrust::stable_sort_by_key calls).
// Here one stable sort of (code, face index) replaces the two payload sorts
// and the permutation is kept, so faces are gathered once into a 16-byte
// record (v0, v1, v2, original index). Keys are the reference's 30 bits, or
// 63 bits (21 per axis) as an option, sorted 8 bits a pass.
#include "oibvh_common.cuh"
#include "oibvh_launch.h"
#include "refit_device.cuh"

#include <atomic>

namespace oibvh {

// Floats as unsigned keys of the same order.
__device__ __forceinline__ uint32_t float_to_ordered(float f)
{
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ordered_to_float(uint32_t k)
{
    const uint32_t b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(b);
}

// Positions as given (x, y, z) to the device layout (x, y, z, 0): one
// 16-byte vector load per vertex everywhere else.
// Positions in the tree's vertex order: tree vertex v is the caller's vertex
// vperm[v] (vperm == nullptr: the caller's order).
__global__ void __launch_bounds__(256) k_xyz_to_pos4(const float* __restrict__ xyz, const uint32_t* __restrict__ vperm,
                                                     uint32_t nV, float4* __restrict__ pos)
{
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nV) return;
    const size_t u = vperm ? __ldg(vperm + v) : v;
    pos[v] = make_float4(__ldg(xyz + 3 * u), __ldg(xyz + 3 * u + 1), __ldg(xyz + 3 * u + 2), 0.0f);
}
__global__ void __launch_bounds__(256) k_gather_pos4(const float4* __restrict__ src, const uint32_t* __restrict__ vperm,
                                                     uint32_t nV, float4* __restrict__ pos)
{
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nV) return;
    pos[v] = __ldg(src + (vperm ? __ldg(vperm + v) : v));
}

// Morton codes (src/cuda/oibvh.cu:6-22).
__device__ __forceinline__ uint32_t stretch3(uint32_t x)
{
    x &= 0x3ffu;
    x = (x | (x << 16)) & 0x30000ffu;
    x = (x | (x << 8)) & 0x300f00fu;
    x = (x | (x << 4)) & 0x30c30c3u;
    x = (x | (x << 2)) & 0x9249249u;
    return x;
}

// 21 bits -> every third bit of 63 (the wide key: 21 bits per axis)
__device__ __forceinline__ uint64_t stretch3_21(uint32_t v)
{
    uint64_t x = v & 0x1fffffu;
    x = (x | (x << 32)) & 0x1f00000000ffffull;
    x = (x | (x << 16)) & 0x1f0000ff0000ffull;
    x = (x | (x << 8)) & 0x100f00f00f00f00full;
    x = (x | (x << 4)) & 0x10c30c30c30c30c3ull;
    x = (x | (x << 2)) & 0x1249249249249249ull;
    return x;
}

// The wide key's quantisation: as quant1024 with 2^21 cells per axis (the
// scaling by 2^21 is exact, the clamp bound 2^21 - 1 is a float).
__device__ __forceinline__ uint32_t quant2m(float u)
{
    float v = __fmul_rn(u, 2097152.0f);
    v = (v < 0.0f) ? 0.0f : v;
    v = (2097151.0f < v) ? 2097151.0f : v;
    return __float2uint_rz(v);  // NaN -> 0
}

// The key of a leaf from its three cell coordinates: 30 bits (the
// reference's morton3D, x << 2 | y << 1 | z) in `lo`, or 63 bits (same
// interleave, 21 bits per axis) split into `lo` (bits 0..31) and `hi`.
__device__ __forceinline__ void morton_key(const float u[3], bool wide, uint32_t& lo, uint32_t& hi);

__device__ __forceinline__ uint32_t quant1024(float u)
{
    float v = __fmul_rn(u, 1024.0f);
    v = (v < 0.0f) ? 0.0f : v;        // thrust::max(v, 0.0f)
    v = (1023.0f < v) ? 1023.0f : v;  // thrust::min(v, 1023.0f)
    return __float2uint_rz(v);        // NaN -> 0
}

__device__ __forceinline__ void morton_key(const float u[3], bool wide, uint32_t& lo, uint32_t& hi)
{
    if (!wide) {
        lo = (stretch3(quant1024(u[0])) << 2) | (stretch3(quant1024(u[1])) << 1) | stretch3(quant1024(u[2]));
        hi = 0;
        return;
    }
    const uint64_t k = (stretch3_21(quant2m(u[0])) << 2) | (stretch3_21(quant2m(u[1])) << 1) | stretch3_21(quant2m(u[2]));
    lo = (uint32_t)k;
    hi = (uint32_t)(k >> 32);
}

// ---------------------------------------------------------------------------
// The build of any number of trees: every stage is one launch for all of them
// (a scene build) or for one (a tree build). Faces and vertices are cut into
// tiles of 4096 that never straddle trees; a host-built map names a tile's
// tree.
//
//   k_build_vertices  mesh bounds; first-use slots cleared
//   k_build_codes     Morton codes, and the digit histograms of every pass
//   k_build_sort x 4  one stable radix pass over 8 bits each (x 8 for 63-bit
//                     keys); the last one writes the sorted face records and
//                     each vertex's first use instead of keys
//   k_build_mark, k_build_count, k_build_place
//                     new vertex numbers in order of first use
//   k_build_apply     faces and positions in the new numbering
//
// A tile's share of a running count (digits of a pass, first uses) is its
// tree's sum over the tiles before it, taken by decoupled look-back (Merrill
// and Garland, "Single-pass parallel prefix scan with decoupled look-back",
// 2016; for radix passes Adinets and Merrill, "Onesweep", 2022): a tile
// publishes its own count, then adds up its predecessors' from the nearest on
// until one has published its whole sum. CTAs take their tiles from a counter,
// so the tiles waited for are running or done; a wait has a limit, after which
// the build is given up (BuildScratch::fail).
// ---------------------------------------------------------------------------
constexpr uint32_t kNoUse = 0xffffffffu;
constexpr uint32_t kTileWords = 3 * kBuildTile / 32;  // a bit per face corner of a tile
constexpr uint32_t kStateSum = 1u << 30, kStateTotal = 2u << 30, kStateValue = kStateSum - 1u;

__device__ __forceinline__ const BuildJob& job_of(const BuildArgs& a, const uint32_t* map, uint32_t tile, uint32_t& j)
{
    j = a.jobs ? __ldg(map + tile) : 0u;
    return a.jobs ? a.jobs[j] : a.one;
}
__device__ __forceinline__ uint32_t ld_state(const uint32_t* p) { return *(const volatile uint32_t*)p; }
__device__ __forceinline__ void st_state(uint32_t* p, uint32_t v) { *(volatile uint32_t*)p = v; }
__device__ __forceinline__ void give_up(const BuildArgs& a)
{
    st_state(a.sc.fail, 1u);
    *(volatile uint32_t*)a.host_error = 1u;  // pinned host memory
    __threadfence_system();
}

// Bounds of each mesh (src/utils/mesh.cpp:91-98) as order-preserving keys:
// maxima of the coordinates and of their complements (so 0 is neutral for
// both). One atomic per CTA and bound: with one per warp the 14 M vertices of
// 128 meshes took 573 us, queueing at six words a mesh.
__global__ void __launch_bounds__(256) k_build_vertices(const __grid_constant__ BuildArgs a)
{
    __shared__ uint32_t s_red[6][8];
    uint32_t j;
    const BuildJob& job = job_of(a, a.vtile_job, blockIdx.x >> 2, j);
    const uint32_t base = ((blockIdx.x >> 2) - job.vtile_begin) * kBuildTile + (blockIdx.x & 3u) * 1024u;
    if (base >= job.nV) return;
    uint32_t red[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        const uint32_t v = base + k * 256u + threadIdx.x;
        if (v >= job.nV) continue;
        const float4 p = __ldg(job.pos + v);
        const float c[3] = {p.x, p.y, p.z};
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const uint32_t o = float_to_ordered(c[i]);
            red[i] = max(red[i], ~o);
            red[3 + i] = max(red[3 + i], o);
        }
        a.sc.first[job.vert_off + v] = kNoUse;
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        red[i] = __reduce_max_sync(0xffffffffu, red[i]);
        if ((threadIdx.x & 31) == 0) s_red[i][threadIdx.x >> 5] = red[i];
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        uint32_t m = 0;
        for (int w = 0; w < 8; ++w) m = max(m, s_red[threadIdx.x][w]);
        atomicMax(a.sc.bounds + 6 * j + threadIdx.x, m);
    }
}

// The leaf's Morton code (src/cuda/oibvh.cu:6-22,42-70): the float operations
// are the reference's, each rounded on its own (the *0.5f and the quantiser's
// scaling are exact, the one division is IEEE round-to-nearest).
__device__ __forceinline__ void leaf_code(const float va[3], const float vb[3], const float vc[3], const float bmin[3],
                                          const float bmax[3], bool wide, uint32_t& lo, uint32_t& hi)
{
    float u[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float mn = gmin(gmin(va[k], vb[k]), vc[k]), mx = gmax(gmax(va[k], vb[k]), vc[k]);
        const float centroid = __fmul_rn(__fadd_rn(mn, mx), 0.5f);
        u[k] = __fdiv_rn(__fsub_rn(centroid, bmin[k]), __fsub_rn(bmax[k], bmin[k]));
    }
    morton_key(u, wide, lo, hi);
}

template <bool kWide>
__global__ void __launch_bounds__(256) k_build_codes(const __grid_constant__ BuildArgs a)
{
    constexpr uint32_t P = kWide ? 8 : 4;
    __shared__ uint32_t s_hist[P * 256];
    uint32_t j;
    const BuildJob& job = job_of(a, a.ftile_job, blockIdx.x >> 2, j);
    const uint32_t base = ((blockIdx.x >> 2) - job.ftile_begin) * kBuildTile + (blockIdx.x & 3u) * 1024u;
    if (base >= job.nT) return;
    for (uint32_t i = threadIdx.x; i < P * 256; i += 256) s_hist[i] = 0;
    float bmin[3], bmax[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        bmin[k] = ordered_to_float(~a.sc.bounds[6 * j + k]);
        bmax[k] = ordered_to_float(a.sc.bounds[6 * j + 3 + k]);
    }
    uint32_t f[4][3];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        const uint32_t i = base + k * 256u + threadIdx.x;
        const uint32_t* t = job.tri + 3 * (size_t)(i < job.nT ? i : 0u);
        f[k][0] = __ldg(t);
        f[k][1] = __ldg(t + 1);
        f[k][2] = __ldg(t + 2);
    }
    __syncthreads();
#pragma unroll
    for (uint32_t h = 0; h < 4; h += 2) {
        float4 p[2][3];
#pragma unroll
        for (uint32_t k = 0; k < 2; ++k)
#pragma unroll
            for (uint32_t c = 0; c < 3; ++c) p[k][c] = __ldg(job.pos + f[h + k][c]);
#pragma unroll
        for (uint32_t k = 0; k < 2; ++k) {
            const uint32_t i = base + (h + k) * 256u + threadIdx.x;
            if (i >= job.nT) continue;
            const float va[3] = {p[k][0].x, p[k][0].y, p[k][0].z}, vb[3] = {p[k][1].x, p[k][1].y, p[k][1].z},
                        vc[3] = {p[k][2].x, p[k][2].y, p[k][2].z};
            uint32_t lo, hi;
            leaf_code(va, vb, vc, bmin, bmax, kWide, lo, hi);
            a.sc.keys[0][job.face_off + i] = lo;
            if (kWide) a.sc.hi[job.face_off + i] = hi;
#pragma unroll
            for (uint32_t p = 0; p < P; ++p) atomicAdd(&s_hist[p * 256 + (((p < 4 ? lo : hi) >> (8 * (p & 3))) & 255u)], 1u);
        }
    }
    __syncthreads();
    uint32_t* hist = a.sc.hist + (size_t)j * P * 256;
    for (uint32_t i = threadIdx.x; i < P * 256; i += 256)
        if (s_hist[i]) atomicAdd(hist + i, s_hist[i]);
}

// Exclusive scan of one value per thread over threads 0..255 of the CTA (every
// thread calls; the others pass anything and get garbage).
__device__ __forceinline__ uint32_t scan_256(uint32_t v, uint32_t* sh /*[8]*/)
{
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, s);
        if ((int)lane >= s) x += y;
    }
    if (lane == 31 && w < 8) sh[w] = x;
    __syncthreads();
    uint32_t pre = 0;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) pre += i < w ? sh[i] : 0u;
    __syncthreads();
    return pre + x - v;
}

// One pass of the stable LSD radix sort: a CTA ranks a tile of 4096 or 2048 items
// (groups of equal digits in item order), reorders them in shared memory
// so that each digit's items leave as one run, and writes them behind those of
// the tree's earlier tiles. kFirst: the values are the item numbers (not read);
// kLast: the sorted faces are gathered and written with each vertex's first
// use, instead of keys and values. `swap_hi`: the key written is the item's
// high word (the pass between the two halves of a 63-bit key).
// Builds whose tiles are fewer than the SMs' share cut each in two for the
// passes (kHalf), so that twice as many CTAs work half as long.
constexpr uint32_t kSortThreads = 512, kSortWarps = kSortThreads / 32;

template <bool kFirst, bool kLast, bool kHalf>
__global__ void __launch_bounds__(kSortThreads, 2) k_build_sort(const __grid_constant__ BuildArgs a, uint32_t pass, bool swap_hi)
{
    constexpr uint32_t kTile = kHalf ? kBuildTile / 2 : kBuildTile, kSortItems = kTile / kSortThreads;
    __shared__ uint16_t s_cnt[kSortWarps][256];
    __shared__ union {
        uint32_t peers[kSortWarps][256];  // of a row of 32 items: the lanes with this digit
        struct {
            uint32_t key[kTile], val[kTile];
        } out;
    } sh;
    uint32_t *s_key = sh.out.key, *s_val = sh.out.val;
    __shared__ uint32_t s_base[256], s_start[256], s_sh[8], s_tile, s_bad;
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const uint32_t shift = 8 * (pass & 3u);
    if (tid == 0) {
        s_tile = atomicAdd(a.sc.tickets + pass, 1u);
        s_bad = ld_state(a.sc.fail);
    }
    for (uint32_t i = tid; i < kSortWarps * 128; i += kSortThreads) ((uint32_t*)s_cnt)[i] = 0;
    for (uint32_t i = tid; i < kSortWarps * 256; i += kSortThreads) (&sh.peers[0][0])[i] = 0;
    __syncthreads();
    if (s_bad) return;
    const uint32_t tile = s_tile;
    uint32_t j;
    const BuildJob& job = job_of(a, a.ftile_job, kHalf ? tile >> 1 : tile, j);
    const uint32_t chain = kHalf ? 2u * job.ftile_begin : job.ftile_begin, t0 = tile - chain;
    const uint32_t n = t0 * kTile < job.nT ? min(kTile, job.nT - t0 * kTile) : 0u;  // (a tree's last half may be empty)
    const uint32_t* kin = a.sc.keys[pass & 1] + job.face_off + t0 * kTile;
    const uint32_t* vin = a.sc.vals[pass & 1] + job.face_off + t0 * kTile;
    uint32_t* state = a.sc.sort_state[pass & 1];
    uint32_t key[kSortItems], val[kSortItems];
    uint16_t rank[kSortItems];
    const uint32_t i0 = w * (32 * kSortItems) + lane;
#pragma unroll
    for (uint32_t r = 0; r < kSortItems; ++r) {
        const uint32_t i = i0 + 32 * r;
        key[r] = i < n ? kin[i] : 0u;
        val[r] = kFirst ? t0 * kTile + i : i < n ? vin[i] : 0u;
    }
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (uint32_t r = 0; r < kSortItems; ++r) {
        const bool valid = i0 + 32 * r < n;
        const uint32_t d = (key[r] >> shift) & 255u;
        // the row's lanes of the same digit, by a bit each in the digit's word (with eight ballots
        // instead a pass took 100 us, not 92, for 12.9 M faces; __match_any_sync: 140)
        if (valid) atomicOr(&sh.peers[w][d], 1u << lane);
        __syncwarp();
        uint32_t peers = 0, b = 0;
        if (valid) {
            peers = sh.peers[w][d];
            b = s_cnt[w][d];
        }
        rank[r] = (uint16_t)(b + __popc(peers & lt));
        __syncwarp();
        if (valid && (peers & lt) == 0) {
            s_cnt[w][d] = (uint16_t)(b + __popc(peers));
            sh.peers[w][d] = 0;
        }
        __syncwarp();
    }
    __syncthreads();
    uint32_t cnt = 0, digits = 0;
    if (tid < 256) {
#pragma unroll
        for (uint32_t i = 0; i < kSortWarps; ++i) {
            const uint32_t c = s_cnt[i][tid];
            s_cnt[i][tid] = (uint16_t)cnt;
            cnt += c;
        }
        st_state(state + (size_t)tile * 256 + tid, (t0 == 0 ? kStateTotal : kStateSum) | cnt);
        a.sc.sort_state[(pass + 1) & 1][(size_t)tile * 256 + tid] = 0;  // for the next pass
        digits = a.sc.hist[((size_t)j * a.passes + pass) * 256 + tid];
    }
    const uint32_t start = scan_256(cnt, s_sh);
    const uint32_t first = scan_256(digits, s_sh);
    if (tid < 256) s_start[tid] = start;
    __syncthreads();
#pragma unroll
    for (uint32_t r = 0; r < kSortItems; ++r) {
        if (i0 + 32 * r < n) {
            const uint32_t d = (key[r] >> shift) & 255u;
            const uint32_t q = s_start[d] + s_cnt[w][d] + rank[r];
            s_key[q] = key[r];
            s_val[q] = val[r];
        }
    }
    if (tid < 256) {
        // this digit's items in the tree's earlier tiles: eight predecessors per round of loads
        uint32_t before = 0, polls = 0;
        bool done = t0 == 0;
        for (uint32_t k = tile; !done;) {
            uint32_t v[8];
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q)
                v[q] = q < k - chain ? ld_state(state + (size_t)(k - q - 1) * 256 + tid) : 0u;
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q) {
                if (done || v[q] == 0) break;
                before += v[q] & kStateValue;
                done = (v[q] & kStateTotal) != 0;
                --k;
            }
            if (!done && ++polls > a.polls) {
                s_bad = 1;
                break;
            }
        }
        if (t0 != 0 && done) st_state(state + (size_t)tile * 256 + tid, kStateTotal | (before + cnt));
        s_base[tid] = first + before - start;
    }
    __syncthreads();
    if (s_bad) {
        if (tid == 0) give_up(a);
        return;
    }
    uint32_t* kout = a.sc.keys[(pass + 1) & 1] + job.face_off;
    uint32_t* vout = a.sc.vals[(pass + 1) & 1] + job.face_off;
    const uint32_t* hi = a.sc.hi + job.face_off;
#pragma unroll
    for (uint32_t r = 0; r < kSortItems; ++r) {
        const uint32_t q = r * kSortThreads + tid;
        if (q - lane >= n) break;  // (the whole warp: the ballot names every lane)
        const uint32_t row = __ballot_sync(0xffffffffu, q < n);
        if (q >= n) continue;
        const uint32_t k = s_key[q], o = s_val[q], dst = s_base[(k >> shift) & 255u] + q;
        if (kLast) {
            const uint32_t* t = job.tri + 3 * (size_t)o;
            const uint32_t x = __ldg(t), y = __ldg(t + 1), z = __ldg(t + 2);
            job.face_out[dst] = make_uint4(x, y, z, o);
            uint32_t* use = a.sc.first + job.vert_off;
            // (a corner that the face before has too is not its vertex's first use: half of them, on a
            // mesh, and the pass over 12.9 M faces takes 196 us, not 227)
            const uint32_t u = __shfl_up_sync(row, x, 1), v = __shfl_up_sync(row, y, 1), t2 = __shfl_up_sync(row, z, 1);
            if (lane == 0 || (x != u && x != v && x != t2)) atomicMin(use + x, 3u * dst);
            if (lane == 0 || (y != u && y != v && y != t2)) atomicMin(use + y, 3u * dst + 1u);
            if (lane == 0 || (z != u && z != v && z != t2)) atomicMin(use + z, 3u * dst + 2u);
        } else {
            kout[dst] = swap_hi ? __ldg(hi + o) : k;
            vout[dst] = o;
        }
    }
}

// This block's running count: `mine` (of the whole CTA) published, and the sum
// over the chain's earlier blocks [chain, block). Called by warp 0; false: gave up.
__device__ __forceinline__ bool lookback(const BuildArgs& a, uint32_t* state, uint32_t chain, uint32_t block, uint32_t mine,
                                         uint32_t& before)
{
    const uint32_t lane = threadIdx.x & 31;
    before = 0;
    if (block == chain) {
        if (lane == 0) st_state(state + block, kStateTotal | mine);
        return true;
    }
    if (lane == 0) st_state(state + block, kStateSum | mine);
    uint32_t polls = 0;
    for (uint32_t b = block;;) {  // lane l looks at block b - 1 - l
        const bool in = b > chain + lane;
        const uint32_t v = in ? ld_state(state + b - 1 - lane) : kStateTotal;
        const uint32_t empty = __ballot_sync(0xffffffffu, v == 0), total = __ballot_sync(0xffffffffu, (v & kStateTotal) != 0);
        const uint32_t upto = total ? (uint32_t)__ffs(total) - 1u : 31u;  // lanes 0 .. upto count
        if (empty & (0xffffffffu >> (31u - upto))) {
            if (++polls > a.polls) return false;
            continue;
        }
        before += __reduce_add_sync(0xffffffffu, lane <= upto ? v & kStateValue : 0u);
        if (total) break;
        b -= 32;
    }
    if (lane == 0) st_state(state + block, kStateTotal | (before + mine));
    return true;
}

// New vertex numbers, in the order in which the sorted faces first use them (so
// that the refit's and the traversal's vertex gathers for neighbouring leaves
// fall on nearby positions; the caller's order is arbitrary), unused vertices
// last in their previous order. A vertex's number is the count of first uses
// (of unused vertices) before its own: a bit per face corner marks the first
// uses, running counts are kept per 32 corners, and everything that follows
// works vertex by vertex. (Going through the faces instead, each corner looking
// up whether it is its vertex's first use, took 361 us for 12.9 M faces against
// 113 us for these three kernels.) What bounds them is chains of loads with little
// to do in between, so a thread issues those of its four vertices together
// (k_build_place 71 to 63 us, k_build_apply 159 to 151), and the unused are counted
// here, where first uses are read anyway (k_build_count 48 to 23).
__global__ void __launch_bounds__(256) k_build_mark(const __grid_constant__ BuildArgs a)
{
    __shared__ uint32_t s_unused;
    if (ld_state(a.sc.fail)) return;
    if (threadIdx.x == 0) s_unused = 0;
    __syncthreads();
    uint32_t j;
    const BuildJob& job = job_of(a, a.vtile_job, blockIdx.x >> 2, j);
    const uint32_t base = ((blockIdx.x >> 2) - job.vtile_begin) * kBuildTile + (blockIdx.x & 3u) * 1024u + threadIdx.x;
    uint32_t* marks = a.sc.marks + (size_t)job.ftile_begin * kTileWords;
    uint32_t n_unused = 0;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        const uint32_t v = base + 256u * k;
        const uint32_t s = v < job.nV ? __ldg(a.sc.first + job.vert_off + v) : 0u;
        if (v >= job.nV) continue;
        if (s != kNoUse) atomicOr(marks + (s >> 5), 1u << (s & 31));
        else ++n_unused;
    }
    n_unused = __reduce_add_sync(0xffffffffu, n_unused);
    if ((threadIdx.x & 31) == 0 && n_unused) atomicAdd(&s_unused, n_unused);
    __syncthreads();
    if (threadIdx.x == 0) a.sc.unused[blockIdx.x] = s_unused;
}

// Running counts: CTAs [0, f_tiles) of the marks (per word), the rest of the
// unused vertices (per 1024), in ticket order.
__global__ void __launch_bounds__(128) k_build_count(const __grid_constant__ BuildArgs a)
{
    __shared__ uint32_t s_w[4], s_tile, s_before, s_bad;
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid == 0) {
        s_tile = atomicAdd(a.sc.tickets + 8, 1u);
        s_bad = ld_state(a.sc.fail);
    }
    __syncthreads();
    if (s_bad) return;
    const bool faces = s_tile < a.f_tiles;
    const uint32_t tile = faces ? s_tile : s_tile - a.f_tiles;
    uint32_t j;
    const BuildJob& job = faces ? job_of(a, a.ftile_job, tile, j) : job_of(a, a.vtile_job, tile, j);
    const uint32_t chain = faces ? job.ftile_begin : job.vtile_begin;
    constexpr uint32_t kPer = kTileWords / 128;  // words of a thread
    uint32_t c[kPer] = {}, cnt = 0;
    if (faces) {
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) {
            c[k] = __popc(a.sc.marks[(size_t)tile * kTileWords + kPer * tid + k]);
            cnt += c[k];
        }
    } else {
        // a warp: one block (1024 vertices) of k_build_mark and k_build_place
        if (lane == 0) cnt = a.sc.unused[4 * tile + w];
    }
    uint32_t x = cnt;  // inclusive scan over the CTA
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, s);
        if ((int)lane >= s) x += y;
    }
    if (lane == 31) s_w[w] = x;
    __syncthreads();
    uint32_t pre = 0, sum = 0;
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) {
        pre += i < w ? s_w[i] : 0u;
        sum += s_w[i];
    }
    if (w == 0) {
        uint32_t before;
        const bool ok = lookback(a, a.sc.order_state + (faces ? 0u : a.f_tiles), chain, tile, sum, before);
        if (lane == 0) {
            s_before = before;
            s_bad = ok ? 0u : 1u;
        }
    }
    __syncthreads();
    if (s_bad) {
        if (tid == 0) give_up(a);
        return;
    }
    uint32_t run = s_before + pre + x - cnt;
    if (faces) {
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) {
            a.sc.counts[(size_t)tile * kTileWords + kPer * tid + k] = run;
            run += c[k];
        }
    } else if (lane == 0) {
        a.sc.unused[4 * tile + w] = run;
    }
}

// Every vertex to its number: the map from old to new, positions and the
// caller-order map in the new order (to the scratch).
__global__ void __launch_bounds__(256) k_build_place(const __grid_constant__ BuildArgs a)
{
    __shared__ uint32_t s_w[8];
    if (ld_state(a.sc.fail)) return;
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    uint32_t j;
    const BuildJob& job = job_of(a, a.vtile_job, blockIdx.x >> 2, j);
    const uint32_t base = ((blockIdx.x >> 2) - job.vtile_begin) * kBuildTile + (blockIdx.x & 3u) * 1024u;
    const uint32_t* marks = a.sc.marks + (size_t)job.ftile_begin * kTileWords;
    const uint32_t* counts = a.sc.counts + (size_t)job.ftile_begin * kTileWords;
    uint32_t s[4], v[4], unused = 0;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        v[k] = base + 256u * k + tid;
        s[k] = v[k] < job.nV ? __ldg(a.sc.first + job.vert_off + v[k]) : 0u;
        unused |= v[k] < job.nV && s[k] == kNoUse ? 1u << k : 0u;
    }
    float4 p[4];
    uint32_t u[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {  // (early: they wait for nothing)
        const uint32_t at = min(v[k], job.nV - 1u);
        p[k] = __ldg(job.pos_out + at);
        u[k] = job.vperm ? __ldg(job.vperm + at) : at;
    }
    if (__syncthreads_or(unused)) {
        // number the unused ones after the used ones: in vertex order, 256 at a time
        const uint32_t last = job.ftile_begin + (job.nT + kBuildTile - 1) / kBuildTile;
        uint32_t run = (ld_state(a.sc.order_state + last - 1) & kStateValue) + a.sc.unused[blockIdx.x];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            const uint32_t m = __ballot_sync(0xffffffffu, (unused >> k) & 1u);
            if (lane == 0) s_w[w] = __popc(m);
            __syncthreads();
            uint32_t pre = 0, sum = 0;
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                pre += i < w ? s_w[i] : 0u;
                sum += s_w[i];
            }
            __syncthreads();
            if ((unused >> k) & 1u) s[k] = run + pre + __popc(m & ((1u << lane) - 1u));
            run += sum;
        }
    }
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
        if (!((unused >> k) & 1u))
            s[k] = __ldg(counts + (s[k] >> 5)) + __popc(__ldg(marks + (s[k] >> 5)) & ((1u << (s[k] & 31)) - 1u));
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        if (v[k] >= job.nV) continue;
        a.sc.inv[job.vert_off + v[k]] = s[k];
        a.sc.pos_new[job.vert_off + s[k]] = p[k];
        a.sc.vperm_new[job.vert_off + s[k]] = u[k];
    }
}

// Face records and the caller-order faces to the new numbering, positions and
// the map back into each tree's own buffers.
__global__ void __launch_bounds__(256) k_build_apply(const __grid_constant__ BuildArgs a)
{
    const bool faces = blockIdx.x < 4 * a.f_tiles;
    const uint32_t block = faces ? blockIdx.x : blockIdx.x - 4 * a.f_tiles;
    uint32_t j;
    const BuildJob& job = faces ? job_of(a, a.ftile_job, block >> 2, j) : job_of(a, a.vtile_job, block >> 2, j);
    const uint32_t base = (block - 4 * (faces ? job.ftile_begin : job.vtile_begin)) * 1024u + threadIdx.x;
    if (ld_state(a.sc.fail)) {
        // the build gave up and its faces may be anything: the refit that follows reads these
        for (uint32_t k = 0; k < 4 && faces; ++k)
            if (base + 256u * k < job.nT) job.face_out[base + 256u * k] = make_uint4(0, 0, 0, 0);
        return;
    }
    if (faces) {
        const uint32_t* inv = a.sc.inv + job.vert_off;
        // (all four faces are loaded before the first is written: one chain of loads, not four)
        uint4 r[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) r[k] = base + 256u * k < job.nT ? job.face_out[base + 256u * k] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            r[k].x = __ldg(inv + r[k].x);
            r[k].y = __ldg(inv + r[k].y);
            r[k].z = __ldg(inv + r[k].z);
        }
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            if (base + 256u * k >= job.nT) break;
            job.face_out[base + 256u * k] = r[k];
            uint32_t* t = job.tri_rw + 3 * (size_t)r[k].w;
            t[0] = r[k].x;
            t[1] = r[k].y;
            t[2] = r[k].z;
        }
    } else {
        float4 p[4];
        uint32_t u[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            const uint32_t v = job.vert_off + min(base + 256u * k, job.nV - 1u);
            p[k] = a.sc.pos_new[v];
            u[k] = a.sc.vperm_new[v];
        }
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            const uint32_t v = base + 256u * k;
            if (v >= job.nV) break;
            job.pos_out[v] = p[k];
            job.vperm_out[v] = u[k];
        }
    }
}

// The scratch of a build: `p` (256-byte aligned) laid out; returns the bytes,
// of which the first `zero_bytes` have to be zero when the build starts.
size_t build_scratch(BuildArgs& a, uint32_t n_jobs, uint32_t n_faces, uint32_t n_verts, void* p)
{
    size_t off = 0;
    auto take = [&](size_t bytes) {
        void* q = (uint8_t*)p + off;
        off += (bytes + 255) / 256 * 256;
        return q;
    };
    BuildScratch& s = a.sc;
    s.fail = (uint32_t*)take(256);
    s.tickets = s.fail + 16;  // one per sort pass (8), one of k_build_count
    s.bounds = (uint32_t*)take(6 * (size_t)n_jobs * 4);
    s.hist = (uint32_t*)take((size_t)n_jobs * a.passes * 256 * 4);
    s.order_state = (uint32_t*)take(((size_t)a.f_tiles + a.v_tiles) * 4);
    s.marks = (uint32_t*)take((size_t)a.f_tiles * kTileWords * 4);
    s.sort_state[0] = (uint32_t*)take((size_t)(a.half_tiles ? 2 : 1) * a.f_tiles * 256 * 4);
    s.zero_bytes = off;
    s.sort_state[1] = (uint32_t*)take((size_t)(a.half_tiles ? 2 : 1) * a.f_tiles * 256 * 4);
    for (int i = 0; i < 2; ++i) {
        s.keys[i] = (uint32_t*)take((size_t)n_faces * 4);
        s.vals[i] = (uint32_t*)take((size_t)n_faces * 4);
    }
    s.hi = a.passes == 8 ? (uint32_t*)take((size_t)n_faces * 4) : s.keys[0];
    s.counts = (uint32_t*)take((size_t)a.f_tiles * kTileWords * 4);
    s.unused = (uint32_t*)take(4 * (size_t)a.v_tiles * 4);
    s.first = (uint32_t*)take((size_t)n_verts * 4);
    s.inv = (uint32_t*)take((size_t)n_verts * 4);
    s.vperm_new = (uint32_t*)take((size_t)n_verts * 4);
    s.pos_new = (float4*)take((size_t)n_verts * 16);
    return off;
}

template <bool kHalf>
static void launch_sort(const BuildArgs& a, uint32_t p, cudaStream_t s)
{
    const uint32_t tiles = kHalf ? 2 * a.f_tiles : a.f_tiles;
    if (p == 0) k_build_sort<true, false, kHalf><<<tiles, kSortThreads, 0, s>>>(a, p, false);
    else if (p + 1 < a.passes) k_build_sort<false, false, kHalf><<<tiles, kSortThreads, 0, s>>>(a, p, p == 3);
    else k_build_sort<false, true, kHalf><<<tiles, kSortThreads, 0, s>>>(a, p, false);
}

cudaError_t launch_build(const BuildArgs& a, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(a.sc.fail, 0, a.sc.zero_bytes, s);
    if (e != cudaSuccess) return e;
    const bool wide = a.passes == 8;
    note_launches(6 + a.passes);
    k_build_vertices<<<4 * a.v_tiles, 256, 0, s>>>(a);
    if (wide) k_build_codes<true><<<4 * a.f_tiles, 256, 0, s>>>(a);
    else k_build_codes<false><<<4 * a.f_tiles, 256, 0, s>>>(a);
    for (uint32_t p = 0; p < a.passes; ++p) {
        if (a.half_tiles) launch_sort<true>(a, p, s);
        else launch_sort<false>(a, p, s);
    }
    k_build_mark<<<4 * a.v_tiles, 256, 0, s>>>(a);
    k_build_count<<<a.f_tiles + a.v_tiles, 128, 0, s>>>(a);
    k_build_place<<<4 * a.v_tiles, 256, 0, s>>>(a);
    k_build_apply<<<4 * (a.f_tiles + a.v_tiles), 256, 0, s>>>(a);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// The whole build of one small tree in one CTA: positions, keys, sort and
// renumbering in shared memory, then every node of the tree. A build of a few
// thousand faces is a chain of a dozen launches otherwise, each a few
// microseconds of latency for less work than one SM has threads for (1,280
// faces: 83 us, against 32 here; up to 4,096 faces and vertices, what the
// shared memory holds).
// ---------------------------------------------------------------------------
constexpr uint32_t kSmallMax = 4096, kSmallThreads = 1024;
struct SmallShared {
    float4 pos[kSmallMax];
    uint32_t first[kSmallMax], lo[kSmallMax], hi[kSmallMax];
    uint16_t idx[2][kSmallMax], inv[kSmallMax];
    uint16_t cnt[kSmallThreads / 32][256];
    uint32_t peers[kSmallThreads / 32][256];
    uint32_t base[256], w[32], red[6][32];
    Box boxes[32];
};

// Exclusive scan of one value per thread over the CTA of 1024; `sum` = the total.
__device__ __forceinline__ uint32_t scan_1024(uint32_t v, uint32_t* sh /*[32]*/, uint32_t& sum)
{
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, s);
        if ((int)lane >= s) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    const uint32_t t = sh[lane];
    const uint32_t pre = __reduce_add_sync(0xffffffffu, lane < w ? t : 0u);
    sum = __reduce_add_sync(0xffffffffu, t);
    __syncthreads();
    return pre + x - v;
}

template <bool kWide>
__global__ void __launch_bounds__(kSmallThreads, 1) k_build_small(const BuildJob job, const TreeShape S, float4* box)
{
    extern __shared__ uint4 s_mem[];
    SmallShared& sh = *(SmallShared*)s_mem;
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const uint32_t nT = job.nT, nV = job.nV;
    // positions and bounds
    uint32_t red[6] = {0, 0, 0, 0, 0, 0}, from[kSmallMax / kSmallThreads];
#pragma unroll
    for (uint32_t k = 0; k < kSmallMax / kSmallThreads; ++k) {
        const uint32_t v = k * kSmallThreads + tid;
        if (v >= nV) break;
        const float4 p = job.pos[v];
        from[k] = job.vperm ? job.vperm[v] : v;
        sh.pos[v] = p;
        sh.first[v] = kNoUse;
        const float c[3] = {p.x, p.y, p.z};
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const uint32_t o = float_to_ordered(c[i]);
            red[i] = max(red[i], ~o);
            red[3 + i] = max(red[3 + i], o);
        }
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        red[i] = __reduce_max_sync(0xffffffffu, red[i]);
        if (lane == 0) sh.red[i][w] = red[i];
    }
    __syncthreads();
    float bmin[3], bmax[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        bmin[k] = ordered_to_float(~__reduce_max_sync(0xffffffffu, sh.red[k][lane]));
        bmax[k] = ordered_to_float(__reduce_max_sync(0xffffffffu, sh.red[3 + k][lane]));
    }
    // keys
    for (uint32_t i = tid; i < nT; i += kSmallThreads) {
        const uint32_t* t = job.tri + 3 * (size_t)i;
        const float4 p0 = sh.pos[t[0]], p1 = sh.pos[t[1]], p2 = sh.pos[t[2]];
        const float va[3] = {p0.x, p0.y, p0.z}, vb[3] = {p1.x, p1.y, p1.z}, vc[3] = {p2.x, p2.y, p2.z};
        uint32_t lo, hi;
        leaf_code(va, vb, vc, bmin, bmax, kWide, lo, hi);
        sh.lo[i] = lo;
        if (kWide) sh.hi[i] = hi;
        sh.idx[0][i] = (uint16_t)i;
    }
    for (uint32_t i = tid; i < kSmallThreads / 32 * 256; i += kSmallThreads) (&sh.peers[0][0])[i] = 0;
    // stable LSD radix sort of the item numbers, 8 bits a pass; warp w ranks the items from w * 32 * rounds on
    const uint32_t rounds = (nT + kSmallThreads - 1) / kSmallThreads, lt = (1u << lane) - 1u;
    for (uint32_t p = 0; p < (kWide ? 8u : 4u); ++p) {
        const uint32_t* key = p < 4 ? sh.lo : sh.hi;
        const uint32_t shift = 8 * (p & 3u);
        for (uint32_t i = tid; i < 32 * 128; i += kSmallThreads) ((uint32_t*)sh.cnt)[i] = 0;
        __syncthreads();
        uint32_t item[4], rank[4], dig[4];
#pragma unroll
        for (uint32_t r = 0; r < 4; ++r) {
            if (r >= rounds) break;
            const uint32_t i = (w * rounds + r) * 32 + lane;
            const bool valid = i < nT;
            item[r] = valid ? sh.idx[p & 1][i] : 0u;
            const uint32_t d = valid ? (key[item[r]] >> shift) & 255u : 0u;
            // (as in k_build_sort; with ballots a build of 1280 faces took 31.2 us, not 29, of 4096 47.6, not 44)
            if (valid) atomicOr(&sh.peers[w][d], 1u << lane);
            __syncwarp();
            const uint32_t peers = valid ? sh.peers[w][d] : 0u;
            const uint32_t before = valid ? sh.cnt[w][d] : 0u;
            rank[r] = before + __popc(peers & lt);
            dig[r] = valid ? d : 256u;
            __syncwarp();
            if (valid && (peers & lt) == 0) {
                sh.cnt[w][d] = (uint16_t)(before + __popc(peers));
                sh.peers[w][d] = 0;
            }
            __syncwarp();
        }
        __syncthreads();
        // four threads a digit, eight warps each: counts to exclusive sums over the warps, then over the digits
        const uint32_t d = tid >> 2, w0 = 8 * (tid & 3u);
        uint32_t c[8], sum = 0;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            c[k] = sh.cnt[w0 + k][d];
            sum += c[k];
        }
        uint32_t x = sum;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, s);
            if ((int)lane >= s) x += y;
        }
        if (lane == 31) sh.w[w] = x;
        const uint32_t group = __shfl_sync(0xffffffffu, x - sum, lane & ~3u);  // the digit's start within the warp
        uint32_t run = x - sum - group;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            sh.cnt[w0 + k][d] = (uint16_t)run;
            run += c[k];
        }
        __syncthreads();
        const uint32_t pre = __reduce_add_sync(0xffffffffu, lane < w ? sh.w[lane] : 0u);
        if ((tid & 3u) == 0) sh.base[d] = pre + group;
        __syncthreads();
#pragma unroll
        for (uint32_t r = 0; r < 4; ++r)
            if (r < rounds && dig[r] < 256u)
                sh.idx[(p + 1) & 1][sh.base[dig[r]] + sh.cnt[w][dig[r]] + rank[r]] = (uint16_t)item[r];
        __syncthreads();
    }
    // first uses; four consecutive sorted faces a thread
    uint32_t f[4][4], m[4], cnt = 0, used, unused;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        const uint32_t i = 4 * tid + k;
        if (i >= nT) continue;
        f[k][3] = sh.idx[0][i];  // an even number of passes
#pragma unroll
        for (uint32_t c = 0; c < 3; ++c) {
            f[k][c] = job.tri[3 * (size_t)f[k][3] + c];
            atomicMin(&sh.first[f[k][c]], 3 * i + c);
        }
    }
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        const uint32_t i = 4 * tid + k;
        m[k] = 0;
        if (i < nT)
#pragma unroll
            for (uint32_t c = 0; c < 3; ++c) m[k] |= sh.first[f[k][c]] == 3 * i + c ? 1u << c : 0u;
        cnt += __popc(m[k]);
    }
    uint32_t nv = scan_1024(cnt, sh.w, used);
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
#pragma unroll
        for (uint32_t c = 0; c < 3; ++c)
            if ((m[k] >> c) & 1u) sh.inv[f[k][c]] = (uint16_t)nv++;
    cnt = 0;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) cnt += 4 * tid + k < nV && sh.first[4 * tid + k] == kNoUse ? 1u : 0u;
    nv = scan_1024(cnt, sh.w, unused) + used;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
        if (4 * tid + k < nV && sh.first[4 * tid + k] == kNoUse) sh.inv[4 * tid + k] = (uint16_t)nv++;
    __syncthreads();  // (also: every thread has read its part of the map before it is rewritten)
#pragma unroll
    for (uint32_t k = 0; k < kSmallMax / kSmallThreads; ++k) {
        const uint32_t v = k * kSmallThreads + tid;
        if (v >= nV) break;
        job.pos_out[sh.inv[v]] = sh.pos[v];
        job.vperm_out[sh.inv[v]] = from[k];
    }
    // faces, and the leaves' boxes
    Box b[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        b[k] = Box{0, 0, 0, 0, 0, 0};
        const uint32_t i = 4 * tid + k;
        if (i >= nT) continue;
        const uint4 r = make_uint4(sh.inv[f[k][0]], sh.inv[f[k][1]], sh.inv[f[k][2]], f[k][3]);
        job.face_out[i] = r;
        uint32_t* t = job.tri_rw + 3 * (size_t)r.w;
        t[0] = r.x;
        t[1] = r.y;
        t[2] = r.z;
        b[k] = box_of(sh.pos[f[k][0]], sh.pos[f[k][1]], sh.pos[f[k][2]]);
    }
    if (S.L > 0) reduce_block<12>(b, S, box, S.L, 0, S.L, sh.boxes);
}

bool build_is_small(uint32_t nT, uint32_t nV) { return nT <= kSmallMax && nV <= kSmallMax; }

cudaError_t launch_build_small(const BuildJob& job, const TreeShape& shape, float4* box, bool wide, cudaStream_t s)
{
    static std::atomic<unsigned long long> configured[64];  // the context it was done for
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long ctx = current_context_id();
    if (dev < 0 || dev >= 64 || ctx == 0 || configured[dev].load(std::memory_order_acquire) != ctx) {
        e = cudaFuncSetAttribute(k_build_small<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmallShared));
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_build_small<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmallShared));
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) configured[dev].store(ctx, std::memory_order_release);
    }
    note_launches(1);
    if (wide) k_build_small<true><<<1, kSmallThreads, sizeof(SmallShared), s>>>(job, shape, box);
    else k_build_small<false><<<1, kSmallThreads, sizeof(SmallShared), s>>>(job, shape, box);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
cudaError_t launch_xyz_to_pos4(const float* xyz, const uint32_t* vperm, uint32_t nV, float4* pos, cudaStream_t s)
{
    note_launches(1);
    k_xyz_to_pos4<<<(nV + 255) / 256, 256, 0, s>>>(xyz, vperm, nV, pos);
    return cudaGetLastError();
}

cudaError_t launch_gather_pos4(const float4* src, const uint32_t* vperm, uint32_t nV, float4* pos, cudaStream_t s)
{
    note_launches(1);
    k_gather_pos4<<<(nV + 255) / 256, 256, 0, s>>>(src, vperm, nV, pos);
    return cudaGetLastError();
}

__device__ __forceinline__ uint32_t find_job(const BuildJob* jobs, uint32_t n, uint32_t block,
                                             const uint32_t* __restrict__ table)
{
    if (table) return __ldg(table + block);  // host-built block -> job map: one load
    uint32_t lo = 0, hi = n - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (jobs[mid].vblock_begin <= block) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Rigid transforms of every tree: pos = M * rest, M a row-major 3x4 matrix per tree.
// Four 256-vertex blocks per CTA (vertex v of block k at thread v): the four
// loads are issued before any arithmetic, for more bytes in flight.
constexpr uint32_t kTransformUnroll = 4;

__global__ void __launch_bounds__(256, 8) k_transform_multi(const BuildJob* __restrict__ jobs, uint32_t n_jobs,
                                                         const uint32_t* __restrict__ vjob,
                                                         const float4* __restrict__ rest,
                                                         const float* __restrict__ mats, uint32_t v_blocks,
                                                         bool rest_tree_order)
{
    float4 p[kTransformUnroll];
    uint32_t jj[kTransformUnroll], vv[kTransformUnroll];
#pragma unroll
    for (uint32_t k = 0; k < kTransformUnroll; ++k) {
        const uint32_t vb = blockIdx.x * kTransformUnroll + k;
        jj[k] = 0xffffffffu;
        if (vb >= v_blocks) continue;
        const uint32_t j = find_job(jobs, n_jobs, vb, vjob);
        const uint32_t v = (vb - jobs[j].vblock_begin) * 256u + threadIdx.x;
        if (v >= jobs[j].nV) continue;
        jj[k] = j;
        vv[k] = v;
        // packed rest positions of all jobs, in the caller's vertex order (through vperm) or the trees',
        // or (rest == nullptr) each job's own source in the tree's order
        const uint32_t* vp = rest_tree_order ? nullptr : jobs[j].vperm;
        p[k] = rest ? __ldg(rest + jobs[j].vert_off + (vp ? __ldg(vp + v) : v)) : __ldg(jobs[j].pos + v);
    }
#pragma unroll
    for (uint32_t k = 0; k < kTransformUnroll; ++k) {
        if (jj[k] == 0xffffffffu) continue;
        const float* m = mats + 12 * (size_t)jj[k];
        jobs[jj[k]].pos_out[vv[k]] = rigid_move([&](int i) { return __ldg(m + i); }, p[k]);
    }
}

cudaError_t launch_transform_multi(const BuildJob* d_jobs, uint32_t n_jobs, uint32_t v_blocks, const uint32_t* vjob,
                                   const float4* rest, const float* mats, bool rest_tree_order, cudaStream_t s)
{
    note_launches(1);
    k_transform_multi<<<(v_blocks + kTransformUnroll - 1) / kTransformUnroll, 256, 0, s>>>(d_jobs, n_jobs, vjob, rest,
                                                                                            mats, v_blocks,
                                                                                            rest_tree_order);
    return cudaGetLastError();
}

// Packed rest positions (caller's vertex order per tree) into each tree's
// vertex order: out[vert_off + v] = rest[vert_off + vperm[v]].
__global__ void __launch_bounds__(256) k_gather_rest_multi(const BuildJob* __restrict__ jobs, uint32_t n_jobs,
                                                           const uint32_t* __restrict__ vjob,
                                                           const float4* __restrict__ rest, float4* __restrict__ out)
{
    const uint32_t j = find_job(jobs, n_jobs, blockIdx.x, vjob);
    const uint32_t v = (blockIdx.x - jobs[j].vblock_begin) * 256u + threadIdx.x;
    if (v >= jobs[j].nV) return;
    const uint32_t* vp = jobs[j].vperm;
    out[jobs[j].vert_off + v] = __ldg(rest + jobs[j].vert_off + (vp ? __ldg(vp + v) : v));
}

cudaError_t launch_gather_rest_multi(const BuildJob* d_jobs, uint32_t n_jobs, uint32_t v_blocks, const uint32_t* vjob,
                                     const float4* rest, float4* out, cudaStream_t s)
{
    if (v_blocks == 0) return cudaSuccess;
    note_launches(1);
    k_gather_rest_multi<<<v_blocks, 256, 0, s>>>(d_jobs, n_jobs, vjob, rest, out);
    return cudaGetLastError();
}


} // namespace oibvh
