// The level reduction shared by the refit and the small build.
#pragma once

#include "oibvh_common.cuh"

namespace oibvh {

__device__ __forceinline__ Box shfl_down(const Box& b, int d)
{
    return Box{__shfl_down_sync(0xffffffffu, b.nx, d), __shfl_down_sync(0xffffffffu, b.ny, d),
               __shfl_down_sync(0xffffffffu, b.nz, d), __shfl_down_sync(0xffffffffu, b.xx, d),
               __shfl_down_sync(0xffffffffu, b.xy, d), __shfl_down_sync(0xffffffffu, b.xz, d)};
}

__device__ __forceinline__ void store_node(float4* box, uint32_t real, const Box& b)
{
    store_node_v8(box + 2 * (size_t)real, b);
}

// Reduce the 2^kLog-node block whose four nodes per thread are v[0..3]
// (level `lvl`, global indices base + 4*tid + k, real when < level_count(lvl))
// by `levels` levels, writing each produced node. Thread 0 ends holding the
// block root (level lvl - levels, index base >> levels).
template <int kLog>
__device__ __forceinline__ void reduce_block(Box v[4], const TreeShape& S, float4* box, uint32_t lvl, uint32_t base,
                                             uint32_t levels, Box* sm8)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t cnt = S.level_count(lvl);
    uint32_t idx = base + 4 * tid;  // index of v[0]
    uint32_t done = 0;
    // two levels inside the thread
    if (done < levels) {
        const uint32_t off = S.level_offset(lvl - 1);
        const Box n0 = (idx + 1 < cnt) ? merge(v[0], v[1]) : v[0];
        const Box n1 = (idx + 3 < cnt) ? merge(v[2], v[3]) : v[2];
        if (idx < cnt) store_node(box, off + (idx >> 1), n0);
        if (idx + 2 < cnt) store_node(box, off + (idx >> 1) + 1, n1);
        v[0] = n0;
        v[1] = n1;
        cnt = (cnt + 1) >> 1;
        idx >>= 1;
        --lvl;
        ++done;
    }
    if (done < levels) {
        const uint32_t off = S.level_offset(lvl - 1);
        const Box n0 = (idx + 1 < cnt) ? merge(v[0], v[1]) : v[0];
        if (idx < cnt) store_node(box, off + (idx >> 1), n0);
        v[0] = n0;
        cnt = (cnt + 1) >> 1;
        --lvl;
        ++done;
    }
    // five levels across the warp: lane holds node idx0 + lane (idx0 = base/4 + 32*warp)
    const uint32_t idx0 = (base >> 2) + 32 * warp;
#pragma unroll
    for (int s = 0; s < 5; ++s) {
        if (done < levels) {  // uniform over the CTA
            const Box r = shfl_down(v[0], 1 << s);
            const uint32_t j = (idx0 + lane) >> s;  // this lane's node (when lane % 2^(s+1) == 0)
            if ((lane & ((2u << s) - 1u)) == 0) {
                if (j + 1 < cnt) v[0] = merge(v[0], r);
                if (j < cnt) store_node(box, S.level_offset(lvl - 1) + (j >> 1), v[0]);
            }
            cnt = (cnt + 1) >> 1;
            --lvl;
            ++done;
        }
    }
    // the last kLog - 7 levels across the CTA: one root per warp
    constexpr int kWarpLog = kLog - 7, kWarps = 1 << kWarpLog;
    if (done < levels) {
        if (lane == 0) sm8[warp] = v[0];
        __syncthreads();
        if (warp == 0) {
            if (lane < kWarps) v[0] = sm8[lane];
            const uint32_t b0 = base >> 7;  // index of warp 0's root
#pragma unroll
            for (int s = 0; s < kWarpLog; ++s) {
                if (done < levels) {
                    const Box r = shfl_down(v[0], 1 << s);
                    const uint32_t j = (b0 + lane) >> s;
                    if (lane < kWarps && (lane & ((2u << s) - 1u)) == 0) {
                        if (j + 1 < cnt) v[0] = merge(v[0], r);
                        if (j < cnt) store_node(box, S.level_offset(lvl - 1) + (j >> 1), v[0]);
                    }
                    cnt = (cnt + 1) >> 1;
                    --lvl;
                    ++done;
                }
            }
        }
    }
}

} // namespace oibvh
