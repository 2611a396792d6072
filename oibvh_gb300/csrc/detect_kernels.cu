// Broad phase (BVTT front expansion) and narrow phase (17-axis SAT).
//
// Reference: Scene::expandBvttNodes (src/cuda/scene.cu:192-223),
// traversal_kernel (src/cuda/collide.cu:76-246) driven by the host loop of
// Scene::detectCollisionOnGPU (src/cuda/scene.cu:270-311), and
// triangle_intersect_kernel (src/cuda/collide.cu:248-299) with
// triangleIntersection2 (third/gProximity/cuda_intersect_tritri.h:350-434).
//
// The broad phase is one kernel, k_walk, after k_begin has set its counters:
// warps claim start-level node pairs 32 at a time, test them, and walk the
// overlapping ones down through a private ring in shared memory. It goes in
// rounds of a launch each: a warp that has nothing more to claim goes on for a
// few levels only and leaves the rest to the next round's list, which all warps
// share out anew. No CTA waits for another one. Appends
// (next list, hits, candidates) are warp-aggregated: one atomic per warp,
// positions from ballot/shuffle prefix sums.
//
// Narrow phase: overlapping leaf pairs are buffered per warp in shared memory
// and, 32 at a time, tested inside the traversal (the kernels' <true>
// instantiation, the float test) or stored for a separate kernel (<false>,
// fewer registers): k_narrow (float test, split API) or, in precision mode,
// the FP64-filtered test's passes (k_prec_classify, k_prec_recheck,
// k_prec_settle, k_prec_df, k_prec_fp64_setup, k_prec_fp64).
//
// The float triangle test reproduces the reference's CPU arithmetic
// (src/utils/utils.cpp:71-169, glm scalar dot/cross): every product, sum and
// difference is rounded on its own (__fmul_rn/__fadd_rn/__fsub_rn, never
// contracted to FMA), so the GPU pair set is the CPU pair set bit for bit.
#include "oibvh_common.cuh"
#include "oibvh_launch.h"

#include <algorithm>
#include <atomic>

namespace oibvh {

constexpr int kDetectThreads = 256;

// ---------------------------------------------------------------------------
// Exact-rounding SAT
// ---------------------------------------------------------------------------
struct V3 {
    float x, y, z;
};
__device__ __forceinline__ V3 vsub(const V3& a, const V3& b)
{
    return V3{__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)};
}
// glm::cross: (x.y*y.z - y.y*x.z, x.z*y.x - y.z*x.x, x.x*y.y - y.x*x.y)
__device__ __forceinline__ V3 vcross(const V3& x, const V3& y)
{
    return V3{__fsub_rn(__fmul_rn(x.y, y.z), __fmul_rn(y.y, x.z)), __fsub_rn(__fmul_rn(x.z, y.x), __fmul_rn(y.z, x.x)),
              __fsub_rn(__fmul_rn(x.x, y.y), __fmul_rn(y.x, x.y))};
}
// glm::dot: (a.x*b.x + a.y*b.y) + a.z*b.z, each op rounded
__device__ __forceinline__ float vdot(const V3& a, const V3& b)
{
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
// project6 (src/utils/utils.cpp:71-95)
__device__ __forceinline__ bool project6(const V3& ax, const V3& p1, const V3& p2, const V3& p3, const V3& q1,
                                         const V3& q2, const V3& q3)
{
    const float P1 = vdot(ax, p1), P2 = vdot(ax, p2), P3 = vdot(ax, p3);
    const float Q1 = vdot(ax, q1), Q2 = vdot(ax, q2), Q3 = vdot(ax, q3);
    const float mx1 = fmaxf(fmaxf(P1, P2), P3), mn1 = fminf(fminf(P1, P2), P3);
    const float mx2 = fmaxf(fmaxf(Q1, Q2), Q3), mn2 = fminf(fminf(Q1, Q2), Q3);
    if (mn1 > mx2) return false;
    if (mn2 > mx1) return false;
    return true;
}
// triangleIntersect (src/utils/utils.cpp:97-169); the 17 tests are a
// conjunction, so evaluating the axes lazily, or in two goes, does not change
// the result. kPart: all axes, the two face normals, or the 15 others.
enum SatPart { kSatAll = 0, kSatNormals = 1, kSatEdges = 2 };
template <int kPart = kSatAll>
__device__ __forceinline__ bool tri_intersect_exact(const V3& P1, const V3& P2, const V3& P3, const V3& Q1,
                                                    const V3& Q2, const V3& Q3)
{
    const V3 p1{0.0f, 0.0f, 0.0f};
    const V3 p2 = vsub(P2, P1), p3 = vsub(P3, P1);
    const V3 q1 = vsub(Q1, P1), q2 = vsub(Q2, P1), q3 = vsub(Q3, P1);
    const V3 e1 = vsub(p2, p1), e2 = vsub(p3, p2), e3 = vsub(p1, p3);
    const V3 f1 = vsub(q2, q1), f2 = vsub(q3, q2), f3 = vsub(q1, q3);
    const V3 n1 = vcross(e1, e2);
    if (kPart != kSatEdges && !project6(n1, p1, p2, p3, q1, q2, q3)) return false;
    const V3 m1 = vcross(f1, f2);
    if (kPart != kSatEdges && !project6(m1, p1, p2, p3, q1, q2, q3)) return false;
    if (kPart == kSatNormals) return true;
    if (!project6(vcross(e1, f1), p1, p2, p3, q1, q2, q3)) return false;
    if (!project6(vcross(e1, f2), p1, p2, p3, q1, q2, q3)) return false;
    if (!project6(vcross(e1, f3), p1, p2, p3, q1, q2, q3)) return false;
    if (!project6(vcross(e2, f1), p1, p2, p3, q1, q2, q3)) return false;
    if (!project6(vcross(e2, f2), p1, p2, p3, q1, q2, q3)) return false;
    if (!project6(vcross(e2, f3), p1, p2, p3, q1, q2, q3)) return false;
    if (!project6(vcross(e3, f1), p1, p2, p3, q1, q2, q3)) return false;
    if (!project6(vcross(e3, f2), p1, p2, p3, q1, q2, q3)) return false;
    if (!project6(vcross(e3, f3), p1, p2, p3, q1, q2, q3)) return false;
    if (!project6(vcross(e1, n1), p1, p2, p3, q1, q2, q3)) return false;
    if (!project6(vcross(e2, n1), p1, p2, p3, q1, q2, q3)) return false;
    if (!project6(vcross(e3, n1), p1, p2, p3, q1, q2, q3)) return false;
    if (!project6(vcross(f1, m1), p1, p2, p3, q1, q2, q3)) return false;
    if (!project6(vcross(f2, m1), p1, p2, p3, q1, q2, q3)) return false;
    if (!project6(vcross(f3, m1), p1, p2, p3, q1, q2, q3)) return false;
    return true;
}

__device__ __forceinline__ V3 vpick(bool p, const V3& a, const V3& b)
{
    return V3{p ? a.x : b.x, p ? a.y : b.y, p ? a.z : b.z};
}
// Whether axis k (0, 1: the normals, 2 + 3 i + j: E_i x F_j, 11 + i: E_i x n1,
// 14 + j: F_j x m1) does not separate: the same arithmetic, for a k of the
// lane's own. Every axis is a cross product (the normals e1 x e2 and f1 x f2).
__device__ __forceinline__ bool axis_overlaps(uint32_t k, const V3& P1, const V3& P2, const V3& P3, const V3& Q1,
                                              const V3& Q2, const V3& Q3)
{
    const V3 p1{0.0f, 0.0f, 0.0f};
    const V3 p2 = vsub(P2, P1), p3 = vsub(P3, P1);
    const V3 q1 = vsub(Q1, P1), q2 = vsub(Q2, P1), q3 = vsub(Q3, P1);
    const V3 e1 = vsub(p2, p1), e2 = vsub(p3, p2), e3 = vsub(p1, p3);
    const V3 f1 = vsub(q2, q1), f2 = vsub(q3, q2), f3 = vsub(q1, q3);
    const bool pairs = k >= 2u && k < 11u;
    const uint32_t i = pairs ? (k - 2u) / 3u : k >= 11u ? (k - 11u) % 3u : 0u, j = pairs ? (k - 2u) % 3u : i;
    const V3 E = vpick(i == 0, e1, vpick(i == 1, e2, e3)), F = vpick(j == 0, f1, vpick(j == 1, f2, f3));
    const bool of_f = k == 1u || k >= 14u;  // F_j x .. (else E_i x ..)
    const V3 n = vcross(vpick(of_f, f1, e1), vpick(of_f, f2, e2));  // the normal of that side
    const V3 c = vcross(vpick(of_f, F, E), vpick(pairs, F, n));
    return project6(vpick(k < 2u, n, c), p1, p2, p3, q1, q2, q3);
}

// ---------------------------------------------------------------------------
// Precision mode: the same 17 tests with an FP64 filter.
//
// Each axis test compares two margins, d1 = mn1 - mx2 and d2 = mn2 - mx1
// (the axis separates when either is > 0). Every float quantity of the test
// carries a running forward error bound against its exact value over the
// same float inputs (u = 2^-24; c = fl(a - b): e_c = e_a + e_b + u|c|;
// c = fl(a b): e_c = |a| e_b + |b| e_a + e_a e_b + u|c| + 2^-149), so each projection
// P has a bound e_P and each margin the bound E = max e_P + max e_Q. The
// FP64 formula obeys the same recurrences with u = 2^-53, so its margin lies
// within 2^-29 E (plus second-order terms) of the exact one. A margin with
// |d| > 2E therefore has the same sign in float, exact and FP64 arithmetic.
//
// The test runs in two passes. Pass 1 evaluates all 17 axes in float: an
// axis whose margin is > 2E separates in every arithmetic and ends the
// test; an axis with both margins < -2E separates in none; the rest are
// undecided. Pass 2 evaluates only the undecided axes again in FP64, with
// the FP64 formula's own operations in its own order (no contraction),
// until one separates. The pair set then equals the all-FP64 pair set by
// construction, while the float answer (the reference arithmetic) is known
// for every candidate, so the disagreements between the two are counted.
//
// Shortcut: two triangles that share a vertex (equal coordinates) are never
// separated by this test in any arithmetic: the shared vertex gives the same
// projection in both triangles' sets, so mn1 <= s <= mx2 and mn2 <= s <= mx1
// on every axis. Relative extents outside [2^-20, 2^20] and non-finite
// inputs take the full FP64 test (the bounds could under- or overflow).
// ---------------------------------------------------------------------------
struct D3 {
    double x, y, z;
};
__device__ __forceinline__ D3 to_d(const V3& v) { return D3{(double)v.x, (double)v.y, (double)v.z}; }
__device__ __forceinline__ D3 dsub(const D3& a, const D3& b)
{
    return D3{__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y), __dsub_rn(a.z, b.z)};
}
__device__ __forceinline__ D3 dcross(const D3& x, const D3& y)
{
    return D3{__dsub_rn(__dmul_rn(x.y, y.z), __dmul_rn(y.y, x.z)), __dsub_rn(__dmul_rn(x.z, y.x), __dmul_rn(y.z, x.x)),
              __dsub_rn(__dmul_rn(x.x, y.y), __dmul_rn(y.x, x.y))};
}
__device__ __forceinline__ double ddot(const D3& a, const D3& b)
{
    return __dadd_rn(__dadd_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)), __dmul_rn(a.z, b.z));
}
// Relative vertices of the FP64 formula: p_i = P_i - P1, q_j = Q_j - P1.
struct D6 {
    D3 p2, p3, q1, q2, q3;
};
__device__ __forceinline__ D6 fp64_relative(const V3& P1, const V3& P2, const V3& P3, const V3& Q1, const V3& Q2,
                                            const V3& Q3)
{
    const D3 dP1 = to_d(P1);
    return D6{dsub(to_d(P2), dP1), dsub(to_d(P3), dP1), dsub(to_d(Q1), dP1), dsub(to_d(Q2), dP1), dsub(to_d(Q3), dP1)};
}

// A float vector with a componentwise bound on its error.
struct EV3 {
    V3 v, e;
};
constexpr float kU = 0x1p-24f;
constexpr float kEta = 0x1p-149f;  // a product that underflows is off by up to half the smallest subnormal
// (a sum or difference whose result is subnormal is exact)
__device__ __forceinline__ float err_sub(float c, float ea, float eb) { return ea + eb + kU * fabsf(c); }
__device__ __forceinline__ float err_mul(float a, float b, float c, float ea, float eb)
{
    return fabsf(a) * eb + fabsf(b) * ea + ea * eb + kU * fabsf(c) + kEta;
}
__device__ __forceinline__ EV3 esub(const EV3& a, const EV3& b)
{
    const V3 c = vsub(a.v, b.v);
    return EV3{c, V3{err_sub(c.x, a.e.x, b.e.x), err_sub(c.y, a.e.y, b.e.y), err_sub(c.z, a.e.z, b.e.z)}};
}
// glm::cross with bounds: c = fl(fl(a b) - fl(d g)) per component
__device__ __forceinline__ float ecross1(float a, float b, float d, float g, float ea, float eb, float ed, float eg,
                                         float& err)
{
    const float m1 = __fmul_rn(a, b), m2 = __fmul_rn(d, g), c = __fsub_rn(m1, m2);
    err = err_sub(c, err_mul(a, b, m1, ea, eb), err_mul(d, g, m2, ed, eg));
    return c;
}
__device__ __forceinline__ EV3 ecross(const EV3& x, const EV3& y)
{
    EV3 r;
    r.v.x = ecross1(x.v.y, y.v.z, y.v.y, x.v.z, x.e.y, y.e.z, y.e.y, x.e.z, r.e.x);
    r.v.y = ecross1(x.v.z, y.v.x, y.v.z, x.v.x, x.e.z, y.e.x, y.e.z, x.e.x, r.e.y);
    r.v.z = ecross1(x.v.x, y.v.y, y.v.x, x.v.y, x.e.x, y.e.y, y.e.x, x.e.y, r.e.z);
    return r;
}
// glm::dot with a bound: fl(fl(fl(ax px) + fl(ay py)) + fl(az pz))
__device__ __forceinline__ float edot(const EV3& a, const EV3& p, float& err)
{
    const float t0 = __fmul_rn(a.v.x, p.v.x), t1 = __fmul_rn(a.v.y, p.v.y), t2 = __fmul_rn(a.v.z, p.v.z);
    const float s = __fadd_rn(t0, t1), r = __fadd_rn(s, t2);
    const float e0 = err_mul(a.v.x, p.v.x, t0, a.e.x, p.e.x);
    const float e1 = err_mul(a.v.y, p.v.y, t1, a.e.y, p.e.y);
    const float e2 = err_mul(a.v.z, p.v.z, t2, a.e.z, p.e.z);
    err = err_sub(r, err_sub(s, e0, e1), e2);
    return r;
}
// One float axis test with bounds: 0 = separates in every arithmetic,
// 1 = separates in none, 2 = undecided; `sep32` is the plain float answer.
__device__ __forceinline__ uint32_t project6_bounded(const EV3& ax, const EV3& p1, const EV3& p2, const EV3& p3,
                                                     const EV3& q1, const EV3& q2, const EV3& q3, bool& sep32)
{
    float eP1, eP2, eP3, eQ1, eQ2, eQ3;
    const float P1 = edot(ax, p1, eP1), P2 = edot(ax, p2, eP2), P3 = edot(ax, p3, eP3);
    const float Q1 = edot(ax, q1, eQ1), Q2 = edot(ax, q2, eQ2), Q3 = edot(ax, q3, eQ3);
    const float mx1 = fmaxf(fmaxf(P1, P2), P3), mn1 = fminf(fminf(P1, P2), P3);
    const float mx2 = fmaxf(fmaxf(Q1, Q2), Q3), mn2 = fminf(fminf(Q1, Q2), Q3);
    sep32 = mn1 > mx2 || mn2 > mx1;
    // 2 E: covers the FP64 error (2^-29 E), second-order terms and the
    // rounding of the margins and of the bound itself
    const float tau = 2.0f * (fmaxf(fmaxf(eP1, eP2), eP3) + fmaxf(fmaxf(eQ1, eQ2), eQ3));
    const float d1 = __fsub_rn(mn1, mx2), d2 = __fsub_rn(mn2, mx1);
    if (d1 > tau || d2 > tau) return 0u;
    if (d1 < -tau && d2 < -tau) return 1u;
    return 2u;
}

__device__ __forceinline__ bool veq(const V3& a, const V3& b) { return a.x == b.x && a.y == b.y && a.z == b.z; }

enum : uint32_t { kPass1Separated = 0, kPass1Hit = 1, kPass1Undecided = 2 };

// Pass 1 of the filtered test: every axis in float with error bounds.
// Returns kPass1Separated / kPass1Hit when the float and FP64 answers are
// known to agree, else kPass1Undecided with the axes to settle in FP64 in
// `mask` and the plain float answer in `hit32`.
__device__ __forceinline__ uint32_t tri_pass1(const V3& P1, const V3& P2, const V3& P3, const V3& Q1, const V3& Q2,
                                              const V3& Q3, uint32_t& mask, bool& hit32)
{
    const EV3 p1{V3{0.0f, 0.0f, 0.0f}, V3{0.0f, 0.0f, 0.0f}};
    const V3 p2v = vsub(P2, P1), p3v = vsub(P3, P1);
    const V3 q1v = vsub(Q1, P1), q2v = vsub(Q2, P1), q3v = vsub(Q3, P1);
    float A = fmaxf(fmaxf(fmaxf(fabsf(p2v.x), fabsf(p2v.y)), fmaxf(fabsf(p2v.z), fabsf(p3v.x))),
                    fmaxf(fmaxf(fabsf(p3v.y), fabsf(p3v.z)), fmaxf(fabsf(q1v.x), fabsf(q1v.y))));
    A = fmaxf(A, fmaxf(fmaxf(fabsf(q1v.z), fabsf(q2v.x)), fmaxf(fabsf(q2v.y), fabsf(q2v.z))));
    A = fmaxf(A, fmaxf(fmaxf(fabsf(q3v.x), fabsf(q3v.y)), fabsf(q3v.z)));
    if (!(A >= 0x1p-20f && A <= 0x1p20f)) {
        // the bounds could under- or overflow: every axis in FP64
        hit32 = tri_intersect_exact(P1, P2, P3, Q1, Q2, Q3);
        mask = (1u << 17) - 1u;
        return kPass1Undecided;
    }
    if (veq(P1, Q1) || veq(P1, Q2) || veq(P1, Q3) || veq(P2, Q1) || veq(P2, Q2) || veq(P2, Q3) || veq(P3, Q1) ||
        veq(P3, Q2) || veq(P3, Q3))
        return kPass1Hit;  // a shared vertex: never separated
    // relative vertices: one rounding each
    const EV3 p2{p2v, V3{kU * fabsf(p2v.x), kU * fabsf(p2v.y), kU * fabsf(p2v.z)}};
    const EV3 p3{p3v, V3{kU * fabsf(p3v.x), kU * fabsf(p3v.y), kU * fabsf(p3v.z)}};
    const EV3 q1{q1v, V3{kU * fabsf(q1v.x), kU * fabsf(q1v.y), kU * fabsf(q1v.z)}};
    const EV3 q2{q2v, V3{kU * fabsf(q2v.x), kU * fabsf(q2v.y), kU * fabsf(q2v.z)}};
    const EV3 q3{q3v, V3{kU * fabsf(q3v.x), kU * fabsf(q3v.y), kU * fabsf(q3v.z)}};
    const EV3 e1 = esub(p2, p1), e2 = esub(p3, p2), e3 = esub(p1, p3);
    const EV3 f1 = esub(q2, q1), f2 = esub(q3, q2), f3 = esub(q1, q3);
    const EV3 n1 = ecross(e1, e2), m1 = ecross(f1, f2);
    bool sep32 = false;
    uint32_t undecided = 0;
#define OIBVH_AXIS(K, AX)                                                        \
    {                                                                            \
        bool s32;                                                                \
        const uint32_t c = project6_bounded((AX), p1, p2, p3, q1, q2, q3, s32);  \
        if (c == 0u) return kPass1Separated;                                     \
        sep32 |= s32;                                                            \
        if (c == 2u) undecided |= 1u << (K);                                     \
    }
    OIBVH_AXIS(0, n1)
    OIBVH_AXIS(1, m1)
    OIBVH_AXIS(2, ecross(e1, f1))
    OIBVH_AXIS(3, ecross(e1, f2))
    OIBVH_AXIS(4, ecross(e1, f3))
    OIBVH_AXIS(5, ecross(e2, f1))
    OIBVH_AXIS(6, ecross(e2, f2))
    OIBVH_AXIS(7, ecross(e2, f3))
    OIBVH_AXIS(8, ecross(e3, f1))
    OIBVH_AXIS(9, ecross(e3, f2))
    OIBVH_AXIS(10, ecross(e3, f3))
    OIBVH_AXIS(11, ecross(e1, n1))
    OIBVH_AXIS(12, ecross(e2, n1))
    OIBVH_AXIS(13, ecross(e3, n1))
    OIBVH_AXIS(14, ecross(f1, m1))
    OIBVH_AXIS(15, ecross(f2, m1))
    OIBVH_AXIS(16, ecross(f3, m1))
#undef OIBVH_AXIS
    if (undecided == 0) return kPass1Hit;  // no axis separates, in any arithmetic
    mask = undecided;
    hit32 = !sep32;
    return kPass1Undecided;
}

__device__ __forceinline__ V3 load_vertex(const float4* __restrict__ pos, uint32_t v)
{
    const float4 p = __ldg(pos + v);
    return V3{p.x, p.y, p.z};
}

// The record of mesh pair `p`. kOne: the pass holds one pair, which comes with
// the kernel's arguments (constant cache) instead of the pair table: one
// dependent load less per step, and no table to upload.
template <bool kOne>
__device__ __forceinline__ void pair_refs(const DetectArgs& a, uint32_t p, TreeRef& TA, TreeRef& TB)
{
    if constexpr (kOne) {
        TA = tree_ref(a.one.ta);
        TB = tree_ref(a.one.tb);
    } else {
        TA = load_tree_ref(a.pairs[p].ta);
        TB = load_tree_ref(a.pairs[p].tb);
    }
}

__device__ __forceinline__ uint32_t warp_append(uint32_t* counter, bool pred, uint32_t lane)
{
    const uint32_t mask = __ballot_sync(0xffffffffu, pred);
    if (mask == 0) return 0;
    const int leader = __ffs(mask) - 1;
    uint32_t base = 0;
    if ((int)lane == leader) base = atomicAdd(counter, (uint32_t)__popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    return base + __popc(mask & ((1u << lane) - 1u));
}

// Descendant x of implicit node i (level l), d levels down (d = 0: the node
// itself, for x = 0); false: there is none (x past the 2^d, or past the level's
// last real node).
__device__ __forceinline__ bool child_of(const TreeRef& T, uint32_t i, uint32_t l, uint32_t d, uint32_t x, uint32_t& c,
                                         uint32_t& lc)
{
    lc = l + d;
    c = ((i + 1u) << d) - 1u + x;
    // implicit nodes of level lc: [2^lc - 1, 2^(lc+1) - 2 - virtual ones]
    return x >> d == 0 && c <= (2u << lc) - 2u - (T.vl >> (T.L - lc));
}

// ---------------------------------------------------------------------------
// Per-warp candidate buffer: leaf pairs whose boxes overlap are queued in
// shared memory and tested 32 at a time, one per lane, so the 17-axis test
// runs at full SIMT width however sparse the candidates are.
// ---------------------------------------------------------------------------
constexpr int kCandBuf = 160;  // <= 31 left over + up to 4 per lane added by one expansion step
constexpr uint32_t kWalkCap = 128;      // default per-warp capacity of the walkers (node pairs)
constexpr uint32_t kWalkCapMax = 512;
constexpr uint32_t kWarps = kDetectThreads / 32;
// Ring entries per warp for a requested capacity (0: the default): a power of
// two (slots by masking), twice the capacity: a step's children are appended
// beside up to 32 pairs that are still queued. 256 entries against 128 take
// the walk of 512 mesh pairs from 1.75 to 1.63 ms (less goes to the lists).
__host__ __device__ __forceinline__ uint32_t walk_ring(uint32_t cap)
{
    cap = cap ? cap : kWalkCap;
    return cap <= 64u ? 128u : cap <= 128u ? 256u : 512u;
}

// Candidates are tested in two goes: the face normals first, which separate four
// of five (batched meshes: 78 %), and what is left, 32 at a time again, against
// the other 15 axes. In one go a warp ran all 17 axes nearly always, for the
// one lane in nine that needs them: 900 instructions for 32 candidates, against
// about 360 so.
constexpr int kLateBuf = 64;  // <= 31 left over + up to 32 that pass the normals
struct WarpCands {
    uint64_t* buf;       // kCandBuf entries
    uint64_t* late;      // kLateBuf entries: past the normals
    uint32_t n;          // warp-uniform
    uint32_t n_late = 0;
    uint32_t found = 0;  // candidates found by this warp (added to the counter once a round)
};

// `count` buffered candidates, one per lane: against kPart's axes. Hits go to
// the hit list (not with kSatNormals alone); returns whether this lane's passed.
template <bool kOne, int kPart>
__device__ __forceinline__ bool test_candidates(const DetectArgs& a, const uint64_t* buf, uint32_t count, uint32_t lane)
{
    bool hit = false;
    uint4 rec = make_uint4(0, 0, 0, 0);
    if (lane < count) {
        const uint64_t c = buf[lane];
        const PairView& pv = kOne ? a.one : a.pairs[bvtt_pair(c)];
        TreeRef TA, TB;
        pair_refs<kOne>(a, bvtt_pair(c), TA, TB);
        const uint4 fa = __ldg(TA.face + bvtt_a(c));
        const uint4 fb = __ldg(TB.face + bvtt_b(c));
        hit = tri_intersect_exact<kPart>(load_vertex(TA.pos, fa.x), load_vertex(TA.pos, fa.y), load_vertex(TA.pos, fa.z),
                                         load_vertex(TB.pos, fb.x), load_vertex(TB.pos, fb.y), load_vertex(TB.pos, fb.z));
        if (kPart != kSatNormals) rec = make_uint4(pv.a, pv.b, fa.w, fb.w);
    }
    if (kPart != kSatNormals) {
        const uint32_t pos = warp_append(a.counts + kCountHits, hit, lane);
        if (hit) {
            if (pos < a.hit_cap) a.hits[pos] = rec;
            else atomicOr(a.counts + kCountFlags, (uint32_t)kFlagHitOverflow);
        }
    }
    return hit;
}

// Up to 16 candidates, g = 2, 4, .. 32 lanes each: lane q of a candidate's tests the
// axes q, q + g, ... What is left in the buffers at a round's end is waited for
// by every warp: one candidate per lane and its 17 axes take 2 us (a few
// candidates 4, in two lists), so they take about 1.
template <bool kOne>
__device__ __forceinline__ void test_few(const DetectArgs& a, const WarpCands& wc, uint32_t lane)
{
    const uint32_t count = wc.n + wc.n_late;
    const uint32_t lg = 5u - (count > 1u ? 32u - __clz(count - 1u) : 0u), g = 1u << lg, item = lane >> lg;
    bool over = true;
    uint4 rec = make_uint4(0, 0, 0, 0);
    if (item < count) {
        const uint64_t c = item < wc.n ? wc.buf[item] : wc.late[item - wc.n];
        const PairView& pv = kOne ? a.one : a.pairs[bvtt_pair(c)];
        TreeRef TA, TB;
        pair_refs<kOne>(a, bvtt_pair(c), TA, TB);
        const uint4 fa = __ldg(TA.face + bvtt_a(c));
        const uint4 fb = __ldg(TB.face + bvtt_b(c));
        const V3 P1 = load_vertex(TA.pos, fa.x), P2 = load_vertex(TA.pos, fa.y), P3 = load_vertex(TA.pos, fa.z);
        const V3 Q1 = load_vertex(TB.pos, fb.x), Q2 = load_vertex(TB.pos, fb.y), Q3 = load_vertex(TB.pos, fb.z);
        rec = make_uint4(pv.a, pv.b, fa.w, fb.w);
        for (uint32_t k = lane & (g - 1u); over && k < 17u; k += g) over = axis_overlaps(k, P1, P2, P3, Q1, Q2, Q3);
    }
    const uint32_t m = __ballot_sync(0xffffffffu, over) >> (item << lg);  // this candidate's lanes
    const uint32_t all = g == 32u ? 0xffffffffu : (1u << g) - 1u;
    const bool hit = item < count && (lane & (g - 1u)) == 0 && (m & all) == all;
    const uint32_t pos = warp_append(a.counts + kCountHits, hit, lane);
    if (hit) {
        if (pos < a.hit_cap) a.hits[pos] = rec;
        else atomicOr(a.counts + kCountFlags, (uint32_t)kFlagHitOverflow);
    }
}

// Broad phase only: `count` buffered candidates (one per lane) to the global
// candidate queue with one atomic for the warp.
__device__ __forceinline__ void store_candidates(const DetectArgs& a, const uint64_t* buf, uint32_t count,
                                                 uint32_t lane)
{
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(a.counts + kCountCandSlots, count);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (lane < count) {
        if (base + lane < a.cand_cap) a.cand[base + lane] = buf[lane];
        else atomicOr(a.counts + kCountFlags, (uint32_t)kFlagCandOverflow);
    }
}

// 32 buffered candidates: tested (kFused: the narrow phase is compiled into the
// traversal) or stored (the kernel carries no triangle-test code).
template <bool kFused, bool kOne>
__device__ __forceinline__ void take_candidates(const DetectArgs& a, WarpCands& wc, const uint64_t* buf, uint32_t lane)
{
    if constexpr (kFused) {
        const bool pass = test_candidates<kOne, kSatNormals>(a, buf, 32, lane);
        const uint32_t m = __ballot_sync(0xffffffffu, pass);
        if (pass) wc.late[wc.n_late + __popc(m & ((1u << lane) - 1u))] = buf[lane];
        wc.n_late += __popc(m);
        __syncwarp();
        if (wc.n_late >= 32) {
            test_candidates<kOne, kSatEdges>(a, wc.late + wc.n_late - 32, 32, lane);
            wc.n_late -= 32;
            __syncwarp();
        }
    } else {
        store_candidates(a, buf, 32, lane);
    }
}

// What is left in the buffers (fewer than 32 each).
template <bool kFused, bool kOne>
__device__ __forceinline__ void flush_candidates(const DetectArgs& a, WarpCands& wc, uint32_t lane)
{
    const uint32_t n = wc.n + wc.n_late;
    if (kFused && n <= 16) {
        if (n > 0) test_few<kOne>(a, wc, lane);
    } else {
        if (wc.n > 0) {
            if constexpr (kFused) test_candidates<kOne, kSatAll>(a, wc.buf, wc.n, lane);
            else store_candidates(a, wc.buf, wc.n, lane);
        }
        if constexpr (kFused)
            if (wc.n_late > 0) test_candidates<kOne, kSatEdges>(a, wc.late, wc.n_late, lane);
    }
    wc.n = wc.n_late = 0;
    __syncwarp();
}

// Queue one candidate per lane where `pred` in the warp's buffer (at most 4
// per lane between two drains).
__device__ __forceinline__ void push_candidate(WarpCands& wc, bool pred, uint64_t cval,
                                               uint32_t lane)
{
    const uint32_t mask = __ballot_sync(0xffffffffu, pred);
    if (mask == 0) return;
    wc.found += __popc(mask);
    if (pred) wc.buf[wc.n + __popc(mask & ((1u << lane) - 1u))] = cval;
    wc.n += __popc(mask);
    __syncwarp();
}

// Every 32 queued candidates are tested (fused narrow phase) or stored (broad
// phase only) at once; called once per step, where little else is live.
template <bool kFused, bool kOne>
__device__ __forceinline__ void drain_candidates(const DetectArgs& a, WarpCands& wc, uint32_t lane)
{
    while (wc.n >= 32) {
        take_candidates<kFused, kOne>(a, wc, wc.buf + wc.n - 32, lane);
        wc.n -= 32;
        __syncwarp();
    }
}

// One BVTT pair per lane, one level down on the sides its key names (both,
// or the larger box's; a leaf never descends): the up to 2 + 2 boxes (a side
// that stays contributes its own node) are loaded first (independent loads)
// and the up to 4 child pairs are tested. `m`: the overlapping ones (bit 2x + y:
// first child of A + x, of B + y); child pair k's key is `key` + child_step(k)
// and, in bits 2k and 2k + 1 of `dm`, how it expands next. Leaf pairs
// (`leaves`): keys of candidates, with leaf indices. `tested` gets the warp's
// number of child pairs tested (lane 0 only).
struct Expansion {
    uint64_t key;
    uint32_t m, dm;
    bool leaves;
};
__device__ __forceinline__ uint64_t child_step(uint32_t k) { return (uint64_t)(k >> 1) << 24 | (k & 1u); }

// A side of an expansion: the first child (or the node itself), its level, whether
// there is a second one, and the first's place among the level's real nodes.
struct Side {
    uint32_t first, level, real;
    bool two;
};
__device__ __forceinline__ Side side_of(const TreeRef& T, uint32_t i, uint32_t l, bool down)
{
    Side s;
    s.level = down ? l + 1u : l;
    s.first = down ? 2u * i + 1u : i;
    const uint32_t w = T.vl >> (T.L - s.level);  // virtual nodes of the level
    s.two = down && s.first < (2u << s.level) - 2u - w;
    s.real = s.first - ((w & ~1u) - __popc(w >> 1));  // less the virtual nodes above it
    return s;
}

// Boxes of a side's first child and, where there is one, its second.
// Leaves: sibling leaves 2j and 2j+1 have adjacent 16-byte face records, read
// as one 32-byte load (face arrays hold one record past the last face, so the
// load stays inside the array when the sibling is virtual); an odd leaf index
// only occurs for a leaf that stays put, read on its own.
__device__ __forceinline__ void side_boxes(const TreeRef& T, const Side& s, Box& b0, Box& b1)
{
    if (s.level == T.L) {
        const uint32_t i = s.first - ((1u << s.level) - 1u);
        uint4 f0, f1;
        if ((i & 1u) == 0) {
            load_face_pair(T.face + i, f0, f1);
        } else {
            f0 = __ldg(T.face + i);
            f1 = f0;
        }
        b0 = leaf_box(T.pos, f0);
        if (s.two) b1 = leaf_box(T.pos, f1);
    } else {
        const float4* p = T.box + 2 * (size_t)s.real;
        b0 = load_node_nc(p);
        if (s.two) b1 = load_node_nc(p + 2);  // same level: the next real node
    }
}

template <bool kOne>
__device__ __forceinline__ Expansion expand_test(const DetectArgs& a, bool valid, uint64_t node, uint32_t lane,
                                                 uint32_t& tested)
{
    Expansion e{0, 0, 0, false};
    uint32_t n = 0;
    if (valid) {
        const uint32_t pair = bvtt_pair(node), ia = bvtt_a(node), ib = bvtt_b(node);
        TreeRef TA, TB;
        pair_refs<kOne>(a, pair, TA, TB);
        const uint32_t la = ilog2(ia + 1u), lb = ilog2(ib + 1u);
        // the sides to descend: the key's, never a leaf (a leaf side stays and
        // the other one descends), so every expansion goes one level down
        const uint32_t d = bvtt_desc(node);
        const Side sa = side_of(TA, ia, la, la != TA.L && (d != kDescendB || lb == TB.L));
        const Side sb = side_of(TB, ib, lb, lb != TB.L && (d != kDescendA || la == TA.L));
        Box A0, A1{}, B0, B1{};
        side_boxes(TA, sa, A0, A1);
        side_boxes(TB, sb, B0, B1);
        n = (sa.two ? 2u : 1u) * (sb.two ? 2u : 1u);
        e.m = (overlap(A0, B0) ? 1u : 0u) | (sb.two && overlap(A0, B1) ? 2u : 0u) | (sa.two && overlap(A1, B0) ? 4u : 0u) |
              (sa.two && sb.two && overlap(A1, B1) ? 8u : 0u);
        const bool a_leaf = sa.level == TA.L, b_leaf = sb.level == TB.L;
        e.leaves = a_leaf && b_leaf;
        if (e.leaves) {  // leaf indices, in Morton order
            e.key = bvtt_pack(pair, sa.first - ((1u << sa.level) - 1u), sb.first - ((1u << sb.level) - 1u));
        } else {
            e.key = bvtt_pack(pair, sa.first, sb.first);
            const float r = a.descend_ratio;
            const float za0 = box_size2(A0), za1 = box_size2(A1), zb0 = box_size2(B0), zb1 = box_size2(B1);
            e.dm = a_leaf   ? 0x55u * kDescendB
                   : b_leaf ? 0x55u * kDescendA
                            : descend_of(za0, zb0, r) | descend_of(za0, zb1, r) << 2 | descend_of(za1, zb0, r) << 4 |
                                descend_of(za1, zb1, r) << 6;
        }
    }
    const uint32_t t = __reduce_add_sync(0xffffffffu, n);
    tested = lane == 0 ? t : 0u;
    return e;
}

// The same for up to 8 pairs, four lanes each: lane 2x + y of an item tests its
// child pair (first child of A + x, of B + y), so a lane has one overlap test,
// one descent rule and one ballot where a lane with all four child pairs has
// them four times over, a scan and loops: 2.2x fewer cycles from a step's start
// to its end. Warps of small traversals mostly hold fewer than 8 pairs.
// Returns whether `child` is an overlapping pair to expand next.
constexpr uint32_t kFewPairs = 8, kDeepPairs = 2;
template <bool kOne>
__device__ __forceinline__ bool expand_few(const DetectArgs& a, WarpCands& wc, bool valid, uint64_t node, uint32_t lane,
                                           uint64_t& child, uint32_t& tested)
{
    bool ov = false, leaves = false, active = false;
    uint64_t cval = 0;
    child = 0;
    if (valid) {
        const uint32_t pair = bvtt_pair(node), ia = bvtt_a(node), ib = bvtt_b(node);
        TreeRef TA, TB;
        pair_refs<kOne>(a, pair, TA, TB);
        const uint32_t la = ilog2(ia + 1u), lb = ilog2(ib + 1u);
        const uint32_t d = bvtt_desc(node);
        const bool down_a = la != TA.L && (d != kDescendB || lb == TB.L);
        const bool down_b = lb != TB.L && (d != kDescendA || la == TA.L);
        uint32_t ca, lca, cb, lcb;
        const bool va = child_of(TA, ia, la, down_a, (lane >> 1) & 1u, ca, lca);
        const bool vb = child_of(TB, ib, lb, down_b, lane & 1u, cb, lcb);
        active = va && vb;
        if (active) {
            const Box A = node_box(TA, ca, lca), B = node_box(TB, cb, lcb);
            ov = overlap(A, B);
            const bool a_leaf = lca == TA.L, b_leaf = lcb == TB.L;
            leaves = a_leaf && b_leaf;
            // leaf indices in Morton order, or the pair to expand next
            cval = bvtt_pack(pair, ca - ((1u << lca) - 1u), cb - ((1u << lcb) - 1u));
            child = bvtt_pack(pair, ca, cb, descend_side(A, a_leaf, B, b_leaf, a.descend_ratio));
        }
    }
    const uint32_t t = __popc(__ballot_sync(0xffffffffu, active));
    tested = lane == 0 ? t : 0u;
    push_candidate(wc, ov && leaves, cval, lane);
    return ov && !leaves;
}

// Up to 2 pairs, 16 lanes each and two levels at once, so that a warp with a
// pair or two, as most in small traversals, is down in half the steps: lane
// 4x + y of an item follows child x / 2 of A and then its child x % 2, and so in
// B. The loads of both levels are issued together, but the pair in between is
// tested and decides how it descends, as in two steps: a box does not hold its
// children's where positions are NaN or were set without a refit, and the
// candidates must not depend on how many pairs a warp happens to hold.
// Internal nodes only, as two_levels_left() says for the warp: next to the leaves,
// whose boxes are two loads away, the four boxes of a lane in a row took longer
// than two steps (two meshes of 1.31 M triangles 72.5 us a detect, 70.7 so; 67.1
// with the pairs in between not tested).
template <bool kOne>
__device__ __forceinline__ bool two_levels_left(const DetectArgs& a, bool valid, uint64_t node)
{
    bool left = true;
    if (valid) {
        TreeRef TA, TB;
        pair_refs<kOne>(a, bvtt_pair(node), TA, TB);
        left = ilog2(bvtt_a(node) + 1u) + 2u < TA.L && ilog2(bvtt_b(node) + 1u) + 2u < TB.L;
    }
    return __all_sync(0xffffffffu, left);
}
template <bool kOne>
__device__ __forceinline__ bool expand_two_levels(const DetectArgs& a, bool valid, uint64_t node, uint32_t lane,
                                                  uint64_t& child, uint32_t& tested)
{
    const uint32_t x = (lane >> 2) & 3u, y = lane & 3u;
    bool ov = false;
    uint32_t n = 0;  // pairs tested by this lane
    child = 0;
    if (valid) {
        TreeRef TA, TB;
        pair_refs<kOne>(a, bvtt_pair(node), TA, TB);
        const uint32_t la = ilog2(bvtt_a(node) + 1u), lb = ilog2(bvtt_b(node) + 1u), d = bvtt_desc(node);
        uint32_t ca, lca, cb, lcb, ga, lga, gb, lgb;  // the pair in between, and its children
        const bool va = child_of(TA, bvtt_a(node), la, d != kDescendB, x >> 1, ca, lca);
        const bool vb = child_of(TB, bvtt_b(node), lb, d != kDescendA, y >> 1, cb, lcb);
        if (va && vb) {
            const bool wa = child_of(TA, ca, lca, 1u, x & 1u, ga, lga), wb = child_of(TB, cb, lcb, 1u, y & 1u, gb, lgb);
            Box A = load_node_nc(TA.box + 2 * (size_t)TA.shape().real_index(ca));
            Box B = load_node_nc(TB.box + 2 * (size_t)TB.shape().real_index(cb));
            const Box A2 = load_node_nc(TA.box + 2 * (size_t)TA.shape().real_index(wa ? ga : ca));
            const Box B2 = load_node_nc(TB.box + 2 * (size_t)TB.shape().real_index(wb ? gb : cb));
            n = ((x | y) & 1u) == 0 ? 1u : 0u;  // (one lane counts the pair in between)
            const uint32_t side = descend_side(A, false, B, false, a.descend_ratio);
            const bool sa = side != kDescendB, sb = side != kDescendA;
            if (overlap(A, B) && (sa ? wa : (x & 1u) == 0) && (sb ? wb : (y & 1u) == 0)) {
                ++n;
                if (sa) A = A2;
                if (sb) B = B2;
                ov = overlap(A, B);
                child = bvtt_pack(bvtt_pair(node), sa ? ga : ca, sb ? gb : cb, descend_side(A, false, B, false, a.descend_ratio));
            }
        }
    }
    const uint32_t t = __reduce_add_sync(0xffffffffu, n);
    tested = lane == 0 ? t : 0u;
    return ov;
}

// Exclusive prefix over the warp of each lane's count; `total` = the warp's sum.
__device__ __forceinline__ uint32_t child_prefix(uint32_t cnt, uint32_t lane, uint32_t& total)
{
    uint32_t incl = cnt;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, s);
        if ((int)lane >= s) incl += y;
    }
    total = __shfl_sync(0xffffffffu, incl, 31);
    return incl - cnt;
}

// ---------------------------------------------------------------------------
// The traversal's rounds. Round 0 takes the start tests, round r >= 1 the list
// that round r - 1 appended (two arrays in turn). A round's words (list size,
// items claimed) are one of four slots in turn: round r appends to slot r + 1 and
// clears slot r + 2, which nobody looks at then.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t* round_slot(uint32_t* counts, uint32_t r)
{
    return counts + kCtlRound + (r & 3u) * kCtlRoundWords;
}

// Counters before a traversal.
__global__ void __launch_bounds__(256) k_begin(DetectArgs a, uint32_t hits_before)
{
    for (uint32_t i = threadIdx.x; i < kCountTotal; i += blockDim.x) a.counts[i] = i == kCountHits ? hits_before : 0u;
}

// The counters and, when there are at most host_hit_cap, the hits to pinned
// host memory (one CTA): a result that a program reads at once is then there
// without a copy of its own (about 18 us a call, for a few hundred records).
__device__ __forceinline__ void publish(const DetectArgs& a)
{
    for (uint32_t i = threadIdx.x; i < kCountHost; i += blockDim.x) a.host[i] = __ldcg(a.counts + i);
    const uint32_t n = __ldcg(a.counts + kCountHits);
    if (n > a.host_hit_cap || n > a.hit_cap) return;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) a.host_hits[i] = __ldcg(a.hits + i);
}
__global__ void __launch_bounds__(256) k_publish(DetectArgs a) { publish(a); }

// One start pair per lane (test i of the start-level cross products, the
// reference's Scene::expandBvttNodes, src/cuda/scene.cu:192-223): overlapping
// internal pairs are appended to the ring, overlapping leaf pairs are
// candidates. Returns the number appended.
template <bool kOne>
__device__ __forceinline__ uint32_t start_pairs(const DetectArgs& a, WarpCands& wc, uint32_t i, bool valid,
                                                uint64_t* ring, uint32_t mask, uint32_t at, uint32_t lane)
{
    bool ov = false, leafpair = false;
    uint64_t node = 0, cval = 0;
    if (valid) {
        uint32_t lo = 0, hi = kOne ? 0u : a.n_pairs - 1;
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if (a.pairs[mid].front_off <= i) lo = mid;
            else hi = mid - 1;
        }
        const PairView& pv = kOne ? a.one : a.pairs[lo];
        const uint32_t k = i - pv.front_off;
        const uint32_t x = k / pv.front_cnt_b, y = k - x * pv.front_cnt_b;
        const uint32_t ia = (1u << pv.entry_a) - 1u + x, ib = (1u << pv.entry_b) - 1u + y;
        TreeRef TA, TB;
        pair_refs<kOne>(a, lo, TA, TB);
        const Box ba = node_box(TA, ia, pv.entry_a), bb = node_box(TB, ib, pv.entry_b);
        ov = overlap(ba, bb);
        leafpair = ov && pv.entry_a == TA.L && pv.entry_b == TB.L;
        node = bvtt_pack(lo, ia, ib, descend_side(ba, pv.entry_a == TA.L, bb, pv.entry_b == TB.L, a.descend_ratio));
        cval = bvtt_pack(lo, x, y);
    }
    push_candidate(wc, leafpair, cval, lane);
    const uint32_t m = __ballot_sync(0xffffffffu, ov && !leafpair);
    if (ov && !leafpair) ring[(at + __popc(m & ((1u << lane) - 1u))) & mask] = node;
    __syncwarp();
    return __popc(m);
}

// Pairs per warp from which a round's list is claimed: below it, a warp's few
// pairs are better spread out than walked together (16 against 1: two pairs of
// meshes 94 to 81 us a detect, 24 bodies 92 to 80, 64 pairs 306 to 297).
constexpr uint32_t kClaimMin = 16;

// Round r of the traversal. Each step pops up to 32 pairs of the warp's ring (one
// per lane), expands them and appends the overlapping children at the tail, with
// no barrier between tree levels. `last`: the last round that the host has
// launched; its CTA that finishes last writes what is left for a next one, and
// hands over the results.
//
// A round is a launch, not a barrier in one launch: the CTAs of a grid barrier
// all have to be resident at once (a cooperative launch starts when they can be),
// so a detect waited for the end of whatever else held the SMs. The next round's
// CTAs are scheduled while this one's last warps finish (programmatic launch:
// they wait at the start for its end), which a round's launch latency hides
// behind: two meshes of 20 k triangles 31.6 us a detect with the barrier, 35.0
// with plain launches, 31.5 so; of 1.31 M 67, 72 and 65; a scene of 64 pairs 275,
// 276 and 268 (all three before the pairs between two levels were tested).
//
// What bounds it is latency: a step's chain of loads (ring entry, boxes, at the
// leaves faces and then vertices), 1.1 to 1.5 us, times the steps in a row of the
// busiest warp in small traversals; in large ones the same chain at the warps that 64
// registers leave. Four CTAs an SM keep 45 to 47 % of the warps active, the schedulers
// issue in 41 to 51 % of the cycles, and a warp waits 7 to 10 cycles of 14 to 17 for a
// load between two instructions (a frame of 64 pairs; DRAM 2 to 12 %, the L1's data
// pipe 18 to 47 %). Fewer instructions a step help all the same, as each is in the
// chain: about 450 for 32 pairs, 554 before a side's arithmetic was written out and a
// step's children and candidates were given their places by one scan (a frame of 64
// pairs 228 to 197 us, of 512 pairs 1254 to 1088). A warp cuts its walk six steps
// after it has last claimed something and the rest is shared out anew: the next round
// costs about 2 us, a warp left alone with a deep subtree tens (2, 4, 6, 8, 12 steps:
// two meshes of 1.31 M triangles 141, 104, 96, 103, 119 us a detect); three steps after
// start tests that were dealt out, which leave pairs to one warp in ten (six against
// three: 1.31 M triangles 77 to 71 us, 24 bodies 72 to 66, 20 k triangles 39 to 36, with
// pairs taken two levels at once). Measured, whole detects, against one kernel for the
// start tests, one CTA for the top levels and several launches that each walk to
// the leaves: two meshes of 20 k triangles 91 to 34 us, of 1.31 M 158 to 68, 24
// bodies 115 to 67. A queue that idle warps wait on, instead of rounds, was slower
// (20 k: 112 us): a hand-over costs its giver about 3 us.
template <bool kFused, bool kOne>
__global__ void __launch_bounds__(kDetectThreads, 4) k_walk(DetectArgs a, uint32_t total0, uint32_t r, bool last)
{
    extern __shared__ uint64_t s_ring[];  // [warp][walk_ring(cap)]
    __shared__ uint64_t s_cand[kWarps][kCandBuf], s_late[kFused ? kWarps : 1][kLateBuf];
    __shared__ uint32_t s_last, s_found, s_tested;
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_found = s_tested = 0;
    // (with a programmatic launch only: the round before is done and its writes are here; then
    // the next round's CTAs may come as this one's leave)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __syncthreads();
    WarpCands wc{s_cand[wib], s_late[kFused ? wib : 0], 0};
    const uint32_t R = walk_ring(a.walk_cap), mask = R - 1u;
    uint64_t* ring = s_ring + (size_t)wib * R;
    const uint32_t W = gridDim.x * kWarps;
    const uint32_t w = wib * gridDim.x + blockIdx.x;  // neighbouring items go to different SMs
    const uint32_t listed = r == 0 ? total0 : *(volatile uint32_t*)round_slot(a.counts, r);
    // (a list that was too small: the pass is given up here, and runs again or fails)
    const uint32_t n_src = r == 0 || listed <= a.work_cap ? listed : 0u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        round_slot(a.counts, r + 2)[0] = 0;
        round_slot(a.counts, r + 2)[kCtlRoundClaim] = 0;
        if (listed > 0) a.counts[kCountRounds] = r + 1u;
        if (r > 0) a.counts[kCountPeak] = max(a.counts[kCountPeak], listed);
    }
    if (n_src > 0) {
        uint32_t* claim = round_slot(a.counts, r) + kCtlRoundClaim;
        uint32_t* spill_cnt = round_slot(a.counts, r + 1);
        // (where they are used: kept, the two pointers are spilled, 28 B a thread and more)
        auto src = [&]() { return r & 1u ? a.work[1] : a.work[0]; };
        auto spill = [&]() { return r & 1u ? a.work[0] : a.work[1]; };
        // A long list is claimed `chunk` consecutive items at a time; a short one (start tests:
        // at most a warp's worth per warp; pairs: fewer than kClaimMin per warp) is dealt out
        // statically, items w, w + W, .., so that it spreads over all warps.
        const uint32_t per_warp = n_src / W;
        const bool claiming = r == 0 ? per_warp >= 32u : per_warp >= max(kClaimMin, a.claim_min);
        const uint32_t chunk = claiming ? min(32u, max(1u, per_warp)) : 0u;
        uint32_t next = w;  // static share: the next item
        bool more = claiming ? n_src > 0 : w < n_src;
        // pairs a warp may queue (the rest goes to the next round): few items, few pairs each
        const uint32_t cap = claiming || a.stay ? R - 32u : 32u;
        const uint32_t limit = r == 0 && !claiming ? a.start_steps : a.walk_steps;
        uint32_t head = 0, live = 0, steps = 0, tested = 0;
        for (;;) {
            while (live < 32u && more) {
                uint32_t i, n_take;  // this lane's item; items taken
                steps = 0;
                if (claiming) {
                    uint32_t base = 0;
                    if (lane == 0) base = atomicAdd(claim, chunk);
                    base = __shfl_sync(0xffffffffu, base, 0);
                    n_take = base < n_src ? min(chunk, n_src - base) : 0u;
                    i = base + lane;
                    more = base + chunk < n_src;
                } else {
                    const uint32_t left = (n_src - next + W - 1u) / W;
                    n_take = min(32u, left);
                    i = next + lane * W;
                    next += n_take * W;
                    more = left > 32u;
                }
                if (r == 0) {
                    live += start_pairs<kOne>(a, wc, i, lane < n_take, ring, mask, head + live, lane);
                    drain_candidates<kFused, kOne>(a, wc, lane);
                } else {
                    if (lane < n_take) ring[(head + live + lane) & mask] = __ldcg(src() + i);
                    live += n_take;
                    __syncwarp();
                }
            }
            if (live == 0) break;
            bool cut = false;
            // some steps since the last claim (two more with few pairs, which may be about to end):
            // is anything left to claim?
            if (steps >= limit && (live > kFewPairs || steps >= limit + 2u)) {
                if (more && claiming) {
                    uint32_t c = 0;
                    if (lane == 0) c = *(volatile uint32_t*)claim;
                    more = __shfl_sync(0xffffffffu, c, 0) < n_src;
                }
                cut = !more;
                steps = 0;
            }
            ++steps;
            if (cut) {
                // no: other warps may be idle, and what this one holds is shared out anew
                uint32_t base = 0;
                if (lane == 0) base = atomicAdd(spill_cnt, live);
                base = __shfl_sync(0xffffffffu, base, 0);
                for (uint32_t k = lane; k < live; k += 32)
                    if (base + k < a.work_cap) spill()[base + k] = ring[(head + k) & mask];
                if (lane == 0 && base + live > a.work_cap) atomicOr(a.counts + kCountFlags, (uint32_t)kFlagFrontOverflow);
                break;
            }
            uint32_t t;
            if (live <= kFewPairs) {
                const bool two = live <= kDeepPairs && two_levels_left<kOne>(a, lane >> 4 < live, ring[(head + (lane >> 4)) & mask]);
                const uint32_t item = lane >> (two ? 4 : 2);
                const uint64_t node = ring[(head + item) & mask];
                const uint32_t n = live;
                __syncwarp();  // every lane has read its entry before the slots are reused
                head += n;
                uint64_t child;
                const bool keep = two ? expand_two_levels<kOne>(a, item < n, node, lane, child, t)
                                      : expand_few<kOne>(a, wc, item < n, node, lane, child, t);
                const uint32_t km = __ballot_sync(0xffffffffu, keep);
                live = __popc(km);  // at most 32: fits any ring
                if (keep) ring[(head + __popc(km & ((1u << lane) - 1u))) & mask] = child;
            } else {
                const uint32_t n = min(32u, live);
                const bool valid = lane < n;
                const uint64_t node = valid ? ring[(head + lane) & mask] : 0ull;
                __syncwarp();
                head += n;
                live -= n;
                const Expansion e = expand_test<kOne>(a, valid, node, lane, t);
                // places for both kinds at once: children in the low half, candidates in the high one
                uint32_t total;
                const uint32_t cnt = (uint32_t)__popc(e.m);
                const uint32_t ex = child_prefix(e.leaves ? cnt << 16 : cnt, lane, total);
                const uint32_t kids = total & 0xffffu, cands = total >> 16;
                const uint32_t fit = live < cap ? min(kids, cap - live) : 0u;
                uint32_t sbase = 0;
                if (kids > fit) {
                    if (lane == 31) sbase = atomicAdd(spill_cnt, kids - fit);
                    sbase = __shfl_sync(0xffffffffu, sbase, 31);
                    if (sbase + (kids - fit) > a.work_cap && lane == 0) atomicOr(a.counts + kCountFlags, (uint32_t)kFlagFrontOverflow);
                }
                if (e.leaves) {
                    uint64_t* to = wc.buf + wc.n + (ex >> 16);
#pragma unroll
                    for (uint32_t k = 0; k < 4; ++k)
                        if ((e.m >> k) & 1u) *to++ = e.key + child_step(k);
                } else {
                    uint32_t at = ex & 0xffffu;
#pragma unroll
                    for (uint32_t k = 0; k < 4; ++k) {
                        if (!((e.m >> k) & 1u)) continue;
                        const uint64_t child = e.key + child_step(k) + ((uint64_t)((e.dm >> (2 * k)) & 3u) << 48);
                        if (at < fit) ring[(head + live + at) & mask] = child;
                        else if (sbase + (at - fit) < a.work_cap) spill()[sbase + (at - fit)] = child;
                        ++at;
                    }
                }
                wc.n += cands;
                wc.found += cands;
                live += fit;
            }
            tested += t;
            __syncwarp();  // appended entries are visible to the lanes that pop them
            // the step's candidates are tested (or stored) after its children are
            // queued, where little else is live
            drain_candidates<kFused, kOne>(a, wc, lane);
        }
        flush_candidates<kFused, kOne>(a, wc, lane);
        if (lane == 0 && (tested | wc.found)) {
            atomicAdd(&s_tested, tested);
            atomicAdd(&s_found, wc.found);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            if (r == 0 && blockIdx.x == 0) s_tested += total0;
            if (s_tested) atomicAdd(a.counts + kCountTested, s_tested);
            if (s_found) atomicAdd(a.counts + kCountCands, s_found);
        }
    }
    if (!last) return;
    // the CTA that is last to finish hands over the results, and clears the other
    // counter block for the next traversal (nobody uses it now)
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicInc(a.counts + kCtlDone, gridDim.x - 1u) == gridDim.x - 1u;  // (wraps to 0)
        if (s_last) {
            __threadfence();
            const uint32_t left = __ldcg(round_slot(a.counts, r + 1));
            a.counts[kCountLeft] = left;
            a.counts[kCountPeak] = max(__ldcg(a.counts + kCountPeak), left);  // (no next round to note it)
            __threadfence();
        }
    }
    __syncthreads();
    if (!s_last || !a.host) return;
    publish(a);
    if (a.counts_next)
        for (uint32_t i = threadIdx.x; i < kCountTotal; i += blockDim.x) a.counts_next[i] = 0;
}

// Narrow phase over stored candidates (the split broad/narrow API):
// triangle_intersect_kernel (src/cuda/collide.cu:248-299).
__global__ void __launch_bounds__(kDetectThreads) k_narrow(DetectArgs a)
{
    __shared__ uint64_t s_late[kWarps][kLateBuf];
    const uint32_t n = min(a.counts[kCountCandSlots], a.cand_cap);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t n_warps = (gridDim.x * blockDim.x) >> 5;
    WarpCands wc{nullptr, s_late[threadIdx.x >> 5], 0};
    for (uint32_t base = warp * 32; base < n; base += n_warps * 32) {
        if (n - base >= 32) take_candidates<true, false>(a, wc, a.cand + base, lane);
        else test_candidates<false, kSatAll>(a, a.cand + base, n - base, lane);
    }
    flush_candidates<true, false>(a, wc, lane);
}

// Precision mode's narrow phase over stored candidates: one candidate's
// triangles, and a hit appended with one atomic per warp.
__device__ __forceinline__ void load_tris(const DetectArgs& a, uint64_t c, V3& P1, V3& P2, V3& P3, V3& Q1, V3& Q2,
                                          V3& Q3, uint4& rec)
{
    const PairView& pv = a.pairs[bvtt_pair(c)];
    const TreeRef TA = load_tree_ref(pv.ta);
    const TreeRef TB = load_tree_ref(pv.tb);
    const uint4 fa = __ldg(TA.face + bvtt_a(c));
    const uint4 fb = __ldg(TB.face + bvtt_b(c));
    P1 = load_vertex(TA.pos, fa.x);
    P2 = load_vertex(TA.pos, fa.y);
    P3 = load_vertex(TA.pos, fa.z);
    Q1 = load_vertex(TB.pos, fb.x);
    Q2 = load_vertex(TB.pos, fb.y);
    Q3 = load_vertex(TB.pos, fb.z);
    rec = make_uint4(pv.a, pv.b, fa.w, fb.w);
}

__device__ __forceinline__ void append_hit(const DetectArgs& a, bool hit, const uint4& rec, uint32_t lane)
{
    const uint32_t pos = warp_append(a.counts + kCountHits, hit, lane);
    if (hit) {
        if (pos < a.hit_cap) a.hits[pos] = rec;
        else atomicOr(a.counts + kCountFlags, (uint32_t)kFlagHitOverflow);
    }
}

// One candidate's relative vertices and face normals (with error bounds),
// from which axis_of forms any of the 17 axes with selects only.
struct LaneTri {
    V3 p2, p3, q1, q2, q3;  // relative vertices (p1 = 0); their bound is u|x|
    EV3 n1, m1;             // face normals with error bounds
};

__device__ __forceinline__ EV3 ev_rel(const V3& v)
{
    return EV3{v, V3{kU * fabsf(v.x), kU * fabsf(v.y), kU * fabsf(v.z)}};
}
__device__ __forceinline__ V3 vsel(bool c, const V3& a, const V3& b)
{
    return V3{c ? a.x : b.x, c ? a.y : b.y, c ? a.z : b.z};
}
__device__ __forceinline__ EV3 esel(bool c, const EV3& a, const EV3& b) { return EV3{vsel(c, a.v, b.v), vsel(c, a.e, b.e)}; }

// Axis `k` (0..16, the reference numbering) of the lane's candidate, built
// with selects only (no divergence between lanes on different axes).
__device__ __forceinline__ EV3 axis_of(uint32_t k, const LaneTri& t)
{
    const EV3 zero{V3{0.0f, 0.0f, 0.0f}, V3{0.0f, 0.0f, 0.0f}};
    const EV3 p2 = ev_rel(t.p2), p3 = ev_rel(t.p3), q1 = ev_rel(t.q1), q2 = ev_rel(t.q2), q3 = ev_rel(t.q3);
    // edges as the reference forms them: e1 = p2 - p1, e2 = p3 - p2, e3 = p1 - p3,
    // f1 = q2 - q1, f2 = q3 - q2, f3 = q1 - q3
    const uint32_t ei = k < 11 ? (k - 2) / 3 : k - 11;  // edge of A (axes 2..13)
    const uint32_t fj = k < 11 ? (k - 2) % 3 : k - 14;  // edge of B (axes 2..10, 14..16)
    const EV3 E = esub(esel(ei == 0, p2, esel(ei == 1, p3, zero)), esel(ei == 0, zero, esel(ei == 1, p2, p3)));
    const EV3 F = esub(esel(fj == 0, q2, esel(fj == 1, q3, q1)), esel(fj == 0, q1, esel(fj == 1, q2, q3)));
    const bool ef = k >= 2 && k < 11, en = k >= 11 && k < 14;
    const EV3 X = esel(ef || en, E, F);
    const EV3 Y = esel(ef, F, esel(en, t.n1, t.m1));
    return esel(k == 0, t.n1, esel(k == 1, t.m1, ecross(X, Y)));
}

// ---------------------------------------------------------------------------
// Precision narrow phase in passes, grouping candidates by how much of the
// filtered test they need, so that the lanes of a warp run the same code:
//  1. k_prec_classify: the plain float SAT (the reference's arithmetic), which
//     also names the first separating axis. A float-separated candidate needs
//     only that axis bounded: a margin above its error bound separates in every
//     arithmetic (no hit, float and FP64 agree); otherwise it goes to the
//     recheck list with the axis. Shared vertices are hits at once, and so is a
//     float hit whose every axis overlaps beyond a static bound on the float
//     and FP64 errors; other float hits go to the float-hit list, whose members
//     need all 17 bounded axes.
//     Then k_prec_recheck: the recheck list's one axis in double-float
//     arithmetic (3.). Where FP64 separates there too, which is nearly always,
//     the candidate is done; the others join the float hits.
//  2. k_prec_settle over the float hits and what the recheck left, one per
//     lane: pass 1 of the filtered test (all 17 axes bounded, straight-line
//     for float hits: no lane leaves early); what it leaves undecided goes to
//     the FP64 list with the mask of its undecided axes.
//  3. k_prec_df evaluates those axes in double-float arithmetic with a bound
//     on its own and FP64's errors, deciding each axis as FP64 would where
//     the bound allows; the axes it leaves open go on.
//  4. k_prec_fp64_setup forms each remaining entry's FP64 vertices and
//     normals with every lane busy; k_prec_fp64 then evaluates the open axes
//     in FP64, one axis per lane per iteration, lanes refilled from the list
//     as their candidates are decided.
// The pair set is the all-FP64 one by construction.
// ---------------------------------------------------------------------------

// project6 of the float test, which also clears `robust` unless both of the
// axis' margins are below -B (used only when no axis separates).
__device__ __forceinline__ bool project6_robust(const V3& ax, const V3& p1, const V3& p2, const V3& p3, const V3& q1,
                                                const V3& q2, const V3& q3, float B, bool& robust)
{
    const float P1 = vdot(ax, p1), P2 = vdot(ax, p2), P3 = vdot(ax, p3);
    const float Q1 = vdot(ax, q1), Q2 = vdot(ax, q2), Q3 = vdot(ax, q3);
    const float mx1 = fmaxf(fmaxf(P1, P2), P3), mn1 = fminf(fminf(P1, P2), P3);
    const float mx2 = fmaxf(fmaxf(Q1, Q2), Q3), mn2 = fminf(fminf(Q1, Q2), Q3);
    if (mn1 > mx2) return false;
    if (mn2 > mx1) return false;
    robust = robust && __fsub_rn(mn1, mx2) < -B && __fsub_rn(mn2, mx1) < -B;
    return true;
}

// The first of the 17 axes (reference order) that separates the triangles
// in float, 17 when none does (then they intersect in float). When none
// does, `robust` tells whether every axis overlaps by more than a bound on
// the float and FP64 errors: then the triangles intersect in FP64 as well.
//
// The bound follows from the largest relative coordinate A (|p_i|, |q_j| <=
// A; relative extents in [2^-20, 2^20], else never robust) by propagating
// the rounding of each operation (u = 2^-24): edges |e| <= 2A (error 4uA),
// edge x edge and the normals |c| <= 8A^2 (48uA^2), edge x normal 32A^3
// (320uA^3); a projection onto a degree-2 axis errs by at most 232uA^3, a
// margin by 512uA^3 = 2^-15 A^3; onto a degree-3 axis 1312uA^4, a margin by
// 2816uA^4 < 2^-12 A^4. FP64 errs by 2^-29 of that. B = twice (2^-14 A^3)
// and four times (2^-10 A^4) these, covering second-order terms, underflow
// (2^-149 per product, far below 2^-90) and the rounding of B itself.
__device__ __forceinline__ uint32_t tri_first_separating_axis(const V3& P1, const V3& P2, const V3& P3, const V3& Q1,
                                                              const V3& Q2, const V3& Q3, bool& robust)
{
    const V3 p1{0.0f, 0.0f, 0.0f};
    const V3 p2 = vsub(P2, P1), p3 = vsub(P3, P1);
    const V3 q1 = vsub(Q1, P1), q2 = vsub(Q2, P1), q3 = vsub(Q3, P1);
    float A = fmaxf(fmaxf(fmaxf(fabsf(p2.x), fabsf(p2.y)), fmaxf(fabsf(p2.z), fabsf(p3.x))),
                    fmaxf(fmaxf(fabsf(p3.y), fabsf(p3.z)), fmaxf(fabsf(q1.x), fabsf(q1.y))));
    A = fmaxf(A, fmaxf(fmaxf(fabsf(q1.z), fabsf(q2.x)), fmaxf(fabsf(q2.y), fabsf(q2.z))));
    A = fmaxf(A, fmaxf(fmaxf(fabsf(q3.x), fabsf(q3.y)), fabsf(q3.z)));
    robust = A >= 0x1p-20f && A <= 0x1p20f;
    const float A3 = A * A * A;
    const float B3 = 0x1p-14f * A3, B4 = 0x1p-10f * A3 * A;
    const V3 e1 = vsub(p2, p1), e2 = vsub(p3, p2), e3 = vsub(p1, p3);
    const V3 f1 = vsub(q2, q1), f2 = vsub(q3, q2), f3 = vsub(q1, q3);
    const V3 n1 = vcross(e1, e2);
    if (!project6_robust(n1, p1, p2, p3, q1, q2, q3, B3, robust)) return 0;
    const V3 m1 = vcross(f1, f2);
    if (!project6_robust(m1, p1, p2, p3, q1, q2, q3, B3, robust)) return 1;
    const V3 E[3] = {e1, e2, e3}, F[3] = {f1, f2, f3};
#pragma unroll
    for (uint32_t i = 0; i < 3; ++i)
#pragma unroll
        for (uint32_t j = 0; j < 3; ++j)
            if (!project6_robust(vcross(E[i], F[j]), p1, p2, p3, q1, q2, q3, B3, robust)) return 2 + 3 * i + j;
#pragma unroll
    for (uint32_t i = 0; i < 3; ++i)
        if (!project6_robust(vcross(E[i], n1), p1, p2, p3, q1, q2, q3, B4, robust)) return 11 + i;
#pragma unroll
    for (uint32_t j = 0; j < 3; ++j)
        if (!project6_robust(vcross(F[j], m1), p1, p2, p3, q1, q2, q3, B4, robust)) return 14 + j;
    return 17;
}

// Axis k with error bounds (kPass1Separated: its margin separates in every
// arithmetic; otherwise undecided). Relative extents outside [2^-20, 2^20]
// are never decided here (the bounds could under- or overflow).
__device__ __forceinline__ uint32_t bounded_axis_separates(uint32_t k, const V3& P1, const V3& P2, const V3& P3,
                                                           const V3& Q1, const V3& Q2, const V3& Q3)
{
    const V3 p2v = vsub(P2, P1), p3v = vsub(P3, P1);
    const V3 q1v = vsub(Q1, P1), q2v = vsub(Q2, P1), q3v = vsub(Q3, P1);
    float A = fmaxf(fmaxf(fmaxf(fabsf(p2v.x), fabsf(p2v.y)), fmaxf(fabsf(p2v.z), fabsf(p3v.x))),
                    fmaxf(fmaxf(fabsf(p3v.y), fabsf(p3v.z)), fmaxf(fabsf(q1v.x), fabsf(q1v.y))));
    A = fmaxf(A, fmaxf(fmaxf(fabsf(q1v.z), fabsf(q2v.x)), fmaxf(fabsf(q2v.y), fabsf(q2v.z))));
    A = fmaxf(A, fmaxf(fmaxf(fabsf(q3v.x), fabsf(q3v.y)), fabsf(q3v.z)));
    if (!(A >= 0x1p-20f && A <= 0x1p20f)) return kPass1Undecided;
    const EV3 zero{V3{0.0f, 0.0f, 0.0f}, V3{0.0f, 0.0f, 0.0f}};
    const EV3 p2 = ev_rel(p2v), p3 = ev_rel(p3v), q1 = ev_rel(q1v), q2 = ev_rel(q2v), q3 = ev_rel(q3v);
    LaneTri t;
    t.p2 = p2v;
    t.p3 = p3v;
    t.q1 = q1v;
    t.q2 = q2v;
    t.q3 = q3v;
    t.n1 = (k == 0 || (k >= 11 && k < 14)) ? ecross(esub(p2, zero), esub(p3, p2)) : zero;
    t.m1 = (k == 1 || k >= 14) ? ecross(esub(q2, q1), esub(q3, q2)) : zero;
    bool s32;
    return project6_bounded(axis_of(k, t), zero, p2, p3, q1, q2, q3, s32) == 0u ? kPass1Separated : kPass1Undecided;
}

// The lists of the precision passes, in prec_lists (4 x cand_cap words): the
// float hits (words), what the recheck leaves (words), and the recheck list
// ((candidate, axis) pairs), whose room the FP64 list takes once it is done.
struct PrecLists {
    uint32_t *hits, *left;
    uint2 *recheck, *fp64;
    __device__ __forceinline__ explicit PrecLists(const DetectArgs& a)
        : hits(a.prec_lists), left(a.prec_lists + a.cand_cap), recheck((uint2*)(a.prec_lists + 2 * (size_t)a.cand_cap)),
          fp64(recheck)
    {
    }
};

// A warp's entries for a global list, gathered in shared memory and appended 32
// at a time: an atomic for each list and 32 candidates queued up at the counters
// (3.2 M candidates of 16 pairs of sheets: 140 us so, 127 with this. The test in
// two goes, the walk's way, took 128, and 18 in place of 15 for 239 k).
template <typename T>
struct WarpList {
    T* buf;          // 64 entries in shared memory
    uint32_t n = 0;  // warp-uniform
    template <typename Store>
    __device__ __forceinline__ void flush(uint32_t count, uint32_t* counter, uint32_t lane, Store store)
    {
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(counter, count);
        at = __shfl_sync(0xffffffffu, at, 0);
        if (lane < count) store(at + lane, buf[n - count + lane]);
        n -= count;
        __syncwarp();
    }
    template <typename Store>
    __device__ __forceinline__ void push(bool pred, const T& v, uint32_t* counter, uint32_t lane, Store store)
    {
        const uint32_t m = __ballot_sync(0xffffffffu, pred);
        if (m == 0) return;
        if (pred) buf[n + __popc(m & ((1u << lane) - 1u))] = v;
        n += __popc(m);
        __syncwarp();
        if (n >= 32) flush(32, counter, lane, store);
    }
};

__global__ void __launch_bounds__(kDetectThreads) k_prec_classify(DetectArgs a)
{
    __shared__ uint4 s_hit[kWarps][64];
    __shared__ uint2 s_recheck[kWarps][64], s_other[kWarps][64];
    __shared__ uint32_t s_float[kWarps][64];
    const uint32_t n = min(a.counts[kCountCandSlots], a.cand_cap);
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const PrecLists lists(a);
    WarpList<uint4> hits{s_hit[w]};
    WarpList<uint2> rechecks{s_recheck[w]}, others{s_other[w]};
    WarpList<uint32_t> floats{s_float[w]};
    auto put_hit = [&](uint32_t at, const uint4& rec) {
        if (at < a.hit_cap) a.hits[at] = rec;
        else atomicOr(a.counts + kCountFlags, (uint32_t)kFlagHitOverflow);
    };
    // (the normals from the front, the other axes from the back: together no more than there are candidates)
    auto put_recheck = [&](uint32_t at, const uint2& e) { lists.recheck[at] = e; };
    auto put_other = [&](uint32_t at, const uint2& e) { lists.recheck[a.cand_cap - 1u - at] = e; };
    auto put_float = [&](uint32_t at, uint32_t i) { lists.hits[at] = i; };
    for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n; base += gridDim.x * blockDim.x) {
        const uint32_t i = base + lane;
        bool robust = false, hit = false, to_floats = false, to_recheck = false;
        uint4 rec = make_uint4(0, 0, 0, 0);
        uint32_t k = 17;
        if (i < n) {
            V3 P1, P2, P3, Q1, Q2, Q3;
            load_tris(a, a.cand[i], P1, P2, P3, Q1, Q2, Q3, rec);
            if (veq(P1, Q1) || veq(P1, Q2) || veq(P1, Q3) || veq(P2, Q1) || veq(P2, Q2) || veq(P2, Q3) || veq(P3, Q1) ||
                veq(P3, Q2) || veq(P3, Q3)) {
                hit = true;  // a shared vertex: never separated, in any arithmetic
            } else {
                k = tri_first_separating_axis(P1, P2, P3, Q1, Q2, Q3, robust);
                if (k != 17) to_recheck = bounded_axis_separates(k, P1, P2, P3, Q1, Q2, Q3) != kPass1Separated;
                else if (robust) hit = true;  // every axis overlaps beyond the error bounds
                else to_floats = true;
            }
        }
        hits.push(hit, rec, a.counts + kCountHits, lane, put_hit);
        floats.push(to_floats, i, a.counts + kCountPrecHits, lane, put_float);
        rechecks.push(to_recheck && k < 2u, make_uint2(i, k), a.counts + kCountPrecRecheck, lane, put_recheck);
        others.push(to_recheck && k >= 2u, make_uint2(i, k), a.counts + kCountPrecOther, lane, put_other);
    }
    if (hits.n > 0) hits.flush(hits.n, a.counts + kCountHits, lane, put_hit);
    if (floats.n > 0) floats.flush(floats.n, a.counts + kCountPrecHits, lane, put_float);
    if (rechecks.n > 0) rechecks.flush(rechecks.n, a.counts + kCountPrecRecheck, lane, put_recheck);
    if (others.n > 0) others.flush(others.n, a.counts + kCountPrecOther, lane, put_other);
}

__global__ void __launch_bounds__(kDetectThreads) k_prec_settle(DetectArgs a)
{
    const uint32_t n_hits = min(a.counts[kCountPrecHits], a.cand_cap);
    const uint32_t n = n_hits + min(a.counts[kCountPrecAgain], a.cand_cap);
    const PrecLists lists(a);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t n_warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t base = warp * 32; base < n; base += n_warps * 32) {
        const uint32_t j = base + lane;
        bool hit = false, queue = false;
        uint4 rec = make_uint4(0, 0, 0, 0);
        uint32_t i = 0, mask = 0;
        if (j < n) {
            i = j < n_hits ? lists.hits[j] : lists.left[j - n_hits];
            V3 P1, P2, P3, Q1, Q2, Q3;
            load_tris(a, a.cand[i], P1, P2, P3, Q1, Q2, Q3, rec);
            bool hit32 = false;
            const uint32_t r = tri_pass1(P1, P2, P3, Q1, Q2, Q3, mask, hit32);
            if (r == kPass1Hit) hit = true;
            else if (r == kPass1Undecided) {
                queue = true;
                mask |= hit32 ? 0x80000000u : 0u;
            }
        }
        append_hit(a, hit, rec, lane);
        const uint32_t q = warp_append(a.counts + kCountPrecFp64, queue, lane);
        if (queue) lists.fp64[q] = make_uint2(i, mask);
    }
}

// FP64 axis evaluation with every lane on the same instructions whatever its
// axis: the face normals n1 = e1 x e2 and m1 = f1 x f2 are formed once per
// candidate (FP64Tri), and per axis the cross product's two factors are
// picked by selects (integer work) before ONE FP64 cross product and the
// projections, so lanes on different kinds of axes do not issue their FP64
// instructions apart (each FP64 warp instruction takes the SM's FP64 pipe for
// many cycles). The operations and their order are the FP64 formula's
// (axis_overlaps_fp64); the projection of p1 = 0 is 0 in any order.
struct FP64Tri {
    D6 r;
    D3 n1, m1;
};
__device__ __forceinline__ FP64Tri fp64_tri(const V3& P1, const V3& P2, const V3& P3, const V3& Q1, const V3& Q2,
                                            const V3& Q3)
{
    FP64Tri t;
    t.r = fp64_relative(P1, P2, P3, Q1, Q2, Q3);
    t.n1 = dcross(t.r.p2, dsub(t.r.p3, t.r.p2));  // e1 = p2 - p1 = p2 exactly (p1 = +0)
    t.m1 = dcross(dsub(t.r.q2, t.r.q1), dsub(t.r.q3, t.r.q2));
    return t;
}
// A finite double as an unsigned key with the same order (-0 and +0 equal).
__device__ __forceinline__ uint64_t ordered_key(double d)
{
    uint64_t b = (uint64_t)__double_as_longlong(d);
    if (b == 0x8000000000000000ull) b = 0;
    return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ D3 dsel(bool c, const D3& a, const D3& b)
{
    return D3{c ? a.x : b.x, c ? a.y : b.y, c ? a.z : b.z};
}
// `edges`: some lane of the warp is on an edge axis (k >= 2); when none is,
// the warp skips the edge cross product (the plane axes are n1 and m1).
__device__ __forceinline__ bool axis_overlaps_fp64_uniform(uint32_t k, const FP64Tri& t, bool edges)
{
    const D3 z{0.0, 0.0, 0.0};
    const D6& r = t.r;
    D3 c = z;
    if (edges) {
        // e_i = (p2 - p1, p3 - p2, p1 - p3), f_j = (q2 - q1, q3 - q2, q1 - q3)
        const uint32_t i = k < 11 ? (k - 2) / 3 : k - 11;
        const uint32_t j = k < 11 ? (k - 2) % 3 : k - 14;
        const D3 E = dsub(dsel(i == 0, r.p2, dsel(i == 1, r.p3, z)), dsel(i == 0, z, dsel(i == 1, r.p2, r.p3)));
        const D3 F = dsub(dsel(j == 0, r.q2, dsel(j == 1, r.q3, r.q1)), dsel(j == 0, r.q1, dsel(j == 1, r.q2, r.q3)));
        const D3 X = dsel(k >= 14, F, E);
        const D3 Y = dsel(k < 11, F, dsel(k < 14, t.n1, t.m1));
        c = dcross(X, Y);
    }
    const D3 ax = dsel(k == 0, t.n1, dsel(k == 1, t.m1, c));
    // the comparisons on integer keys: the projections are finite, and after
    // -0 is made +0 the key order is the double order
    const uint64_t P1 = ordered_key(0.0), P2 = ordered_key(ddot(ax, r.p2)), P3 = ordered_key(ddot(ax, r.p3));
    const uint64_t Q1 = ordered_key(ddot(ax, r.q1)), Q2 = ordered_key(ddot(ax, r.q2)), Q3 = ordered_key(ddot(ax, r.q3));
    const uint64_t mx1 = max(max(P1, P2), P3), mn1 = min(min(P1, P2), P3);
    const uint64_t mx2 = max(max(Q1, Q2), Q3), mn2 = min(min(Q1, Q2), Q3);
    return !(mn1 > mx2) && !(mn2 > mx1);
}

// Idle lanes that trigger a refill: with the setups formed ahead a refill is
// loads only, so the lanes are refilled early (4 measured best of 4 / 8 / 12
// / 16 on the sheets; 16 was best while the refills formed the setups).
#ifndef OIBVH_FP64_REFILL
#define OIBVH_FP64_REFILL 4
#endif
constexpr uint32_t kFp64Refill = OIBVH_FP64_REFILL;

// ---------------------------------------------------------------------------
// Double-float pass: the FP64 list's undecided axes evaluated with pairs of
// floats on the FP32 pipe (the FP64 pipe of this part runs at 1/64 of its
// rate), with a bound W on |double-float value - exact| + |FP64 value -
// exact| for every quantity. The FP64 value of each projection then lies
// within W of the double-float one, so the FP64 comparisons of an axis are
// known whenever the intervals [v - W, v + W] of the two triangles' sets do
// not straddle: the axis separates in FP64, or overlaps in FP64, exactly as
// the FP64 pass would find. What stays undecided (nearly or exactly coplanar
// triangles, whose FP64 projections are rounding noise) goes on to FP64.
//
// Arithmetic (Joldes, Muller, Popescu, "Tight and rigorous error bounds for
// basic building blocks of double-word arithmetic", ACM TOMS 2017): exact
// TwoSum and Fast2Sum, the FMA-based exact product, AccurateDWPlusDW
// (relative error <= 3u^2/(1-4u)) and DWTimesDW3 (<= 4u^2), u = 2^-24. The
// relative coordinates are exact (TwoSum of two floats); the FP64 formula
// rounds them once (2^-53). Each operation then adds at most U|c| to W with
// U = 2^-44 (> 5u^2 + 2^-53, double-float and FP64 rounding together), and
// a product the propagated |a| W_b + |b| W_a + W_a W_b; 2^-140 per step covers
// underflowing low parts. The decision doubles W.
// ---------------------------------------------------------------------------
struct DF {
    float h, l;
};
struct DFB {  // a double-float value and its bound
    DF v;
    float w;
};
constexpr float kDfU = 0x1p-44f, kDfEta = 0x1p-140f;
__device__ __forceinline__ DF two_sum(float a, float b)
{
    const float s = __fadd_rn(a, b);
    const float ap = __fsub_rn(s, b), bp = __fsub_rn(s, ap);
    return DF{s, __fadd_rn(__fsub_rn(a, ap), __fsub_rn(b, bp))};
}
__device__ __forceinline__ DF fast_two_sum(float a, float b)  // |a| >= |b| (or a's exponent at least b's)
{
    const float s = __fadd_rn(a, b);
    return DF{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ DF df_add(const DF& x, const DF& y)  // AccurateDWPlusDW
{
    const DF s = two_sum(x.h, y.h), t = two_sum(x.l, y.l);
    const DF v = fast_two_sum(s.h, __fadd_rn(s.l, t.h));
    return fast_two_sum(v.h, __fadd_rn(t.l, v.l));
}
__device__ __forceinline__ DF df_neg(const DF& x) { return DF{-x.h, -x.l}; }
__device__ __forceinline__ DF df_mul(const DF& x, const DF& y)  // DWTimesDW3
{
    const float ch = __fmul_rn(x.h, y.h), cl1 = __fmaf_rn(x.h, y.h, -ch);
    const float tl1 = __fmaf_rn(x.h, y.l, __fmul_rn(x.l, y.l));
    const float cl2 = __fmaf_rn(x.l, y.h, tl1);
    return fast_two_sum(ch, __fadd_rn(cl1, cl2));
}
__device__ __forceinline__ float df_abs(const DF& x) { return __fadd_ru(fabsf(x.h), fabsf(x.l)); }
// The propagated part is scaled by 1 + 2^-20, which covers the FP64
// rounding of the propagated error itself (2^-53 of it, second order).
constexpr float kDfGrow = 1.0f + 0x1p-20f;
__device__ __forceinline__ float dfb_w_sum(const DFB& a, const DFB& b, const DF& c)
{
    return __fadd_ru(__fmaf_ru(kDfU, df_abs(c), __fmul_ru(kDfGrow, __fadd_ru(a.w, b.w))), kDfEta);
}
__device__ __forceinline__ DFB dfb_sub(const DFB& a, const DFB& b)
{
    const DF c = df_add(a.v, df_neg(b.v));
    return DFB{c, dfb_w_sum(a, b, c)};
}
__device__ __forceinline__ DFB dfb_add(const DFB& a, const DFB& b)
{
    const DF c = df_add(a.v, b.v);
    return DFB{c, dfb_w_sum(a, b, c)};
}
// |ab - exact| + |FP64 ab - exact| <= |a| W_b + |b| W_a + 2 W_a W_b, plus the
// two roundings of the product
__device__ __forceinline__ DFB dfb_mul(const DFB& a, const DFB& b)
{
    const DF c = df_mul(a.v, b.v);
    float w = __fmaf_ru(df_abs(a.v), b.w, __fmul_ru(df_abs(b.v), a.w));
    w = __fmaf_ru(__fmul_ru(2.0f, a.w), b.w, w);
    w = __fadd_ru(__fmaf_ru(kDfU, df_abs(c), __fmul_ru(kDfGrow, w)), kDfEta);
    return DFB{c, w};
}
struct DFB3 {
    DFB x, y, z;
};
__device__ __forceinline__ DFB3 dfb3_sub(const DFB3& a, const DFB3& b)
{
    return DFB3{dfb_sub(a.x, b.x), dfb_sub(a.y, b.y), dfb_sub(a.z, b.z)};
}
// the FP64 formula's cross product: (x.y*y.z - y.y*x.z, x.z*y.x - y.z*x.x, x.x*y.y - y.x*x.y)
__device__ __forceinline__ DFB3 dfb3_cross(const DFB3& x, const DFB3& y)
{
    return DFB3{dfb_sub(dfb_mul(x.y, y.z), dfb_mul(y.y, x.z)), dfb_sub(dfb_mul(x.z, y.x), dfb_mul(y.z, x.x)),
                dfb_sub(dfb_mul(x.x, y.y), dfb_mul(y.x, x.y))};
}
// (a.x*b.x + a.y*b.y) + a.z*b.z
__device__ __forceinline__ DFB dfb3_dot(const DFB3& a, const DFB3& b)
{
    return dfb_add(dfb_add(dfb_mul(a.x, b.x), dfb_mul(a.y, b.y)), dfb_mul(a.z, b.z));
}
// A relative coordinate P - P1: exact as a double-float; FP64 rounds it once.
__device__ __forceinline__ DFB dfb_rel(float a, float b)
{
    const DF d = two_sum(a, -b);
    return DFB{d, __fmul_ru(0x1p-53f, df_abs(d))};
}
__device__ __forceinline__ DFB3 dfb3_rel(const V3& p, const V3& o)
{
    return DFB3{dfb_rel(p.x, o.x), dfb_rel(p.y, o.y), dfb_rel(p.z, o.z)};
}
struct DFTri {
    DFB3 p2, p3, q1, q2, q3, n1, m1;
};
__device__ __forceinline__ DFB3 dfb3_sel(bool c, const DFB3& a, const DFB3& b)
{
    auto s = [c](const DFB& x, const DFB& y) {
        return DFB{DF{c ? x.v.h : y.v.h, c ? x.v.l : y.v.l}, c ? x.w : y.w};
    };
    return DFB3{s(a.x, b.x), s(a.y, b.y), s(a.z, b.z)};
}
// Axis k (0: n1, 1: m1, 2 + 3i + j: e_i x f_j, 11 + i: e_i x n1, 14 + j: f_j x
// m1), e_i = (p2 - 0, p3 - p2, 0 - p3), f_j = (q2 - q1, q3 - q2, q1 - q3) as
// the FP64 formula forms them (p2 - 0 and 0 - p3 are exact; their bounds
// grow by one rounding's share, which only widens the intervals). The two
// factors of the cross product are picked by selects, so the lanes of a warp
// run one cross product whatever their axes; `edges` (warp-uniform) is false
// when no lane of the warp is on a cross-product axis.
__device__ __forceinline__ DFB3 dfb_axis(uint32_t k, const DFTri& t, bool edges)
{
    if (!edges) return dfb3_sel(k == 0, t.n1, t.m1);
    const DFB z{DF{0.0f, 0.0f}, 0.0f};
    const DFB3 Z{z, z, z};
    const uint32_t i = k < 11 ? (k - 2) / 3 : k - 11;  // edge of A (axes 2..13)
    const uint32_t j = k < 11 ? (k - 2) % 3 : k - 14;  // edge of B (axes 2..10, 14..16)
    const DFB3 E = dfb3_sub(dfb3_sel(i == 0, t.p2, dfb3_sel(i == 1, t.p3, Z)),
                            dfb3_sel(i == 0, Z, dfb3_sel(i == 1, t.p2, t.p3)));
    const DFB3 F = dfb3_sub(dfb3_sel(j == 0, t.q2, dfb3_sel(j == 1, t.q3, t.q1)),
                            dfb3_sel(j == 0, t.q1, dfb3_sel(j == 1, t.q2, t.q3)));
    const bool ef = k >= 2 && k < 11, en = k >= 11 && k < 14;
    const DFB3 c = dfb3_cross(dfb3_sel(ef || en, E, F), dfb3_sel(ef, F, dfb3_sel(en, t.n1, t.m1)));
    return dfb3_sel(k == 0, t.n1, dfb3_sel(k == 1, t.m1, c));
}
// What FP64 finds on the axis, known from double-floats: 0 = separates, 1 =
// overlaps, 2 = undecided.
__device__ __forceinline__ uint32_t dfb_decide(const DFB3& ax, const DFTri& t)
{
    const DFB P[3] = {DFB{DF{0.0f, 0.0f}, 0.0f}, dfb3_dot(ax, t.p2), dfb3_dot(ax, t.p3)};
    const DFB Q[3] = {dfb3_dot(ax, t.q1), dfb3_dot(ax, t.q2), dfb3_dot(ax, t.q3)};
    // intervals that hold the FP64 values: value as hi + lo (the sum's rounding
    // is inside the doubled bound)
    float pl = 3.4e38f, ph = -3.4e38f, ql = 3.4e38f, qh = -3.4e38f;  // min of lows, max of highs, ...
    float plh = -3.4e38f, phl = 3.4e38f, qlh = -3.4e38f, qhl = 3.4e38f;  // max of lows, min of highs
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float v = __fadd_rn(P[i].v.h, P[i].v.l), w = __fmul_ru(2.0f, __fadd_ru(P[i].w, __fmul_ru(0x1p-23f, fabsf(v))));
        const float lo = __fsub_rd(v, w), hi = __fadd_ru(v, w);
        pl = fminf(pl, lo); ph = fmaxf(ph, hi); plh = fmaxf(plh, lo); phl = fminf(phl, hi);
        const float u = __fadd_rn(Q[i].v.h, Q[i].v.l), x = __fmul_ru(2.0f, __fadd_ru(Q[i].w, __fmul_ru(0x1p-23f, fabsf(u))));
        const float ulo = __fsub_rd(u, x), uhi = __fadd_ru(u, x);
        ql = fminf(ql, ulo); qh = fmaxf(qh, uhi); qlh = fmaxf(qlh, ulo); qhl = fminf(qhl, uhi);
    }
    // FP64 mn1 lies in [pl, phl], mx1 in [plh, ph], mn2 in [ql, qhl], mx2 in [qlh, qh]
    if (pl > qh || ql > ph) return 0u;             // mn1 > mx2 or mn2 > mx1 for sure
    if (phl < qlh && qhl < plh) return 1u;         // mn1 < mx2 and mn2 < mx1 for sure
    return 2u;
}
__device__ __forceinline__ uint32_t dfb_axis_fp64(uint32_t k, const DFTri& t, bool edges)
{
    return dfb_decide(dfb_axis(k, t, edges), t);
}
__device__ __forceinline__ float max_abs_diff(const V3& a, const V3& b)
{
    return fmaxf(fmaxf(fabsf(__fsub_rn(a.x, b.x)), fabsf(__fsub_rn(a.y, b.y))), fabsf(__fsub_rn(a.z, b.z)));
}

// The recheck list: candidates that an axis separates in float by less than the
// bound. The same axis with double-floats: where FP64 separates there too the
// candidate is done, else it needs every axis. (Sending them all through the 17
// bounded axes and then through the double-float pass took 190 us for the
// 553 k of 16 pairs of sheets, whose margins of 1e-8 to 1e-7 no float bound
// decides; with this pass 62 us, 35 of them here.) Normals take one cross product
// with its factors picked by selects; they and the other axes are listed from the
// two ends, so that a warp has one kind (57 us mixed, half the lanes idle).
__global__ void __launch_bounds__(kDetectThreads) k_prec_recheck(DetectArgs a)
{
    const uint32_t n = min(a.counts[kCountPrecRecheck], a.cand_cap), n_other = min(a.counts[kCountPrecOther], a.cand_cap - n);
    const uint32_t lane = threadIdx.x & 31, rows = (n + 31u) / 32u, all_rows = rows + (n_other + 31u) / 32u;
    const PrecLists lists(a);
    for (uint32_t row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < all_rows; row += gridDim.x * (blockDim.x >> 5)) {
        const bool normals = row < rows;  // a row's lanes have the same kind of axis
        const uint32_t at = 32u * (normals ? row : row - rows) + lane;
        bool again = false;
        uint2 item = make_uint2(0, 0);
        if (at < (normals ? n : n_other)) {
            item = lists.recheck[normals ? at : a.cand_cap - 1u - at];
            V3 P1, P2, P3, Q1, Q2, Q3;
            uint4 rec;
            load_tris(a, a.cand[item.x], P1, P2, P3, Q1, Q2, Q3, rec);
            const float A = fmaxf(fmaxf(max_abs_diff(P2, P1), max_abs_diff(P3, P1)),
                                  fmaxf(fmaxf(max_abs_diff(Q1, P1), max_abs_diff(Q2, P1)), max_abs_diff(Q3, P1)));
            // (fmaxf drops a NaN, this sum does not)
            const float sum = (P2.x + P2.y + P2.z) + (P3.x + P3.y + P3.z) + (Q1.x + Q1.y + Q1.z) + (Q2.x + Q2.y + Q2.z) +
                              (Q3.x + Q3.y + Q3.z) + (P1.x + P1.y + P1.z);
            again = true;
            if (A >= 0x1p-20f && A <= 0x1p20f && fabsf(sum) <= 3e38f) {  // (else the bounds could under- or overflow)
                DFTri t;
                t.p2 = dfb3_rel(P2, P1);
                t.p3 = dfb3_rel(P3, P1);
                t.q1 = dfb3_rel(Q1, P1);
                t.q2 = dfb3_rel(Q2, P1);
                t.q3 = dfb3_rel(Q3, P1);
                if (normals) {
                    const bool nrm = item.y == 0;  // n1 = p2 x (p3 - p2), m1 = (q2 - q1) x (q3 - q2)
                    const DFB3 c = dfb3_cross(dfb3_sel(nrm, t.p2, dfb3_sub(t.q2, t.q1)),
                                              dfb3_sub(dfb3_sel(nrm, t.p3, t.q3), dfb3_sel(nrm, t.p2, t.q2)));
                    again = dfb_decide(c, t) != 0u;
                } else {
                    t.n1 = dfb3_cross(t.p2, dfb3_sub(t.p3, t.p2));
                    t.m1 = dfb3_cross(dfb3_sub(t.q2, t.q1), dfb3_sub(t.q3, t.q2));
                    again = dfb_axis_fp64(item.y, t, true) != 0u;
                }
            }
        }
        const uint32_t q = warp_append(a.counts + kCountPrecAgain, again, lane);
        if (again) lists.left[q] = item.x;
    }
}

// Idle lanes that trigger a refill of the double-float pass (a refill forms
// the new candidates' double-float vertices and normals with only the idle
// lanes active, so refilling early costs setups, late costs idle steps).
#ifndef OIBVH_DF_REFILL
#define OIBVH_DF_REFILL 12
#endif
constexpr uint32_t kDfRefill = OIBVH_DF_REFILL;

// The FP64 list through the double-float pass: each lane holds a candidate
// and evaluates one of its undecided axes per step, all lanes of a warp on
// the same instructions (dfb_axis picks the axis with selects), until an
// axis separates for sure or the mask is done; the axes still open (and the
// float answer) go to the list the FP64 passes take. A lane whose candidate
// is decided is refilled from the warp's share of the list once enough lanes
// are idle: the masks differ in length (most candidates end at their first
// axis, coplanar ones run all of theirs), so a lane per candidate for the
// whole walk would idle most lanes. The warp's share is chunks of 32
// consecutive entries, grid-strided.
__global__ void __launch_bounds__(kDetectThreads) k_prec_df(DetectArgs a)
{
    const uint32_t n = min(a.counts[kCountPrecFp64], a.cand_cap);
    const uint2* list = (const uint2*)(a.prec_lists + 2 * (size_t)a.cand_cap);
    uint2* left = (uint2*)a.prec_lists;  // the room of the float hits and the recheck's rest, free after the bounded pass
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t W = (gridDim.x * blockDim.x) >> 5;
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    // the t-th entry of this warp's share (increasing in t)
    auto entry = [&](uint32_t t) { return (w + (t >> 5) * W) * 32u + (t & 31u); };
    uint32_t t_next = 0, dis = 0;
    bool more = entry(0) < n;
    bool live = false;
    uint2 item = make_uint2(0, 0);
    uint4 rec = make_uint4(0, 0, 0, 0);
    uint32_t mask = 0, open = 0;
    bool separated = false;
    DFTri t;
    const DFB z{DF{0.0f, 0.0f}, 0.0f};
    t.p2 = t.p3 = t.q1 = t.q2 = t.q3 = t.n1 = t.m1 = DFB3{z, z, z};
    for (;;) {
        const uint32_t idle = __ballot_sync(0xffffffffu, !live);
        if (more && (__popc(idle) >= kDfRefill || idle == 0xffffffffu)) {
            if (!live) {
                const uint32_t j = entry(t_next + __popc(idle & ((1u << lane) - 1u)));
                if (j < n) {
                    item = list[j];
                    V3 P1, P2, P3, Q1, Q2, Q3;
                    load_tris(a, a.cand[item.x], P1, P2, P3, Q1, Q2, Q3, rec);
                    live = true;
                    mask = item.y & 0x1ffffu;
                    open = 0;
                    separated = false;
                    const float A =
                        fmaxf(fmaxf(fmaxf(fabsf(__fsub_rn(P2.x, P1.x)), fabsf(__fsub_rn(P2.y, P1.y))),
                                    fmaxf(fabsf(__fsub_rn(P2.z, P1.z)), fabsf(__fsub_rn(P3.x, P1.x)))),
                              fmaxf(fmaxf(fabsf(__fsub_rn(P3.y, P1.y)), fabsf(__fsub_rn(P3.z, P1.z))),
                                    fmaxf(fabsf(__fsub_rn(Q1.x, P1.x)), fabsf(__fsub_rn(Q1.y, P1.y)))));
                    const float A2 =
                        fmaxf(fmaxf(fmaxf(fabsf(__fsub_rn(Q1.z, P1.z)), fabsf(__fsub_rn(Q2.x, P1.x))),
                                    fmaxf(fabsf(__fsub_rn(Q2.y, P1.y)), fabsf(__fsub_rn(Q2.z, P1.z)))),
                              fmaxf(fmaxf(fabsf(__fsub_rn(Q3.x, P1.x)), fabsf(__fsub_rn(Q3.y, P1.y))),
                                    fabsf(__fsub_rn(Q3.z, P1.z))));
                    const float Am = fmaxf(A, A2);
                    if (!(Am >= 0x1p-20f && Am <= 0x1p20f)) {
                        open = mask;  // the bounds could under- or overflow: all to FP64
                        mask = 0;
                    } else {
                        t.p2 = dfb3_rel(P2, P1);
                        t.p3 = dfb3_rel(P3, P1);
                        t.q1 = dfb3_rel(Q1, P1);
                        t.q2 = dfb3_rel(Q2, P1);
                        t.q3 = dfb3_rel(Q3, P1);
                        t.n1 = dfb3_cross(t.p2, dfb3_sub(t.p3, t.p2));
                        t.m1 = dfb3_cross(dfb3_sub(t.q2, t.q1), dfb3_sub(t.q3, t.q2));
                    }
                }
            }
            t_next += __popc(idle);
            more = entry(t_next) < n;
        }
        if (!__any_sync(0xffffffffu, live)) {
            if (!more) break;
            continue;
        }
        const bool busy = live && mask != 0u;
        if (__any_sync(0xffffffffu, busy)) {
            const uint32_t k = busy ? __ffs(mask) - 1 : 0u;
            const bool edges = __any_sync(0xffffffffu, busy && k >= 2);
            const uint32_t r = dfb_axis_fp64(k, t, edges);
            if (busy) {
                mask &= mask - 1;
                if (r == 0u) {
                    separated = true;
                    mask = 0;
                } else if (r == 2u) {
                    open |= 1u << k;
                }
            }
        }
        // decided lanes: the hit, or the entry with its open axes for FP64
        const bool done = live && mask == 0u;
        const bool hit = done && !separated && open == 0u;  // every axis overlaps in FP64
        const bool keep = done && !separated && open != 0u;
        if (done && !keep) dis += (hit != ((item.y >> 31) != 0u)) ? 1u : 0u;
        append_hit(a, hit, rec, lane);
        const uint32_t q = warp_append(a.counts + kCountPrecLeft, keep, lane);
        if (keep) left[q] = make_uint2(item.x, open | (item.y & 0x80000000u));
        if (done) live = false;
    }
    const uint32_t nd = __reduce_add_sync(0xffffffffu, dis);
    if (lane == 0 && nd) atomicAdd(a.counts + kCountDisagree, nd);
}

// FP64 setups (fp64_tri and the hit record) of the FP64 list's first
// fp64_tri_cap entries, one entry per lane: formed here with every lane of a
// warp busy, where k_prec_fp64 would form them in its refills with only the
// refilling lanes. Structure of arrays: row r of entry i at r * cap + i.
__device__ __forceinline__ void fp64_tri_store(double* base, uint32_t cap, uint32_t i, const FP64Tri& t, const uint4& rec)
{
    const double v[21] = {t.r.p2.x, t.r.p2.y, t.r.p2.z, t.r.p3.x, t.r.p3.y, t.r.p3.z, t.r.q1.x,
                          t.r.q1.y, t.r.q1.z, t.r.q2.x, t.r.q2.y, t.r.q2.z, t.r.q3.x, t.r.q3.y,
                          t.r.q3.z, t.n1.x, t.n1.y, t.n1.z, t.m1.x, t.m1.y, t.m1.z};
#pragma unroll
    for (uint32_t r = 0; r < 21; ++r) base[(size_t)r * cap + i] = v[r];
    uint64_t* w = (uint64_t*)base;
    w[(size_t)21 * cap + i] = ((uint64_t)rec.y << 32) | rec.x;
    w[(size_t)22 * cap + i] = ((uint64_t)rec.w << 32) | rec.z;
}
__device__ __forceinline__ void fp64_tri_load(const double* base, uint32_t cap, uint32_t i, FP64Tri& t, uint4& rec)
{
    double v[21];
#pragma unroll
    for (uint32_t r = 0; r < 21; ++r) v[r] = __ldcg(base + (size_t)r * cap + i);
    t.r.p2 = D3{v[0], v[1], v[2]};
    t.r.p3 = D3{v[3], v[4], v[5]};
    t.r.q1 = D3{v[6], v[7], v[8]};
    t.r.q2 = D3{v[9], v[10], v[11]};
    t.r.q3 = D3{v[12], v[13], v[14]};
    t.n1 = D3{v[15], v[16], v[17]};
    t.m1 = D3{v[18], v[19], v[20]};
    const uint64_t* w = (const uint64_t*)base;
    const uint64_t r0 = __ldcg(w + (size_t)21 * cap + i), r1 = __ldcg(w + (size_t)22 * cap + i);
    rec = make_uint4((uint32_t)r0, (uint32_t)(r0 >> 32), (uint32_t)r1, (uint32_t)(r1 >> 32));
}
__global__ void __launch_bounds__(kDetectThreads) k_prec_fp64_setup(DetectArgs a)
{
    const uint32_t n = min(min(a.counts[kCountPrecLeft], a.cand_cap), a.fp64_tri_cap);
    const uint2* list = (const uint2*)a.prec_lists;  // what the double-float pass left open
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        V3 P1, P2, P3, Q1, Q2, Q3;
        uint4 rec;
        load_tris(a, a.cand[list[i].x], P1, P2, P3, Q1, Q2, Q3, rec);
        fp64_tri_store(a.fp64_tri, a.fp64_tri_cap, i, fp64_tri(P1, P2, P3, Q1, Q2, Q3), rec);
    }
}

// The FP64 list in lockstep: every lane holds one undecided candidate and
// evaluates ONE of its undecided axes (in order) per iteration, so the FP64
// pipe sees full warps however many axes each candidate needs; a lane whose
// candidate is decided (an axis separates: no hit; none left: hit) takes the
// next one from the warp's range, once kFp64Refill lanes are idle (a refill
// costs the setup's loads, or, past the setup buffer, the chain candidate ->
// faces -> vertices and the setup's FP64 work).
__global__ void __launch_bounds__(kDetectThreads) k_prec_fp64(DetectArgs a)
{
    const uint32_t n = min(a.counts[kCountPrecLeft], a.cand_cap);
    const uint2* list = (const uint2*)a.prec_lists;  // what the double-float pass left open
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t n_warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t per = (n + n_warps - 1) / n_warps;
    const uint32_t lo = min(n, warp * per), hi = min(n, lo + per);
    uint32_t next = lo;  // warp-uniform
    bool busy = false;
    uint32_t mask = 0, evaluated = 0, dis = 0, cands = 0;
    FP64Tri t{};
    uint4 rec = make_uint4(0, 0, 0, 0);
    for (;;) {
        const uint32_t idle = __ballot_sync(0xffffffffu, !busy);
        const bool refill = __popc(idle) >= kFp64Refill || idle == 0xffffffffu;
        const uint32_t take = refill ? min((uint32_t)__popc(idle), hi - next) : 0u;
        const uint32_t rank = __popc(idle & ((1u << lane) - 1u));
        if (!busy && rank < take) {
            const uint32_t i = next + rank;
            const uint2 item = list[i];
            if (i < a.fp64_tri_cap) {  // formed by k_prec_fp64_setup
                fp64_tri_load(a.fp64_tri, a.fp64_tri_cap, i, t, rec);
            } else {
                V3 P1, P2, P3, Q1, Q2, Q3;
                load_tris(a, a.cand[item.x], P1, P2, P3, Q1, Q2, Q3, rec);
                t = fp64_tri(P1, P2, P3, Q1, Q2, Q3);
            }
            mask = item.y;
            busy = true;
            ++cands;
        }
        next += take;
        bool hit = false;
        const uint32_t k = busy ? __ffs(mask & 0x1ffffu) - 1 : 0u;
        const bool edges = __any_sync(0xffffffffu, busy && k >= 2);
        if (busy) {
            mask &= mask - 1;  // the lowest set bit is the axis just taken
            ++evaluated;
            const bool overlaps = axis_overlaps_fp64_uniform(k, t, edges);
            if (!overlaps || (mask & 0x1ffffu) == 0) {
                busy = false;
                hit = overlaps;
                dis += hit != ((mask >> 31) != 0u) ? 1u : 0u;
            }
        }
        append_hit(a, hit, rec, lane);
        if (!__any_sync(0xffffffffu, busy) && next >= hi) break;
    }
    const uint32_t axes = __reduce_add_sync(0xffffffffu, evaluated);
    const uint32_t nc = __reduce_add_sync(0xffffffffu, cands);
    const uint32_t nd = __reduce_add_sync(0xffffffffu, dis);
    if (lane == 0) {
        if (axes) atomicAdd(a.counts + kCountFp64Axes, axes);
        if (nc) atomicAdd(a.counts + kCountFp64Cands, nc);
        if (nd) atomicAdd(a.counts + kCountDisagree, nd);
    }
}

// The traversal kernels' fused narrow phase is the float test only; precision
// mode runs the broad phase alone and then its narrow-phase passes.
static inline bool fused_precision(const DetectArgs& a) { return a.precision && a.fuse_narrow; }

cudaError_t launch_begin(const DetectArgs& a, uint32_t hits_before, cudaStream_t s)
{
    if (fused_precision(a)) return cudaErrorInvalidValue;
    note_launches(1);
    k_begin<<<1, 256, 0, s>>>(a, hits_before);
    return cudaGetLastError();
}

cudaError_t launch_publish(const DetectArgs& a, cudaStream_t s)
{
    note_launches(1);
    k_publish<<<1, 256, 0, s>>>(a);
    return cudaGetLastError();
}

static size_t walk_smem(uint32_t cap) { return (size_t)kWarps * walk_ring(cap) * 8; }  // one ring per warp

typedef void (*WalkKernel)(DetectArgs, uint32_t, uint32_t, bool);
static WalkKernel walk_kernel(bool fused, bool one)
{
    return fused ? (one ? k_walk<true, true> : k_walk<true, false>) : (one ? k_walk<false, true> : k_walk<false, false>);
}

static cudaError_t walk_configure()
{
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && configured[dev]) return cudaSuccess;
    const int smem = (int)walk_smem(kWalkCapMax);
    for (int k = 0; k < 4; ++k) {
        const cudaError_t e = cudaFuncSetAttribute(walk_kernel(k & 1, k & 2), cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
    }
    if (dev >= 0 && dev < 64) configured[dev] = true;
    return cudaSuccess;
}

cudaError_t launch_walk(const DetectArgs& a, uint32_t total0, uint32_t from, uint32_t to, bool hand_over, cudaStream_t s)
{
    if (fused_precision(a)) return cudaErrorInvalidValue;
    if (a.walk_cap > kWalkCapMax || (a.walk_cap % 32) != 0) return cudaErrorInvalidValue;
    cudaError_t e = walk_configure();
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)a.grid);
    cfg.blockDim = dim3(kDetectThreads);
    cfg.dynamicSmemBytes = walk_smem(a.walk_cap);
    cfg.stream = s;
    cfg.attrs = &attr;
    for (uint32_t r = from; r < to && e == cudaSuccess; ++r) {
        note_launches(1);
        cfg.numAttrs = a.ahead && r > 0 ? 1 : 0;  // (round 0 waits for all before it, as does one behind anything but a round)
        e = cudaLaunchKernelEx(&cfg, walk_kernel(a.fuse_narrow, a.n_pairs == 1), a, total0, r, hand_over && r + 1 == to);
    }
    return e;
}

int walk_blocks_per_sm(uint32_t walk_cap, bool fused)
{
    static std::atomic<int> known[64][2][kWalkCapMax / 32 + 1];
    int dev = 0;
    if (walk_cap > kWalkCapMax || cudaGetDevice(&dev) != cudaSuccess || walk_configure() != cudaSuccess) return 1;
    std::atomic<int>* cached = dev >= 0 && dev < 64 ? &known[dev][fused][walk_cap / 32] : nullptr;
    if (cached && cached->load(std::memory_order_relaxed)) return cached->load(std::memory_order_relaxed);
    int n = 0, m = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, walk_kernel(fused, false), kDetectThreads, walk_smem(walk_cap));
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&m, walk_kernel(fused, true), kDetectThreads, walk_smem(walk_cap));
    n = std::min(n, m);
    if (e != cudaSuccess || n < 1) return 1;
    if (cached) cached->store(n, std::memory_order_relaxed);
    return n;
}

uint32_t narrow_kernels(const DetectArgs& a) { return a.precision ? (a.fp64_tri_cap ? 6u : 5u) : 1u; }

cudaError_t launch_narrow(const DetectArgs& a, cudaStream_t s)
{
    if (a.precision) {
        if (a.prec_lists == nullptr || (a.fp64_tri_cap && a.fp64_tri == nullptr)) return cudaErrorInvalidValue;
        note_launches(narrow_kernels(a));
        k_prec_classify<<<a.grid, kDetectThreads, 0, s>>>(a);
        k_prec_recheck<<<a.grid, kDetectThreads, 0, s>>>(a);
        k_prec_settle<<<a.grid, kDetectThreads, 0, s>>>(a);
        k_prec_df<<<a.grid, kDetectThreads, 0, s>>>(a);
        if (a.fp64_tri_cap) k_prec_fp64_setup<<<a.grid, kDetectThreads, 0, s>>>(a);
        k_prec_fp64<<<a.grid, kDetectThreads, 0, s>>>(a);
        return cudaGetLastError();
    }
    note_launches(1);
    k_narrow<<<a.grid, kDetectThreads, 0, s>>>(a);
    return cudaGetLastError();
}

} // namespace oibvh
