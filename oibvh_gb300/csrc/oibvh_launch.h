// Host-side launchers of the device kernels (one translation unit per stage).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "oibvh_common.cuh"

namespace oibvh {

// Count of this library's kernel launches (all devices), for benchmarks.
void note_launches(uint64_t n);

// One tree of a (possibly multi-tree) refit launch.
struct RefitJob {
    float4* box;           // internal nodes
    const uint4* face;
    const float4* pos;
    TreeShape shape;
    uint32_t block_begin;  // first CTA of this tree in the launch
    uint32_t n_blocks;
    uint32_t* counters;    // refit_counters_per_tree() words, zero before the first refit (each leaves them zero)
    uint32_t pad0;
};

// A refit's positions as the caller gave them (xyz; tree vertex v is the
// caller's vperm[v]); xyz == nullptr: the tree's own positions.
struct RefitSource {
    const float* xyz;
    const uint32_t* vperm;
    uint32_t nV;
};

// Rigid transforms done by the refit that follows them (launch_transform_refit):
// the trees' transform jobs, one for each refit job, the packed rest positions
// in the trees' vertex order (nullptr: each job's own source) and the matrices.
struct BuildJob;
struct RefitRest {
    const BuildJob* jobs;
    const float4* rest;
    const float* mats;
};

// One tree of a multi-tree build / transform launch.
struct BuildJob {
    const float4* pos;      // positions to build from (transform source when no packed rest array is given)
    const uint32_t* tri;    // faces as given (3 * nT)
    uint4* face_out;        // Morton-ordered face records
    float4* pos_out;        // transform target (the tree's own positions)
    uint32_t nV, nT;
    uint32_t vblock_begin;  // first CTA of this tree in vertex-chunk launches (256 vertices per CTA)
    uint32_t ftile_begin;   // first tile of this tree in the build's face tiles (kBuildTile faces each)
    uint32_t vtile_begin;   // the same for its vertex tiles
    uint32_t face_off;      // first face of this tree in the build's keys
    uint32_t vert_off;      // first vertex of this tree in packed rest positions
    uint32_t pad0;
    const uint32_t* vperm;  // tree vertex v is the caller's vertex vperm[v] (nullptr: the same order)
    uint32_t* vperm_out;    // the tree's map buffer (nV entries), rewritten by the renumbering
    uint32_t* tri_rw;       // the tree's faces (3 * nT), rewritten by the renumbering (tri, writable)
};

// Id of the current context, 0 when it cannot be read (host.cu). What lives as
// long as a context (pools, pinned pages, kernel attributes, symbol addresses) is
// kept under it: after cudaDeviceReset the next context starts without them.
unsigned long long current_context_id();

// build_kernels.cu
constexpr uint32_t kBuildTile = 4096;  // faces (vertices) of a tile
struct BuildScratch {
    uint32_t* fail;           // a wait ran out: the build's later kernels return at once
    uint32_t* tickets;        // next tile of each sort pass, next block of the renumbering
    uint32_t* bounds;         // 6 words per job
    uint32_t* hist;           // per job and pass: 256 digit counts
    uint32_t* order_state;    // per face tile, then per vertex tile: look-back states
    uint32_t* marks;          // a bit per face corner (sorted faces): a vertex's first use
    uint32_t* counts;         // per word of marks: the tree's marks before it
    uint32_t* unused;         // per 1024 vertices: the tree's unused vertices before them
    uint32_t* sort_state[2];  // per sort tile: 256 look-back states, in turn between passes
    size_t zero_bytes;
    uint32_t *keys[2], *vals[2], *hi;  // n_faces each (hi: 63-bit keys only)
    uint32_t *first, *inv, *vperm_new; // n_verts: first-use slot, new number, caller-order map in the new order
    float4* pos_new;                   // n_verts
};
constexpr uint32_t kLookbackPolls = 1u << 20;
struct BuildArgs {
    const BuildJob* jobs;   // one job: nullptr, and the job in `one`
    BuildJob one;
    const uint32_t *ftile_job, *vtile_job;  // tile -> job
    uint32_t f_tiles, v_tiles;
    uint32_t half_tiles;    // the sort's tiles are of kBuildTile / 2 faces
    uint32_t passes;        // 4: the reference's 30-bit keys; 8: 63 bits (21 per axis)
    uint32_t* host_error;   // pinned word, set when the build gave up
    uint32_t polls;         // looks at a tile's predecessors before it gives up (kLookbackPolls: about a second)
    BuildScratch sc;
};
// Bytes of the build's scratch, and its parts set from `p`.
size_t build_scratch(BuildArgs& a, uint32_t n_jobs, uint32_t n_faces, uint32_t n_verts, void* p);
// Bounds, codes, sort, sorted faces and vertex renumbering of every job: face
// records, `tri` and positions get the new vertex numbers, vperm_out the new
// caller-order map.
cudaError_t launch_build(const BuildArgs& a, cudaStream_t s);
// The whole build of one tree, boxes included, in one launch, for trees that
// build_is_small() (up to 4,096 faces and vertices).
bool build_is_small(uint32_t nT, uint32_t nV);
cudaError_t launch_build_small(const BuildJob& job, const TreeShape& shape, float4* box, bool wide, cudaStream_t s);
// rest: packed positions of all jobs in each caller's vertex order (read
// through the jobs' vperm), or in each tree's order (rest_tree_order); nullptr: each job's own pos.
// Writes each job's pos_out.
cudaError_t launch_transform_multi(const BuildJob* d_jobs, uint32_t n_jobs, uint32_t v_blocks, const uint32_t* vjob,
                                   const float4* rest, const float* mats, bool rest_tree_order, cudaStream_t s);
cudaError_t launch_gather_rest_multi(const BuildJob* d_jobs, uint32_t n_jobs, uint32_t v_blocks, const uint32_t* vjob,
                                     const float4* rest, float4* out, cudaStream_t s);
// pos[v] = (xyz of the caller's vertex vperm[v], 0); vperm == nullptr: the same order
cudaError_t launch_xyz_to_pos4(const float* xyz, const uint32_t* vperm, uint32_t nV, float4* pos, cudaStream_t s);
// pos[v] = src[vperm[v]] (vperm == nullptr: a copy)
cudaError_t launch_gather_pos4(const float4* src, const uint32_t* vperm, uint32_t nV, float4* pos, cudaStream_t s);
// refit_kernels.cu
// refit CTAs of a tree of nT leaves with level groups of group_log2 levels
// (9, 10 or 11; 0 = 10, the single-tree refit's)
uint32_t refit_blocks_for(uint32_t nT, uint32_t group_log2 = 0);
uint32_t refit_counters_per_tree();
bool refit_takes_xyz(uint32_t nT, uint32_t nV);  // whether launch_refit_one should be given `src` rather than converted positions
cudaError_t launch_refit_one(const RefitJob& job, const RefitSource& src, cudaStream_t s);
cudaError_t launch_leaf_boxes(const uint4* face, const float4* pos, uint32_t nT, float4* out, cudaStream_t s);
// block_job: optional host-built map from a refit CTA to its job (nullptr:
// each CTA binary-searches the job table).
cudaError_t launch_refit(const RefitJob* d_jobs, uint32_t n_jobs, uint32_t total_blocks, const uint32_t* block_job,
                         uint32_t group_log2, cudaStream_t s);
// launch_transform_multi and launch_refit in one
cudaError_t launch_transform_refit(const RefitJob* d_jobs, uint32_t n_jobs, uint32_t total_blocks,
                                   const uint32_t* block_job, uint32_t group_log2, const RefitRest& rest, cudaStream_t s);
bool transform_refit_pays(uint64_t n_faces);  // whether a captured frame should
bool transform_refit_takes(uint32_t nT, uint32_t nV);  // whether it should with such a tree (and a server batch)

// detect_kernels.cu
struct DetectArgs {
    const PairView* pairs;  // n_pairs records (the walk of one pair reads `one` instead)
    uint32_t n_pairs;
    PairView one;           // the record of the only pair when n_pairs == 1
    uint64_t* work[2];     // traversal work lists (ping-pong between rounds)
    uint32_t work_cap;
    uint64_t* cand;        // broad-only mode: candidate leaf pairs
    uint32_t cand_cap;
    uint4* hits;
    uint32_t hit_cap;
    uint32_t* counts;      // see kCount* below
    uint32_t* host;        // pinned: where the last walk round (or launch_publish) puts the counters; nullptr: nowhere
    uint4* host_hits;      // pinned: and the hits, when there are at most host_hit_cap
    uint32_t host_hit_cap;
    uint32_t* counts_next; // with host: the counter block that the walk clears for the next traversal (nullptr: none)
    uint32_t* prec_lists;  // precision mode, 4 x cand_cap words: the passes' lists (PrecLists)
    double* fp64_tri;      // precision mode: the FP64 list's setups, kFp64TriRows rows of fp64_tri_cap
                           // (structure of arrays; nullptr: each is formed where it is used)
    uint32_t fp64_tri_cap;
    uint32_t fuse_narrow;  // 1: test candidates in the traversal; 0: store them
    int grid;              // CTAs of the grid-stride / persistent kernels
    uint32_t precision;    // 0: float triangle test (reference arithmetic); 1: FP64-filtered
    uint32_t walk_cap;     // per-warp ring entries of the walkers (multiple of 32, <= 512; 0: the default)
    uint32_t walk_steps = 6;   // steps a warp goes on for when its round has nothing more to claim
    uint32_t start_steps = 3;  // the same in a round 0 that is dealt out
    uint32_t claim_min = 1;   // a round's pairs are claimed dynamically from this many per warp
    uint32_t stay = 0;        // 1: warps keep what their rings hold, also of items dealt out (with steps without end:
                              // the lists take the fewest pairs, and a pass the longest)
    uint32_t ahead = 1;       // a round's CTAs are scheduled while the round before still runs (launch_walk)
    float descend_ratio = kDescendRatio;  // both sides descend while the boxes' squared diagonals are within it
};
// A traversal of `total0` start pairs: counters cleared (launch_begin, which
// sets the hits to hits_before, or the traversal before), then rounds 0, 1, .. in any number of calls of
// launch_walk (rounds from .. to - 1), until one leaves nothing. hand_over: the last of them writes kCountLeft,
// and the counters and few hits to the pinned host memory where there is any.
cudaError_t launch_begin(const DetectArgs& a, uint32_t hits_before, cudaStream_t s);
cudaError_t launch_walk(const DetectArgs& a, uint32_t total0, uint32_t from, uint32_t to, bool hand_over, cudaStream_t s);
// the counters (and few hits) to the pinned host memory
cudaError_t launch_publish(const DetectArgs& a, cudaStream_t s);
// walker CTAs that fit on one SM with rings of `walk_cap` entries (0:
// default), for the fused (narrow phase inside) or the broad-only walker
int walk_blocks_per_sm(uint32_t walk_cap = 0, bool fused = true);
cudaError_t launch_narrow(const DetectArgs& a, cudaStream_t s);
uint32_t narrow_kernels(const DetectArgs& a);  // kernels launch_narrow launches
// Rows of a precision-mode FP64 setup: the relative vertices p2, p3, q1, q2,
// q3 and the normals n1, m1 (x, y, z each), then the hit record (2 words).
constexpr uint32_t kFp64TriRows = 23;

// counts[]: hits, flags, candidates found, candidate slots used (broad-only),
// BVTT pairs tested, (precision mode) axes evaluated in FP64, candidates with
// at least one such axis, candidates whose float and FP64 answers differ,
// the sizes of the float-hit, recheck and FP64 lists of the precision narrow phase
// of the list its double-float pass leaves to FP64, of what its recheck
// leaves to the bounded pass, and of the rechecks of axes other than normals
// (not counted with the others); then the largest list
// of a walk round, the rounds that had anything to walk, and what the last round
// that was launched has left to a next one. Past the words that the host reads:
// the walk's control words, each on a cache line of its own.
constexpr uint32_t kCountHits = 0, kCountFlags = 1, kCountCands = 2, kCountCandSlots = 3, kCountTested = 4,
                   kCountFp64Axes = 5, kCountFp64Cands = 6, kCountDisagree = 7, kCountPrecHits = 8,
                   kCountPrecRecheck = 9, kCountPrecFp64 = 10, kCountPrecLeft = 11, kCountPrecAgain = 12,
                   kCountPrecOther = 13, kCountNarrowEnd = 14, kCountPeak = 14, kCountRounds = 15, kCountLeft = 16,
                   kCountHost = 17, kCtlDone = 32,
                   kCtlRound = 64, kCtlRoundWords = 64, kCtlRoundClaim = 32,  // four slots
                   kCountTotal = kCtlRound + 4 * kCtlRoundWords;

} // namespace oibvh
