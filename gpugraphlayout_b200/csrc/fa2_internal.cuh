// fa2_internal.cuh -- device data layout and kernel entry points of the B200
// ForceAtlas2 engine.  Host code in fa2_capi.cu enqueues one iteration as
//
//   stream A: build (the quadtree) -> [join B] -> traverse (+ speed)
//             -> displace (+ next bounding box)
//   stream B: attract (gravity + attraction)
//
// which replaces the eleven launches of CUDAForceAtlas2::doStep
// (src/RPGPUForceAtlas2.cu:206-248 of the reference).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace fa2 {

constexpr int kWarp = 32;
constexpr int kLevels = 32;        // quadrant digits in a 64-bit Morton key
constexpr int kBodyLevel = 63;     // level code of a body (leaf) node
constexpr int kMetaShift = 6;      // node meta = next_index << 6 | level code
constexpr uint32_t kMaxTreeNodes = (1u << 26) - 1;  // next index fits the 26 meta bits
constexpr int kMaxRun = 1024;      // longest run of equal 64-bit keys handled
constexpr int kDeepLevels = 64;    // levels past 32 used to order such a run

// Device error bits (DevState::err).  Any of them stops the iteration.
enum : int {
    kErrScanWait = 2,      // a block of the tree build waited too long
    kErrRunTooLong = 4,    // more than kMaxRun bodies share a 64-bit key
    kErrTreeTooLarge = 8,  // the quadtree needs more nodes than allocated
    kErrNonFinite = 16,    // a position is NaN or infinite
};

// Scalars that live on the device for the whole run.
struct DevState {
    float minx, maxx, miny, maxy;        // bounding box of the positions
    float radius, rootx, rooty;          // root cell (src/RPBHKernels.cu:140-148)
    float global_speed, speed_efficiency; // src/RPFA2Kernels.cu:29-33, per context here
    float jitter_tolerance, k_s_max;
    int poison;          // coincident bodies seen: this iteration is replayed
    int err;             // kErr* bits
    int iters_done;      // completed iterations
    int resorts;         // sorts done again on every digit
    uint32_t tree_nodes; // nodes of the last quadtree
    int max_level;
    float swg_sum, etra_sum;
    unsigned long long interactions;  // body-node force terms of the last traversal
    unsigned long long visits;        // body-node acceptance tests of the last traversal
    float trav_radius;                // root radius the last traversal used
    int resort;                       // this sort skipped low digits that it needs
    int deep;                         // bodies that share a whole 64-bit key
    int cells[6];                     // largest cell of the last tree at levels 12, 16, .., 28, 6
};

constexpr int kBuildBins = 4096;

// Counters at zero between iterations: each is cleared by the kernels that are
// done with it.
struct IterCounters {
    unsigned bbox_done;
    unsigned build_bar;  // barrier arrivals of the tree build
    unsigned trav_ticket;
    unsigned trav_done;
    unsigned disp_done;
    unsigned pad[3];
    unsigned pair_count[16];  // (group, cell) pairs of a learned walk, per pair segment
    unsigned hist[kBuildBins];  // keys per bin of the tree build's bucket sort
};

// Blocks of the tree build: 512 bodies or more each, at most one per SM; fewer
// where the context holds fewer (Buffers::build_blocks).  The build with 256, 512
// and 1024 bodies as the least: 300 bodies 30.5, 18.0 and 18.3 us (one block needs
// no barrier in global memory), 800 32.8, 32.8 and 24.1, 3000 34.4, 34.9 and 42.7,
// 30000 37.7, 38.5 and 45.2.
constexpr int kBuildMinTile = 512;
inline int build_blocks(int n, int nsm) {
    const int b = (n + kBuildMinTile - 1) / kBuildMinTile;
    return b < 1 ? 1 : (b > nsm ? nsm : b);
}
// A cooperative grid has to be resident as a whole, and a context can hold less
// than the device (an MPS client's share of the SMs): launch(blocks) with half
// as many blocks until they fit, which a launch says before anything runs.
template <class Launch>
cudaError_t launch_fitting(int &blocks, Launch launch) {
    for (;;) {
        const cudaError_t e = launch(blocks);
        if (e != cudaErrorCooperativeLaunchTooLarge || blocks <= 1) return e;
        cudaGetLastError();  // refused, not failed
        blocks = (blocks + 1) / 2;
    }
}
// Digit counts of the sort passes: [8][blocks][256].
inline size_t build_counts(int blocks) { return (size_t)8 * blocks * 256; }

// Attraction work split: rows (nodes in degree-descending order) with the
// same number of lanes per row form one contiguous bucket.
struct AttractBucket {
    int row_begin, row_end;  // rows [row_begin, row_end)
    int lanes;               // lanes per row: 256 (one block), 32, 16, ..., 1
    int block_begin;         // first block index of this bucket
};
constexpr int kMaxBuckets = 8;
constexpr int kAttractBatch = 2;  // row groups per warp in short-row buckets
struct AttractPlan {
    AttractBucket b[kMaxBuckets];
    int nbuckets;
    int nblocks;
};

// Exact moments of a run of sorted bodies on the fixed-point grid of 2^-44
// root radii (q = offset from the root centre): sum m q_x, sum m q_y,
// sum m (q_x^2 - q_y^2), sum m q_x q_y.  With the total mass below 2^32 and
// |q| <= 2^45 every sum stays below 2^123.
struct Moments {
    __int128 x, y, re, im;
};

struct Buffers {
    int n;
    // per node, internal (degree-descending) order
    float2 *pos, *fprev, *f, *fag;
    float *mass;
    const uint32_t *csr_off;  // n + 1, padded-row offsets (multiples of 4)
    const int4 *csr_col4;     // neighbour ids in fours
    const float4 *csr_w4;     // w^delta beside each id (null: unweighted, w^delta = 1)
    const uint32_t *ref_of;   // internal id -> reference id
    // sort
    uint64_t *keys[2];
    uint32_t *vals[2];
    // tree
    float4 *sbody;            // n: sorted bodies, x, y, mass, id
    uint8_t *lcp;             // n, padded to 64: digits shared with the next sorted body, + 1
    uint8_t *rowmin;          // rows of 32 bodies, padded to 64: the least of lcp
    uint8_t *tilemin;         // tree-build tiles, padded to 64: the least of lcp
    uint32_t *defer;          // 33 per row: the tree build's cells that end in a later row
    uint32_t *group;          // n: first preorder node of body k's group
    uint32_t *body_node;      // n: preorder node of sorted body k
    uint32_t *owner;          // capacity: per node, sorted body k << 6 | cell offset (63: body)
    float2 *quad;             // capacity: per cell, complex 2nd moment about its centre of mass
    Moments *pmom;            // n + 1: exclusive prefix of the body moments (quadrupole only)
    Moments *mom_totals;      // [build blocks]: their bodies' moments (quadrupole only)
    float4 *nodes;            // capacity + 1: x, y, mass, meta
    uint32_t capacity;
    long long *pm;            // n + 1: exclusive prefix of mass over sorted bodies
    __int128 *pxy;            // 2(n + 1): prefix of mass x fixed-point offset, x and y
    int build_blocks;         // blocks of the tree build, at most build_blocks(n, SMs)
    void *build_totals;       // tree-build blocks: their tiles' sums (NodeSums)
    // reductions
    float4 *bbox_partial;     // bbox blocks
    float2 *warp_partial;     // one per 32 sorted bodies
    DevState *st;
    IterCounters *ctr;
    uint32_t *sort_counts;    // [8][tree-build blocks][256]: digit counts per tile and pass
    const float *size;        // n: node sizes for prevent_overlap (null: off)
    float *ssize;             // n: the same in sorted order, per iteration
};

struct Params {
    float k_r, k_g, itolsq, epssq;
    int strong_gravity;
    int linlog;     // linear-log attraction
    int multipole;  // 1: monopole cells (the reference); 2: + quadrupole term
    int nsm;
    int overlap;    // prevent_overlap: node sizes in Buffers::size
};

constexpr int kBBoxThreads = 512;
constexpr int kTravThreads = 256;
constexpr int kTravWarpsPerSm = 32;
constexpr int kDispThreads = 512;

// ---------------------------------------------------------------- kernels --
void launch_bbox(const Buffers &b, int nblocks, cudaStream_t s);
// The quadtree of the current positions, one cooperative launch of
// b.build_blocks blocks.  With an error bit set it returns at once.
cudaError_t launch_build(const Buffers &b, bool moments, cudaStream_t s);
size_t build_totals_bytes(int blocks);
void build_set_smem_attr();
// Bytes padded for vector loads of 64.
inline size_t pad64(size_t x) { return (x + 63) & ~(size_t)63; }
void launch_runs(const Buffers &b, int perturb, int nsm, cudaStream_t s);
void launch_quad_cells(const Buffers &b, int nsm, cudaStream_t s);
void launch_traverse(const Buffers &b, const Params &p, int nblocks, cudaStream_t s);
void launch_displace(const Buffers &b, int nsm, cudaStream_t s);
void launch_count_interactions(const Buffers &b, const Params &p, int nblocks, cudaStream_t s);
void launch_exact_f64(const Buffers &b, const Params &p, const uint32_t *ids, int n_ids,
                      double2 *out, cudaStream_t s);
// The accuracy guard's sums for ns samples: exact (FP64), the reference walk's
// (plain) and the applied repulsion (cur); part holds guard_part_count(ns)
// partial sums.
size_t guard_part_count(int ns);
void launch_guard(const Buffers &b, const Params &p, int ns, double2 *exact, float2 *plain,
                  float2 *cur, double2 *part, cudaStream_t s);
void launch_attract(const Buffers &b, const Params &p, const AttractPlan &plan, cudaStream_t s);
// prevent_overlap: node sizes in sorted order (before the walk)
void launch_sorted_sizes(const Buffers &b, cudaStream_t s);
void launch_scatter_xy(int n, const uint32_t *ref_of, const float2 *src_ref, float2 *dst_int,
                       cudaStream_t s);
// Positions from reference order, and in reference order; with host_st, the
// device state to that pinned host copy as well.
void launch_place(const Buffers &b, const float2 *src_ref, int nblocks, cudaStream_t s);
void launch_gather_xy(int n, const uint32_t *ref_of, const float2 *src_int, float2 *dst_ref,
                      const DevState *st, DevState *host_st, cudaStream_t s);
void launch_sorted_ref_ids(int n, const uint32_t *ref_of, const uint32_t *vals, uint32_t *out,
                           cudaStream_t s);
int traverse_blocks_per_sm();

}  // namespace fa2
