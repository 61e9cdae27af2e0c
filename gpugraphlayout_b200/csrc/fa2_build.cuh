// fa2_build.cuh -- the quadtree of one graph, from the positions to the node
// array, by a team of thread blocks in one kernel.
//
// The reference inserts bodies into its quadtree with locks
// (TreeBuildingKernel, src/RPBHKernels.cu:184-329) and sums cells bottom-up
// with spin-waits (SummarizationKernel, :357-506).  The tree's shape does not
// depend on insertion order: its cells are exactly the quadrant prefixes that
// hold at least two bodies.  With the bodies sorted by key (the reference's
// in-order sortd), body k starts the cells at levels L[k-1]+1 .. L[k], where
// L[k] is the number of leading digits keys k and k+1 share.  The phases, with
// a barrier of the team between them:
//
//   keys    each body's 64-bit Morton key (morton_key);
//   buckets for up to 1024 bodies per block: the keys to 4096 bins by their top
//           bits, then each to its place among its bin's keys; else, or when
//           a bin is too full:
//   passes  a stable LSD radix sort of (key, id) by 8-bit digits.  Each block
//           owns a fixed tile of the array.  A pass needs, per digit, how many
//           keys with it lie in the tiles before: the counts of the first
//           pass come from the keys phase, those of the next from the pass
//           before, which counts a key's next digit for the tile it goes to;
//   fix     the sort leaves out the low digits that the last tree's cells
//           hardly needed (sort_plan); every run of keys equal in the sorted
//           digits is then put in the order of the full key, stably, which is
//           exactly the full sort's order.  A run longer than kFixRun sorts
//           again on every digit;
//   count   L[k], the bodies' records in sorted order, and the sums of each
//           tile: nodes (a body's cells plus itself), mass and mass x position
//           (integers: mass is degree + 1; positions in 2^-48 steps of the
//           root radius; 128-bit sums).  Runs of equal 64-bit keys (trees
//           deeper than 32 levels) are ordered by deeper digits, and exactly
//           coincident bodies flagged (poison);
//   nodes   a warp takes 32 sorted bodies, a row, at a time: their exclusive
//           prefixes (every node's preorder index; any cell's mass and centre
//           of mass are two prefix differences), the body nodes, and the cells
//           that start and end in the row, found and summed in the lanes;
//   rest    the cells that end in a later row, one per lane: the first row,
//           in this tile or a later one, with fewer shared digits, then the
//           prefix difference.
//
// Against the reference's float summation in quadrant order
// (src/RPBHKernels.cu:461-494) the centres agree to float rounding; the sums
// here are exact and do not depend on thread timing.
//
// Why one kernel: a tree of up to 10^5 bodies is a chain of a dozen small
// dependent steps.  As a kernel each, a step takes 8 to 10 us (launch, ramp,
// the loads of its own prefix, tail); a barrier of 148 blocks takes about 1 us.
#pragma once

#include <stdint.h>

#include "fa2_device.cuh"

namespace fa2 {

constexpr int kBuildRounds = 9;  // keys per thread in a sort chunk, at most
// Levels whose largest cell is tracked, for the next build's plan: 12, 16, 20,
// 24, 28, and the bins' level (there only cells that end in a later row).
constexpr int kCellLevels = 6;
constexpr int kBinLevel = 6;

struct NodeSums {
    uint32_t g;  // nodes (cells + body)
    long long m;
    i128 x, y;
};

__device__ __forceinline__ void sums_add(NodeSums &a, const NodeSums &b) {
    a.g += b.g;
    a.m += b.m;
    a.x += b.x;
    a.y += b.y;
}

__device__ __forceinline__ NodeSums shfl_up_sums(const NodeSums &v, int o) {
    NodeSums t;
    t.g = __shfl_up_sync(kFullMask, v.g, o);
    t.m = __shfl_up_sync(kFullMask, v.m, o);
    t.x = shfl_up_i128(v.x, o);
    t.y = shfl_up_i128(v.y, o);
    return t;
}

__device__ __forceinline__ NodeSums shfl_xor_sums(const NodeSums &v, int o) {
    NodeSums t;
    t.g = __shfl_xor_sync(kFullMask, v.g, o);
    t.m = __shfl_xor_sync(kFullMask, v.m, o);
    t.x = shfl_xor_i128(v.x, o);
    t.y = shfl_xor_i128(v.y, o);
    return t;
}

// What a team works on.  Arrays that one phase writes and another reads are
// plain pointers: between them lies a barrier, and no load may go through the
// read-only path.
struct BuildArgs {
    int n;
    float2 *pos;
    const float *mass;
    const uint32_t *ref_of;  // null: the ids are reference ids
    uint64_t *keys[2];       // the order ends in keys[0], vals[0]
    uint32_t *vals[2];
    float4 *sbody;        // sorted bodies: x, y, mass, id
    uint8_t *lcp;         // n: digits shared with the next sorted body, + 1 (0: the last)
    uint8_t *rowmin;      // per 32 sorted bodies: the least of lcp
    uint8_t *tilemin;     // per tile: the least of lcp
    uint32_t *defer;      // 33 per row: cells that end in a later row, body << 6 | level
    uint32_t *group;      // first preorder node of body k's group
    uint32_t *body_node;  // preorder node of sorted body k
    uint32_t *owner;      // per node: sorted body k << 6 | cell offset (63: body)
    float4 *nodes;
    uint32_t capacity;
    long long *pm;
    i128 *pxy;
    Moments *pmom;        // n + 1 (MOM): exclusive prefix of the sorted bodies' moments
    Moments *mom_totals;  // [team size] (MOM)
    uint32_t *counts;     // [8][team size][256]
    uint32_t *hist;       // [kBinsPerThread x threads], zero between builds
    NodeSums *totals;     // [team size]
    float rootx, rooty, radius;
    // results and flags, in global memory
    int *err, *poison;
    int *resort;          // set by a run too long for the fix phase
    int *resorts;         // counts the sorts repeated for one
    int *deep;            // set by two bodies sharing all 64 bits of their keys
    int *cells;           // [kCellLevels]: the last tree's largest cells
    uint32_t *tree_nodes;
    int *max_level;
};

// The lowest 8-bit digit the sort starts at: the fewest digits after which
// the last tree's cells held at most kThinCell bodies, so that the runs the
// fix phase puts in order are short.  Measured on the scale-20 R-MAT layout
// and 10^4- to 10^5-node graphs: 3 or 4 passes instead of 8.
constexpr int kThinCell = 32;
// The longest run the fix phase puts in order, and the keys it loads at a time.
// A body looks through its whole run, so long runs cost more than the sort on
// every digit that follows a longer one.  The build of positions that share
// level-12 cells after a tree that had none, one key at a time up to 1024 and
// this way: one cell of 3000 bodies 182 and 85 us, of 10^5 382 and 194, of 6 10^5
// 920 and 285; 10^5 bodies in cells of 500 197 and 134, of 250 136 and 116, of
// 150 103 and 94.  A limit of 128 takes 40 % longer for cells of 150, one of 512
// 15 % longer for cells of 500; eight loads at a time 0 to 4 %.
constexpr int kFixRun = 256;
constexpr int kFixLoads = 4;
static_assert(kThinCell % kFixLoads == 0, "where build_fix looks for a long run");
__device__ __forceinline__ int sort_plan(const volatile int *cells) {
#pragma unroll
    for (int i = 0; i < 5; ++i)
        if (cells[i] <= kThinCell) return 5 - i;
    return 0;
}

// Bodies per tile: whole rows of 32, so that a row lies in one tile.
__host__ __device__ inline int build_tile(int n, int size) {
    return ((n + size - 1) / size + 31) & ~31;
}

constexpr int kMinRows = 256;

// The bucket sort: bins by the keys' top bits (12 with 512 threads, 11 with
// 256), the fullest bin it takes, and the keys per thread of a team.  Two
// moves and two barriers instead of four of each: 4 us less for the build of
// 300 nodes (23 us with the passes) and of 10^4 (44), 5 to 7 us less for an
// iteration of 46717 (87) to 10^5 nodes (117, learned 144).  Placing a key
// reads its whole bin: with bins of 128 bodies the two ways meet (46000 normal
// positions: 49.6 us both; with 512 allowed, 10^5 of them take 96 us instead
// of 70).  At four keys per thread a 1.7 10^5-node iteration takes 205 us
// instead of 181.  The last tree's cells tell most crowded layouts beforehand;
// the others lose 4 us (4000 bodies) to 25 us (10^5) in their first build.  One
// atomic per warp and bin (match) costs every other layout 1 us.
constexpr int kBinsPerThread = 8;
constexpr uint32_t kBinMax = 128;
constexpr int kBucketKeys = 2;  // keys per thread of a team's bucket sort

// T: threads per block (256 or 512).
template <int T>
struct BuildSmem {
    static constexpr int kThreads = T, kWarps = T / kWarp;
    union {
        uint32_t whist[kWarps][256];  // per-warp digit counts, then offsets
        uint32_t bins[T * kBinsPerThread];  // the bins' counts, then first places
        struct {
            uint4 before[T / 64][64], all[T / 64][64];  // partial sums over the count rows
        } rows;
        struct {
            NodeSums warp[kWarps];
            NodeSums prefix;
            Moments mom[kWarps], mom_prefix;
            uint32_t least[kWarps];
            int deepest[kWarps];
        } scan;
    };
    uint32_t base[256];      // next output position of each digit
    uint32_t tile_off[256];  // exclusive scan of the chunk's digit counts
    uint32_t qsum[T / 256][256];
    uint32_t scan_w[kWarps], max_w[kWarps];
    int cells[kCellLevels + 3];
    // the tile's least shared digits per row (up to kMinRows rows), and every
    // tile's, where the search for the cells' ends looks first
    __align__(64) uint8_t rowmin[kMinRows];
    __align__(64) uint8_t tilemin[256];
    // staging of `chunk` keys, then as many ids (launch-sized)
    __device__ __forceinline__ uint64_t *stage_keys() {
        return reinterpret_cast<uint64_t *>(this + 1);
    }
};
// Keys a tile's sort stages at a time: the tile where it fits.
inline int build_chunk(int tile, int threads) {
    const int most = threads * kBuildRounds;
    return tile > most ? most : (tile < threads ? threads : tile);
}
template <int T>
size_t build_smem_bytes(int chunk) {
    return sizeof(BuildSmem<T>) + (size_t)chunk * 12;
}

// Exclusive scan of v over threads 0..255 (every thread of the block calls;
// the others' results are unused).
template <int T>
__device__ __forceinline__ uint32_t scan256(uint32_t v, BuildSmem<T> &S) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFullMask, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31 && wid < 8) S.scan_w[wid] = inc;
    __syncthreads();
    uint32_t b = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w)
        if (w < wid) b += S.scan_w[w];
    __syncthreads();
    return b + inc - v;
}

// The fix phase of this block's tile: every key of a run of keys equal above
// `low` bits goes to its place by (key, input position), the others keep
// theirs.  A run longer than kFixRun needs the sort on every digit: nearly all
// of its keys see that from the keys kFixRun and half as many places away, and
// read no further.
template <int T>
__device__ __forceinline__ void build_fix(const BuildArgs &A, int low, const uint64_t *kin,
                                          const uint32_t *vin, uint64_t *kout, uint32_t *vout,
                                          int t0, int t1) {
    const int n = A.n;
    bool resort = false;
    for (int i = t0 + (int)threadIdx.x; i < t1; i += T) {
        const uint64_t key = kin[i];
        const uint32_t v = vin[i];
        const uint64_t hk = key >> low;
        int to = i;
        const bool left = low > 0 && i > 0 && (kin[i - 1] >> low) == hk;
        const bool right = low > 0 && i + 1 < n && (kin[i + 1] >> low) == hk;
        if (left || right) {
            int s = i, e = i + 1, smaller = 0;
            bool over = false, down = left, up = right;
            // a key that has seen kThinCell of its run looks for a long one
            auto same = [&](int j) { return j >= 0 && j < n && (kin[j] >> low) == hk; };
            auto is_long = [&]() {
                return same(i - kFixRun) || same(i + kFixRun) ||
                       (same(i - kFixRun / 2) && same(i + kFixRun / 2));
            };
            while (down) {
                uint64_t o[kFixLoads];
                const int j = s - 1;
#pragma unroll
                for (int u = 0; u < kFixLoads; ++u) o[u] = kin[max(j - u, 0)];
#pragma unroll
                for (int u = 0; u < kFixLoads; ++u) {
                    down = down && j - u >= 0 && (o[u] >> low) == hk;
                    s -= down;
                    smaller += down && o[u] <= key;
                }
                if (down && i - s == kThinCell && is_long()) {
                    over = true;
                    down = up = false;
                }
            }
            while (up) {
                uint64_t o[kFixLoads];
                const int j = e;
#pragma unroll
                for (int u = 0; u < kFixLoads; ++u) o[u] = kin[min(j + u, n - 1)];
#pragma unroll
                for (int u = 0; u < kFixLoads; ++u) {
                    up = up && j + u < n && (o[u] >> low) == hk;
                    e += up;
                    smaller += up && o[u] < key;
                }
                if (up && e - 1 - i == kThinCell && is_long()) {
                    over = true;
                    up = false;
                }
            }
            over |= e - s > kFixRun;
            if (over)
                resort = true;
            else
                to = s + smaller;
        }
        kout[to] = key;
        vout[to] = v;
    }
    // one store per block, not one per key
    if (__syncthreads_or(resort) && threadIdx.x == 0) *(volatile int *)A.resort = 1;
}

// Where each of a chunk's keys goes by the digit at `shift`, stably: at[r] for
// the thread's key k[r], the (w0 + 32 r + lane)-th, valid below `end`.  Warps
// hold consecutive keys.  Leaves the digits' first places in S.tile_off and
// returns the count of digit threadIdx.x & 255.
template <int T>
__device__ __forceinline__ uint32_t chunk_order(const uint64_t (&k)[kBuildRounds], int rounds,
                                                int w0, int end, int shift,
                                                uint32_t (&at)[kBuildRounds], BuildSmem<T> &S) {
    constexpr int kWarps = T / kWarp, kQ = T / 256;  // threads per digit
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    for (int j = tid; j < kWarps * 256; j += T) (&S.whist[0][0])[j] = 0;
    __syncthreads();
    // rank by digit per warp, in key order: the lanes that share a digit are
    // the AND of eight ballots
#pragma unroll
    for (int r = 0; r < kBuildRounds; ++r) {
        if (r < rounds) {
            const bool valid = w0 + r * 32 + lane < end;
            const uint32_t d = (uint32_t)(k[r] >> shift) & 255u;
            unsigned peers = __ballot_sync(kFullMask, valid);
            if (!valid) peers = ~peers;
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const bool bit = (d >> b) & 1u;
                const unsigned m = __ballot_sync(kFullMask, bit);
                peers &= bit ? m : ~m;
            }
            uint32_t before = 0;
            if (valid) before = S.whist[wid][d];
            at[r] = before + __popc(peers & lt);
            __syncwarp();
            if (valid && (peers & lt) == 0) S.whist[wid][d] = before + __popc(peers);
            __syncwarp();
        }
    }
    __syncthreads();
    // per digit: offsets across the warps, eight warps per thread
    const int dg = tid & 255, part = tid >> 8;
    uint32_t q = 0;
#pragma unroll
    for (int w = 0; w < kWarps / kQ; ++w) q += S.whist[part * (kWarps / kQ) + w][dg];
    S.qsum[part][dg] = q;
    __syncthreads();
    uint32_t run = 0, total = 0;
#pragma unroll
    for (int h = 0; h < kQ; ++h) {
        const uint32_t c = S.qsum[h][dg];
        if (h < part) run += c;
        total += c;
    }
#pragma unroll
    for (int w = 0; w < kWarps / kQ; ++w) {
        const uint32_t c = S.whist[part * (kWarps / kQ) + w][dg];
        S.whist[part * (kWarps / kQ) + w][dg] = run;
        run += c;
    }
    const uint32_t ex = scan256(total, S);
    if (part == 0) S.tile_off[dg] = ex;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kBuildRounds; ++r) {
        if (r < rounds && w0 + r * 32 + lane < end) {
            const uint32_t d = (uint32_t)(k[r] >> shift) & 255u;
            at[r] += S.tile_off[d] + S.whist[wid][d];
        }
    }
    return total;
}

// One stable pass over this block's tile [t0, t1): digit `pass` from kin/vin
// to kout/vout.  counts rows of `pass` are complete; the next pass's rows get
// the counts of its digits per output tile.
template <int T, class Team>
__device__ __forceinline__ void build_pass(const BuildArgs &A, const Team &team, int pass,
                                           const uint64_t *kin, const uint32_t *vin,
                                           uint64_t *kout, uint32_t *vout, int t0, int t1,
                                           int tile, int chunk, BuildSmem<T> &S) {
    uint64_t *stage_k = S.stage_keys();
    uint32_t *stage_v = reinterpret_cast<uint32_t *>(stage_k + chunk);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int shift = 8 * pass;
    // the digits' starts: keys of smaller digits anywhere, and of this digit
    // in the tiles before
    {
        const uint4 *row = reinterpret_cast<const uint4 *>(A.counts) +
                           (size_t)pass * team.size * 64 + (tid & 63);
        uint4 before = make_uint4(0, 0, 0, 0), all = before;
#pragma unroll 4
        for (int t = tid >> 6; t < team.size; t += T / 64) {
            const uint4 c = __ldcg(row + (size_t)t * 64);
            all.x += c.x;
            all.y += c.y;
            all.z += c.z;
            all.w += c.w;
            if (t < team.rank) {
                before.x += c.x;
                before.y += c.y;
                before.z += c.z;
                before.w += c.w;
            }
        }
        S.rows.before[tid >> 6][tid & 63] = before;
        S.rows.all[tid >> 6][tid & 63] = all;
        __syncthreads();
        uint32_t b = 0, a = 0;
        if (tid < 256) {
#pragma unroll
            for (int g = 0; g < T / 64; ++g) {
                b += reinterpret_cast<const uint32_t *>(S.rows.before[g])[tid];
                a += reinterpret_cast<const uint32_t *>(S.rows.all[g])[tid];
            }
        }
        const uint32_t ex = scan256(a, S);
        if (tid < 256) S.base[tid] = ex + b;
    }
    uint32_t *next = pass < 7 ? A.counts + (size_t)(pass + 1) * team.size * 256 : nullptr;
    for (int c0 = t0; c0 < t1; c0 += chunk) {
        const int cn = min(chunk, t1 - c0);
        const int rounds = (cn + T - 1) / T;
        const int w0 = c0 + wid * rounds * 32;
        uint64_t k[kBuildRounds];
        uint32_t v[kBuildRounds], at[kBuildRounds];
#pragma unroll
        for (int r = 0; r < kBuildRounds; ++r) {
            const int i = w0 + r * 32 + lane;
            const bool in = r < rounds && i < t1;
            k[r] = in ? kin[i] : 0ull;
            v[r] = in ? vin[i] : 0u;
        }
        const uint32_t total = chunk_order(k, rounds, w0, t1, shift, at, S);
        // regroup by digit in shared memory, write digit runs, count the next
        // pass's digits per output tile
#pragma unroll
        for (int r = 0; r < kBuildRounds; ++r) {
            if (r < rounds && w0 + r * 32 + lane < t1) {
                stage_k[at[r]] = k[r];
                stage_v[at[r]] = v[r];
            }
        }
        __syncthreads();
        for (int j = tid; j < cn; j += T) {
            const uint64_t key = stage_k[j];
            const uint32_t d = (uint32_t)(key >> shift) & 255u;
            const uint32_t out = S.base[d] + (uint32_t)j - S.tile_off[d];
            kout[out] = key;
            vout[out] = stage_v[j];
            if (next)
                atomicAdd(&next[(size_t)(out / (uint32_t)tile) * 256 +
                                ((uint32_t)(key >> (shift + 8)) & 255u)],
                          1u);
        }
        __syncthreads();
        if (tid < 256) S.base[tid] += total;
        __syncthreads();
    }
}

// The bins' counts, eight per thread, to their first places in S.bins; returns
// the fullest bin's count.  Every thread calls it.
template <int T>
__device__ __forceinline__ uint32_t bin_starts(uint4 a, uint4 b, BuildSmem<T> &S) {
    constexpr int kWarps = T / kWarp;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t most = max(max(max(a.x, a.y), max(a.z, a.w)), max(max(b.x, b.y), max(b.z, b.w)));
    const uint32_t sum = (a.x + a.y) + (a.z + a.w) + ((b.x + b.y) + (b.z + b.w));
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFullMask, inc, o);
        if (lane >= o) inc += t;
    }
    const uint32_t wmax = __reduce_max_sync(kFullMask, most);
    if (lane == 31) {
        S.scan_w[wid] = inc;
        S.max_w[wid] = wmax;
    }
    __syncthreads();
    uint32_t at = inc - sum, top = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        if (w < wid) at += S.scan_w[w];
        top = max(top, S.max_w[w]);
    }
    uint4 first, second;
    first.x = at;
    first.y = first.x + a.x;
    first.z = first.y + a.y;
    first.w = first.z + a.z;
    second.x = first.w + a.w;
    second.y = second.x + b.x;
    second.z = second.y + b.y;
    second.w = second.z + b.z;
    reinterpret_cast<uint4 *>(S.bins)[2 * tid] = first;
    reinterpret_cast<uint4 *>(S.bins)[2 * tid + 1] = second;
    __syncthreads();
    return top;
}

// A bucketed key to its place among its bin's keys by (key, id): the order of
// the stable sort.
template <int T>
__device__ __forceinline__ void place_in_bin(const BuildArgs &A, const uint64_t *kin,
                                             const uint32_t *vin, int j, const BuildSmem<T> &S) {
    constexpr int kBins = T * kBinsPerThread, kShift = T == 512 ? 52 : 53;
    const uint64_t key = kin[j];
    const uint32_t v = vin[j];
    const uint32_t bin = (uint32_t)(key >> kShift);
    const int b0 = (int)S.bins[bin], b1 = bin + 1 < kBins ? (int)S.bins[bin + 1] : A.n;
    int to = b0;
#pragma unroll 4
    for (int q = b0; q < b1; ++q) {
        const uint64_t o = kin[q];
        to += o < key;
        if (o == key && q != j) to += vin[q] < v;
    }
    A.keys[0][to] = key;
    A.vals[0][to] = v;
}

// Keys and sort by buckets: every key to its bin (top bits of the key, any
// order), then to its place in the bin.  Two moves instead of the radix
// passes; a bin too full (bodies crowded into one of 4096 squares) goes back
// to those.  One block, in shared memory; false: nothing done.
template <int T>
__device__ __forceinline__ bool bucket_sort_local(const BuildArgs &A, int chunk,
                                                  BuildSmem<T> &S) {
    constexpr int kShift = T == 512 ? 52 : 53;
    const int n = A.n, tid = threadIdx.x;
    uint64_t *stage_k = S.stage_keys();
    uint32_t *stage_v = reinterpret_cast<uint32_t *>(stage_k + chunk);
    reinterpret_cast<uint4 *>(S.bins)[2 * tid] = make_uint4(0, 0, 0, 0);
    reinterpret_cast<uint4 *>(S.bins)[2 * tid + 1] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    uint64_t key[kBuildRounds];
    uint32_t slot[kBuildRounds];
#pragma unroll
    for (int r = 0; r < kBuildRounds; ++r) {
        const int i = r * T + tid;
        if (i < n) {
            const float2 p = A.pos[i];
            key[r] = morton_key(p.x, p.y, A.rootx, A.rooty, A.radius);
            slot[r] = atomicAdd(&S.bins[(uint32_t)(key[r] >> kShift)], 1u);
        }
    }
    __syncthreads();
    const uint4 a = reinterpret_cast<const uint4 *>(S.bins)[2 * tid];
    const uint4 b = reinterpret_cast<const uint4 *>(S.bins)[2 * tid + 1];
    if (bin_starts(a, b, S) > kBinMax) return false;
#pragma unroll
    for (int r = 0; r < kBuildRounds; ++r) {
        const int i = r * T + tid;
        if (i < n) {
            const uint32_t at = S.bins[(uint32_t)(key[r] >> kShift)] + slot[r];
            stage_k[at] = key[r];
            stage_v[at] = (uint32_t)i;
        }
    }
    __syncthreads();
    for (int j = tid; j < n; j += T) place_in_bin<T>(A, stage_k, stage_v, j, S);
    __syncthreads();
    return true;
}

// The same by a team, through global memory: the bins' counts in A.hist.
enum BucketResult { kBucketFailed, kBucketDone, kBucketTooFull };
template <int T, class Team>
__device__ __forceinline__ BucketResult bucket_sort(const BuildArgs &A, Team &team, int t0, int t1,
                                                    BuildSmem<T> &S) {
    constexpr int kBins = T * kBinsPerThread, kShift = T == 512 ? 52 : 53;
    const int tid = threadIdx.x;
    uint64_t key[kBucketKeys];
    uint32_t slot[kBucketKeys];
#pragma unroll
    for (int r = 0; r < kBucketKeys; ++r) {
        const int i = t0 + r * T + tid;
        if (i < t1) {
            const float2 p = A.pos[i];
            key[r] = morton_key(p.x, p.y, A.rootx, A.rooty, A.radius);
            slot[r] = atomicAdd(&A.hist[(uint32_t)(key[r] >> kShift)], 1u);
        }
    }
    if (!team.sync()) return kBucketFailed;
    const uint4 *h = reinterpret_cast<const uint4 *>(A.hist) + 2 * tid;
    // every block sees the same counts, so all of them turn back or none
    if (bin_starts(__ldcg(h), __ldcg(h + 1), S) > kBinMax) return kBucketTooFull;
#pragma unroll
    for (int r = 0; r < kBucketKeys; ++r) {
        const int i = t0 + r * T + tid;
        if (i < t1) {
            const uint32_t at = S.bins[(uint32_t)(key[r] >> kShift)] + slot[r];
            A.keys[1][at] = key[r];
            A.vals[1][at] = (uint32_t)i;
        }
    }
    if (!team.sync()) return kBucketFailed;
    for (int j = team.rank * T + tid; j < kBins; j += team.size * T) A.hist[j] = 0;
    for (int j = t0 + tid; j < t1; j += T) place_in_bin<T>(A, A.keys[1], A.vals[1], j, S);
    return team.sync() ? kBucketDone : kBucketFailed;
}

// The keys and every pass of a graph that one block's staging holds, in
// registers and shared memory; the order goes to keys[0], vals[0].
template <int T>
__device__ __forceinline__ void build_sort_local(const BuildArgs &A, int first, int chunk,
                                                 BuildSmem<T> &S) {
    const int n = A.n, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    uint64_t *stage_k = S.stage_keys();
    uint32_t *stage_v = reinterpret_cast<uint32_t *>(stage_k + chunk);
    const int rounds = (n + T - 1) / T, w0 = wid * rounds * 32;
    uint64_t k[kBuildRounds];
    uint32_t v[kBuildRounds], at[kBuildRounds];
#pragma unroll
    for (int r = 0; r < kBuildRounds; ++r) {
        const int i = w0 + r * 32 + lane;
        k[r] = 0ull;
        v[r] = (uint32_t)i;
        if (r < rounds && i < n) {
            const float2 p = A.pos[i];
            k[r] = morton_key(p.x, p.y, A.rootx, A.rooty, A.radius);
        }
    }
    for (;;) {
        for (int pass = first; pass < 8; ++pass) {
            chunk_order(k, rounds, w0, n, 8 * pass, at, S);
#pragma unroll
            for (int r = 0; r < kBuildRounds; ++r) {
                if (r < rounds && w0 + r * 32 + lane < n) {
                    stage_k[at[r]] = k[r];
                    stage_v[at[r]] = v[r];
                }
            }
            __syncthreads();
#pragma unroll
            for (int r = 0; r < kBuildRounds; ++r) {
                const int i = w0 + r * 32 + lane;
                if (r < rounds && i < n) {
                    k[r] = stage_k[i];
                    v[r] = stage_v[i];
                }
            }
            __syncthreads();
        }
        // with every digit sorted there is nothing to put in order
        build_fix<T>(A, 8 * first, stage_k, stage_v, A.keys[0], A.vals[0], 0, n);
        __syncthreads();
        if (first == 0 || !*(volatile int *)A.resort) break;
        // a run too long: every digit, from the order the partial sort left
        if (tid == 0) *A.resorts += 1;
        first = 0;
    }
}

// This block's row of the counts of digit `first` from `keys`, and zeros in
// its rows of the later passes.
template <int T, class Team>
__device__ __forceinline__ void build_count_rows(const BuildArgs &A, const Team &team, int first,
                                                 BuildSmem<T> &S) {
    for (int j = threadIdx.x; j < (8 - first) * 256; j += T) {
        const int p = first + (j >> 8);
        A.counts[((size_t)p * team.size + team.rank) * 256 + (j & 255)] =
            p == first ? S.base[j & 255] : 0u;
    }
}

// An offset on the 2^-48 grid moved to the 2^-44 grid of the moment sums
// (positions lie inside the root box, so |q| <= 2^44; the clamp only bounds
// the sums for inputs that do not).
__device__ __forceinline__ long long mom_grid(long long q48) {
    const long long q = q48 >> 4;
    constexpr long long kMax = 1ll << 45;
    return q > kMax ? kMax : (q < -kMax ? -kMax : q);
}

__device__ __forceinline__ void mom_add(Moments &a, const Moments &b) {
    a.x += b.x;
    a.y += b.y;
    a.re += b.re;
    a.im += b.im;
}

__device__ __forceinline__ Moments mom_shfl_up(const Moments &v, int o) {
    return Moments{shfl_up_i128(v.x, o), shfl_up_i128(v.y, o), shfl_up_i128(v.re, o),
                   shfl_up_i128(v.im, o)};
}

__device__ __forceinline__ Moments mom_shfl_xor(const Moments &v, int o) {
    return Moments{shfl_xor_i128(v.x, o), shfl_xor_i128(v.y, o), shfl_xor_i128(v.re, o),
                   shfl_xor_i128(v.im, o)};
}

// Moments of one body from its grid offset and mass.
__device__ __forceinline__ Moments body_moments(longlong2 q, uint32_t m) {
    const i128 mx = (i128)(long long)m * q.x, my = (i128)(long long)m * q.y;
    return Moments{mx, my, mx * q.x - my * q.y, mx * q.y};
}

// The moments of the body in this lane of row r (none: 0).
__device__ __forceinline__ Moments row_moments(const BuildArgs &A, int k, double scale) {
    if (k >= A.n) return Moments{0, 0, 0, 0};
    const float4 me = A.sbody[k];
    return body_moments(make_longlong2(mom_grid(fixed_offset(me.x, A.rootx, scale)),
                                       mom_grid(fixed_offset(me.y, A.rooty, scale))),
                        (uint32_t)me.z);
}

// The sum of the rows' moments, by one warp that wrote their records.
__device__ __forceinline__ Moments sum_moments(const BuildArgs &A, int r0, int r1, double scale) {
    const int lane = threadIdx.x & 31;
    Moments sum{0, 0, 0, 0};
    for (int r = r0; r < r1; ++r) mom_add(sum, row_moments(A, r * 32 + lane, scale));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mom_add(sum, mom_shfl_xor(sum, o));
    return sum;
}

// The rows' exclusive prefixes, from `base` on.
__device__ __forceinline__ void scan_moments(const BuildArgs &A, int r0, int r1, double scale,
                                             Moments base) {
    const int lane = threadIdx.x & 31;
    for (int r = r0; r < r1; ++r) {
        const int k = r * 32 + lane;
        const Moments own = row_moments(A, k, scale);
        Moments inc = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const Moments t = mom_shfl_up(inc, o);
            if (lane >= o) mom_add(inc, t);
        }
        mom_add(inc, base);
        if (k < A.n)
            A.pmom[k] = Moments{inc.x - own.x, inc.y - own.y, inc.re - own.re, inc.im - own.im};
        if (k == A.n - 1) A.pmom[A.n] = inc;
        base = Moments{shfl_i128(inc.x, 31), shfl_i128(inc.y, 31), shfl_i128(inc.re, 31),
                       shfl_i128(inc.im, 31)};
    }
}

// First index in [a, b) of a byte below t (t <= 128), b if there is none.
// Bytes are below 128; `base` is 16-byte aligned and readable up to the next
// multiple of 16 past b.  One lane searches alone, so its instructions count:
// 32 bytes a step with one mask for the start instead of 64 with a mask per
// word took the build of 10^4 bodies from 40.0 to 37.5 us, of 93000 from 59.7
// to 53.0, of 6.5 10^5 from 142.6 to 135.
__device__ __forceinline__ int first_below(const uint8_t *base, int a, int b, uint32_t t) {
    const uint32_t tt = t * 0x01010101u;
    int i = a & ~15;
    uint32_t skip = 8u * (uint32_t)(a - i);  // bits of the bytes before a
    for (; i < b; i += 32) {
        const uint4 w0 = *reinterpret_cast<const uint4 *>(base + i);
        const uint4 w1 = i + 16 < b ? *reinterpret_cast<const uint4 *>(base + i + 16)
                                    : make_uint4(~0u, ~0u, ~0u, ~0u);
        const uint32_t x[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
        uint32_t hit = 0, word = 0;
#pragma unroll
        for (int j = 7; j >= 0; --j) {
            // bit 7 of a byte: the byte is below t
            uint32_t m = ~((x[j] | 0x80808080u) - tt) & 0x80808080u;
            if (j < 4) {
                const uint32_t s = skip > 32u * j ? skip - 32u * j : 0u;
                m = s >= 32u ? 0u : m & (~0u << s);
            }
            if (m) {
                hit = m;
                word = (uint32_t)j;
            }
        }
        if (hit) return min(b, i + 4 * (int)word + ((__ffs(hit) - 1) >> 3));
        skip = 0;
    }
    return b;
}

// A row of 32 sorted bodies in a warp's lanes: sums that fit 32 bits (mass
// below 2^25) or 96 bits (mass x offset below 2^80).
struct RowSums {
    uint32_t g, m;
    i128 x, y;
};

__device__ __forceinline__ i128 shfl96(i128 v, int src) {
    const uint32_t a = __shfl_sync(kFullMask, (uint32_t)v, src);
    const uint32_t b = __shfl_sync(kFullMask, (uint32_t)(v >> 32), src);
    const int c = __shfl_sync(kFullMask, (int)(v >> 64), src);
    return ((i128)c << 64) | (i128)(((unsigned long long)b << 32) | a);
}

__device__ __forceinline__ RowSums row_scan(RowSums v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t g = __shfl_up_sync(kFullMask, v.g, o);
        const uint32_t m = __shfl_up_sync(kFullMask, v.m, o);
        const int src = max(lane - o, 0);
        const i128 x = shfl96(v.x, src), y = shfl96(v.y, src);
        if (lane >= o) {
            v.g += g;
            v.m += m;
            v.x += x;
            v.y += y;
        }
    }
    return v;
}

// Cell record from the sums over its bodies (src/RPBHKernels.cu:461-494: the
// centre of mass and the mass; here exact sums, rounded once).
__device__ __forceinline__ float4 cell_record(double cm, double sx, double sy, double rx,
                                              double ry, double inv_scale, uint32_t next,
                                              int lvl) {
    return make_float4((float)(rx + sx / cm * inv_scale), (float)(ry + sy / cm * inv_scale),
                       (float)cm, make_meta(next, lvl));
}

// First part of the count, over this warp's rows [r0, r1) of 32 sorted bodies:
// the bodies' records and shared digits in sorted order, the rows' and the
// tile's least shared digits, and the warp's sums (in every lane).
struct CountOut {
    NodeSums sum;
    int deepest;     // most shared digits
    uint32_t least;  // least shared digits + 1
};
template <int T>
__device__ __forceinline__ CountOut build_count(const BuildArgs &A, int r0, int r1, int tile_r0,
                                                double scale, BuildSmem<T> &S) {
    const int n = A.n, lane = threadIdx.x & 31;
    CountOut out{{0, 0, 0, 0}, 0, 255u};
    constexpr int kB = 3;  // rows whose loads are in flight together
    for (int r = r0; r < r1; r += kB) {
        uint64_t key[kB], edge[kB];
        uint32_t id[kB];
        float2 p[kB];
        float m[kB];
#pragma unroll
        for (int u = 0; u < kB; ++u) {
            const int k = (r + u) * 32 + lane;
            const bool in = r + u < r1 && k < n;
            key[u] = in ? A.keys[0][k] : 0ull;
            id[u] = in ? A.vals[0][k] : 0u;
            edge[u] = 0ull;
            if (in && lane == 0 && k > 0) edge[u] = A.keys[0][k - 1];
            if (in && lane == 31 && k + 1 < n) edge[u] = A.keys[0][k + 1];
        }
#pragma unroll
        for (int u = 0; u < kB; ++u) {
            p[u] = A.pos[id[u]];
            m[u] = A.mass[id[u]];
        }
#pragma unroll
        for (int u = 0; u < kB; ++u) {
            if (r + u >= r1) break;
            const int k = (r + u) * 32 + lane;
            const bool in = k < n;
            uint64_t after = __shfl_down_sync(kFullMask, key[u], 1);
            if (lane == 31) after = edge[u];
            const int Lk = k >= n - 1 ? -1 : lcp_digits(key[u], after);
            int Lkm1 = __shfl_up_sync(kFullMask, Lk, 1);
            if (lane == 0) Lkm1 = k == 0 ? -1 : lcp_digits(edge[u], key[u]);
            const uint32_t least = __reduce_min_sync(kFullMask, in ? (uint32_t)(Lk + 1) : 255u);
            out.least = min(out.least, least);
            if (lane == 0) {
                A.rowmin[r + u] = (uint8_t)least;
                const int at = r + u - tile_r0;
                if (at < kMinRows) S.rowmin[at] = (uint8_t)least;
            }
            if (!in) continue;
            out.deepest = max(out.deepest, Lk);
            A.lcp[k] = (uint8_t)(Lk + 1);
            A.sbody[k] = make_float4(p[u].x, p[u].y, m[u], __uint_as_float(id[u]));
            const long long im = (long long)m[u];
            const long long qx = fixed_offset(p[u].x, A.rootx, scale);
            const long long qy = fixed_offset(p[u].y, A.rooty, scale);
            sums_add(out.sum, NodeSums{(uint32_t)cells_at(k, Lk, Lkm1) + 1u, im, (i128)im * qx,
                                       (i128)im * qy});
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sums_add(out.sum, shfl_xor_sums(out.sum, o));
    out.deepest = __reduce_max_sync(kFullMask, out.deepest);
    return out;
}

// The whole build.  Team: rank, size and sync(), a barrier of its blocks that
// orders their global memory accesses and returns false when it gave up.
// `chunk` is the number of keys the shared memory stages.
// MOM: also the prefix sums of the bodies' second moments (pmom), for the
// quadrupole option: 10 us of the build of 1.7 10^5 bodies, where a scan of its
// own behind the build took 22 (an iteration: 172 and 180 us).
template <int T, bool MOM, class Team>
__device__ __forceinline__ void build_tree(const BuildArgs &A, Team &team, BuildSmem<T> &S,
                                           int chunk) {
    constexpr int kWarps = T / kWarp;
    const int n = A.n, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int tile = build_tile(n, team.size);
    const int t0 = min(n, team.rank * tile), t1 = min(n, t0 + tile);
    const int first = sort_plan(A.cells);
    // a bin is a cell of level 6 (with 11 bits, two of them)
    const bool thin = ((const volatile int *)A.cells)[5] <= (int)kBinMax;
    // an odd number of moves (passes and the fix) starts in buffer 1
    int cur = ((8 - first) + (first > 0)) & 1;
    auto K = [&](int c) { return c ? A.keys[1] : A.keys[0]; };
    auto V = [&](int c) { return c ? A.vals[1] : A.vals[0]; };
    if (team.rank == 0 && tid == 0) {  // set after the first barrier at the earliest
        *A.resort = 0;
        *A.deep = 0;
    }
    if (tid < kCellLevels) S.cells[tid] = 0;
    BucketResult bucket = kBucketDone;
    if (team.size == 1 && n <= chunk) {
        // ---- keys and sort within the block
        __syncthreads();  // every thread has read the plan
        if (tid < kCellLevels) A.cells[tid] = 0;
        if (!thin || !bucket_sort_local(A, chunk, S)) build_sort_local(A, first, chunk, S);
    } else if (thin && tile <= kBucketKeys * T &&
               (bucket = bucket_sort(A, team, t0, t1, S)) != kBucketTooFull) {
        if (bucket == kBucketFailed) return;
        // every block has read the plan
        if (team.rank == 0 && tid < kCellLevels) A.cells[tid] = 0;
    } else {
        // ---- keys
        if (tid < 256) S.base[tid] = 0;
        __syncthreads();
        for (int i = t0 + tid; i < t1; i += T) {
            const float2 p = A.pos[i];
            const uint64_t key = morton_key(p.x, p.y, A.rootx, A.rooty, A.radius);
            K(cur)[i] = key;
            V(cur)[i] = (uint32_t)i;
            atomicAdd(&S.base[(uint32_t)(key >> (8 * first)) & 255u], 1u);
        }
        __syncthreads();
        build_count_rows(A, team, first, S);
        if (!team.sync()) return;
        // every block has read the plan, and the bins that were too full
        if (team.rank == 0 && tid < kCellLevels) A.cells[tid] = 0;
        if (bucket == kBucketTooFull)
            for (int j = team.rank * T + tid; j < T * kBinsPerThread; j += team.size * T) A.hist[j] = 0;
        // ---- sort
        for (int pass = first; pass < 8; ++pass, cur ^= 1) {
            build_pass(A, team, pass, K(cur), V(cur), K(cur ^ 1), V(cur ^ 1), t0, t1, tile, chunk, S);
            if (!team.sync()) return;
        }
        if (first > 0) {
            build_fix<T>(A, 8 * first, K(cur), V(cur), K(cur ^ 1), V(cur ^ 1), t0, t1);
            cur ^= 1;
            if (!team.sync()) return;
            if (*(volatile int *)A.resort) {
                if (team.rank == 0 && tid == 0) *A.resorts += 1;
                // every digit, from the order the partial sort left: equal keys
                // keep their input order through both, so this is the full
                // sort's order
                if (tid < 256) S.base[tid] = 0;
                __syncthreads();
                for (int i = t0 + tid; i < t1; i += T)
                    atomicAdd(&S.base[(uint32_t)K(cur)[i] & 255u], 1u);
                __syncthreads();
                build_count_rows(A, team, 0, S);
                if (!team.sync()) return;
                for (int pass = 0; pass < 8; ++pass, cur ^= 1) {
                    build_pass(A, team, pass, K(cur), V(cur), K(cur ^ 1), V(cur ^ 1), t0, t1, tile,
                               chunk, S);
                    if (!team.sync()) return;
                }
            }
        }
    }
    // ---- count: the warps' and tiles' sums
    const double scale = A.radius > 0.0f ? kFixedScale / (double)A.radius : 1.0;
    const int rows = (t1 - t0 + 31) >> 5, per = (rows + kWarps - 1) / kWarps;
    const int r0 = (t0 >> 5) + min(rows, wid * per), r1 = (t0 >> 5) + min(rows, (wid + 1) * per);
    for (bool fixed = false;; fixed = true) {
        const CountOut c = build_count(A, r0, r1, t0 >> 5, scale, S);
        if (MOM) {
            const Moments v = sum_moments(A, r0, r1, scale);
            if (lane == 0) S.scan.mom[wid] = v;
        }
        if (lane == 0) {
            S.scan.warp[wid] = c.sum;
            S.scan.least[wid] = c.least;
            S.scan.deepest[wid] = c.deepest;
        }
        __syncthreads();
        if (wid == 0) {
            // the warps' exclusive sums, and the tile's
            const NodeSums zero{0, 0, 0, 0};
            const NodeSums w = lane < kWarps ? S.scan.warp[lane] : zero;
            NodeSums wi = w;
#pragma unroll
            for (int o = 1; o < kWarps; o <<= 1) {
                const NodeSums t = shfl_up_sums(wi, o);
                if (lane >= o) sums_add(wi, t);
            }
            if (lane == kWarps - 1) A.totals[team.rank] = wi;
            wi.g -= w.g;
            wi.m -= w.m;
            wi.x -= w.x;
            wi.y -= w.y;
            if (lane < kWarps) S.scan.warp[lane] = wi;
            const uint32_t least =
                __reduce_min_sync(kFullMask, lane < kWarps ? S.scan.least[lane] : 255u);
            const int deepest =
                __reduce_max_sync(kFullMask, lane < kWarps ? S.scan.deepest[lane] : 0);
            if (lane == 0) {
                A.tilemin[team.rank] = (uint8_t)least;
                atomicMax(A.max_level, deepest);
                if (deepest == kLevels) atomicExch(A.deep, 1);
            }
        }
        if (MOM && wid == 1) {
            Moments run{0, 0, 0, 0};
            if (lane == 0) {
                for (int w = 0; w < kWarps; ++w) {
                    const Moments v = S.scan.mom[w];
                    S.scan.mom[w] = run;
                    mom_add(run, v);
                }
                A.mom_totals[team.rank] = run;
            }
        }
        if (!team.sync()) return;
        if (fixed || !*(volatile int *)A.deep) break;
        // runs of equal 64-bit keys: in the order of the digits below, then
        // the count again
        for (int k = t0 + tid; k < t1; k += T)
            if (A.lcp[k] == kLevels + 1 && (k == 0 || A.lcp[k - 1] != kLevels + 1))
                fix_run(k, n, A.keys[0], A.vals[0], A.pos, A.ref_of, A.rootx, A.rooty, A.radius,
                        A.err, A.poison, 0);
        if (!team.sync()) return;
    }
    // the same in every block: the bit that the next phase sets does not count
    if ((*(volatile int *)A.err & ~kErrTreeTooLarge) || *(volatile int *)A.poison) return;
    // ---- prefixes and nodes, a row at a time
    if (wid == 0) {
        NodeSums p{0, 0, 0, 0};
        for (int t = lane; t < team.rank; t += 32) {
            const NodeSums *q = &A.totals[t];
            NodeSums v;
            v.g = __ldcg(&q->g);
            v.m = __ldcg(&q->m);
            v.x = ldcg_i128(&q->x);
            v.y = ldcg_i128(&q->y);
            sums_add(p, v);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sums_add(p, shfl_xor_sums(p, o));
        if (lane == 0) S.scan.prefix = p;
    }
    if (MOM && wid == 1) {
        Moments p{0, 0, 0, 0};
        for (int t = lane; t < team.rank; t += 32) {
            const Moments *q = &A.mom_totals[t];
            mom_add(p, Moments{ldcg_i128(&q->x), ldcg_i128(&q->y), ldcg_i128(&q->re),
                               ldcg_i128(&q->im)});
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mom_add(p, mom_shfl_xor(p, o));
        if (lane == 0) S.scan.mom_prefix = p;
    }
    if (tid < team.size) S.tilemin[tid] = A.tilemin[tid];  // at most 256 tiles
    __syncthreads();
    NodeSums base = S.scan.prefix;
    sums_add(base, S.scan.warp[wid]);
    const double inv_scale = A.radius > 0.0f ? (double)A.radius / kFixedScale : 1.0;
    const double rx = A.rootx, ry = A.rooty;
    uint32_t *defer = A.defer + (size_t)r0 * (kLevels + 1);
    int deferred = 0;
    // the next row's loads go out before this row's sums
    auto body = [&](int r) {
        const int k = r * 32 + lane;
        return r < r1 && k < n ? A.sbody[k] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    };
    auto shared = [&](int r) {
        const int k = r * 32 + lane;
        return r < r1 && k < n ? (int)A.lcp[k] - 1 : -1;
    };
    float4 me_next = body(r0);
    int L_next = shared(r0);
    for (int r = r0; r < r1; ++r) {
        const int k = r * 32 + lane;
        const bool in = k < n;
        const float4 me = me_next;
        const int Lk = L_next;
        me_next = body(r + 1);
        L_next = shared(r + 1);
        int Lkm1 = __shfl_up_sync(kFullMask, Lk, 1);
        if (lane == 0) Lkm1 = k == 0 ? -1 : (int)A.lcp[k - 1] - 1;
        const int c = in ? cells_at(k, Lk, Lkm1) : 0;
        const long long im = (long long)me.z;
        const RowSums own{in ? (uint32_t)c + 1u : 0u, (uint32_t)im,
                          (i128)im * fixed_offset(me.x, A.rootx, scale),
                          (i128)im * fixed_offset(me.y, A.rooty, scale)};
        const RowSums inc = row_scan(own, lane);
        const RowSums ex{inc.g - own.g, inc.m - own.m, inc.x - own.x, inc.y - own.y};
        // this body's prefix, record and node
        if (in) {
            const uint32_t g = base.g + ex.g, gb = g + (uint32_t)c;
            A.group[k] = g;
            A.pm[k] = base.m + ex.m;
            A.pxy[2 * (size_t)k] = base.x + ex.x;
            A.pxy[2 * (size_t)k + 1] = base.y + ex.y;
            if (gb < A.capacity) {
                A.nodes[gb] = make_float4(me.x, me.y, me.z, make_meta(gb + 1, kBodyLevel));
                A.owner[gb] = ((uint32_t)k << 6) | 63u;
            }
            A.body_node[k] = gb;
            if (k == n - 1) {
                A.pm[n] = base.m + inc.m;
                A.pxy[2 * (size_t)n] = base.x + inc.x;
                A.pxy[2 * (size_t)n + 1] = base.y + inc.y;
                *A.tree_nodes = base.g + inc.g;
                if (base.g + inc.g > A.capacity) atomicOr(A.err, kErrTreeTooLarge);
            }
        }
        // the cells that start in this row, one per lane: lane o's cells are
        // the numbers ci - c .. ci - 1 (ci: inclusive count)
        const uint32_t ci = inc.g - (uint32_t)min(lane + 1, n - r * 32);
        const uint32_t cells = __shfl_sync(kFullMask, ci, 31);
        // least shared digits over the 2^s bodies from each lane on
        int low[5];
        low[0] = Lk;
#pragma unroll
        for (int s = 1; s < 5; ++s)
            low[s] = min(low[s - 1], __shfl_down_sync(kFullMask, low[s - 1], 1 << (s - 1)));
        const int l0 = k == 0 ? 0 : Lkm1 + 1;
        for (uint32_t j0 = 0; j0 < cells; j0 += 32) {
            const uint32_t j = j0 + (uint32_t)lane;
            const bool valid = j < cells;
            int o = 0;  // the lane whose cell this is
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) {
                const uint32_t v = __shfl_sync(kFullMask, ci, o + s - 1);
                if (v <= j && o + s < 32) o += s;
            }
            const uint32_t q = j - (__shfl_sync(kFullMask, ci, o) - __shfl_sync(kFullMask, (uint32_t)c, o));
            const int lvl = __shfl_sync(kFullMask, l0, o) + (int)q;
            // its last body: the first from o on that shares fewer digits
            // with the next
            int e = o;
#pragma unroll
            for (int s = 5; s >= 0; --s) {
                const int w = s == 0 ? 0 : s - 1;  // widths 16, 8, 4, 2, 1, 1
                const int v = __shfl_sync(kFullMask, low[w], e & 31);
                if (e < 32 && v >= lvl) e += 1 << w;
            }
            const bool here = e < 32;
            const int eb = e & 31;
            const uint32_t dm = __shfl_sync(kFullMask, inc.m, eb) - __shfl_sync(kFullMask, ex.m, o);
            const i128 dx = shfl96(inc.x, eb) - shfl96(ex.x, o);
            const i128 dy = shfl96(inc.y, eb) - shfl96(ex.y, o);
            const uint32_t next = base.g + __shfl_sync(kFullMask, inc.g, eb);
            const uint32_t g = base.g + __shfl_sync(kFullMask, ex.g, o) + q;
            const int kb = r * 32 + o;
            if (valid && g < A.capacity) {
                A.owner[g] = ((uint32_t)kb << 6) | q;
                if (here) {
                    A.nodes[g] = cell_record((double)dm, i128_to_double(dx), i128_to_double(dy),
                                             rx, ry, inv_scale, next, lvl);
                    if (lvl >= 12 && lvl <= 28 && (lvl & 3) == 0)
                        atomicMax(&S.cells[(lvl - 12) >> 2], e - o + 1);
                }
            }
            // the others after the barrier
            const unsigned dmask = __ballot_sync(kFullMask, valid && !here);
            if (valid && !here)
                defer[deferred + __popc(dmask & ((1u << lane) - 1u))] = ((uint32_t)kb << 6) | (uint32_t)lvl;
            deferred += __popc(dmask);
        }
        base.g += __shfl_sync(kFullMask, inc.g, 31);
        base.m += __shfl_sync(kFullMask, inc.m, 31);
        base.x += shfl96(inc.x, 31);
        base.y += shfl96(inc.y, 31);
    }
    if (MOM) {
        Moments p = S.scan.mom_prefix;
        mom_add(p, S.scan.mom[wid]);
        scan_moments(A, r0, r1, scale, p);
    }
    if (!team.sync()) return;
    if (*(volatile int *)A.err) return;
    // ---- cells that end in a later row
    const uint32_t nodes = *(volatile uint32_t *)A.tree_nodes;
    const int tile_rows = tile >> 5, all_rows = (n + 31) >> 5;
    for (int j = lane; j < deferred; j += 32) {
        const uint32_t w = defer[j];
        const int k = (int)(w >> 6), lvl = (int)(w & 63u);
        const uint32_t t = (uint32_t)lvl + 1u;  // bytes hold shared digits + 1
        const long long pmk = A.pm[k];
        const i128 pxk = A.pxy[2 * (size_t)k], pyk = A.pxy[2 * (size_t)k + 1];
        const uint32_t gk = A.group[k];
        const int lk = k == 0 ? 0 : (int)A.lcp[k - 1];
        // the row with its last body: in this tile, or in the first later
        // tile that has one
        const int tr0 = t0 >> 5;
        int row = rows <= kMinRows ? tr0 + first_below(S.rowmin, (k >> 5) + 1 - tr0, rows, t)
                                   : first_below(A.rowmin, (k >> 5) + 1, tr0 + rows, t);
        if (row == tr0 + rows) {
            const int u = first_below(S.tilemin, team.rank + 1, team.size, t);
            row = first_below(A.rowmin, u * tile_rows, min((u + 1) * tile_rows, all_rows), t);
        }
        const int b = first_below(A.lcp, row * 32, min(row * 32 + 32, n), t);
        const double cm = (double)(A.pm[b + 1] - pmk);
        const double sx = i128_to_double(A.pxy[2 * (size_t)(b + 1)] - pxk);
        const double sy = i128_to_double(A.pxy[2 * (size_t)(b + 1) + 1] - pyk);
        const uint32_t next = b == n - 1 ? nodes : A.group[b + 1];
        // cells of body k in order: the first one's level is the shared
        // digits with the body before, plus one
        const uint32_t g = gk + (uint32_t)(lvl - lk);
        A.nodes[g] = cell_record(cm, sx, sy, rx, ry, inv_scale, next, lvl);
        if (lvl >= 12 && lvl <= 28 && (lvl & 3) == 0)
            atomicMax(&S.cells[(lvl - 12) >> 2], b - k + 1);
        if (lvl == kBinLevel) atomicMax(&S.cells[kCellLevels - 1], b - k + 1);  // full bins end here
    }
    __syncthreads();
    if (tid < kCellLevels && S.cells[tid]) atomicMax(&A.cells[tid], S.cells[tid]);
}

}  // namespace fa2
