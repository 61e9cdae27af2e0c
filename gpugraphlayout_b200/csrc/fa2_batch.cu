// fa2_batch.cu -- many independent graphs laid out in one persistent launch.
//
// Each graph is small next to the GPU (tens to tens of thousands of nodes),
// so one team, a block or a cluster of up to eight, runs the whole ForceAtlas2
// iteration of one graph: gravity and attraction, bounding box, the tree
// (build_tree), the walk (walk_group), the speed rule and the displacement --
// the same code and arithmetic as the single-graph kernels.  Only the blocks
// of a cluster wait on one another, at the cluster's hardware barrier.  The
// teams of a grid that fills the GPU take graphs from a queue, largest first,
// and run `iters` iterations of a graph before taking the next, so a graph's
// working set stays in L2 across its iterations.  A team's scratch is one
// slot, sized for the largest graph of its class.
//
// Why clusters: with one block per graph a batch takes as long as its largest
// graph (3.4 ms for 512 graphs of up to 20,000 nodes, 1.2 with clusters) while
// the other SMs run dry.
//
// The reference has no batched mode: it lays out one graph per process, with
// its speed and tree state in device statics (src/RPFA2Kernels.cu:29-33,
// src/RPBHKernels.cu:54-62), so a batch is a sequence of separate runs.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <numeric>
#include <vector>

#include "../../include/fa2b200.h"
#include "fa2_build.cuh"
#include "fa2_device.cuh"
#include "fa2_walk.cuh"

namespace fa2 {

namespace {

// Every result is the same for each team (stable sort, exact integer sums,
// per-warp walks, fixed-order speed sums); only the speed differs.
constexpr int kMaxTeam = 8;                       // blocks per graph (a portable cluster)
constexpr uint32_t kBatchMaxNodes = FA2_BATCH_MAX_NODES;  // nodes per graph
constexpr int kErrPoisonRounds = 1 << 9;          // coincident bodies kept reappearing

struct BatchGraph {
    uint32_t node_base;  // first node of the graph in the batch arrays
    uint32_t n;          // nodes
};

struct BatchSpeed {
    float global_speed, speed_efficiency;
    int err;             // kErr* bits of this graph; its iterations stop
    int perturb_rounds;  // .99 re-insertion rounds of its last iteration
};

// Control block of one team's slot, in global memory: what its blocks share.
struct BatchCtl {
    int graph;     // index in the queue order
    int ticket;    // groups handed out in the walk
    int err, poison, resort, resorts, deep;
    int cells[kCellLevels];
    uint32_t tree_nodes;
    int max_level;
    int bad;       // a block saw a NaN or infinite position
    float4 box[kMaxTeam];  // the blocks' boxes: min x, max x, min y, max y
};

// Offsets of one team's scratch slot, in bytes, each 256-byte aligned.
struct SlotLayout {
    size_t ctl, keys0, keys1, vals0, vals1, sbody, lcp, rowmin, tilemin, defer, group, body_node,
        owner, nodes, pm, pxy, counts, hist, totals, fa, f, gpart;
    size_t bytes;
    uint32_t cap;  // tree nodes a slot holds
};

struct BatchArgs {
    const BatchGraph *graphs;
    const uint32_t *order;  // graphs, largest first
    int num_graphs;
    float2 *pos, *fprev;
    const float *mass;
    const uint32_t *off, *col;  // CSR over batch node ids
    BatchSpeed *speed;
    float2 *f_tot, *f_ag;       // last iteration's forces (diagnostics)
    uint32_t *sortd;            // last iteration's body order, graph-local ids
    unsigned *queue;
    char *slots;
    SlotLayout L;
    Params prm;
    float jitter_tolerance, k_s_max;
    int iters;
    int chunk;                  // keys the sort stages in shared memory
};

// The blocks of one cluster, or one block alone.
struct ClusterTeam {
    int rank, size;
    __device__ __forceinline__ bool sync() {
        if (size == 1)
            __syncthreads();
        else
            asm volatile(
                "barrier.cluster.arrive.release;\n\t"
                "barrier.cluster.wait.acquire;" ::
                    : "memory");
        return true;
    }
};

// Shared memory of the batch kernel (dynamic).  The build and the warps' walks
// take turns.
template <int T>
struct BatchShared {
    float dq[64];
    float4 wbox[T / kWarp];
    float rx, ry, radius;
    float gs, se;
};
template <int T>
constexpr size_t kBatchHead = (sizeof(BatchShared<T>) + 63) & ~(size_t)63;
template <int T>
size_t batch_smem_bytes(int chunk) {
    return kBatchHead<T> + std::max(build_smem_bytes<T>(chunk),
                                            sizeof(WalkWarp<false, false>) * (T / kWarp));
}

template <typename U>
__device__ __forceinline__ U *slot_ptr(char *slot, size_t off) {
    return reinterpret_cast<U *>(slot + off);
}

// --------------------------------------------------------------- phases --

// Gravity + attraction of the graph's nodes (8 lanes per row), into fa.
template <int T, bool LINLOG>
__device__ void phase_attract(const BatchArgs &A, const ClusterTeam &team, uint32_t base,
                              uint32_t n, float2 *fa) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int sub = lane >> 3, l8 = lane & 7;
    const uint32_t warp = (uint32_t)(team.rank * (T / kWarp) + wid);
    for (uint32_t r0 = warp * 4; r0 < n; r0 += (uint32_t)team.size * (T / kWarp) * 4) {
        const uint32_t row = r0 + (uint32_t)sub;
        const bool valid = row < n;
        float ax = 0.0f, ay = 0.0f;
        float2 p = make_float2(0.0f, 0.0f);
        if (valid) {
            p = A.pos[base + row];
            const uint32_t e1 = A.off[base + row + 1];
            // two of the lane's edges in flight at a time, added in order
            for (uint32_t e = A.off[base + row] + (uint32_t)l8; e < e1; e += 16) {
                const bool two = e + 8 < e1;
                const uint32_t c0 = A.col[e], c1 = two ? A.col[e + 8] : c0;
                const float2 p0 = A.pos[c0], p1 = A.pos[c1];
                const float2 q0 = pull<LINLOG>(p0, p);
                ax += q0.x;
                ay += q0.y;
                if (two) {
                    const float2 q1 = pull<LINLOG>(p1, p);
                    ax += q1.x;
                    ay += q1.y;
                }
            }
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            ax += __shfl_xor_sync(kFullMask, ax, o);
            ay += __shfl_xor_sync(kFullMask, ay, o);
        }
        if (valid && l8 == 0) {
            const float2 g = with_gravity(p, A.mass[base + row], ax, ay, A.prm);
            fa[row] = g;
            A.f_ag[base + row] = g;
        }
    }
}

// Bounding box and root cell of the graph (BoundingBoxKernel,
// src/RPBHKernels.cu:70-157), into S.rx, S.ry, S.radius of every block.
template <int T>
__device__ void phase_bbox(const BatchArgs &A, ClusterTeam &team, uint32_t base, uint32_t n,
                           BatchCtl *ctl, BatchShared<T> &S) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float4 a = make_float4(FLT_MAX, -FLT_MAX, FLT_MAX, -FLT_MAX);
    bool bad = false;
    for (uint32_t i = (uint32_t)(team.rank * T) + threadIdx.x; i < n; i += (uint32_t)team.size * T) {
        const float2 p = A.pos[base + i];
        a = make_float4(fminf(a.x, p.x), fmaxf(a.y, p.x), fminf(a.z, p.y), fmaxf(a.w, p.y));
        bad |= !(isfinite(p.x) && isfinite(p.y));
    }
    if (__any_sync(kFullMask, bad) && lane == 0) ctl->bad = 1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a.x = fminf(a.x, __shfl_xor_sync(kFullMask, a.x, o));
        a.y = fmaxf(a.y, __shfl_xor_sync(kFullMask, a.y, o));
        a.z = fminf(a.z, __shfl_xor_sync(kFullMask, a.z, o));
        a.w = fmaxf(a.w, __shfl_xor_sync(kFullMask, a.w, o));
    }
    if (lane == 0) S.wbox[wid] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        float4 b = S.wbox[0];
        for (int w = 1; w < T / kWarp; ++w) {
            const float4 c = S.wbox[w];
            b = make_float4(fminf(b.x, c.x), fmaxf(b.y, c.y), fminf(b.z, c.z), fmaxf(b.w, c.w));
        }
        ctl->box[team.rank] = b;
    }
    team.sync();
    if (threadIdx.x == 0) {
        float4 b = ctl->box[0];
        for (int r = 1; r < team.size; ++r) {
            const float4 c = ctl->box[r];
            b = make_float4(fminf(b.x, c.x), fmaxf(b.y, c.y), fminf(b.z, c.z), fmaxf(b.w, c.w));
        }
        S.radius = fmaxf(b.y - b.x, b.w - b.z) * 0.5f;
        S.rx = (b.x + b.y) * 0.5f;
        S.ry = (b.z + b.w) * 0.5f;
    }
    __syncthreads();
}

// The walk over this graph's tree, the total force, swing and traction per
// group of 32 bodies.
template <int T>
__device__ void phase_traverse(const BatchArgs &A, const ClusterTeam &team, uint32_t base,
                               uint32_t n, char *slot, BatchCtl *ctl, BatchShared<T> &S,
                               WalkWarp<false, false> *walk) {
    const float4 *nodes = slot_ptr<float4>(slot, A.L.nodes);
    const float4 *sbody = slot_ptr<float4>(slot, A.L.sbody);
    const float2 *fa = slot_ptr<float2>(slot, A.L.fa);
    float2 *f = slot_ptr<float2>(slot, A.L.f);
    float2 *gpart = slot_ptr<float2>(slot, A.L.gpart);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) walk_thresholds(S.radius, A.prm, S.dq);
    __syncthreads();
    const uint32_t end = *(volatile uint32_t *)&ctl->tree_nodes;
    const int ngroups = (int)((n + 31) >> 5);
    // a warp's first group spreads the groups over the blocks, the others come
    // from the ticket
    int w = wid * team.size + team.rank;
    while (w < ngroups) {
        const int k = w * 32 + lane;
        const bool active = k < (int)n;
        const float4 me = sbody[active ? k : (int)n - 1];
        const float px = active ? me.x : 1e30f, py = active ? me.y : 1e30f;
        auto none = [](bool, const float4 &, float, uint32_t) {};
        const float2 a =
            A.prm.epssq >= FLT_MIN
                ? walk_group<false, false, false, true, false>(walk[wid], S.dq, nodes, nullptr, nullptr,
                                                        nullptr, end, px, py, 0.0f, A.prm.epssq,
                                                        none)
                : walk_group<false, false, false, false, false>(walk[wid], S.dq, nodes, nullptr, nullptr,
                                                         nullptr, end, px, py, 0.0f, A.prm.epssq,
                                                         none);
        const float kmi = A.prm.k_r * me.z;
        const float ax = __fmul_rn(a.x, kmi), ay = __fmul_rn(a.y, kmi);
        float sw = 0.0f, tr = 0.0f;
        if (active) {
            const uint32_t i = __float_as_uint(me.w);
            const float2 g = fa[i], fp = A.fprev[base + i];
            const float fx = g.x + ax, fy = g.y + ay;
            f[i] = make_float2(fx, fy);
            A.f_tot[base + i] = make_float2(fx, fy);
            float dx = fx - fp.x, dy = fy - fp.y;
            sw = me.z * sqrtf(dx * dx + dy * dy);
            dx = fx + fp.x;
            dy = fy + fp.y;
            tr = me.z * (float)(sqrtf(dx * dx + dy * dy) / 2.0);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sw += __shfl_xor_sync(kFullMask, sw, o);
            tr += __shfl_xor_sync(kFullMask, tr, o);
        }
        if (lane == 0) {
            gpart[w] = make_float2(sw, tr);
            w = team.size * (T / kWarp) + atomicAdd(&ctl->ticket, 1);
        }
        w = __shfl_sync(kFullMask, w, 0);
    }
}

// The speed rule from the group partials, summed in a fixed order (by each
// block for itself).
template <int T>
__device__ void phase_speed(const BatchArgs &A, uint32_t n, char *slot, BatchShared<T> &S) {
    const float2 *gpart = slot_ptr<float2>(slot, A.L.gpart);
    const int lane = threadIdx.x & 31, ngroups = (int)((n + 31) >> 5);
    if (threadIdx.x < 32) {
        float sw = 0.0f, tr = 0.0f;
        for (int w = lane; w < ngroups; w += 32) {
            const float2 v = gpart[w];
            sw += v.x;
            tr += v.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sw += __shfl_xor_sync(kFullMask, sw, o);
            tr += __shfl_xor_sync(kFullMask, tr, o);
        }
        if (lane == 0) {
            float se = S.se, gs = S.gs;
            speed_update(sw, tr, (int)n, A.jitter_tolerance, A.k_s_max, se, gs);
            S.se = se;
            S.gs = gs;
        }
    }
    __syncthreads();
}

// Displacement (DisplacementKernel, src/RPFA2Kernels.cu:223-251).
template <int T>
__device__ void phase_displace(const BatchArgs &A, const ClusterTeam &team, uint32_t base,
                               uint32_t n, char *slot, float gs) {
    const float2 *f = slot_ptr<float2>(slot, A.L.f);
    for (uint32_t i = (uint32_t)(team.rank * T) + threadIdx.x; i < n; i += (uint32_t)team.size * T) {
        const float2 fi = f[i], fp = A.fprev[base + i];
        const float factor = displacement_factor(fi, fp, gs);
        float2 p = A.pos[base + i];
        p.x += fi.x * factor;
        p.y += fi.y * factor;
        A.pos[base + i] = p;
        A.fprev[base + i] = fi;
    }
}

// 1024 threads per SM, 64 registers a thread: a warp's walk has 32 loads in
// flight, so it needs few warps, and at 32 registers it spills.  Measured with
// 1024, 1536 and 2048 threads per SM: 512 graphs of 50 to 20,000 nodes 0.99, 0.98
// and 1.12 ms an iteration (one 256-thread block each 4.18, 5.13 and 5.99), 96
// graphs of 50 to 600 nodes 63, 72 and 80 us.
constexpr int kBatchThreadsPerSm = 1024;

// Launched in clusters of the team's size.
template <int T, bool LINLOG>
__global__ void __launch_bounds__(T, kBatchThreadsPerSm / T) k_batch(BatchArgs A) {
    extern __shared__ __align__(64) unsigned char smem_raw[];
    BatchShared<T> &S = *reinterpret_cast<BatchShared<T> *>(smem_raw);
    unsigned char *turns = smem_raw + kBatchHead<T>;
    BuildSmem<T> &B = *reinterpret_cast<BuildSmem<T> *>(turns);
    auto *walk = reinterpret_cast<WalkWarp<false, false> *>(turns);
    uint32_t crank, csize;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));
    ClusterTeam team{(int)crank, (int)csize};
    char *slot = A.slots + (size_t)(blockIdx.x / csize) * A.L.bytes;
    BatchCtl *ctl = slot_ptr<BatchCtl>(slot, A.L.ctl);
    float2 *fa = slot_ptr<float2>(slot, A.L.fa);
    const bool leader = team.rank == 0 && threadIdx.x == 0;
    const int tid0 = team.rank * T + (int)threadIdx.x, stride = team.size * T;
    auto flag = [](const int *p) { return *(const volatile int *)p; };
    for (;;) {
        if (leader) ctl->graph = (int)atomicAdd(A.queue, 1u);
        team.sync();
        const int qi = flag(&ctl->graph);
        if (qi >= A.num_graphs) break;
        const int gi = (int)A.order[qi];
        const BatchGraph G = A.graphs[gi];
        const uint32_t base = G.node_base, n = G.n;
        const BatchSpeed sp = A.speed[gi];
        if (threadIdx.x == 0) {
            S.gs = sp.global_speed;
            S.se = sp.speed_efficiency;
        }
        if (leader) {
            ctl->err = sp.err;
            ctl->poison = 0;
            ctl->bad = 0;
            ctl->resorts = 0;
            for (int l = 0; l < kCellLevels; ++l) ctl->cells[l] = 0;  // no last tree
        }
        BuildArgs T_{};
        T_.n = (int)n;
        T_.pos = A.pos + base;
        T_.mass = A.mass + base;
        T_.ref_of = nullptr;
        T_.keys[0] = slot_ptr<uint64_t>(slot, A.L.keys0);
        T_.keys[1] = slot_ptr<uint64_t>(slot, A.L.keys1);
        T_.vals[0] = slot_ptr<uint32_t>(slot, A.L.vals0);
        T_.vals[1] = slot_ptr<uint32_t>(slot, A.L.vals1);
        T_.sbody = slot_ptr<float4>(slot, A.L.sbody);
        T_.lcp = slot_ptr<uint8_t>(slot, A.L.lcp);
        T_.rowmin = slot_ptr<uint8_t>(slot, A.L.rowmin);
        T_.tilemin = slot_ptr<uint8_t>(slot, A.L.tilemin);
        T_.defer = slot_ptr<uint32_t>(slot, A.L.defer);
        T_.group = slot_ptr<uint32_t>(slot, A.L.group);
        T_.body_node = slot_ptr<uint32_t>(slot, A.L.body_node);
        T_.owner = slot_ptr<uint32_t>(slot, A.L.owner);
        T_.nodes = slot_ptr<float4>(slot, A.L.nodes);
        T_.capacity = A.L.cap;
        T_.pm = slot_ptr<long long>(slot, A.L.pm);
        T_.pxy = slot_ptr<i128>(slot, A.L.pxy);
        T_.counts = slot_ptr<uint32_t>(slot, A.L.counts);
        T_.hist = slot_ptr<uint32_t>(slot, A.L.hist);
        T_.totals = slot_ptr<NodeSums>(slot, A.L.totals);
        for (int j = tid0; j < kBuildBins; j += stride) T_.hist[j] = 0;
        T_.err = &ctl->err;
        T_.poison = &ctl->poison;
        T_.resort = &ctl->resort;
        T_.resorts = &ctl->resorts;
        T_.deep = &ctl->deep;
        T_.cells = ctl->cells;
        T_.tree_nodes = &ctl->tree_nodes;
        T_.max_level = &ctl->max_level;
        team.sync();
        int rounds = 0, err = flag(&ctl->err);
        for (int it = 0; it < A.iters && n > 0 && !err; ++it) {
            phase_attract<T, LINLOG>(A, team, base, n, fa);
            phase_bbox(A, team, base, n, ctl, S);
            // a NaN or infinite position stops this graph's iterations
            if (flag(&ctl->bad)) {
                err = kErrNonFinite;
                break;
            }
            T_.rootx = S.rx;
            T_.rooty = S.ry;
            T_.radius = S.radius;
            // Exactly coincident bodies: scale the later ones by .99 (the
            // reference's re-insertion, src/RPBHKernels.cu:271-278) and build
            // again, keeping gravity, attraction and the box of before.
            for (rounds = 0;; ++rounds) {
                if (leader) ctl->ticket = 0;
                build_tree<T, false>(T_, team, B, A.chunk);
                team.sync();
                err = flag(&ctl->err);
                if (err || !flag(&ctl->poison)) break;
                if (rounds >= 64) {
                    err = kErrPoisonRounds;
                    break;
                }
                for (int k = tid0; k + 1 < (int)n; k += stride)
                    if (T_.keys[0][k + 1] == T_.keys[0][k] &&
                        !(k > 0 && T_.keys[0][k - 1] == T_.keys[0][k]))
                        fix_run(k, (int)n, T_.keys[0], T_.vals[0], T_.pos, nullptr, S.rx, S.ry,
                                S.radius, &ctl->err, &ctl->poison, 1);
                team.sync();
                if (leader) ctl->poison = 0;
                team.sync();
            }
            if (err) break;
            phase_traverse(A, team, base, n, slot, ctl, S, walk);
            team.sync();
            phase_speed(A, n, slot, S);
            phase_displace<T>(A, team, base, n, slot, S.gs);
            team.sync();
        }
        // the body order of the last iteration, graph-local ids
        for (int k = tid0; k < (int)n; k += stride) A.sortd[base + k] = T_.vals[0][k];
        if (leader) {
            BatchSpeed out;
            out.global_speed = S.gs;
            out.speed_efficiency = S.se;
            out.err = err;
            out.perturb_rounds = rounds;
            A.speed[gi] = out;
        }
        team.sync();
    }
}

__global__ void k_clear_errors(int n, BatchSpeed *__restrict speed) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < n) speed[g].err = 0;
}

size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

SlotLayout make_layout(uint32_t nmax, int team) {
    SlotLayout L;
    const uint64_t cap64 = 33ull * nmax + 64, rows = (nmax + 31) / 32;
    L.cap = (uint32_t)cap64;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o = up256(o + bytes);
        return at;
    };
    L.ctl = take(sizeof(BatchCtl));
    L.keys0 = take(8ull * nmax);
    L.keys1 = take(8ull * nmax);
    L.vals0 = take(4ull * nmax);
    L.vals1 = take(4ull * nmax);
    L.sbody = take(16ull * nmax);
    L.lcp = take(pad64(nmax));
    L.rowmin = take(pad64(rows));
    L.tilemin = take(pad64((size_t)team));
    L.defer = take(4ull * (kLevels + 1) * rows);
    L.group = take(4ull * nmax);
    L.body_node = take(4ull * nmax);
    L.owner = take(4ull * cap64);
    L.nodes = take(16ull * (cap64 + 1));
    L.pm = take(8ull * (nmax + 1));
    L.pxy = take(32ull * (nmax + 1));
    L.counts = take(4ull * build_counts(team));
    L.hist = take(4ull * kBuildBins);
    L.totals = take(build_totals_bytes(team));
    L.fa = take(8ull * nmax);
    L.f = take(8ull * nmax);
    L.gpart = take(8ull * rows);
    L.bytes = o;
    return L;
}

}  // namespace

}  // namespace fa2

using namespace fa2;

// One size class of the batch: its graphs (a slice of the queue order), the
// teams that run them, and its grid with one scratch slot per team.
struct BatchClass {
    BatchArgs args{};
    int threads = 0;        // per block; 0: the class is empty
    int team = 1;           // blocks per graph, one cluster
    int grid = 0;           // teams
    size_t smem = 0;
    void *slots = nullptr;  // grid x args.L.bytes
    size_t slot_cap = 0;    // bytes allocated at slots
};

// A split's two sides, each of one class or one per team size.
constexpr int kMaxClasses = 6;

// How many 512-thread blocks (one cluster) run a graph: one up to `base` nodes,
// four up to four times as many, eight above.  A cluster of four does the work of
// about 2.8 blocks, so it is for graphs that would outlast the others: those of
// more than half the nodes a resident block has on average, at least kTeamNodes.
// A batch that one wave of single blocks holds, none of its graphs much above
// that average, has none; where four blocks for every graph are resident at once
// the line is kFewNodes.  Measured, ms an iteration, lines at 2048 / at the
// average's half / at the average; 512, 1024 and 4096 graphs of 50 to 20,000
// nodes: 1.19 / 1.19 / 1.34, 1.96 / 1.87 / 1.97, 7.94 / 6.74 / 6.74; 600 of 2500
// nodes 1.01 / 0.83 / 0.83, 300 of 20,000 3.95 / 3.61 / 5.06, 296 of 4000 (one
// wave) 0.71 / 0.71 / 0.56.  Lines at 2048 and 768: 8 of 2000 nodes 0.168 and
// 0.067, 64 of 2000 0.170 and 0.089, of 1000 0.088 and 0.061, of 800 0.076 and
// 0.057; 148 of 1500, more than fit at once, 0.131 and 0.193.
constexpr uint32_t kTeamNodes = 2048, kFewNodes = 768;
constexpr int kTeams[3] = {1, 4, 8};
uint32_t team_base(uint64_t total_nodes, uint32_t graphs, uint32_t largest, int nsm) {
    const uint64_t blocks = (uint64_t)nsm * (kBatchThreadsPerSm / 512);
    if (graphs <= blocks && 3ull * largest * blocks <= 4 * total_nodes)
        return std::max(largest, kTeamNodes);
    const uint64_t least = 4ull * graphs <= blocks ? kFewNodes : kTeamNodes;
    return (uint32_t)std::min<uint64_t>(std::max(total_nodes / (2 * blocks), least),
                                        kBatchMaxNodes);
}

struct fa2_batch {
    int device = 0;
    int nsm = 0;
    uint32_t num_graphs = 0;
    uint64_t total_nodes = 0;
    fa2_params prm{};
    Params kp{};
    std::vector<uint32_t> base;   // node base per graph
    std::vector<uint32_t> count;  // nodes per graph
    std::vector<uint32_t> order;  // graphs, largest first
    std::vector<void *> allocs;
    BatchArgs args{};             // the fields every class shares
    uint32_t *d_order = nullptr;  // the queue order of the current classes
    unsigned *queues = nullptr;   // one ticket counter per class
    // Graphs of at most `split` nodes run on `small_threads`, the others on
    // `large_threads`: 256 is one block of 256 threads per graph, 512 and 1024
    // are blocks of 512 threads, one or a cluster of them by the graph's size
    // and the batch's (team_base).  The classes that makes, small graphs first.
    uint32_t split = 0;
    int small_threads = 256, large_threads = 1024;
    std::vector<BatchClass> cls;
    // the launch of one step call, captured for its iteration count
    cudaGraphExec_t exec = nullptr;
    int exec_iters = -1;
    cudaStream_t stream = nullptr, side[kMaxClasses] = {};
    cudaEvent_t ev0 = nullptr, ev1 = nullptr, evFork = nullptr, evJoin[kMaxClasses] = {};
};

namespace {

int cuda_status_b(cudaError_t e) {
    if (e == cudaSuccess) return FA2_OK;
    if (e == cudaErrorMemoryAllocation) return FA2_ERR_OUT_OF_MEMORY;
    return FA2_ERR_CUDA;
}

#define BCK(x)                                       \
    do {                                             \
        cudaError_t e_ = (x);                        \
        if (e_ != cudaSuccess) return cuda_status_b(e_); \
    } while (0)

template <typename T>
int balloc(fa2_batch *b, T **p, size_t count) {
    void *q = nullptr;
    BCK(cudaMalloc(&q, count * sizeof(T) + 16));
    b->allocs.push_back(q);
    *p = static_cast<T *>(q);
    return FA2_OK;
}

void drop_graph(fa2_batch *b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
    b->exec_iters = -1;
}

void bfree(fa2_batch *b) {
    drop_graph(b);
    if (b->ev0) cudaEventDestroy(b->ev0);
    if (b->ev1) cudaEventDestroy(b->ev1);
    if (b->evFork) cudaEventDestroy(b->evFork);
    for (cudaEvent_t e : b->evJoin)
        if (e) cudaEventDestroy(e);
    if (b->stream) cudaStreamDestroy(b->stream);
    for (cudaStream_t t : b->side)
        if (t) cudaStreamDestroy(t);
    for (BatchClass &c : b->cls)
        if (c.slots) cudaFree(c.slots);
    for (void *p : b->allocs) cudaFree(p);
    b->allocs.clear();
}

// The launch of a class on a stream (or, with teams, only how many of its
// teams the GPU holds at once).
template <int T, bool LINLOG>
int launch_class(const BatchClass &c, cudaStream_t s, int *teams) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)c.team;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(c.team * std::max(1, c.grid)));
    cfg.blockDim = dim3(T);
    cfg.dynamicSmemBytes = c.smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = c.team > 1 ? 1 : 0;
    if (teams) {
        // the most any class of this kernel asks for
        BCK(cudaFuncSetAttribute(k_batch<T, LINLOG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)batch_smem_bytes<T>(T * kBuildRounds)));
        if (c.team > 1)
            return cuda_status_b(cudaOccupancyMaxActiveClusters(teams, k_batch<T, LINLOG>, &cfg));
        int per_sm = 0;
        BCK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch<T, LINLOG>, T, c.smem));
        *teams = per_sm * c.args.prm.nsm;
        return FA2_OK;
    }
    return cuda_status_b(cudaLaunchKernelEx(&cfg, k_batch<T, LINLOG>, c.args));
}

int launch_class(const BatchClass &c, bool linlog, cudaStream_t s, int *teams) {
    if (c.threads == 256)
        return linlog ? launch_class<256, true>(c, s, teams) : launch_class<256, false>(c, s, teams);
    return linlog ? launch_class<512, true>(c, s, teams) : launch_class<512, false>(c, s, teams);
}

// Splits the graphs into classes, uploads the queue order (class after class,
// each largest first) and sizes each class's grid and slots.
int configure(fa2_batch *b, uint32_t split, int small_threads, int large_threads) {
    drop_graph(b);  // the classes' grids and arguments are part of the graph
    // {largest graph of the class, threads per block, blocks per graph}
    struct Kind {
        uint32_t upto;
        int threads, team;
    };
    std::vector<Kind> kinds;
    uint32_t largest = 0;
    for (uint32_t n : b->count) largest = std::max(largest, n);
    const uint32_t base = team_base(b->total_nodes, b->num_graphs, largest, b->nsm);
    auto add = [&](uint32_t upto, int threads) {
        if (threads > 256)
            for (int team : kTeams)
                kinds.push_back(Kind{team == 8 ? upto : std::min(upto, base * (uint32_t)team), 512,
                                     team});
        else
            kinds.push_back(Kind{upto, 256, 1});
    };
    if (split) add(split, small_threads);
    add(kBatchMaxNodes, large_threads);
    std::vector<std::vector<uint32_t>> members(kinds.size());
    for (uint32_t g : b->order) {
        // the first kind that takes it: the small side's come first
        size_t k = 0;
        while (b->count[g] > kinds[k].upto) ++k;
        members[k].push_back(g);
    }
    std::vector<uint32_t> q;
    for (const auto &m : members) q.insert(q.end(), m.begin(), m.end());
    if (!q.empty())
        BCK(cudaMemcpyAsync(b->d_order, q.data(), q.size() * 4, cudaMemcpyHostToDevice,
                            b->stream));
    b->cls.resize(std::max(b->cls.size(), kinds.size()));
    for (BatchClass &c : b->cls) c.threads = 0;
    uint32_t first = 0;
    for (size_t k = 0; k < kinds.size(); ++k) {
        const std::vector<uint32_t> &m = members[k];
        if (m.empty()) continue;
        BatchClass &c = b->cls[k];
        c.args = b->args;
        c.threads = kinds[k].threads;
        c.team = kinds[k].team;
        uint32_t nmax = 1;
        for (uint32_t g : m) nmax = std::max(nmax, b->count[g]);
        c.args.order = b->d_order + first;
        first += (uint32_t)m.size();
        c.args.num_graphs = (int)m.size();
        c.args.queue = b->queues + k;
        int teams = 0;
        for (;; c.team /= 2) {
            c.args.L = make_layout(nmax, c.team);
            c.args.chunk = build_chunk(build_tile((int)nmax, c.team), c.threads);
            c.smem = c.threads == 256 ? batch_smem_bytes<256>(c.args.chunk)
                                      : batch_smem_bytes<512>(c.args.chunk);
            const int s = launch_class(c, b->kp.linlog != 0, b->stream, &teams);
            if (s) return s;
            // a context with a share of the SMs may hold no cluster of a size
            if (teams > 0 || c.team == 1) break;
        }
        c.grid = std::max(1, std::min<int>(teams, (int)m.size()));
        const size_t need = c.args.L.bytes * (size_t)c.grid;
        if (need > c.slot_cap) {
            if (c.slots) cudaFree(c.slots);
            c.slots = nullptr;
            c.slot_cap = 0;
            BCK(cudaMalloc(&c.slots, need));
            c.slot_cap = need;
        }
        c.args.slots = static_cast<char *>(c.slots);
    }
    b->split = split;
    b->small_threads = small_threads;
    b->large_threads = large_threads;
    BCK(cudaStreamSynchronize(b->stream));
    return FA2_OK;
}

// All classes at once, the largest graphs' first: that one on the batch
// stream, the others on side streams joined back into it.
int launch_batch(fa2_batch *b, int iters) {
    BCK(cudaMemsetAsync(b->queues, 0, kMaxClasses * sizeof(unsigned), b->stream));
    BCK(cudaEventRecord(b->evFork, b->stream));
    bool main = true;
    for (int k = (int)b->cls.size() - 1; k >= 0; --k) {
        BatchClass &c = b->cls[k];
        if (!c.threads) continue;
        c.args.iters = iters;
        cudaStream_t t = main ? b->stream : b->side[k];
        if (!main) BCK(cudaStreamWaitEvent(t, b->evFork, 0));
        const int s = launch_class(c, b->kp.linlog != 0, t, nullptr);
        if (s) return s;
        if (!main) BCK(cudaEventRecord(b->evJoin[k], t));
        main = false;
    }
    bool first = true;
    for (int k = (int)b->cls.size() - 1; k >= 0; --k) {
        if (!b->cls[k].threads) continue;
        if (!first) BCK(cudaStreamWaitEvent(b->stream, b->evJoin[k], 0));
        first = false;
    }
    return FA2_OK;
}

// One step call as a CUDA graph: the queue reset, the fork, a persistent
// launch per class and the join, captured once per iteration count and
// replayed.
int run_batch(fa2_batch *b, int iters) {
    if (!b->exec || b->exec_iters != iters) {
        drop_graph(b);
        BCK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
        const int s = launch_batch(b, iters);
        cudaGraph_t g = nullptr;
        const cudaError_t e = cudaStreamEndCapture(b->stream, &g);
        if (s) {
            if (g) cudaGraphDestroy(g);
            return s;
        }
        BCK(e);
        const cudaError_t e2 = cudaGraphInstantiate(&b->exec, g, 0);
        cudaGraphDestroy(g);
        BCK(e2);
        b->exec_iters = iters;
    }
    BCK(cudaGraphLaunch(b->exec, b->stream));
    return FA2_OK;
}

int check_errors(fa2_batch *b) {
    std::vector<BatchSpeed> sp(b->num_graphs);
    BCK(cudaMemcpyAsync(sp.data(), b->args.speed, sp.size() * sizeof(BatchSpeed),
                        cudaMemcpyDeviceToHost, b->stream));
    BCK(cudaStreamSynchronize(b->stream));
    for (const BatchSpeed &s : sp)
        if (s.err) return FA2_ERR_DEVICE_LIMIT;
    return FA2_OK;
}

}  // namespace

extern "C" {

fa2_batch *fa2_batch_create(uint32_t num_graphs, const fa2_graph_desc *graphs,
                            const fa2_params *prm, int *status) {
    int dummy;
    if (!status) status = &dummy;
    *status = FA2_ERR_INVALID_ARGUMENT;
    if (!prm || (num_graphs && !graphs)) return nullptr;
    // the batched walk uses cells as point masses only
    if (!prm->use_barneshut || prm->multipole > 1) {
        *status = FA2_ERR_UNSUPPORTED;
        return nullptr;
    }
    if (!(prm->theta > 0.0f)) return nullptr;
    uint64_t total_n = 0, total_m = 0;
    for (uint32_t g = 0; g < num_graphs; ++g) {
        const fa2_graph_desc &d = graphs[g];
        if (d.num_edges && (!d.sources || !d.targets)) return nullptr;
        // the batched attraction has no edge weights (w^0 = 1 is accepted)
        if (d.weights && prm->delta != 0.0f) {
            *status = FA2_ERR_UNSUPPORTED;
            return nullptr;
        }
        for (uint64_t e = 0; e < d.num_edges; ++e)
            if (d.sources[e] >= d.num_nodes || d.targets[e] >= d.num_nodes ||
                d.sources[e] == d.targets[e])
                return nullptr;
        if (d.num_nodes > kBatchMaxNodes) {
            *status = FA2_ERR_TOO_LARGE;
            return nullptr;
        }
        total_n += d.num_nodes;
        total_m += d.num_edges;
    }
    if (total_n >= (1ull << 31) || 2 * total_m >= (1ull << 32)) {
        *status = FA2_ERR_TOO_LARGE;
        return nullptr;
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || prm->device < 0 || prm->device >= ndev) {
        *status = FA2_ERR_NO_DEVICE;
        return nullptr;
    }
    cudaDeviceProp dp;
    if (cudaGetDeviceProperties(&dp, prm->device) != cudaSuccess || dp.major < 10) {
        *status = FA2_ERR_NO_DEVICE;
        return nullptr;
    }
    if (cudaSetDevice(prm->device) != cudaSuccess) {
        *status = FA2_ERR_CUDA;
        return nullptr;
    }
    fa2_batch *b = new fa2_batch();
    auto fail = [&](int s) {
        *status = s;
        bfree(b);
        delete b;
        return (fa2_batch *)nullptr;
    };
    b->device = prm->device;
    b->nsm = dp.multiProcessorCount;
    b->num_graphs = num_graphs;
    b->total_nodes = total_n;
    b->prm = *prm;
    b->kp.k_r = prm->scale;
    b->kp.k_g = prm->gravity;
    b->kp.itolsq = 1.0f / (prm->theta * prm->theta);  // src/RPForceAtlas2.cpp:47
    b->kp.epssq = prm->epssq;
    b->kp.strong_gravity = prm->strong_gravity;
    b->kp.linlog = prm->linlog != 0;
    b->kp.multipole = 1;
    b->kp.nsm = b->nsm;

    // host layout: graphs back to back, each graph's nodes in id order;
    // symmetric CSR over batch ids; mass = degree + 1 (src/RPForceAtlas2.cpp:74-77)
    const size_t N = (size_t)total_n;
    b->base.resize(num_graphs);
    b->count.resize(num_graphs);
    std::vector<BatchGraph> hg(num_graphs);
    std::vector<uint32_t> deg(N, 0);
    uint64_t nb = 0;
    for (uint32_t g = 0; g < num_graphs; ++g) {
        b->base[g] = (uint32_t)nb;
        b->count[g] = graphs[g].num_nodes;
        hg[g] = BatchGraph{(uint32_t)nb, graphs[g].num_nodes};
        for (uint64_t e = 0; e < graphs[g].num_edges; ++e) {
            deg[nb + graphs[g].sources[e]]++;
            deg[nb + graphs[g].targets[e]]++;
        }
        nb += graphs[g].num_nodes;
    }
    std::vector<uint32_t> off(N + 1, 0);
    for (size_t i = 0; i < N; ++i) off[i + 1] = off[i] + deg[i];
    std::vector<uint32_t> col(std::max<size_t>(off[N], 1));
    std::vector<uint32_t> fill(off.begin(), off.end() - 1);
    for (uint32_t g = 0; g < num_graphs; ++g) {
        const uint32_t bs = b->base[g];
        for (uint64_t e = 0; e < graphs[g].num_edges; ++e) {
            const uint32_t s = bs + graphs[g].sources[e], t = bs + graphs[g].targets[e];
            col[fill[s]++] = t;
            col[fill[t]++] = s;
        }
    }
    std::vector<float> mass(N);
    for (size_t i = 0; i < N; ++i) mass[i] = (float)deg[i] + 1.0f;
    // largest first (nodes + edges), so the long graphs start early
    std::vector<uint32_t> &order = b->order;
    order.resize(num_graphs);
    std::iota(order.begin(), order.end(), 0u);
    std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t c) {
        return (uint64_t)graphs[a].num_nodes + graphs[a].num_edges >
               (uint64_t)graphs[c].num_nodes + graphs[c].num_edges;
    });

    BatchArgs &A = b->args;

    BatchGraph *d_graphs = nullptr;
    uint32_t *d_off = nullptr, *d_col = nullptr;
    float *d_mass = nullptr;
    int s = FA2_OK;
    if ((s = balloc(b, &d_graphs, std::max<size_t>(num_graphs, 1))) ||
        (s = balloc(b, &b->d_order, std::max<size_t>(num_graphs, 1))) ||
        (s = balloc(b, &A.pos, std::max<size_t>(N, 1))) ||
        (s = balloc(b, &A.fprev, std::max<size_t>(N, 1))) ||
        (s = balloc(b, &d_mass, std::max<size_t>(N, 1))) || (s = balloc(b, &d_off, N + 1)) ||
        (s = balloc(b, &d_col, col.size())) ||
        (s = balloc(b, &A.speed, std::max<size_t>(num_graphs, 1))) ||
        (s = balloc(b, &A.f_tot, std::max<size_t>(N, 1))) ||
        (s = balloc(b, &A.f_ag, std::max<size_t>(N, 1))) ||
        (s = balloc(b, &A.sortd, std::max<size_t>(N, 1))) || (s = balloc(b, &b->queues, kMaxClasses)))
        return fail(s);
    A.graphs = d_graphs;
    A.mass = d_mass;
    A.off = d_off;
    A.col = d_col;
    A.prm = b->kp;
    A.jitter_tolerance = prm->jitter_tolerance;
    A.k_s_max = prm->k_s_max;
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&b->ev0) != cudaSuccess || cudaEventCreate(&b->ev1) != cudaSuccess ||
        cudaEventCreateWithFlags(&b->evFork, cudaEventDisableTiming) != cudaSuccess)
        return fail(FA2_ERR_CUDA);
    for (int k = 0; k < kMaxClasses; ++k)
        if (cudaStreamCreateWithFlags(&b->side[k], cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&b->evJoin[k], cudaEventDisableTiming) != cudaSuccess)
            return fail(FA2_ERR_CUDA);
    std::vector<BatchSpeed> sp(num_graphs);
    for (auto &x : sp) x = BatchSpeed{1.0f, 1.0f, 0, 0};  // src/RPFA2Kernels.cu:30-31
    cudaStream_t st = b->stream;
    if (cudaMemcpyAsync(d_graphs, hg.data(), hg.size() * sizeof(BatchGraph), cudaMemcpyHostToDevice, st) ||
        cudaMemcpyAsync(d_mass, mass.data(), N * 4, cudaMemcpyHostToDevice, st) ||
        cudaMemcpyAsync(d_off, off.data(), (N + 1) * 4, cudaMemcpyHostToDevice, st) ||
        cudaMemcpyAsync(d_col, col.data(), col.size() * 4, cudaMemcpyHostToDevice, st) ||
        cudaMemcpyAsync(A.speed, sp.data(), sp.size() * sizeof(BatchSpeed), cudaMemcpyHostToDevice, st) ||
        cudaMemsetAsync(A.pos, 0, N * 8, st) || cudaMemsetAsync(A.fprev, 0, N * 8, st) ||
        cudaMemsetAsync(A.f_tot, 0, N * 8, st) || cudaMemsetAsync(A.f_ag, 0, N * 8, st) ||
        cudaMemsetAsync(A.sortd, 0, N * 4, st) || cudaStreamSynchronize(st))
        return fail(FA2_ERR_CUDA);
    // every graph on teams by its size until fa2_batch_configure / _autotune
    if ((s = configure(b, 0, 256, 1024))) return fail(s);
    *status = FA2_OK;
    return b;
}

void fa2_batch_destroy(fa2_batch *b) {
    if (!b) return;
    cudaSetDevice(b->device);
    bfree(b);
    delete b;
}

int fa2_batch_set_positions(fa2_batch *b, const float *xy) {
    if (!b || (!xy && b->total_nodes)) return FA2_ERR_INVALID_ARGUMENT;
    BCK(cudaSetDevice(b->device));
    if (!b->total_nodes) return FA2_OK;
    BCK(cudaMemcpyAsync(b->args.pos, xy, b->total_nodes * 8, cudaMemcpyHostToDevice, b->stream));
    // new positions clear the graphs' device errors, which depend on them
    k_clear_errors<<<(b->num_graphs + 255) / 256, 256, 0, b->stream>>>((int)b->num_graphs,
                                                                       b->args.speed);
    BCK(cudaGetLastError());
    BCK(cudaStreamSynchronize(b->stream));
    return FA2_OK;
}

int fa2_batch_get_positions(fa2_batch *b, float *xy) {
    if (!b || (!xy && b->total_nodes)) return FA2_ERR_INVALID_ARGUMENT;
    BCK(cudaSetDevice(b->device));
    if (!b->total_nodes) return FA2_OK;
    BCK(cudaMemcpyAsync(xy, b->args.pos, b->total_nodes * 8, cudaMemcpyDeviceToHost, b->stream));
    BCK(cudaStreamSynchronize(b->stream));
    return FA2_OK;
}

int fa2_batch_step(fa2_batch *b, int32_t n_iters) {
    if (!b || n_iters < 0) return FA2_ERR_INVALID_ARGUMENT;
    BCK(cudaSetDevice(b->device));
    if (!n_iters || !b->num_graphs) return FA2_OK;
    int s = run_batch(b, n_iters);
    if (s) return s;
    return check_errors(b);
}

int fa2_batch_step_timed(fa2_batch *b, int32_t n_iters, float *ms) {
    if (!b || n_iters < 0 || !ms) return FA2_ERR_INVALID_ARGUMENT;
    BCK(cudaSetDevice(b->device));
    *ms = 0.0f;
    if (!n_iters || !b->num_graphs) return FA2_OK;
    BCK(cudaEventRecord(b->ev0, b->stream));
    int s = run_batch(b, n_iters);
    if (s) return s;
    BCK(cudaEventRecord(b->ev1, b->stream));
    BCK(cudaEventSynchronize(b->ev1));
    BCK(cudaEventElapsedTime(ms, b->ev0, b->ev1));
    return check_errors(b);
}

int fa2_batch_configure(fa2_batch *b, uint32_t split, int32_t small_threads,
                        int32_t large_threads) {
    auto ok = [](int32_t t) { return t == 256 || t == 512 || t == 1024; };
    if (!b || !ok(small_threads) || !ok(large_threads)) return FA2_ERR_INVALID_ARGUMENT;
    BCK(cudaSetDevice(b->device));
    BCK(cudaStreamSynchronize(b->stream));
    return configure(b, split, small_threads, large_threads);
}

int fa2_batch_get_config(fa2_batch *b, uint32_t *split, int32_t *small_threads,
                         int32_t *large_threads) {
    if (!b) return FA2_ERR_INVALID_ARGUMENT;
    if (split) *split = b->split;
    if (small_threads) *small_threads = b->small_threads;
    if (large_threads) *large_threads = b->large_threads;
    return FA2_OK;
}

int fa2_batch_autotune(fa2_batch *b, int32_t iters, uint32_t *split_out, int32_t *threads_out,
                       int32_t *large_out, float *ms_out) {
    if (!b || iters <= 0) return FA2_ERR_INVALID_ARGUMENT;
    BCK(cudaSetDevice(b->device));
    if (!b->num_graphs || !b->total_nodes) return FA2_OK;
    BCK(cudaStreamSynchronize(b->stream));
    // The trial steps change the layout state; it is saved here and put back
    // before each trial and at the end.
    const size_t N = b->total_nodes, G = b->num_graphs;
    BatchArgs &A = b->args;
    struct Saved {
        void *dst, *src;
        size_t bytes;
    };
    const Saved parts[] = {{nullptr, A.pos, N * 8},
                           {nullptr, A.fprev, N * 8},
                           {nullptr, A.speed, G * sizeof(BatchSpeed)},
                           {nullptr, A.f_tot, N * 8},
                           {nullptr, A.f_ag, N * 8},
                           {nullptr, A.sortd, N * 4}};
    std::vector<Saved> saved(std::begin(parts), std::end(parts));
    int s = FA2_OK;
    for (Saved &x : saved) {
        if (cudaMalloc(&x.dst, x.bytes) != cudaSuccess) {
            x.dst = nullptr;
            s = FA2_ERR_OUT_OF_MEMORY;
            break;
        }
        if (cudaMemcpyAsync(x.dst, x.src, x.bytes, cudaMemcpyDeviceToDevice, b->stream) !=
            cudaSuccess) {
            s = FA2_ERR_CUDA;
            break;
        }
    }
    auto restore = [&]() {
        for (Saved &x : saved)
            if (x.dst && cudaMemcpyAsync(x.src, x.dst, x.bytes, cudaMemcpyDeviceToDevice,
                                         b->stream) != cudaSuccess)
                return FA2_ERR_CUDA;
        return cudaStreamSynchronize(b->stream) == cudaSuccess ? FA2_OK : FA2_ERR_CUDA;
    };
    // candidates, each with classes of its own (512 and 1024 are the same
    // teams): every graph on teams by size, the graphs up to a size apart from
    // the others on one 256-thread block or teams of their own, or every graph
    // on one 256-thread block
    struct Cand {
        uint32_t split;
        int small, large;
    };
    uint32_t nmax = 1;
    for (uint32_t c : b->count) nmax = std::max(nmax, c);
    std::vector<Cand> cand{Cand{0u, 256, 1024}};
    for (uint32_t sp : {256u, 1024u, 4096u})
        for (int t : {256, 512})
            if (sp < nmax) cand.push_back(Cand{sp, t, 1024});
    cand.push_back(Cand{nmax, 256, 1024});
    const Cand start{b->split, b->small_threads, b->large_threads};
    float best_ms = 0.0f;
    Cand best = start;
    bool found = false;
    for (const Cand &c : cand) {
        if (s) break;
        if ((s = configure(b, c.split, c.small, c.large))) break;
        if ((s = restore())) break;
        float ms = 0.0f;
        if (cudaEventRecord(b->ev0, b->stream) != cudaSuccess) s = FA2_ERR_CUDA;
        if (!s) s = launch_batch(b, iters);
        if (!s && (cudaEventRecord(b->ev1, b->stream) != cudaSuccess ||
                   cudaEventSynchronize(b->ev1) != cudaSuccess ||
                   cudaEventElapsedTime(&ms, b->ev0, b->ev1) != cudaSuccess))
            s = FA2_ERR_CUDA;
        if (!s && (!found || ms < best_ms)) {
            best_ms = ms;
            best = c;
            found = true;
        }
    }
    const Cand pick = found ? best : start;
    const int s2 = configure(b, pick.split, pick.small, pick.large);
    const int s3 = restore();
    for (Saved &x : saved)
        if (x.dst) cudaFree(x.dst);
    if (s) return s;
    if (s2) return s2;
    if (s3) return s3;
    if (split_out) *split_out = b->split;
    if (threads_out) *threads_out = b->small_threads;
    if (large_out) *large_out = b->large_threads;
    if (ms_out) *ms_out = best_ms / (float)iters;
    return FA2_OK;
}

int fa2_batch_get_forces(fa2_batch *b, float *f_total, float *f_attr_grav) {
    if (!b) return FA2_ERR_INVALID_ARGUMENT;
    BCK(cudaSetDevice(b->device));
    const size_t bytes = b->total_nodes * 8;
    if (f_total && bytes)
        BCK(cudaMemcpyAsync(f_total, b->args.f_tot, bytes, cudaMemcpyDeviceToHost, b->stream));
    if (f_attr_grav && bytes)
        BCK(cudaMemcpyAsync(f_attr_grav, b->args.f_ag, bytes, cudaMemcpyDeviceToHost, b->stream));
    BCK(cudaStreamSynchronize(b->stream));
    return FA2_OK;
}

int fa2_batch_get_sort_order(fa2_batch *b, uint32_t *order) {
    if (!b || (!order && b->total_nodes)) return FA2_ERR_INVALID_ARGUMENT;
    BCK(cudaSetDevice(b->device));
    if (!b->total_nodes) return FA2_OK;
    BCK(cudaMemcpyAsync(order, b->args.sortd, b->total_nodes * 4, cudaMemcpyDeviceToHost,
                        b->stream));
    BCK(cudaStreamSynchronize(b->stream));
    return FA2_OK;
}

int fa2_batch_get_speed(fa2_batch *b, float *global_speed, float *speed_efficiency) {
    if (!b) return FA2_ERR_INVALID_ARGUMENT;
    BCK(cudaSetDevice(b->device));
    std::vector<BatchSpeed> sp(b->num_graphs);
    if (!sp.empty()) {
        BCK(cudaMemcpyAsync(sp.data(), b->args.speed, sp.size() * sizeof(BatchSpeed),
                            cudaMemcpyDeviceToHost, b->stream));
        BCK(cudaStreamSynchronize(b->stream));
    }
    for (size_t g = 0; g < sp.size(); ++g) {
        if (global_speed) global_speed[g] = sp[g].global_speed;
        if (speed_efficiency) speed_efficiency[g] = sp[g].speed_efficiency;
    }
    return FA2_OK;
}

}  // extern "C"
