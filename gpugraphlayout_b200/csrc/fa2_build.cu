// fa2_build.cu -- the tree build of the single-graph engine: build_tree by a
// grid of at most one block per SM with a barrier in global memory.
#include <stdint.h>

#include "fa2_build.cuh"

namespace fa2 {

namespace {

constexpr int kBuildThreads = 512;
static_assert(kBuildThreads * kBinsPerThread == kBuildBins, "the bins' counts");

// The blocks of one cooperative launch (all of them resident).  The barrier
// counts arrivals in a word that is zero when the launch starts.  A wait that
// does not end gives up, at once when another block has: the error bit stops
// the iteration.
struct GridTeam {
    int rank, size;
    unsigned *bar;
    unsigned target;
    DevState *st;
    __device__ __forceinline__ bool sync() {
        if (size == 1) {
            __syncthreads();
            return true;
        }
        __shared__ bool s_ok;
        __syncthreads();
        target += (unsigned)size;
        if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
            bool ok = true;
            for (unsigned polls = 1;; ++polls) {
                unsigned seen;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
                if (seen >= target) break;
                if (polls > (1u << 22) ||
                    ((polls & 4095) == 0 && (*(volatile int *)&st->err & kErrScanWait))) {
                    atomicOr(&st->err, kErrScanWait);
                    ok = false;
                    break;
                }
            }
            s_ok = ok;
        }
        __syncthreads();
        return s_ok;
    }
};

// 64 registers and half an SM's threads per block: the attraction's blocks
// share the SMs with it.
template <bool MOM>
__global__ void __launch_bounds__(kBuildThreads, 2) k_build(BuildArgs A, int chunk,
                                                            DevState *st, IterCounters *ctr) {
    extern __shared__ __align__(64) unsigned char smem_raw[];
    BuildSmem<kBuildThreads> &S = *reinterpret_cast<BuildSmem<kBuildThreads> *>(smem_raw);
    if (st->err || st->poison) return;
    A.rootx = st->rootx;
    A.rooty = st->rooty;
    A.radius = st->radius;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->interactions = 0;  // counted by k_count_interactions
        st->visits = 0;
        st->max_level = 0;  // raised in the count, after the first barrier
    }
    // the pairs of the walk that follows (a learned iteration's)
    if (blockIdx.x == 0 && threadIdx.x < 16) ctr->pair_count[threadIdx.x] = 0;
    GridTeam team{(int)blockIdx.x, (int)gridDim.x, &ctr->build_bar, 0u, st};
    build_tree<kBuildThreads, MOM>(A, team, S, chunk);
}

}  // namespace

cudaError_t launch_build(const Buffers &b, bool moments, cudaStream_t s) {
    BuildArgs A{};
    A.n = b.n;
    A.pos = b.pos;
    A.mass = b.mass;
    A.ref_of = b.ref_of;
    for (int i = 0; i < 2; ++i) {
        A.keys[i] = b.keys[i];
        A.vals[i] = b.vals[i];
    }
    A.sbody = b.sbody;
    A.lcp = b.lcp;
    A.rowmin = b.rowmin;
    A.tilemin = b.tilemin;
    A.defer = b.defer;
    A.group = b.group;
    A.body_node = b.body_node;
    A.owner = b.owner;
    A.nodes = b.nodes;
    A.capacity = b.capacity;
    A.pm = b.pm;
    A.pxy = b.pxy;
    A.pmom = b.pmom;
    A.mom_totals = b.mom_totals;
    A.counts = b.sort_counts;
    A.hist = b.ctr->hist;
    A.totals = static_cast<NodeSums *>(b.build_totals);
    A.err = &b.st->err;
    A.poison = &b.st->poison;
    A.resort = &b.st->resort;
    A.resorts = &b.st->resorts;
    A.deep = &b.st->deep;
    A.cells = b.st->cells;
    A.tree_nodes = &b.st->tree_nodes;
    A.max_level = &b.st->max_level;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg{};
    const int blocks = b.build_blocks;
    const int chunk = build_chunk(build_tile(b.n, blocks), kBuildThreads);
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.dynamicSmemBytes = build_smem_bytes<kBuildThreads>(chunk);
    cfg.blockDim = dim3(kBuildThreads);
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return moments ? cudaLaunchKernelEx(&cfg, k_build<true>, A, chunk, b.st, b.ctr)
                   : cudaLaunchKernelEx(&cfg, k_build<false>, A, chunk, b.st, b.ctr);
}

void build_set_smem_attr() {
    const int most = (int)build_smem_bytes<kBuildThreads>(kBuildThreads * kBuildRounds);
    cudaFuncSetAttribute(k_build<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    cudaFuncSetAttribute(k_build<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
}

size_t build_totals_bytes(int blocks) { return (size_t)blocks * sizeof(NodeSums); }

}  // namespace fa2
