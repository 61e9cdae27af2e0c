// fa2_tree.cu -- beside the tree build (fa2_build.cuh): the replay path of
// coincident bodies, and the quadrupole option's cell moments (k_quad_cells),
// which follow from the build's prefix sums the way the centres of mass do.
#include <stdint.h>

#include "fa2_device.cuh"

namespace fa2 {

namespace {

constexpr unsigned kFull = kFullMask;

// ------------------------------------------------------------------- runs --

// Replay path: the runs of the last sort, with the .99 scaling applied.
__global__ void __launch_bounds__(256) k_runs(int n, const uint64_t *__restrict keys,
                                              uint32_t *__restrict vals, float2 *__restrict pos,
                                              const uint32_t *__restrict ref_of, DevState *st,
                                              int perturb) {
    if (st->err || st->poison) return;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k + 1 < n; k += gridDim.x * blockDim.x) {
        if (keys[k + 1] != keys[k] || (k > 0 && keys[k - 1] == keys[k])) continue;
        fix_run(k, n, keys, vals, pos, ref_of, st->rootx, st->rooty, st->radius, &st->err,
                &st->poison, perturb);
    }
}

inline int grid_for(int n, int threads, int cap) {
    int g = (n + threads - 1) / threads;
    return g < 1 ? 1 : (g > cap ? cap : g);
}

// ------------------------------------------------------------ quadrupoles --

// The quadrupole option needs every cell's complex second moment about its
// centre of mass, a2 = sum m (z - Z)^2, the coefficient of the second term of
// its far field: sum_j m_j / (w - d_j) = M / w + a2 / w^3 + ..., w = z - Z,
// d_j = z_j - Z (the dipole term vanishes about Z).  As for the centres of
// mass, a cell's sums are two prefix differences over its run of sorted
// bodies: exact 128-bit prefix sums of m q, m q^2 on a 2^-44 root-radius grid
// (Moments), which the tree build leaves; k_quad_cells forms a2 per cell.

// a - b
__device__ __forceinline__ Moments mom_sub(const Moments &a, const Moments &b) {
    return Moments{a.x - b.x, a.y - b.y, a.re - b.re, a.im - b.im};
}

constexpr double kMomScale = 17592186044416.0;  // 2^44

// a2 of the cell over sorted bodies k..b: exact integer sums about a grid
// point c near the centre of mass, then the centre's own offset in double.
__device__ __forceinline__ float2 cell_quadrupole(const Moments &hi, const Moments &lo,
                                                  long long mass, float radius) {
    const i128 M = mass;
    const Moments S = mom_sub(hi, lo);
    const double inv_m = 1.0 / (double)mass;
    const long long cx = __double2ll_rn(i128_to_double(S.x) * inv_m);
    const long long cy = __double2ll_rn(i128_to_double(S.y) * inv_m);
    // sum m ((q_x - c_x)^2 - (q_y - c_y)^2) and sum m (q_x - c_x)(q_y - c_y),
    // every term below 2^124
    const i128 tre = S.re - 2 * (i128)cx * S.x + 2 * (i128)cy * S.y +
                     ((i128)cx * cx - (i128)cy * cy) * M;
    const i128 tim = S.im - (i128)cx * S.y - (i128)cy * S.x + (i128)cx * cy * M;
    const double dx = i128_to_double(S.x - (i128)cx * M);
    const double dy = i128_to_double(S.y - (i128)cy * M);
    const double are = i128_to_double(tre) - (dx * dx - dy * dy) * inv_m;
    const double aim = i128_to_double(tim) - dx * dy * inv_m;
    const double u = (double)radius / kMomScale;
    return make_float2((float)(are * u * u), (float)(2.0 * aim * u * u));
}

// a2 of every cell.  A cell's bodies are the sorted run from its owner (the
// body that starts it) to the body at the last node of its subtree, the node
// before "next".  Each warp gathers the cells among 32 nodes at a time into a
// queue and works through it 32 cells at a time, so no lane idles on bodies.
constexpr int kQuadThreads = 256;

// 4 blocks per SM (64 registers); the launch puts no more than that on an SM
__global__ void __launch_bounds__(kQuadThreads, 4) k_quad_cells(const float4 *__restrict nodes,
                                                             const uint32_t *__restrict owner,
                                                             const long long *__restrict pm,
                                                             const Moments *__restrict pmom,
                                                             float2 *__restrict quad,
                                                             const DevState *st) {
    __shared__ uint32_t s_q[kQuadThreads / kWarp][64];
    if (st->err || st->poison) return;
    const uint32_t total = st->tree_nodes;
    const float radius = st->radius;
    const int lane = threadIdx.x & 31;
    uint32_t *q = s_q[threadIdx.x >> 5];
    const uint32_t nwarps = gridDim.x * (kQuadThreads / kWarp);
    const uint32_t warp = blockIdx.x * (kQuadThreads / kWarp) + (threadIdx.x >> 5);
    auto one = [&](uint32_t g) {
        const uint32_t w = owner[g];
        const uint32_t next = meta_next(__float_as_int(nodes[g].w));
        const int k = (int)(w >> 6), b = (int)(owner[next - 1] >> 6);
        quad[g] = cell_quadrupole(pmom[b + 1], pmom[k], pm[b + 1] - pm[k], radius);
    };
    int cnt = 0;
    for (uint32_t c0 = warp * 32; c0 < total; c0 += nwarps * 32) {
        const uint32_t g = c0 + lane;
        const bool cell = g < total && (owner[g] & 63u) != 63u;
        const unsigned m = __ballot_sync(kFull, cell);
        if (cell) q[cnt + __popc(m & ((1u << lane) - 1u))] = g;
        cnt += __popc(m);
        __syncwarp();
        if (cnt >= 32) {
            one(q[lane]);
            const uint32_t rest = lane + 32 < cnt ? q[lane + 32] : 0;
            __syncwarp();
            if (lane + 32 < cnt) q[lane] = rest;
            cnt -= 32;
            __syncwarp();
        }
    }
    if (lane < cnt) one(q[lane]);
}

}  // namespace

void launch_runs(const Buffers &b, int perturb, int nsm, cudaStream_t s) {
    k_runs<<<grid_for(b.n, 256, nsm * 8), 256, 0, s>>>(b.n, b.keys[0], b.vals[0], b.pos, b.ref_of,
                                                       b.st, perturb);
}

void launch_quad_cells(const Buffers &b, int nsm, cudaStream_t s) {
    k_quad_cells<<<grid_for(b.n, kQuadThreads, nsm * 4), kQuadThreads, 0, s>>>(
        b.nodes, b.owner, b.pm, b.pmom, b.quad, b.st);
}

}  // namespace fa2
