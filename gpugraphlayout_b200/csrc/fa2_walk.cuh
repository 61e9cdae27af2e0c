// fa2_walk.cuh -- the Barnes-Hut walk of one group of 32 sorted bodies by one
// warp, shared by the single-graph traversal (fa2_kernels.cu) and the batched
// engine (fa2_batch.cu).
//
// The rule is the reference's (src/RPBHKernels.cu:609-685): a cell is used as a
// whole only if every body of the group passes d^2 + eps >= dq[level], else it
// is opened; bodies always interact.  A walk that takes one node after the
// other is a chain of dependent loads (about 250 ns a node, 500 nodes a group)
// with 21 instructions and one vote per node.  Here the 32 lanes take 32 nodes
// at once and the sums are a separate, dense loop:
//
//   * a lane holds an interval [node, end) of the preorder node array and walks
//     it.  When it opens a cell whose interval goes on behind the cell's
//     subtree, and the warp's stack runs low, it puts the rest on the stack and
//     keeps the subtree; a lane that has finished its interval takes the top of
//     the stack.  Every interval can be walked by one lane alone, so a full
//     stack (or none) costs only balance, never correctness;
//   * each lane tests its own node against the group's 32 bodies (two bodies
//     per packed FP32 instruction): min over the bodies of d^2, in the exact
//     roundings of sq_dist, is below dq exactly if some body fails the test
//     (adding eps is monotonic), so the accepted set is the vote's, bit for bit;
//   * accepted nodes go into a list in shared memory; every 64 of them, each
//     lane adds the 64 terms of its own body, two per packed instruction.
//
// The list's order depends only on the tree and the group, so a walk's sums
// are the same on every run, whatever block, grid or batch it runs in.
//
// Measured, k_traverse alone, one node at a time and now: 126 and 33 us on a
// 10,000-node Barabasi-Albert graph (few groups: latency), 148 and 42 us on
// R-MAT scale 16, 401 and 253 us on scale 20 (20,206 groups).  There the walk
// issues 1.8e8 warp instructions at 69 % of the issue rate, with 18 of 32
// lanes holding a node in the mean round.
#pragma once

#include <stdint.h>

#include "fa2_device.cuh"

namespace fa2 {

// Two floats in one 64-bit register pair, and the packed FP32 arithmetic of
// sm_100 on them (each half rounded on its own, to nearest).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// 1 / x; x is at least eps, so flushing subnormal inputs matters only for an
// eps below the smallest normal number (walk_rcp<false>).
template <bool NORMAL_EPS>
__device__ __forceinline__ float walk_rcp(float x) {
    if (!NORMAL_EPS) return __fdividef(1.0f, x);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
template <bool NORMAL_EPS>
__device__ __forceinline__ f32x2 rcp2(f32x2 v) {
    float a, b;
    unpack2(v, a, b);
    return pack2(walk_rcp<NORMAL_EPS>(a), walk_rcp<NORMAL_EPS>(b));
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    return fminf(fminf(a, b), c);
}

constexpr int kWalkList = 128;   // ring of accepted nodes: below 64 + 32 held
constexpr int kWalkChunk = 64;   // nodes summed at a time
constexpr int kWalkStack = 64;   // pushes stop at 32 entries, 32 more at most per round

// Shared memory of one warp's walk.  nx, ny hold negated coordinates, so that
// a difference is a packed addition.
template <bool QUAD, bool OVERLAP>
struct __align__(16) WalkWarp {
    float bx[32], by[32];                      // the group's bodies
    float nx[kWalkList], ny[kWalkList], m[kWalkList];
    float qx[QUAD ? kWalkList : 4];            // second moment, real part
    float nqy[QUAD ? kWalkList : 4];           // and the negated imaginary part
    float size[OVERLAP ? kWalkList : 4];       // a body's size, NaN for a cell
    uint2 stack[kWalkStack];                   // intervals [x, y)
};

// Level thresholds dq (src/RPBHKernels.cu:579-592): dq for the children of the
// root is (2 radius)^2 / theta^2 + eps, quartering per level; 0 for bodies.
__device__ __forceinline__ void walk_thresholds(float radius, const Params &prm,
                                                float (&dqs)[64]) {
    float tmp = radius * 2;
    float dq = tmp * tmp * prm.itolsq;
    dqs[0] = 0.0f;
    for (int l = 1; l <= kLevels; ++l) {
        dqs[l] = dq + prm.epssq;
        dq = dq * 0.25f;
    }
    for (int l = kLevels + 1; l < 64; ++l) dqs[l] = 0.0f;
}

// The sums of one walk: the even and the odd list entries apart.
struct WalkSums {
    f32x2 ax = 0, ay = 0;  // 0: both halves +0.0f
    f32x2 qy = 0;          // the quadrupole's part of -y
    __device__ __forceinline__ float2 total() const {
        float a, b, c, d, e, f;
        unpack2(ax, a, b);
        unpack2(ay, c, d);
        unpack2(qy, e, f);
        return make_float2(a + b, (c + d) - (e + f));
    }
};

// Adds the list entries [at, at + count) (count a multiple of 4) to the
// lane's body at (px, py): sum of m_j d / (d^2 + eps), and with QUAD the
// quadrupole term of the cells.
template <bool QUAD, bool OVERLAP, bool NORMAL_EPS>
__device__ __forceinline__ void walk_sum(const WalkWarp<QUAD, OVERLAP> &W, int at, int count,
                                         float px, float py, float my_size, float eps,
                                         WalkSums &S) {
    if (OVERLAP) {
        float ax, ay, u;
        unpack2(S.ax, ax, u);
        unpack2(S.ay, ay, u);
        for (int j = at; j < at + count; ++j) {
            const float dx = px + W.nx[j], dy = py + W.ny[j], m = W.m[j], sj = W.size[j];
            const float d2 = sq_dist(dx, dy, eps);
            const float c = sj == sj ? overlap_factor(d2, my_size, sj, m) : __fdividef(m, d2);
            ax = fmaf(dx, c, ax);
            ay = fmaf(dy, c, ay);
        }
        S.ax = pack2(ax, 0.0f);
        S.ay = pack2(ay, 0.0f);
        return;
    }
    const f32x2 p2x = pack2(px, px), p2y = pack2(py, py), e2 = pack2(eps, eps);
    const f32x2 m3 = pack2(-3.0f, -3.0f);
#pragma unroll 4
    for (int j = at; j < at + count; j += 4) {
        const ulonglong2 X = *reinterpret_cast<const ulonglong2 *>(&W.nx[j]);
        const ulonglong2 Y = *reinterpret_cast<const ulonglong2 *>(&W.ny[j]);
        const ulonglong2 M = *reinterpret_cast<const ulonglong2 *>(&W.m[j]);
        ulonglong2 Q = make_ulonglong2(0, 0), R = Q;
        if (QUAD) {
            Q = *reinterpret_cast<const ulonglong2 *>(&W.qx[j]);
            R = *reinterpret_cast<const ulonglong2 *>(&W.nqy[j]);
        }
        auto pair = [&](f32x2 nx, f32x2 ny, f32x2 m, f32x2 qx, f32x2 nqy) {
            const f32x2 dx = add2(p2x, nx), dy = add2(p2y, ny);
            const f32x2 inv = rcp2<NORMAL_EPS>(fma2(dx, dx, fma2(dy, dy, e2)));
            if (QUAD) {
                // conj(a2) u^3 with u = 1 / conj(w) = w / |w|^2: |u| <= 1 / sqrt(eps)
                // and |a2 u^3| is below the monopole term's size, so nothing
                // overflows however far apart the bodies are
                const f32x2 ux = mul2(dx, inv), uy = mul2(dy, inv);
                const f32x2 xx = mul2(ux, ux), yy = mul2(uy, uy);
                const f32x2 ur = mul2(ux, fma2(m3, yy, xx)), ui = mul2(uy, fma2(m3, xx, yy));
                S.ax = fma2(m, ux, S.ax);
                S.ay = fma2(m, uy, S.ay);
                S.ax = fma2(qx, ur, fma2(nqy, ui, S.ax));
                S.ay = fma2(nqy, ur, S.ay);
                S.qy = fma2(qx, ui, S.qy);
            } else {
                const f32x2 c = mul2(m, inv);
                S.ax = fma2(dx, c, S.ax);
                S.ay = fma2(dy, c, S.ay);
            }
        };
        pair(X.x, Y.x, M.x, Q.x, R.x);
        pair(X.y, Y.y, M.y, Q.y, R.y);
    }
}

// Whether every body of the group passes the test of a node at (cx, cy) with
// threshold thr: one lane, its own node.
template <class Warp>
__device__ __forceinline__ bool walk_accepts(const Warp &W, float cx, float cy, float thr,
                                             float eps) {
    const f32x2 ncx = pack2(-cx, -cx), ncy = pack2(-cy, -cy);
    float least = __int_as_float(0x7f800000);
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
        const ulonglong2 X = *reinterpret_cast<const ulonglong2 *>(&W.bx[j]);
        const ulonglong2 Y = *reinterpret_cast<const ulonglong2 *>(&W.by[j]);
        const f32x2 dx0 = add2(X.x, ncx), dy0 = add2(Y.x, ncy);
        const f32x2 dx1 = add2(X.y, ncx), dy1 = add2(Y.y, ncy);
        float a, b, c, d;
        unpack2(fma2(dx0, dx0, mul2(dy0, dy0)), a, b);
        unpack2(fma2(dx1, dx1, mul2(dy1, dy1)), c, d);
        least = min3(min3(least, a, b), c, d);
    }
    // !(< ) : a NaN distance accepts, so the walk always ends
    return !(__fadd_rn(least, eps) < thr);
}

// The walk of the group whose lane bodies sit at (px, py) (a lane without a
// body: 1e30, which passes every test) over the tree nodes[0 .. end).  Returns
// the lane's sums.  `on_cells(accepted_cell, cell, thr, node)` is called once
// per round by all lanes when ON_CELLS (the learned walk's pair list).
//
// AHEAD: a lane loads the two nodes that can follow its node, the first child
// and the next one behind the subtree, beside the node's test, and has the
// right one at hand in the next round.
template <bool QUAD, bool OVERLAP, bool ON_CELLS, bool NORMAL_EPS, bool AHEAD, class OnCells>
__device__ __forceinline__ float2 walk_group(WalkWarp<QUAD, OVERLAP> &W, const float (&dqs)[64],
                                             const float4 *nodes, const float2 *quad,
                                             const uint32_t *owner, const float *ssize,
                                             uint32_t end,
                                             float px, float py, float my_size, float eps,
                                             OnCells on_cells) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    __syncwarp();
    W.bx[lane] = px;
    W.by[lane] = py;
    __syncwarp();
    WalkSums S;
    uint32_t node = 1, stop = lane == 0 ? end : 0u;
    int depth = 0;                 // stack entries
    uint32_t head = 0, tail = 0;   // list entries summed and held
    float4 cur;  // AHEAD: the node's record, of a lane that holds one
    if (AHEAD && node < stop) cur = nodes[node];
    for (;;) {
        bool idle = node >= stop;
        unsigned im = __ballot_sync(kFullMask, idle);
        if (im != 0 && depth > 0) {
            const int r = __popc(im & lt);
            if (idle && r < depth) {
                const uint2 e = W.stack[depth - 1 - r];
                node = e.x;
                stop = e.y;
                idle = false;
                if (AHEAD) cur = nodes[node];
            }
            depth = max(0, depth - __popc(im));
            im = __ballot_sync(kFullMask, idle);
        }
        if (im == kFullMask) break;
        const float4 r = AHEAD ? cur : nodes[idle ? 0u : node];
        const int meta = __float_as_int(r.w);
        const int lvl = idle ? kBodyLevel : meta_level(meta);
        const float thr = dqs[lvl];
        const uint32_t next = meta_next(meta);
        float4 behind, child;
        if (AHEAD) {
            behind = nodes[!idle && next < stop ? next : 0u];
            child = nodes[lvl != kBodyLevel ? node + 1 : 0u];
        }
        const bool accept = walk_accepts(W, r.x, r.y, thr, eps) && !idle;
        // accepted nodes to the list
        const unsigned am = __ballot_sync(kFullMask, accept);
        if (accept) {
            const uint32_t at = (tail + (uint32_t)__popc(am & lt)) & (kWalkList - 1);
            W.nx[at] = -r.x;
            W.ny[at] = -r.y;
            W.m[at] = r.z;
            if (QUAD) {
                float2 q = make_float2(0.0f, 0.0f);
                if (lvl != kBodyLevel) q = quad[node];
                W.qx[at] = q.x;
                W.nqy[at] = -q.y;
            }
            if (OVERLAP)
                W.size[at] = lvl == kBodyLevel ? ssize[owner[node] >> 6]
                                               : __int_as_float(0x7fffffff);
        }
        tail += (uint32_t)__popc(am);
        if (ON_CELLS) on_cells(accept && lvl != kBodyLevel, r, thr, node);
        // opened cells: the rest of the interval to the stack while it is low
        const bool open = !accept && !idle;
        const bool push = open && next < stop && depth < 32;
        const unsigned pm = __ballot_sync(kFullMask, push);
        if (push) {
            W.stack[depth + __popc(pm & lt)] = make_uint2(next, stop);
            stop = next;
        }
        depth += __popc(pm);
        if (!idle) node = accept ? next : node + 1;
        if (AHEAD) cur = accept ? behind : child;
        __syncwarp();
        if (tail - head >= (uint32_t)kWalkChunk) {
            walk_sum<QUAD, OVERLAP, NORMAL_EPS>(W, (int)(head & (kWalkList - 1)), kWalkChunk, px,
                                                py, my_size, eps, S);
            head += kWalkChunk;
        }
    }
    // the rest, padded to a multiple of four with massless points far away
    const uint32_t rest = tail - head;
    const uint32_t pad = (0u - rest) & 3u;
    if ((uint32_t)lane < pad) {
        const uint32_t at = (tail + (uint32_t)lane) & (kWalkList - 1);
        W.nx[at] = W.ny[at] = -1e30f;
        W.m[at] = 0.0f;
        if (QUAD) W.qx[at] = W.nqy[at] = 0.0f;
        if (OVERLAP) W.size[at] = __int_as_float(0x7fffffff);
    }
    __syncwarp();
    // head is a multiple of 64, so the rest does not wrap around the ring
    walk_sum<QUAD, OVERLAP, NORMAL_EPS>(W, (int)(head & (kWalkList - 1)), (int)(rest + pad), px,
                                        py, my_size, eps, S);
    return S.total();
}

}  // namespace fa2
