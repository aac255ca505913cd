// dw_dev.cuh - double-word (float-pair) arithmetic and the split-layout
// column map, shared by the single solver (k_dw.cu) and the batched solver
// (k_batch.cu). Error-free transformations after Joldes, Muller and Popescu,
// "Tight and rigorous error bounds for basic building blocks of double-word
// arithmetic" (2017).
#pragma once
#include "kernels.h"
#include "outer_dev.cuh"

namespace ct {
namespace dwdev {

// ---- double-word arithmetic ------------------------------------------------
// A value is float2 v = (hi, lo) with v = hi + lo and |lo| <= ulp(hi) / 2.

__device__ __forceinline__ float2 two_sum(float a, float b) {
    const float s = a + b;
    const float bp = s - a;
    const float ap = s - bp;
    return make_float2(s, (a - ap) + (b - bp));
}

// |a| >= |b| (or a = 0).
__device__ __forceinline__ float2 fast_two_sum(float a, float b) {
    const float s = a + b;
    return make_float2(s, b - (s - a));
}

__device__ __forceinline__ float2 dw_add(float2 a, float2 b) {
    const float2 s = two_sum(a.x, b.x);
    return fast_two_sum(s.x, s.y + (a.y + b.y));
}

__device__ __forceinline__ float2 dw_neg(float2 a) { return make_float2(-a.x, -a.y); }

__device__ __forceinline__ float2 dw_mul(float2 a, float2 b) {
    const float p = a.x * b.x;
    float e = fmaf(a.x, b.x, -p);
    e = fmaf(a.x, b.y, e);
    e = fmaf(a.y, b.x, e);
    return fast_two_sum(p, e);
}

__device__ __forceinline__ float2 dw_of(double d) {
    const float h = __double2float_rn(d);
    return make_float2(h, __double2float_rn(d - (double)h));
}

__device__ __forceinline__ double dw_d(float2 a) { return (double)a.x + (double)a.y; }

// ---- sums of float x double-word products ------------------------------------
// (s, c): s collects the products' high parts through TwoSum, c the exact
// rounding errors of the products and the sums plus the products of the low
// parts; renormalised once at the end (fast_two_sum(s, c)). Each term costs
// eleven FP32 operations instead of the seventeen of a double-word product
// and a double-word sum, with
// an error of the same order (a few units of 2^-48 of the largest term).
struct DwAcc {
    float s, c;
};

// a += h + lo with |lo| << |h|.
__device__ __forceinline__ void acc_add(DwAcc& a, float h, float lo) {
    const float s = a.s + h;
    const float bp = s - a.s;
    const float err = (a.s - (s - bp)) + (h - bp);
    a.s = s;
    a.c += err + lo;
}

// a += g * p.
__device__ __forceinline__ void acc_mul_f(DwAcc& a, float2 p, float g) {
    const float h = g * p.x;
    acc_add(a, h, fmaf(g, p.y, fmaf(g, p.x, -h)));
}

// a += g * z (an exact product).
__device__ __forceinline__ void acc_mul_ff(DwAcc& a, float g, float z) {
    const float h = g * z;
    acc_add(a, h, fmaf(g, z, -h));
}

// a += u * v (both double words; the lo * lo term is below the error).
__device__ __forceinline__ void acc_mul(DwAcc& a, float2 u, float2 v) {
    const float h = u.x * v.x;
    acc_add(a, h, fmaf(u.x, v.y, fmaf(u.y, v.x, fmaf(u.x, v.x, -h))));
}

// ---- block and grid sums of accumulators ----------------------------------------
// The fixed trees of block_sum2 / gather2 (reduce.cuh) on the FP32 pipe: each
// step adds another thread's (s, c) with acc_add (TwoSum on s, c collecting
// the errors), and only thread 0 converts the block's or the grid's total to
// FP64. Summing every thread's value in FP64 instead cost each block about a
// microsecond of FP64 adds and conversions at its end, with the memory
// system idle.
__device__ __forceinline__ void warp_sum_acc(DwAcc& a) {
    for (int o = 16; o > 0; o >>= 1) {
        const float s = __shfl_down_sync(0xffffffffu, a.s, o);
        const float c = __shfl_down_sync(0xffffffffu, a.c, o);
        acc_add(a, s, c);
    }
}

// Block sums of N accumulators over NT threads; valid in thread 0. Warp q adds
// the warps' totals of accumulator q.
template <int N>
__device__ __forceinline__ void block_sum_acc(DwAcc (&a)[N]) {
    constexpr int NW = NT / 32;
    static_assert(N <= NW && NW <= 32, "a warp an accumulator");
    __shared__ float2 s[N][NW], t[N];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < N; ++q) {
        warp_sum_acc(a[q]);
        if (lane == 0) s[q][w] = make_float2(a[q].s, a[q].c);
    }
    __syncthreads();
    if (w < N) {
        const float2 u = lane < NW ? s[w][lane] : make_float2(0.0f, 0.0f);
        DwAcc b = {u.x, u.y};
        warp_sum_acc(b);
        if (lane == 0) t[w] = make_float2(b.s, b.c);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < N; ++q) a[q] = DwAcc{t[q].x, t[q].y};
    }
}

__device__ __forceinline__ double acc_value(const DwAcc& a) { return (double)a.s + (double)a.c; }

// Publishes the block's N sums as float pairs in slots `slot`, `stride` + slot,
// ... of part, takes a ticket, and returns in every thread whether this block
// arrived last of `count`.
template <int N>
__device__ __forceinline__ bool publish_acc(DwAcc (&a)[N], double* part, int stride, unsigned slot, unsigned* ticket,
                                            unsigned count) {
    __shared__ int last;
    block_sum_acc<N>(a);
    if (threadIdx.x == 0) {
        float2* pp = reinterpret_cast<float2*>(part);
#pragma unroll
        for (int q = 0; q < N; ++q) pp[(size_t)q * stride + slot] = make_float2(a[q].s, a[q].c);
        __threadfence();
        last = atomicAdd(ticket, 1u) == count - 1u ? 1 : 0;
    }
    __syncthreads();
    return last != 0;
}

// In the last block: the totals of slots [first, first + count), in slot
// order through the same tree, as FP64 in thread 0. Resets the ticket.
template <int N>
__device__ __forceinline__ void gather_acc(const double* part, int stride, unsigned first, unsigned count,
                                           unsigned* ticket, double (&total)[N]) {
    __threadfence();
    const float2* pp = reinterpret_cast<const float2*>(part);
    DwAcc a[N];
#pragma unroll
    for (int q = 0; q < N; ++q) a[q] = DwAcc{0.0f, 0.0f};
    // four slots' loads in flight, as gather_sums
    for (unsigned k0 = threadIdx.x; k0 < count; k0 += 4 * NT) {
        float2 p[4][N];
#pragma unroll
        for (unsigned u = 0; u < 4; ++u)
#pragma unroll
            for (int q = 0; q < N; ++q)
                p[u][q] = k0 + u * NT < count ? __ldcg(pp + (size_t)q * stride + first + k0 + u * NT)
                                              : make_float2(0.0f, 0.0f);
#pragma unroll
        for (unsigned u = 0; u < 4; ++u)
            if (k0 + u * NT < count)
#pragma unroll
                for (int q = 0; q < N; ++q) acc_add(a[q], p[u][q].x, p[u][q].y);
    }
    block_sum_acc<N>(a);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < N; ++q) total[q] = acc_value(a[q]);
        *ticket = 0u;
    }
}

// ---- the iteration (single solver and batch) -----------------------------------

// (A + C/dt) z at a cell: the stored diagonal times z minus the west, east,
// south, north, down and up neighbour terms (op_apply's order,
// src/operator3d.h:108-112); the products of floats are exact.
__device__ __forceinline__ float2 az_dw(const CellZ<float, float2>& a) {
    DwAcc off = {0.0f, 0.0f};
#pragma unroll
    for (int q = 0; q < 6; ++q) acc_mul_ff(off, a.g[q], a.z[q]);
    const float h = a.dg.x * a.zc;
    DwAcc r = {h, fmaf(a.dg.y, a.zc, fmaf(a.dg.x, a.zc, -h))};
    acc_add(r, -off.s, -off.c);
    return fast_two_sum(r.s, r.c);
}

// w = A z of a pair; v[0] += r.z, v[1] += z.Ap, v[2] += z.w (r, Ap and z of a
// padding slot are zero).
__device__ __forceinline__ void dots_dw(DwAcc (&v)[3], const PairZ<float, float2>& a, float4 r, float4 ap, float2* w) {
    const float2 w0 = az_dw(a.c[0]), w1 = a.second ? az_dw(a.c[1]) : make_float2(0.0f, 0.0f);
    *reinterpret_cast<float4*>(w + a.k) = make_float4(w0.x, w0.y, w1.x, w1.y);
    acc_mul_f(v[0], make_float2(r.x, r.y), a.c[0].zc);
    acc_mul_f(v[1], make_float2(ap.x, ap.y), a.c[0].zc);
    acc_mul_f(v[2], w0, a.c[0].zc);
    acc_mul_f(v[0], make_float2(r.z, r.w), a.c[1].zc);
    acc_mul_f(v[1], make_float2(ap.z, ap.w), a.c[1].zc);
    acc_mul_f(v[2], w1, a.c[1].zc);
}

// The step of a pair of values: p = z + beta p, Ap = w + beta Ap (p = z and
// Ap = w on the first iteration: beta, p and Ap are zero), r -= alpha Ap;
// rr += r.r.
struct StepItem {
    float2 z;
    float4 w, p, a, r;
};
__device__ __forceinline__ void step_item(StepItem& it, float2 alpha, float2 beta, DwAcc& rr) {
    const float2 ma = dw_neg(alpha);
    auto one = [&](float z, float wx, float wy, float& px, float& py, float& ax, float& ay, float& rx, float& ry) {
        const float2 p = dw_add(dw_mul(beta, make_float2(px, py)), make_float2(z, 0.0f));
        const float2 a = dw_add(dw_mul(beta, make_float2(ax, ay)), make_float2(wx, wy));
        const float2 r = dw_add(make_float2(rx, ry), dw_mul(ma, a));
        px = p.x, py = p.y;
        ax = a.x, ay = a.y;
        rx = r.x, ry = r.y;
        acc_mul(rr, r, r);
    };
    one(it.z.x, it.w.x, it.w.y, it.p.x, it.p.y, it.a.x, it.a.y, it.r.x, it.r.y);
    one(it.z.y, it.w.z, it.w.w, it.p.z, it.p.w, it.a.z, it.a.w, it.r.z, it.r.w);
}

// x += alpha p of a pair of values.
__device__ __forceinline__ float4 x_item(const float4& x, const float4& p, float2 alpha) {
    const float2 x0 = dw_add(make_float2(x.x, x.y), dw_mul(alpha, make_float2(p.x, p.y)));
    const float2 x1 = dw_add(make_float2(x.z, x.w), dw_mul(alpha, make_float2(p.z, p.w)));
    return make_float4(x0.x, x0.y, x1.x, x1.y);
}

// ---- column walk (split layout), as in k_outer.cu ----------------------------
struct Col {
    int i, j;
    unsigned s, sw, se, ss, sn;
    bool valid;
};

__device__ __forceinline__ Col col_of_slot(const Geo& g, unsigned s) {
    Col c;
    const unsigned row2 = 2u * (unsigned)g.hx;
    const int j = (int)(s / row2);
    const unsigned rem = s - (unsigned)j * row2;
    const int colour = rem >= (unsigned)g.hx ? 1 : 0;
    const int t = (int)rem - colour * g.hx;
    const int i = 2 * t + ((j + colour) & 1);
    const int oc = colour ^ 1;
    const unsigned row_o = (unsigned)(2 * j + oc) * (unsigned)g.hx;
    c.i = i;
    c.j = j;
    c.s = s;
    c.sw = row_o + (unsigned)((i - 1) >> 1);
    c.se = row_o + (unsigned)((i + 1) >> 1);
    c.ss = (unsigned)(2 * j - 2 + oc) * (unsigned)g.hx + (unsigned)t;
    c.sn = (unsigned)(2 * j + 2 + oc) * (unsigned)g.hx + (unsigned)t;
    c.valid = i < g.nx;
    return c;
}


}  // namespace dwdev
}  // namespace ct
