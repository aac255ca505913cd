// f64_dev.cuh - float <-> double conversions without the FP64 pipe.
//
// On GB300 the hardware conversions F2F.F64.F32 and F2F.F32.F64 issue at the
// FP64 rate (measured with independent chains on 152 SMs: 0.63 T conversions
// per second, against 0.53 T DFMA/s and 38.6 T FFMA/s). The FP64 outer kernels
// convert every float face conductance and every float V-cycle value they
// touch, so those conversions cost as much as their FP64 arithmetic. These
// helpers rebuild the IEEE-754 results with integer operations (which issue on
// the FP32/INT32 pipes) and bit for bit equal the hardware conversion:
//  - widen: a float is exactly representable as a double; for normal floats
//    the exponent is rebiased (+896 = 1023 - 127) and the 23-bit mantissa
//    shifted into the top of the 52-bit one; zeros keep their sign;
//  - narrow: round to nearest, ties to even, of the 52-bit mantissa to 23
//    bits when the result is a normal float (a carry out of the mantissa
//    correctly bumps the exponent, up to infinity); zeros keep their sign.
// Every other input (subnormal, infinite or NaN floats; doubles whose float
// is subnormal or zero-by-underflow, or out of range) takes the hardware
// conversion, so the helpers are exact for every input.
// ct_selftest_conversions checks both against the hardware on the GPU.
#pragma once
#include <cuda_runtime.h>

#include "kernels.h"
#include "outer_dev.cuh"

namespace ct {
namespace f64dev {

__device__ __forceinline__ double widen(float f) {
    const unsigned u = __float_as_uint(f);
    const unsigned e = (u >> 23) & 0xffu;
    if (e - 1u < 254u) {  // normal
        const unsigned hi = (u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20));
        return __hiloint2double((int)hi, (int)(u << 29));
    }
    if ((u & 0x7fffffffu) == 0u) return __hiloint2double((int)(u & 0x80000000u), 0);
    return (double)f;
}

__device__ __forceinline__ float narrow(double d) {
    const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
    const unsigned E = (hi >> 20) & 0x7ffu;
    if (E - 897u < 254u) {  // the float is normal: 1 <= E - 896 <= 254
        const unsigned m = ((hi & 0xfffffu) << 3) | (lo >> 29);
        const unsigned rest = lo & 0x1fffffffu;
        unsigned f = (hi & 0x80000000u) | ((E - 896u) << 23) | m;
        f += (rest > 0x10000000u || (rest == 0x10000000u && (m & 1u))) ? 1u : 0u;
        return __uint_as_float(f);
    }
    if (((hi & 0x7fffffffu) | lo) == 0u) return __uint_as_float(hi & 0x80000000u);
    return (float)d;
}

// A double as a float pair: dw_of (dw_dev.cuh) without its three conversions.
__device__ __forceinline__ float2 split(double d) {
    const float h = narrow(d);
    return make_float2(h, narrow(d - widen(h)));
}

// The V-cycle's values as doubles: T = float (widened) or double (as is).
__device__ __forceinline__ double to_d(float v) { return widen(v); }
__device__ __forceinline__ double to_d(double v) { return v; }
// A double stored in the V-cycle's precision.
template <class T>
__device__ __forceinline__ T from_d(double v);
template <>
__device__ __forceinline__ float from_d<float>(double v) {
    return narrow(v);
}
template <>
__device__ __forceinline__ double from_d<double>(double v) {
    return v;
}

// n 2^x as a double, to nearest even, for |n| < 2^63 and results in the normal
// range, by integer operations (the conversion instruction holds the FP64 pipe).
// Ties are common (sums of a few 48-bit products) and A z is a small difference
// of large sums: rounding them away from zero moved the fields by 1e-12.
__device__ __forceinline__ double fixed_to_double(long long n, int x) {
    const unsigned hi = (unsigned)((unsigned long long)n >> 32);
    unsigned long long u = n < 0 ? 0ull - (unsigned long long)n : (unsigned long long)n;
    const int lz = __clzll((long long)(u | 1ull));
    u <<= lz - 1;  // bit 62 set
    // 53 bits, the leading one adding 1 to the exponent field
    const unsigned long long m = (u + 0x1ffull + ((u >> 10) & 1ull)) >> 10;
    const unsigned long long bits = m + ((unsigned long long)(unsigned)(1023 + 62 - lz + x) << 52);
    return n == 0 ? 0.0 : __longlong_as_double((long long)(bits | ((unsigned long long)(hi & 0x80000000u) << 32)));
}

// ---- A z of the V-cycle's float z ------------------------------------------------
//
// The sum of six float x float products, correctly summed to better than a
// double's rounding without the FP64 pipe (six DFMA a cell would hold the
// operator at 72 us of FP64 issue at 800 x 800 x 10). Each product is split
// exactly into h + l (one multiplication, one fused multiply-add). With 2^k above
// every |h|, adding the constant 1.5 2^23 q rounds a value to a multiple of q and
// leaves that multiple in the sum's mantissa bits, so integer sums of those bits
// add the rounded parts exactly: h at q = 2^(k-19), its remainder and l at
// 2^(k-39), what is left of both at 2^(k-59). The three integers are one 64-bit
// integer in units of 2^(k-59): error at most 6 x 2^(k-60), i.e. 2^-56 of the
// largest term, against 2^-53 of the partial sums for a chain of DFMA. Terms
// outside 2^-91 .. 2^122 (and all six zero) take that chain.
__device__ __forceinline__ double sum6(const float (&g)[6], const float (&z)[6]) {
    float h[6], l[6], m = 0.0f;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        h[i] = __fmul_rn(g[i], z[i]);
        l[i] = __fmaf_rn(g[i], z[i], -h[i]);
        m = fmaxf(m, fabsf(h[i]));
    }
    const unsigned e = __float_as_uint(m) >> 23;  // 2^k has the biased exponent e + 1
    if (e - 36u <= 213u) {
        const unsigned half = 0x400000u;  // 1.5's mantissa
        const unsigned b1 = ((e + 5u) << 23) | half, b2 = ((e - 15u) << 23) | half, b3 = ((e - 35u) << 23) | half;
        const float c1 = __uint_as_float(b1), c2 = __uint_as_float(b2), c3 = __uint_as_float(b3);
        unsigned n1 = 0u - 6u * b1, n2 = 0u - 12u * b2, n3 = 0u - 6u * b3;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const float t1 = __fadd_rn(h[i], c1), r = __fsub_rn(h[i], __fsub_rn(t1, c1));
            const float t2 = __fadd_rn(r, c2), r2 = __fsub_rn(r, __fsub_rn(t2, c2));
            const float t3 = __fadd_rn(l[i], c2), l2 = __fsub_rn(l[i], __fsub_rn(t3, c2));
            const float t4 = __fadd_rn(__fadd_rn(r2, l2), c3);
            n1 += __float_as_uint(t1);
            n2 += __float_as_uint(t2) + __float_as_uint(t3);
            n3 += __float_as_uint(t4);
        }
        const long long n = ((long long)(int)n1 << 40) + ((long long)(int)n2 << 20) + (long long)(int)n3;
        return fixed_to_double(n, (int)e - 185);
    }
    double off = 0.0;
#pragma unroll
    for (int i = 0; i < 6; ++i) off = __fma_rn(widen(g[i]), widen(z[i]), off);
    return off;
}
// The same for the FP64 V-cycle's z (west, east, south, north, down, up).
__device__ __forceinline__ double sum6(const float (&g)[6], const double (&z)[6]) {
    double off = 0.0;
#pragma unroll
    for (int i = 0; i < 6; ++i) off = __fma_rn(widen(g[i]), z[i], off);
    return off;
}

// (A + C/dt) z at a cell.
template <class T>
__device__ __forceinline__ double az64(const CellZ<T, double>& a) {
    return __fma_rn(a.dg, to_d(a.zc), -sum6(a.g, a.z));
}

// w = A z of a pair; v[0] += r.z, v[1] += z.Ap, v[2] += z.w.
template <class T>
__device__ __forceinline__ void dots64(double (&v)[3], const PairZ<T, double>& a, double2 r, double2 ap, double* w) {
    const double z0 = to_d(a.c[0].zc), z1 = to_d(a.c[1].zc);
    const double w0 = az64(a.c[0]), w1 = a.second ? az64(a.c[1]) : 0.0;
    *reinterpret_cast<double2*>(w + a.k) = make_double2(w0, w1);
    v[0] = __fma_rn(r.x, z0, v[0]);
    v[1] = __fma_rn(z0, ap.x, v[1]);
    v[2] = __fma_rn(z0, w0, v[2]);
    if (a.second) {
        v[0] = __fma_rn(r.y, z1, v[0]);
        v[1] = __fma_rn(z1, ap.y, v[1]);
        v[2] = __fma_rn(z1, w1, v[2]);
    }
}

// ---- the FP64 operator apply, one warp per row (single solver and batch) ----

// Operands of one cell, loaded before any is used (absent neighbours stay
// zero and are skipped by the same guards).
struct Cell64 {
    double pc, dg, pw, pe, ps, pn, pd, pu;
    float gw, ge, gs, gn, gd, gu;
};

__device__ __forceinline__ void load64(const OpView& o, const double* __restrict__ diag,
                                       const double* __restrict__ v, unsigned k, unsigned t,
                                       unsigned orow, int i, int e, bool hs, bool hn, bool hd, bool hu,
                                       Cell64& a) {
    const Geo& g = o.g;
    const unsigned hx = (unsigned)g.hx;
    a.pc = v[k];
    a.dg = diag[k];
    a.pw = a.pe = a.ps = a.pn = a.pd = a.pu = 0.0;
    a.gw = a.ge = a.gs = a.gn = a.gd = a.gu = 0.0f;
    if (i > 0) {
        const unsigned w = orow + t - 1u + (unsigned)e;
        a.pw = v[w];
        a.gw = o.gE[w];
    }
    if (i < g.nx - 1) {
        a.pe = v[orow + t + (unsigned)e];
        a.ge = o.gE[k];
    }
    if (hs) {
        const unsigned sl = orow - 2u * hx + t;
        a.ps = v[sl];
        a.gs = o.gN[sl];
    }
    if (hn) {
        a.pn = v[orow + 2u * hx + t];
        a.gn = o.gN[k];
    }
    if (hd) {
        a.pd = v[k - g.plane];
        a.gd = o.gU[k - g.plane];
    }
    if (hu) {
        a.pu = v[k + g.plane];
        a.gu = o.gU[k];
    }
}

// (A + C/dt) v at the cell: the stored diagonal times v minus the west, east,
// south, north, down and up terms, in op_apply's order (src/operator3d.h:
// 100-112), each a DFMA: 7 FP64 instructions.
__device__ __forceinline__ double compute64(const Cell64& a, bool w, bool e, bool s, bool n, bool d,
                                            bool u) {
    double off = 0.0;
    if (w) off = __fma_rn(widen(a.gw), a.pw, off);
    if (e) off = __fma_rn(widen(a.ge), a.pe, off);
    if (s) off = __fma_rn(widen(a.gs), a.ps, off);
    if (n) off = __fma_rn(widen(a.gn), a.pn, off);
    if (d) off = __fma_rn(widen(a.gd), a.pd, off);
    if (u) off = __fma_rn(widen(a.gu), a.pu, off);
    return __fma_rn(a.dg, a.pc, -off);
}

// Row R = l * 2 ny + 2 j + colour: the calling warp strides over the row's hx
// slots, U cells per lane and step (32 slots apart) with every operand of all
// U loaded first, and hands f(slot, valid, (A + C/dt) v, v) for each slot in
// order (padding slots: valid = false, zeros).
template <int U, class F>
__device__ __forceinline__ void row64(const OpView& o, const double* __restrict__ diag,
                                      const double* __restrict__ v, unsigned R, int lane, F&& f) {
    const Geo& g = o.g;
    const unsigned rows = 2u * (unsigned)g.ny;
    const unsigned l = R / rows;
    const unsigned r = R - l * rows;
    const int j = (int)(r >> 1), c = (int)(r & 1u), e = (j + c) & 1;
    const unsigned hx = (unsigned)g.hx;
    const unsigned base = l * g.plane;
    const unsigned row = base + r * hx;
    const unsigned orow = base + (unsigned)(2 * j + (c ^ 1)) * hx;  // other colour, same j
    const bool hs = j > 0, hn = j < g.ny - 1, hd = l > 0, hu = (int)l < g.nz - 1;
    for (unsigned t0 = (unsigned)lane; t0 < hx; t0 += 32u * U) {
        Cell64 a[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const unsigned t = t0 + 32u * u;
            const int i = 2 * (int)t + e;
            if (t < hx && i < g.nx) load64(o, diag, v, row + t, t, orow, i, e, hs, hn, hd, hu, a[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const unsigned t = t0 + 32u * u;
            const int i = 2 * (int)t + e;
            if (t < hx) {
                if (i < g.nx)
                    f(row + t, true, compute64(a[u], i > 0, i < g.nx - 1, hs, hn, hd, hu), a[u].pc);
                else
                    f(row + t, false, 0.0, 0.0);
            }
        }
    }
}

}  // namespace f64dev
}  // namespace ct
