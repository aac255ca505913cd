// outer_dev.cuh - pieces of the outer iteration shared by its FP64 kernels
// (k_fp64.cu, k_batch64.cu) and its double-word kernels (k_dw.cu, k_batch.cu).
#pragma once
#include "kernels.h"

namespace ct {

// Streams the items k = first, first + stride, ... below end, U per step,
// with the next step's loads issued before the current step's arithmetic (two
// register sets): the FP64 pipe, at ~1/70 of the FP32 rate, would otherwise
// hold each warp between its loads, and the memory traffic and the FP64
// instructions of these kernels would not overlap (measured: the dot took the
// sum of its DRAM time and its DFMA time, 42 us at 800 x 800 x 10).
// The double-word kernels keep more bytes in flight by it.
template <int U, class Item, class Load, class Use>
__device__ __forceinline__ void stream_pipelined(unsigned first, unsigned end, unsigned stride, Load load,
                                                 Use use) {
    Item a[U], b[U];
    bool va[U], vb[U];
    auto fetch = [&](unsigned k0, Item* it, bool* v) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const unsigned k = k0 + (unsigned)u * stride;
            v[u] = k < end;
            if (v[u]) it[u] = load(k);
        }
    };
    unsigned k0 = first;
    fetch(k0, a, va);
    while (k0 < end) {
        const unsigned k1 = k0 + (unsigned)U * stride;
        fetch(k1, b, vb);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (va[u]) use(k0 + (unsigned)u * stride, a[u]);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            a[u] = b[u];
            va[u] = vb[u];
        }
        k0 = k1;
    }
}

// Operands of (A + C/dt) z at one cell, loaded before any is used; an absent
// neighbour has a zero face (and a zero value).
template <class T, class D>
struct CellZ {
    T zc, z[6];
    float g[6];
    D dg;
};
template <class T, class D>
__device__ __forceinline__ void load_z(const OpView& o, const D* __restrict__ diag, const T* __restrict__ z, unsigned k,
                                       unsigned t, unsigned orow, int i, int e, bool hs, bool hn, bool hd, bool hu,
                                       CellZ<T, D>& a) {
    const Geo& g = o.g;
    const unsigned hx = (unsigned)g.hx;
    a.zc = z[k];
    a.dg = diag[k];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        a.z[q] = T(0);
        a.g[q] = 0.0f;
    }
    if (i > 0) {
        const unsigned w = orow + t - 1u + (unsigned)e;
        a.z[0] = z[w];
        a.g[0] = o.gE[w];
    }
    if (i < g.nx - 1) {
        a.z[1] = z[orow + t + (unsigned)e];
        a.g[1] = o.gE[k];
    }
    if (hs) {
        const unsigned s = orow - 2u * hx + t;
        a.z[2] = z[s];
        a.g[2] = o.gN[s];
    }
    if (hn) {
        a.z[3] = z[orow + 2u * hx + t];
        a.g[3] = o.gN[k];
    }
    if (hd) {
        a.z[4] = z[k - g.plane];
        a.g[4] = o.gU[k - g.plane];
    }
    if (hu) {
        a.z[5] = z[k + g.plane];
        a.g[5] = o.gU[k];
    }
}

// Row R = l * 2 ny + 2 j + colour: the calling warp strides over its slots, a cell
// a lane; load(slot) brings whatever else f needs, with the operands, and f(slot,
// that, operands) follows. Padding slots are left alone.
template <class T, class D, class Load, class F>
__device__ __forceinline__ void row_z(const OpView& o, const D* __restrict__ diag, const T* __restrict__ z, unsigned R,
                                      int lane, Load&& load, F&& f) {
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
    for (unsigned t = (unsigned)lane; t < hx; t += 32u) {
        const int i = 2 * (int)t + e;
        if (i >= g.nx) continue;
        CellZ<T, D> a;
        load_z(o, diag, z, row + t, t, orow, i, e, hs, hn, hd, hu, a);
        const auto more = load(row + t);
        f(row + t, more, a);
    }
}

template <class T>
struct Two;
template <>
struct Two<float> {
    typedef float2 type;
};
template <>
struct Two<double> {
    typedef double2 type;
};
template <>
struct Two<float2> {
    typedef float4 type;
};
template <class T>
__device__ __forceinline__ typename Two<T>::type load_two(const T* __restrict__ v, unsigned k) {
    return *reinterpret_cast<const typename Two<T>::type*>(v + k);
}
__device__ __forceinline__ double first_of(double2 v) { return v.x; }
__device__ __forceinline__ double second_of(double2 v) { return v.y; }
__device__ __forceinline__ float2 first_of(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 second_of(float4 v) { return make_float2(v.z, v.w); }

// Two cells of A z: slots k and k + 1 of one colour of one row (k even: hx is a
// multiple of 4), pair p of all planes in slot order, with loads of two values
// where the neighbours lie side by side; of the other colour's row the pair needs
// a third value to the west (even rows of the colour) or the east. second: slot
// k + 1 holds a cell (not padding).
template <class T, class D>
struct PairZ {
    CellZ<T, D> c[2];
    unsigned k;
    bool second;
};
// False where both slots are padding.
template <class T, class D>
__device__ __forceinline__ bool load_pair(const OpView& o, const D* __restrict__ diag, const T* __restrict__ z,
                                          unsigned p, PairZ<T, D>& a) {
    typedef typename Two<T>::type T2;
    const Geo& g = o.g;
    const unsigned hx = (unsigned)g.hx;
    const unsigned F = p / hx, q = 2u * (p - F * hx);  // row of both colours, slot in it
    const unsigned l = F / (unsigned)g.ny;
    const int j = (int)(F - l * (unsigned)g.ny);
    const int c = q >= hx ? 1 : 0, e = (j + c) & 1;
    const unsigned t = q - (c ? hx : 0u), k = 2u * p;
    const unsigned ok = c ? k - hx : k + hx;  // the other colour's slot t
    const int i0 = 2 * (int)t + e, i1 = i0 + 2;
    if (i0 >= g.nx) return false;
    a.k = k;
    a.second = i1 < g.nx;
    const T2 zc = load_two(z, k), zo = load_two(z, ok);
    const float2 go = load_two(o.gE, ok), ge = load_two(o.gE, k);
    const auto dg = load_two(diag, k);
    T zx = T(0);  // the third value of the other colour's row
    float gx = 0.0f;
    if (e == 0) {
        if (t > 0) {
            zx = z[ok - 1u];
            gx = o.gE[ok - 1u];
        }
    } else if (t + 2u < hx) {
        zx = z[ok + 2u];
    }
    T2 v[4];
    float2 f[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        v[s].x = v[s].y = T(0);
        f[s] = make_float2(0.0f, 0.0f);
    }
    if (j > 0) {
        v[0] = load_two(z, ok - 2u * hx);
        f[0] = load_two(o.gN, ok - 2u * hx);
    }
    if (j < g.ny - 1) {
        v[1] = load_two(z, ok + 2u * hx);
        f[1] = load_two(o.gN, k);
    }
    if (l > 0) {
        v[2] = load_two(z, k - g.plane);
        f[2] = load_two(o.gU, k - g.plane);
    }
    if ((int)l < g.nz - 1) {
        v[3] = load_two(z, k + g.plane);
        f[3] = load_two(o.gU, k);
    }
    CellZ<T, D>&u = a.c[0], &w = a.c[1];
    u.zc = zc.x, w.zc = zc.y;
    u.dg = first_of(dg), w.dg = second_of(dg);
    u.z[0] = e ? zo.x : zx;
    u.g[0] = e ? go.x : gx;
    u.z[1] = e ? zo.y : zo.x;
    u.g[1] = i0 < g.nx - 1 ? ge.x : 0.0f;
    w.z[0] = e ? zo.y : zo.x;
    w.g[0] = e ? go.y : go.x;
    w.z[1] = e ? zx : zo.y;
    w.g[1] = i1 < g.nx - 1 ? ge.y : 0.0f;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        u.z[2 + s] = v[s].x, w.z[2 + s] = v[s].y;
        u.g[2 + s] = f[s].x, w.g[2 + s] = f[s].y;
    }
    return true;
}

// beta, p.Ap and alpha of the iteration that the V-cycle's z begins, from r.z,
// z.Ap (Ap, pAp, rz of the iteration before) and z.Az: with p' = z + beta p,
// A p' = A z + beta Ap, so p'.Ap' = z.Az + 2 beta z.Ap + beta^2 p.Ap. Flexible
// beta (Polak-Ribiere): z_new.(r_new - r_old) / (z_old . r_old)
// = -(z_new . Ap) / (p . Ap); otherwise Fletcher-Reeves (src/pcg3d_cpu.cpp:179).
// False (a breakdown): a value is not finite, or p.Ap <= 0 (A is SPD).
struct Scalars {
    double beta, pAp, alpha;
};
__device__ __forceinline__ bool next_scalars(bool flex, bool first, double rz, double zAp, double zAz, double rz_old,
                                             double pAp_old, Scalars& s) {
    s.beta = first ? 0.0 : flex ? -zAp / pAp_old : rz / rz_old;
    s.pAp = first ? zAz : __fma_rn(s.beta, __fma_rn(s.beta, pAp_old, 2.0 * zAp), zAz);
    s.alpha = 0.0;
    if (!isfinite(rz) || !isfinite(s.beta) || !(s.pAp > 0.0) || !isfinite(s.pAp)) return false;
    s.alpha = rz / s.pAp;
    return true;
}

}  // namespace ct
