// mg_dev.cuh - device code of the multigrid V-cycle shared by the single
// solver (k_mg.cu) and the batched solver (k_batch.cu): neighbour maps of the
// colour-split layout, the column line solve (mg_line_solve,
// src/mg3d.h:67-84), the fine residual and restriction
// (src/pcg3d_cpu.cpp:87-100), and the shared-memory bottom of the V-cycle.
#pragma once
#include "f64_dev.cuh"
#include "kernels.h"
#include "tma.cuh"

namespace ct {
namespace mgdev {

// Neighbour slots of an active column, and (for fused prolongation) the
// coarse slots of those neighbours' parents.
struct Nbr {
    unsigned s, sw, se, ss, sn;
    unsigned pw, pe, ps, pn;
    bool w, e, so, no;
};

template <bool PRO>
__device__ __forceinline__ Nbr neighbours(const Geo& g, const Geo& cg, int i, int j, int t,
                                          int color) {
    Nbr n;
    const int oc = color ^ 1;
    const unsigned row_o = (unsigned)(2 * j + oc) * (unsigned)g.hx;
    n.s = (unsigned)(2 * j + color) * (unsigned)g.hx + (unsigned)t;
    n.w = i > 0;
    n.e = i < g.nx - 1;
    n.so = j > 0;
    n.no = j < g.ny - 1;
    n.sw = row_o + (unsigned)((i - 1) >> 1);
    n.se = row_o + (unsigned)((i + 1) >> 1);
    n.ss = (unsigned)(2 * j - 2 + oc) * (unsigned)g.hx + (unsigned)t;
    n.sn = (unsigned)(2 * j + 2 + oc) * (unsigned)g.hx + (unsigned)t;
    if (PRO) {
        n.pw = n.w ? scol(cg, (i - 1) >> 1, j >> 1) : 0u;
        n.pe = n.e ? scol(cg, (i + 1) >> 1, j >> 1) : 0u;
        n.ps = n.so ? scol(cg, i >> 1, (j - 1) >> 1) : 0u;
        n.pn = n.no ? scol(cg, i >> 1, (j + 1) >> 1) : 0u;
    }
    return n;
}

// A face conductance in the V-cycle's precision (FP64: widened by integer
// operations, f64_dev.cuh; the hardware conversion issues at the FP64 rate).
template <class T>
__device__ __forceinline__ T face(float f);
template <>
__device__ __forceinline__ float face<float>(float f) {
    return f;
}
template <>
__device__ __forceinline__ double face<double>(float f) {
    return f64dev::widen(f);
}

// The Thomas factor fcp of a cell from its up face and 1/pivot, rounded as
// factor_column rounds it: -gU * finv, one rounding.
__device__ __forceinline__ float fcp_of(float gu, float fi) { return __fmul_rn(-gu, fi); }
__device__ __forceinline__ double fcp_of(float gu, double fi) { return __dmul_rn(-f64dev::widen(gu), fi); }

// Lateral neighbour sum of op_lat_sum (src/operator3d.h:62-78) at plane l:
// west, east, south, north; with PRO each neighbour value carries its
// parent's coarse correction.
template <class T, bool PRO>
__device__ __forceinline__ T lat_sum(const LevelView<T>& L, const LevelView<T>& C, const Nbr& n,
                                     int l) {
    const unsigned base = (unsigned)l * L.g.plane;
    const unsigned cbase = PRO ? (unsigned)l * C.g.plane : 0u;
    T s = 0;
    if (n.w) {
        T xv = L.x[base + n.sw];
        if (PRO) xv = xv + C.x[cbase + n.pw];
        s += face<T>(L.gE[base + n.sw]) * xv;
    }
    if (n.e) {
        T xv = L.x[base + n.se];
        if (PRO) xv = xv + C.x[cbase + n.pe];
        s += face<T>(L.gE[base + n.s]) * xv;
    }
    if (n.so) {
        T xv = L.x[base + n.ss];
        if (PRO) xv = xv + C.x[cbase + n.ps];
        s += face<T>(L.gN[base + n.ss]) * xv;
    }
    if (n.no) {
        T xv = L.x[base + n.sn];
        if (PRO) xv = xv + C.x[cbase + n.pn];
        s += face<T>(L.gN[base + n.s]) * xv;
    }
    return s;
}

// Right-hand side of plane l of a column, branch-free (for levels in shared
// memory, where load latency bounds a sweep): b plus the lateral sum in op_lat_sum's order (west, east, south, north),
// each neighbour value with its parent's coarse correction under PRO; an
// absent neighbour reads the column itself with weight 0.
template <class T, bool PRO>
__device__ __forceinline__ T bf_rhs(const LevelView<T>& L, const LevelView<T>& C, const Nbr& n, unsigned l) {
    const Geo& g = L.g;
    const unsigned base = l * g.plane, id = base + n.s;
    const T rhs = L.b[id];
    const unsigned sw = n.w ? n.sw : n.s, se = n.e ? n.se : n.s;
    const unsigned ss = n.so ? n.ss : n.s, sn = n.no ? n.sn : n.s;
    T xw = L.x[base + sw], xe = L.x[base + se];
    T xs = L.x[base + ss], xn = L.x[base + sn];
    if (PRO) {
        const T* cx = C.x + l * C.g.plane;
        xw = xw + cx[n.pw];
        xe = xe + cx[n.pe];
        xs = xs + cx[n.ps];
        xn = xn + cx[n.pn];
    }
    const float ew = L.gE[base + sw], ee = L.gE[id], ns = L.gN[base + ss], nn = L.gN[id];
    T sum = 0;
    sum += (n.w ? face<T>(ew) : T(0)) * xw;
    sum += (n.e ? face<T>(ee) : T(0)) * xe;
    sum += (n.so ? face<T>(ns) : T(0)) * xs;
    sum += (n.no ? face<T>(nn) : T(0)) * xn;
    return rhs + sum;
}

// The Thomas recurrence of sweep_column on the column at slot s whose
// right-hand sides are src[l * plane + s] (nz <= MZ): every operand loaded
// first, the recurrence on registers, x written once.
template <class T, int MZ>
__device__ __forceinline__ void column_solve(const LevelView<T>& L, const T* src, unsigned s) {
    const Geo& g = L.g;
    T v[MZ], fi[MZ], fc[MZ];
    float gu[MZ];
#pragma unroll
    for (int l = 0; l < MZ; ++l) {
        if (l < g.nz) {
            const unsigned id = (unsigned)l * g.plane + s;
            v[l] = src[id];
            fi[l] = L.finv[id];
            fc[l] = L.fcp[id];
            gu[l] = L.gU[id];
        }
    }
    T prev = 0;
#pragma unroll
    for (int l = 0; l < MZ; ++l) {
        if (l < g.nz) {
            const T lower = l > 0 ? -face<T>(gu[l - 1]) : T(0);
            prev = (v[l] - lower * prev) * fi[l];
            v[l] = prev;
        }
    }
#pragma unroll
    for (int l = MZ - 2; l >= 0; --l)
        if (l < g.nz - 1) v[l] -= fc[l] * v[l + 1];
#pragma unroll
    for (int l = 0; l < MZ; ++l)
        if (l < g.nz) L.x[(unsigned)l * g.plane + s] = v[l];
}

// Line solve of the q-th column of colour `color` (mg_line_solve,
// src/mg3d.h:67-84). With MZ > 0 (nz <= MZ) the column stays in registers:
// every plane's right-hand side (b plus the lateral sum) is gathered first,
// all loads independent of one another, then the Thomas recurrence runs on
// registers and x is written once. MZ = 0 is the general path for deep
// columns, with forward values going through x as in the reference.
template <class T, int MZ, bool ZERO, bool PRO>
__device__ __forceinline__ void sweep_column(const LevelView<T>& L, const LevelView<T>& C,
                                             int color, unsigned q) {
    const Geo& g = L.g;
    const int j = (int)(q / (unsigned)g.hx), t = (int)(q - (unsigned)j * g.hx);
    const int i = 2 * t + ((j + color) & 1);
    if (i >= g.nx) return;
    const Nbr n = neighbours<PRO>(g, C.g, i, j, t, color);
    if constexpr (MZ > 0) {
        // Gather: every operand of every plane, all loads independent, so the
        // whole column costs about one memory latency.
        T v[MZ], fi[MZ], fc[MZ];
        float gu[MZ];
#pragma unroll
        for (int l = 0; l < MZ; ++l) {
            if (l < g.nz) {
                const unsigned id = (unsigned)l * g.plane + n.s;
                T rhs = L.b[id];
                if (!ZERO) rhs = rhs + lat_sum<T, PRO>(L, C, n, l);
                v[l] = rhs;
                fi[l] = L.finv[id];
                gu[l] = L.gU[id];
                // the x = 0 sweep recomputes fcp as factor_column rounded it
                // (one operand stream less)
                if (ZERO)
                    fc[l] = fcp_of(gu[l], fi[l]);
                else
                    fc[l] = L.fcp[id];
            }
        }
        // Thomas recurrence on registers.
        T prev = 0;
#pragma unroll
        for (int l = 0; l < MZ; ++l) {
            if (l < g.nz) {
                const T lower = l > 0 ? -face<T>(gu[l - 1]) : T(0);
                prev = (v[l] - lower * prev) * fi[l];
                v[l] = prev;
            }
        }
#pragma unroll
        for (int l = MZ - 2; l >= 0; --l)
            if (l < g.nz - 1) v[l] -= fc[l] * v[l + 1];
#pragma unroll
        for (int l = 0; l < MZ; ++l)
            if (l < g.nz) L.x[(unsigned)l * g.plane + n.s] = v[l];
    } else {
        T prev = 0;
        float gu_b = 0.0f;
        for (int l = 0; l < g.nz; ++l) {
            const unsigned id = (unsigned)l * g.plane + n.s;
            T rhs = L.b[id];
            if (!ZERO) rhs = rhs + lat_sum<T, PRO>(L, C, n, l);
            const T lower = l > 0 ? -face<T>(gu_b) : T(0);
            prev = (rhs - lower * prev) * L.finv[id];
            L.x[id] = prev;
            gu_b = L.gU[id];
        }
        for (int l = g.nz - 2; l >= 0; --l) {
            const unsigned id = (unsigned)l * g.plane + n.s;
            prev = L.x[id] - L.fcp[id] * prev;
            L.x[id] = prev;
        }
    }
}

// ---- sweep with one thread per column and plane ---------------------------------
//
// Small levels (L2-resident, latency-bound): a block is 32 columns of the active
// colour x nz planes (at most MZ). Each thread gathers its plane's right-hand side
// (b plus the lateral sum, the same operations as sweep_column) and the column's
// factors into shared memory; after one block barrier, one thread per column runs
// sweep_column's recurrence there, and after a second the block writes x plane by
// plane. Same operations in the same order as sweep_column, so the same bits, but a
// thread issues one plane's loads instead of nz planes' (a thread a column: 6.5-7.8
// us per launch on the 100 x 100 to 25 x 25 levels of an 800 x 800 stack). Slots
// q < end; enter() waits for the preceding kernel and begins the test that closed()
// ends once the gathers are issued: false if it says there is nothing to solve.
template <class T, int MZ>
struct SplitShared {
    T v[MZ][32], fi[MZ][32], fc[MZ][32];
    float gu[MZ][32];
};
template <class T, int MZ, bool ZERO, bool PRO, class Enter, class Closed>
__device__ __forceinline__ bool split_columns(const LevelView<T>& L, const LevelView<T>& C, int color, unsigned q,
                                              unsigned end, SplitShared<T, MZ>& S, Enter enter, Closed closed) {
    const Geo& g = L.g;
    const unsigned tx = threadIdx.x;
    const int l = (int)threadIdx.y;
    const int j = (int)(q / (unsigned)g.hx), t = (int)(q - (unsigned)j * g.hx);
    const int i = 2 * t + ((j + color) & 1);
    const bool on = q < end && i < g.nx && l < g.nz;
    const Nbr n = neighbours<PRO>(g, C.g, i, j, t, color);
    const unsigned s = n.s, base = (unsigned)l * g.plane, id = base + s;
    T rhs = 0, fi = 0, fc = 0;
    float gu = 0.0f, gw = 0.0f, ge = 0.0f, gs = 0.0f, gn = 0.0f;
    // before the wait for the preceding kernel (kernels.h): the operator and the
    // factors, which no kernel of the loop writes
    if (on) {
        fi = L.finv[id];
        gu = L.gU[id];
        if (!ZERO) {
            fc = L.fcp[id];
            if (n.w) gw = L.gE[base + n.sw];
            ge = L.gE[id];
            if (n.so) gs = L.gN[base + n.ss];
            gn = L.gN[id];
        }
    }
    const auto flags = enter();
    if (on) {
        rhs = L.b[id];
        if (!ZERO) {
            T xw = 0, xe = 0, xs = 0, xn = 0;
            if (n.w) xw = L.x[base + n.sw];
            if (n.e) xe = L.x[base + n.se];
            if (n.so) xs = L.x[base + n.ss];
            if (n.no) xn = L.x[base + n.sn];
            if (PRO) {
                const T* const cx = C.x + (unsigned)l * C.g.plane;
                if (n.w) xw = xw + cx[n.pw];
                if (n.e) xe = xe + cx[n.pe];
                if (n.so) xs = xs + cx[n.ps];
                if (n.no) xn = xn + cx[n.pn];
            }
            T sum = 0;  // lat_sum's order
            if (n.w) sum += face<T>(gw) * xw;
            if (n.e) sum += face<T>(ge) * xe;
            if (n.so) sum += face<T>(gs) * xs;
            if (n.no) sum += face<T>(gn) * xn;
            rhs = rhs + sum;
        } else {
            fc = fcp_of(gu, fi);  // as factor_column rounded it (one operand stream less)
        }
    }
    if (closed(flags)) return false;  // the same for every thread of the block
    if (on) {
        S.v[l][tx] = rhs;
        S.fi[l][tx] = fi;
        S.fc[l][tx] = fc;
        S.gu[l][tx] = gu;
    }
    __syncthreads();
    const int nz = g.nz;
    if (on && l == 0) {
        // the recurrence of sweep_column, on shared memory; FP32 up to 16 planes
        // on registers, all MZ planes without a test (the ones past nz hold
        // nothing and reach nothing): one warp runs it while the block waits, so
        // its instruction count is the kernel's time. 237 x 181 x 10: an
        // iteration of 105.2 us against 109.4 with the loop over shared memory;
        // 501 x 333 x 10: 167.1 against 169.8
        if constexpr (sizeof(T) == 4 && MZ <= 16) {
            T v[MZ], c[MZ], prev = 0, lower = 0;
#pragma unroll
            for (int k = 0; k < MZ; ++k) {
                prev = (S.v[k][tx] - lower * prev) * S.fi[k][tx];
                v[k] = prev;
                c[k] = S.fc[k][tx];
                lower = -S.gu[k][tx];
            }
#pragma unroll
            for (int k = MZ - 2; k >= 0; --k) {
                const T n = v[k] - c[k] * v[k + 1];
                v[k] = k < nz - 1 ? n : v[k];
            }
#pragma unroll
            for (int k = 0; k < MZ; ++k)
                if (k < nz) S.v[k][tx] = v[k];
        } else {
            T prev = 0;
#pragma unroll 4
            for (int k = 0; k < nz; ++k) {
                const T lower = k > 0 ? -face<T>(S.gu[k - 1][tx]) : T(0);
                prev = (S.v[k][tx] - lower * prev) * S.fi[k][tx];
                S.v[k][tx] = prev;
            }
#pragma unroll 4
            for (int k = nz - 2; k >= 0; --k) {
                prev = S.v[k][tx] - S.fc[k][tx] * prev;
                S.v[k][tx] = prev;
            }
        }
    }
    __syncthreads();
    if (on) L.x[(unsigned)l * g.plane + s] = S.v[l][tx];
    return true;
}

// The two red children's terms of restrict_sum from operands already loaded: west,
// east, south, north of (2I, 2J), then of (2I + 1, 2J + 1).
template <class T>
__device__ __forceinline__ T red_residuals(bool w, bool e, bool so, bool no, bool both, bool e2, bool n2, float gw,
                                           float ge, float gs, float gn, float hw, float he, float hs, float hn, T xw,
                                           T x10, T xs, T x01, T xe, T xn) {
    T sum = 0, two = 0;
    sum += (w ? face<T>(gw) : T(0)) * xw;
    sum += (e ? face<T>(ge) : T(0)) * x10;
    sum += (so ? face<T>(gs) : T(0)) * xs;
    sum += (no ? face<T>(gn) : T(0)) * x01;
    two += (both ? face<T>(hw) : T(0)) * x01;
    two += (e2 ? face<T>(he) : T(0)) * xe;
    two += (both ? face<T>(hs) : T(0)) * x10;
    two += (n2 ? face<T>(hn) : T(0)) * xn;
    return sum + two;
}

// The faces of restrict_sum at coarse cell (I, J, l) and where they and the black
// x beside them lie (an absent neighbour reads a cell beside it).
struct RedFaces {
    float gw, ge, gs, gn, hw, he, hs, hn;
};
struct RedSlots {
    bool w, e, so, no, both, e2, n2;
    unsigned c00, c10, c01, c11, a_w, a_s, a_e, a_n;
};
__device__ __forceinline__ RedSlots red_slots(const Geo& g, int I, int J, int l) {
    RedSlots r;
    const int i0 = 2 * I, j0 = 2 * J;
    r.w = i0 > 0, r.e = i0 + 1 < g.nx, r.so = j0 > 0, r.no = j0 + 1 < g.ny;
    r.both = r.e && r.no, r.e2 = r.both && i0 + 2 < g.nx, r.n2 = r.both && j0 + 2 < g.ny;
    const unsigned hx = (unsigned)g.hx;
    // red (2I, 2J), black (2I + 1, 2J); black (2I, 2J + 1), red (2I + 1, 2J + 1)
    r.c00 = (unsigned)l * g.plane + 4u * (unsigned)J * hx + (unsigned)I;
    r.c10 = r.c00 + hx;
    r.c11 = r.no ? r.c00 + 2u * hx : r.c00;
    r.c01 = r.no ? r.c10 + 2u * hx : r.c10;
    r.a_w = r.w ? r.c10 - 1u : r.c10;
    r.a_s = r.so ? r.c10 - 2u * hx : r.c10;
    r.a_e = r.e2 ? r.c01 + 1u : r.c01;
    r.a_n = r.n2 ? r.c10 + 4u * hx : r.c10;
    return r;
}
template <class T>
__device__ __forceinline__ RedFaces red_faces(const LevelView<T>& F, int I, int J, int l) {
    const RedSlots r = red_slots(F.g, I, J, l);
    return RedFaces{F.gE[r.a_w], F.gE[r.c00], F.gN[r.a_s], F.gN[r.c00], F.gE[r.c01], F.gE[r.c11], F.gN[r.c10], F.gN[r.c11]};
}

// Restriction (src/pcg3d_cpu.cpp:87-100) of coarse cell (I, J, l): the sum over
// its (up to 4) children of the fine residual b - (A + C/dt) x, x being the
// iterate of the V-cycle's way down: the red columns solved from x = 0, then the
// black ones. A black column was solved with the red x it still has: its residual
// is zero. A red column was solved with zeros beside it: of its residual the
// lateral terms of the black x that came since are left. So the residual is the
// faces times the black neighbours' x at the two red children, (2I, 2J) and
// (2I + 1, 2J + 1): 10 bytes a fine cell in FP32 where b, x, the diagonal and
// every face are 24, and no difference of large terms (the vertical ones are up to
// 1e4 of the lateral).
// The residual of all four children on all operands took 35.5 us at 800 x 800 x 10
// (23.0 so) and, in FP64, 47 at 400 x 400 x 10 (13.1); an iteration 382 -> 359 and
// 388 -> 318.
template <class T>
__device__ __forceinline__ T restrict_sum(const LevelView<T>& F, const RedFaces& f, int I, int J, int l) {
    const RedSlots r = red_slots(F.g, I, J, l);
    const T x10 = F.x[r.c10], x01 = F.x[r.c01], xw = F.x[r.a_w], xs = F.x[r.a_s];
    const T xe = F.x[r.a_e], xn = F.x[r.a_n];
    return red_residuals<T>(r.w, r.e, r.so, r.no, r.both, r.e2, r.n2, f.gw, f.ge, f.gs, f.gn, f.hw, f.he, f.hs, f.hn, xw,
                            x10, xs, x01, xe, xn);
}

// W coarse cells (I .. I + W - 1, J) of plane l at once, I a multiple of W: their
// operands lie side by side, so a load brings W of them, and a black column's x
// and faces serve the cells on both its sides.
template <class T, int W>
struct alignas(W * sizeof(T)) Lane {
    T v[W];
};
template <int W>
struct WideFaces {
    Lane<float, W> ge, gb, hw, he, gs, gn, hs, hn;
    float gw;
};
// Where the rows lie: red and black of row 2J, red and black of row 2J + 1, the
// black rows to the south and north (an absent one reads a row beside it).
struct WideRows {
    bool so, no, nn;
    unsigned c00, c10, c11, c01, a_s, a_n;
};
__device__ __forceinline__ WideRows wide_rows(const Geo& g, int I, int J, int l) {
    WideRows r;
    const int j0 = 2 * J;
    const unsigned hx = (unsigned)g.hx;
    r.so = j0 > 0, r.no = j0 + 1 < g.ny, r.nn = j0 + 2 < g.ny;
    r.c00 = (unsigned)l * g.plane + 4u * (unsigned)J * hx + (unsigned)I;
    r.c10 = r.c00 + hx;
    r.c11 = r.no ? r.c00 + 2u * hx : r.c00;
    r.c01 = r.no ? r.c10 + 2u * hx : r.c10;
    r.a_s = r.so ? r.c10 - 2u * hx : r.c10;
    r.a_n = r.nn ? r.c10 + 4u * hx : r.c10;
    return r;
}
template <class T, int W>
__device__ __forceinline__ WideFaces<W> wide_faces(const LevelView<T>& F, int I, int J, int l) {
    const WideRows r = wide_rows(F.g, I, J, l);
    auto at = [&](const float* f, unsigned k) { return *reinterpret_cast<const Lane<float, W>*>(f + k); };
    return WideFaces<W>{at(F.gE, r.c00), at(F.gE, r.c10), at(F.gE, r.c01), at(F.gE, r.c11), at(F.gN, r.a_s),
                        at(F.gN, r.c00), at(F.gN, r.c10), at(F.gN, r.c11), I > 0 ? F.gE[r.c10 - 1u] : 0.0f};
}
template <class T, int W>
__device__ __forceinline__ void restrict_wide(const LevelView<T>& F, const WideFaces<W>& f, int I, int J, int l,
                                              T (&s)[W]) {
    const Geo& g = F.g;
    const int i0 = 2 * I;
    const WideRows r = wide_rows(g, I, J, l);
    auto at = [&](unsigned k) { return *reinterpret_cast<const Lane<T, W>*>(F.x + k); };
    const Lane<T, W> x10 = at(r.c10), x01 = at(r.c01), xs = at(r.a_s), xn = at(r.a_n);
    const bool w0 = I > 0, e0 = i0 + 2 * W < g.nx;  // a column beyond the first and the last cell
    const T xw = w0 ? F.x[r.c10 - 1u] : T(0), xe = r.no && e0 ? F.x[r.c01 + (unsigned)W] : T(0);
#pragma unroll
    for (int c = 0; c < W; ++c) {
        const int b = c > 0 ? c - 1 : 0, d = c + 1 < W ? c + 1 : c;
        const bool e = i0 + 2 * c + 1 < g.nx, both = e && r.no;
        const bool e2 = both && i0 + 2 * c + 2 < g.nx, n2 = both && r.nn;
        s[c] = red_residuals<T>(c > 0 || w0, e, r.so, r.no, both, e2, n2, c > 0 ? f.gb.v[b] : f.gw, f.ge.v[c], f.gs.v[c],
                                f.gn.v[c], f.hw.v[c], f.he.v[c], f.hs.v[c], f.hn.v[c], c > 0 ? x10.v[b] : xw, x10.v[c],
                                xs.v[c], x01.v[c], c + 1 < W ? x01.v[d] : xe, xn.v[c]);
    }
}
// The sums stored as coarse b (cells past the row's end left alone).
template <class T, int W>
__device__ __forceinline__ void store_wide(const LevelView<T>& C, int I, int J, int l, const T (&s)[W]) {
    const Geo& cg = C.g;
    T* const row = C.b + (unsigned)l * cg.plane + 2u * (unsigned)J * (unsigned)cg.hx + (unsigned)(I >> 1);
#pragma unroll
    for (int c = 0; c < W; ++c)
        if (I + c < cg.nx) row[(((c + J) & 1) ? cg.hx : 0) + (c >> 1)] = s[c];
}

// Coarse cell q = J cnx + I, stored as coarse b.
template <class T>
__device__ __forceinline__ void restrict_cell(const LevelView<T>& F, const LevelView<T>& C, unsigned q,
                                              int l) {
    const Geo& cg = C.g;
    const int J = (int)(q / (unsigned)cg.nx), I = (int)(q - (unsigned)J * cg.nx);
    C.b[(unsigned)l * cg.plane + scol(cg, I, J)] = restrict_sum<T>(F, red_faces(F, I, J, l), I, J, l);
}


// Writes the right-hand side (bf_rhs) of every plane of every column of
// colour `color` into that column's x slots; tasks are (plane, column) pairs
// strided over the nth threads of the block.
template <class T, bool PRO>
__device__ __forceinline__ void gather_rhs(const LevelView<T>& L, const LevelView<T>& C, int color, unsigned tid,
                                           unsigned nth) {
    const Geo& g = L.g;
    const unsigned ncol = (unsigned)g.ny * (unsigned)g.hx;
    const unsigned work = ncol * (unsigned)g.nz;
    for (unsigned w = tid; w < work; w += nth) {
        const unsigned l = w / ncol, q = w - l * ncol;
        const int j = (int)(q / (unsigned)g.hx), t = (int)(q - (unsigned)j * g.hx);
        const int i = 2 * t + ((j + color) & 1);
        if (i >= g.nx) continue;
        const Nbr n = neighbours<PRO>(g, C.g, i, j, t, color);
        L.x[l * g.plane + n.s] = bf_rhs<T, PRO>(L, C, n, l);
    }
}

// Level views of the shared-memory bottom: a level's arrays lie at base in
// the order gE, gN, gU, fcp, finv, x, b, each rounded up to 16 bytes
// (small_level_bytes adds the same sizes). The views are rebuilt from the
// block's base and a byte offset wherever they are used, never stored as
// pointers, so every pointer visibly points into shared memory and the
// compiler issues shared-memory loads through them rather than generic ones.
template <class T>
__device__ __forceinline__ LevelView<T> small_view(unsigned char* base, const Geo& g) {
    const unsigned ln = g.plane * (unsigned)g.nz;
    unsigned char* p = base;
    auto take = [&](unsigned bytes) {
        unsigned char* r = p;
        p += small_round16(bytes);
        return r;
    };
    LevelView<T> S;
    S.g = g;
    S.gE = (const float*)take(ln * 4u);
    S.gN = (const float*)take(ln * 4u);
    S.gU = (const float*)take(ln * 4u);
    S.fcp = (T*)take(ln * (unsigned)sizeof(T));
    S.finv = (T*)take(ln * (unsigned)sizeof(T));
    S.x = (T*)take(ln * (unsigned)sizeof(T));
    S.b = (T*)take(ln * (unsigned)sizeof(T));
    return S;
}

// The bottom of the V-cycle (levels k0 .. single column) in ONE block, with
// every one of those levels held in shared memory: operator and factors of
// every level and level k0's b come in by bulk copies (all in flight at once),
// x and the coarser b start at zero, the phases run with block barriers, and
// level k0's x goes back out for the prolongation above it. Same line-solve
// and restriction code as the grid-wide kernels, pointed at shared memory.
//
// The operator and factors do not change during a solve, so their copies are
// issued (one per lane of the first warp) before wait() (every thread calls
// it: it waits for the preceding kernel); level k0's b, the preceding
// kernel's output, is copied after it, and go() (called after that copy is
// issued, so the two latencies overlap) says whether to run the phases at
// all. Returns kSmallDone, kSmallClosed (go() said no: nothing written once
// the copies have landed) or kSmallTimeout (a bounded wait for the copies ran
// out: nothing written). Any block size.
constexpr int kSmallDone = 0, kSmallTimeout = 1, kSmallClosed = 2;

template <class T, int MZ, class Wait, class Go>
__device__ __forceinline__ int vsmall_body(const TailLevels<T>& tl, unsigned char* smem, Wait wait, Go go) {
    __shared__ Geo sg[kMaxTail];      // level geometry
    __shared__ unsigned soff[kMaxTail];  // byte offset of each level in smem
    __shared__ uint64_t bar, barb;    // operator and factors; level k0's b
    const int nl = tl.n;
    if (threadIdx.x == 0) {
        unsigned off = 0, total = 0;
        for (int k = 0; k < nl; ++k) {
            const Geo g = tl.L[k].g;
            sg[k] = g;
            soff[k] = off;
            off += (unsigned)small_level_bytes(g, sizeof(T));
            const unsigned ln = g.plane * (unsigned)g.nz;
            total += 3u * ln * 4u + 2u * ln * (unsigned)sizeof(T);
        }
        tma::mbar_init(&bar, 1);
        tma::mbar_init(&barb, 1);
        tma::fence_barrier_init();
        tma::mbar_arrive_expect_tx(&bar, total);
    }
    __syncthreads();
    if (threadIdx.x < 32u) {
        // copy c of level k = c / 5: gE, gN, gU, fcp, finv
        for (int c = (int)threadIdx.x; c < 5 * nl; c += 32) {
            const int k = c / 5, a = c - 5 * k;
            const LevelView<T>& G = tl.L[k];
            const LevelView<T> S = small_view<T>(smem + soff[k], sg[k]);
            const unsigned ln = sg[k].plane * (unsigned)sg[k].nz;
            const unsigned fb = ln * 4u, tb = ln * (unsigned)sizeof(T);
            if (a == 0) tma::bulk_load((void*)S.gE, G.gE, fb, &bar);
            else if (a == 1) tma::bulk_load((void*)S.gN, G.gN, fb, &bar);
            else if (a == 2) tma::bulk_load((void*)S.gU, G.gU, fb, &bar);
            else if (a == 3) tma::bulk_load(S.fcp, G.fcp, tb, &bar);
            else tma::bulk_load(S.finv, G.finv, tb, &bar);
        }
    }
    // Padding slots are never written by the phases below but go back out
    // with level k0's x: start every slot at zero, as the global arrays'
    // padding is, so no stale shared-memory value (possibly a NaN) reaches
    // the outer iteration.
    for (int k = 0; k < nl; ++k) {
        const LevelView<T> S = small_view<T>(smem + soff[k], sg[k]);
        const unsigned ln = sg[k].plane * (unsigned)sg[k].nz;
        for (unsigned i = threadIdx.x; i < ln; i += blockDim.x) {
            S.x[i] = T(0);
            if (k > 0) S.b[i] = T(0);
        }
    }
    wait();
    if (threadIdx.x == 0) {
        const unsigned bytes = sg[0].plane * (unsigned)sg[0].nz * (unsigned)sizeof(T);
        tma::mbar_arrive_expect_tx(&barb, bytes);
        tma::bulk_load(small_view<T>(smem, sg[0]).b, tl.L[0].b, bytes, &barb);
    }
    if (!__syncthreads_and(go() ? 1 : 0)) {
        if (threadIdx.x == 0) {  // let the copies land before leaving
            tma::mbar_wait(&bar, 0u);
            tma::mbar_wait(&barb, 0u);
        }
        return kSmallClosed;
    }
    const bool got = tma::mbar_wait(&bar, 0u) && tma::mbar_wait(&barb, 0u);
    if (!__syncthreads_and(got)) {
        if (threadIdx.x == 0) {  // let the copies land before leaving
            tma::mbar_wait(&bar, 0u);
            tma::mbar_wait(&barb, 0u);
        }
        return kSmallTimeout;
    }
    const unsigned tid = threadIdx.x, nth = blockDim.x;
    const int last = nl - 1;
    // The phases in V-cycle order, driven by one loop so that each kind of
    // phase (x = 0 sweep, sweep, restriction, prolongating sweep) is one
    // code region, warm in the instruction cache after its first use: down
    // the levels k < last (red x = 0 sweep, black sweep, restriction), the
    // single column (x = 0 sweep), back up (black sweep with the coarse
    // correction, red sweep).
    const int nph = 3 * last + 1 + 2 * last;
    for (int ph = 0; ph < nph; ++ph) {
        int k, kind;  // kind: 0 x = 0 sweep, 1 sweep, 2 restriction, 3 prolongating sweep
        int color = 0;
        if (ph < 3 * last) {
            k = ph / 3;
            kind = ph - 3 * k;
            color = kind == 1 ? 1 : 0;
        } else if (ph == 3 * last) {
            k = last;
            kind = 0;
        } else {
            const int u = ph - 3 * last - 1;
            k = last - 1 - u / 2;
            kind = (u & 1) ? 1 : 3;
            color = (u & 1) ? 0 : 1;
        }
        const LevelView<T> L = small_view<T>(smem + soff[k], sg[k]);
        const unsigned ncol = (unsigned)L.g.ny * (unsigned)L.g.hx;
        if (kind == 2) {
            const LevelView<T> C = small_view<T>(smem + soff[k + 1], sg[k + 1]);
            const unsigned ccols = (unsigned)C.g.nx * (unsigned)C.g.ny;
            const unsigned work = ccols * (unsigned)C.g.nz;
            for (unsigned w = tid; w < work; w += nth) {
                const int l = (int)(w / ccols);
                restrict_cell<T>(L, C, w - (unsigned)l * ccols, l);
            }
        } else if constexpr (MZ > 0) {
            // A sweep in two steps: one task per column and plane gathers
            // that plane's right-hand side into the column's own x slot (the
            // sweep reads only the other colour's x, so no task reads a slot
            // another one writes), then one thread per column runs the
            // recurrence. Same operations as sweep_column, with the gathers
            // spread over the block instead of one thread walking the planes.
            if (kind == 1)
                gather_rhs<T, false>(L, L, color, tid, nth);
            else if (kind == 3)
                gather_rhs<T, true>(L, small_view<T>(smem + soff[k + 1], sg[k + 1]), color, tid, nth);
            if (kind != 0) __syncthreads();
            const T* src = kind == 0 ? L.b : L.x;
            for (unsigned q = tid; q < ncol; q += nth) {
                const int j = (int)(q / (unsigned)L.g.hx), t = (int)(q - (unsigned)j * L.g.hx);
                if (2 * t + ((j + color) & 1) < L.g.nx)
                    column_solve<T, MZ>(L, src, (unsigned)(2 * j + color) * (unsigned)L.g.hx + (unsigned)t);
            }
        } else if (kind == 0) {  // deep columns (MZ = 0): x goes through memory
            for (unsigned q = tid; q < ncol; q += nth) sweep_column<T, MZ, true, false>(L, L, 0, q);
        } else if (kind == 1) {
            for (unsigned q = tid; q < ncol; q += nth) sweep_column<T, MZ, false, false>(L, L, color, q);
        } else {
            const LevelView<T> C = small_view<T>(smem + soff[k + 1], sg[k + 1]);
            for (unsigned q = tid; q < ncol; q += nth) sweep_column<T, MZ, false, true>(L, C, 1, q);
        }
        __syncthreads();
    }
    pdl_trigger();
    const LevelView<T> S0 = small_view<T>(smem, sg[0]);
    const unsigned ln0 = S0.g.plane * (unsigned)S0.g.nz;
    T* out = tl.L[0].x;
    for (unsigned i = tid; i < ln0; i += nth) out[i] = S0.x[i];
    return kSmallDone;
}


}  // namespace mgdev
}  // namespace ct
