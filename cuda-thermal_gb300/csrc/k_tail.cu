// k_tail.cu - the coarse end of the single solver's FP32 V-cycle (every level
// from some level down to the single column) in ONE launch of a thread-block
// cluster, all of it in shared memory.
//
// What bounds these levels is latency: a level of 64 x 64 columns or fewer is
// nothing but launch, first loads and the serial recurrence. As launches of
// their own (four a level, 3.5-6 us each with everything in L2) and a one-block
// kernel below 16 x 16 columns (30 us) they were a quarter of an 800 x 800
// iteration and two thirds of a 200 x 200 one. Measured, us an iteration before
// and after: 64 x 64 x 10 81 -> 63, 237 x 181 x 13 147 -> 129, 501 x 333 x 10
// 208 -> 189, 800 x 800 x 10 439 -> 419, 1024 x 1024 x 16 977 -> 965.
//
// Layout. The finest levels here are split by rows over the CTAs of the
// cluster (`nd` distributed levels, coarse row J with the fine rows 2J and
// 2J + 1); the levels below (at most kTailBottomCells) are one CTA's, which takes
// no rows of the others where the cluster has a CTA to spare. A CTA keeps its
// rows of b, x, 1/pivot, gU, gE and gN, brought in by one tensor copy an array,
// with a halo row of x on each side and one of gN to the south. A
// sweep sends its boundary rows straight into the neighbours' halos (st.async,
// counted by an mbarrier of the receiver that only this sweep uses), so
// neighbours wait for each other's data and nothing else: 0.2 us, against 0.5
// us for stores and a cluster barrier and 1 us and an L2 round trip for a
// dependent launch.
//
// Each phase is one warp's chain of latencies, and index arithmetic and tests
// were most of it (a sweep of a 2 x 2 level: 280 cycles to find a column, 190
// to load it, 140 for its two recurrences, 180 to leave). So a table made at
// set-up gives each column, parent and coarse cell its offsets, a warp works on
// one plane, and clamped reads and zero weights take the place of tests. A sweep
// gathers the right-hand sides with one task per column and plane (into the
// column's own x slots; 32 consecutive slots a warp: no bank conflicts), then
// one thread per column runs the Thomas recurrence on registers. Arithmetic and
// order are the grid kernels' (k_mg.cu): same bits.
#include <algorithm>
#include <climits>
#include <cstring>

#include "kernels.h"
#include "reduce.cuh"
#include "tma.cuh"

namespace ct {

namespace {

constexpr int kTailWarps = 16;  // at most; a block has one warp a plane up to that

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The shared-memory address `a` of this CTA in CTA `rank` of the cluster.
__device__ __forceinline__ unsigned remote(unsigned a, unsigned rank) {
    unsigned o;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(a), "r"(rank));
    return o;
}
// Stores to another CTA's shared memory, counted by its mbarrier `bar`.
__device__ __forceinline__ void send(unsigned a, float v, unsigned bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(a), "f"(v), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void send4(unsigned a, float4 v, unsigned bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(a),
                 "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar)
                 : "memory");
}
// Bounded wait for what peers send (the first phase of `bar`).
__device__ __forceinline__ bool receive(uint64_t* bar, unsigned limit) {
    for (unsigned k = 0; k < limit; ++k) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(tma::smem_addr(bar))
            : "memory");
        if (ok) return true;
    }
    return false;
}

// The CTA's shared memory and, in it, the level descriptors.
__device__ __forceinline__ float* tail_smem() {
    extern __shared__ __align__(128) float tail_dynamic[];
    return tail_dynamic;
}
__device__ __forceinline__ const int* tail_ints() { return reinterpret_cast<const int*>(tail_smem()); }
__device__ __forceinline__ const TailLevel& tail_level(int k) {
    return reinterpret_cast<const TailLevel*>(tail_smem() + kTailDescriptors)[k];
}

// A CTA's place in the work.
struct Cta {
    int nz, tid, lane, rank, nd;
    int warp, warps;
    __device__ __forceinline__ int row0(int k) const { return k < nd ? rank * tail_level(k).rows : 0; }
};
// Where a sweep sends its boundary rows: the neighbours' shared memory and the
// mbarrier there.
struct Halo {
    unsigned south, north, south_bar, north_bar;
};

// Columns of a plane of one colour, the table's entry (column_entry): own slot,
// row, i & 1, i > 0, a column of the level.
constexpr int kOwnBits = 14, kRowBits = 8;
__device__ __forceinline__ int entry_own(int w) { return w & ((1 << kOwnBits) - 1); }
__device__ __forceinline__ int entry_row(int w) { return (w >> kOwnBits) & ((1 << kRowBits) - 1); }
__device__ __forceinline__ bool entry_bit(int w, int b) { return (w >> (kOwnBits + kRowBits + b)) & 1; }

// Right-hand sides (b plus the lateral sum: west, east, south, north, each
// neighbour with its parent's correction under PRO) of every plane of colour
// `color` into the columns' own x slots. xc, xcp: the coarse x's offset and
// plane stride. Slots that hold no column are computed with the others (every
// read stays inside) and not stored.
template <bool PRO>
__device__ __forceinline__ void tail_gather(const Cta& c, const TailLevel& L, int nr, int color, int xc, int xcp) {
    float* const sm = tail_smem();
    const int hx = L.hx, RS = 2 * hx, pl = L.rows * RS, ncol = L.ncol, gnh = L.gnh;
    const int dh = color ? -hx : hx;  // the same slot of the other colour's half-row
    const int* const tab = tail_ints() + L.tcol + (color ? ncol : 0);
    const int* const par = tail_ints() + L.tpar;
    for (int l = c.warp; l < c.nz; l += c.warps) {
        const int lp = l * pl, lx = L.x + lp + (2 * l + 1) * RS, lb = L.b + lp, le = L.ge + lp;
        const int ln = L.gn + lp + (l + 1) * gnh, lc = xc + l * xcp;
#pragma unroll 2
        for (int q0 = c.lane; q0 < ncol + c.lane; q0 += 32) {
            const int q = min(q0, ncol - 1), w = tab[q], own = entry_own(w), o = own + dh;
            const int e = entry_bit(w, 0) ? 1 : 0;
            float xw = sm[lx + o - 1 + e], xe = sm[lx + o + e], xs = sm[lx + o - RS], xn = sm[lx + o + RS];
            float gw = sm[le + o - 1 + e], gs = sm[ln + o - RS];
            const float gee = sm[le + own], gnn = sm[ln + own], bv = sm[lb + own];
            if (PRO) {
                // of the four neighbours' parents two are the column's own
                const int ph = par[2 * q], v = par[2 * q + 1];
                const float cp = sm[lc + (ph & 0xffff)], ch = sm[lc + (ph >> 16)], cv = sm[lc + v];
                xw = xw + (e ? cp : ch);
                xe = xe + (e ? ch : cp);
                xs = xs + (e ? cv : cp);
                xn = xn + (e ? cp : cv);
            }
            gw = entry_bit(w, 1) ? gw : 0.0f;
            gs = gnh || entry_row(w) > 0 ? gs : 0.0f;
            float s = __fmaf_rn(gw, xw, 0.0f);
            s = __fmaf_rn(gee, xe, s);
            s = __fmaf_rn(gs, xs, s);
            s = __fmaf_rn(gnn, xn, s);
            s = __fadd_rn(bv, s);
            if (q0 == q && entry_bit(w, 2) && entry_row(w) < nr) sm[lx + own] = s;
        }
    }
}

// The Thomas recurrences of colour `color` on the right-hand sides in b (ZERO:
// the sweep from x = 0) or in the columns' x slots, on registers: MZ planes at
// once, those past nz reading the last one (their values are not used), because
// a test of l < nz per plane costs more than the plane (10 planes, one warp: 664
// cycles with the tests, 865 in a rolled loop, 295 so). push: the boundary rows
// also go to the neighbours' halos.
template <int MZ, bool ZERO>
__device__ __forceinline__ void tail_recur(const Cta& c, const TailLevel& L, int nr, int color, const Halo& h,
                                           bool push, int bar) {
    float* const sm = tail_smem();
    const int hx = L.hx, RS = 2 * hx, rows = L.rows, ncol = L.ncol, pl = rows * RS, xpl = pl + 2 * RS, nz = c.nz;
    const int* const tab = tail_ints() + L.tcol + (color ? ncol : 0);
#pragma unroll 1
    for (int q = c.tid; q < ncol; q += 32 * c.warps) {
        const int w = tab[q], r = entry_row(w), own = entry_own(w);
        if (!entry_bit(w, 2) || r >= nr) continue;
        const float *const pf = sm + L.fi + own, *const pg = sm + L.gu + own;
        float* const px = sm + L.x + own + RS;
        const float* const pv = ZERO ? sm + L.b + own : px;
        const int sp = ZERO ? pl : xpl;
        float v[MZ], f[MZ], g[MZ];
#pragma unroll
        for (int l = 0; l < MZ; ++l) {
            const int lc = min(l, nz - 1);
            v[l] = pv[lc * sp];
            f[l] = pf[lc * pl];
            g[l] = pg[lc * pl];
        }
        float prev = 0.0f, below = 0.0f;
#pragma unroll
        for (int l = 0; l < MZ; ++l) {
            prev = __fmul_rn(__fmaf_rn(below, prev, v[l]), f[l]);
            v[l] = prev;
            below = g[l];
        }
#pragma unroll
        for (int l = MZ - 2; l >= 0; --l) {
            const float s = __fmaf_rn(__fmul_rn(g[l], f[l]), v[l + 1], v[l]);  // -fcp = gU finv, rounded once
            v[l] = l < nz - 1 ? s : v[l];
        }
#pragma unroll
        for (int l = 0; l < MZ; ++l)
            if (l < nz) px[l * xpl] = v[l];
        if (!push) continue;
        // row 0 to the south's north halo, the last row to the north's south halo
        if (r == 0 && h.south) {
            const unsigned a = h.south + 4u * (unsigned)(L.x + own + (rows + 1) * RS);
#pragma unroll
            for (int l = 0; l < MZ; ++l)
                if (l < nz) send(a + 4u * (unsigned)(l * xpl), v[l], h.south_bar + 8u * (unsigned)bar);
        }
        if (r == rows - 1 && h.north) {
            const unsigned a = h.north + 4u * (unsigned)(L.x + own - r * RS);
#pragma unroll
            for (int l = 0; l < MZ; ++l)
                if (l < nz) send(a + 4u * (unsigned)(l * xpl), v[l], h.north_bar + 8u * (unsigned)bar);
        }
    }
}

// Restriction of level k (mgdev::restrict_sum: the faces times the black
// neighbours' x at the two red children): one task per coarse cell and plane,
// consecutive cells on consecutive lanes. far: the coarse b lies in another CTA's shared memory (at `far`,
// counted by far_bar), by global rows.
__device__ __forceinline__ void tail_restrict(const Cta& c, const TailLevel& L, const TailLevel& C, int j0,
                                              unsigned far, unsigned far_bar) {
    float* const sm = tail_smem();
    const int hx = L.hx, RS = 2 * hx, rows = L.rows, pl = rows * RS, xpl = pl + 2 * RS, nz = c.nz, ncell = L.ncell;
    const int J0 = j0 >> 1, RC = 2 * C.hx, cpl = C.rows * RC, gnh = L.gnh;
    const int* const tab = tail_ints() + L.tcell;
    for (int l = c.warp; l < nz; l += c.warps) {
        const int lp = l * pl, lx = L.x + l * xpl + RS, le = L.ge + lp, ln = L.gn + lp + (l + 1) * gnh;
#pragma unroll 1
        for (int q0 = c.lane; q0 < ncell + c.lane; q0 += 32) {
            const int q = min(q0, ncell - 1), w = tab[2 * q], at = tab[2 * q + 1], rl = entry_row(w);
            const bool hi = entry_bit(w, 0), hw = entry_bit(w, 1), hj = 2 * (J0 + rl) + 1 < L.ny;
            // the children's slots: (2I, 2J) red, (2I + 1, 2J) black, and a row up;
            // a child row past the level's reads the row below (weight zero)
            const int c00 = entry_own(w), c10 = c00 + hx, R1 = 2 * rl + 1 < rows ? RS : 0;
            const int c01 = c10 + R1, c11 = c00 + R1;
            const bool hs = gnh || rl > 0, both = hi && hj;
            const float x10 = sm[lx + c10], x01 = sm[lx + c01], xw = sm[lx + c10 - 1], xs = sm[lx + c10 - RS];
            const float xe = sm[lx + c01 + 1], xn = sm[lx + c10 + 2 * R1];
            const float gw = sm[le + c10 - 1], ge = sm[le + c00], gs = sm[ln + c10 - RS], gn = sm[ln + c00];
            const float gw1 = sm[le + c01], ge1 = sm[le + c11], gs1 = sm[ln + c10], gn1 = sm[ln + c11];
            float v = __fmaf_rn(hw ? gw : 0.0f, xw, 0.0f);
            v = __fmaf_rn(hi ? ge : 0.0f, x10, v);
            v = __fmaf_rn(hs ? gs : 0.0f, xs, v);
            v = __fmaf_rn(hj ? gn : 0.0f, x01, v);
            float u = __fmaf_rn(both ? gw1 : 0.0f, x01, 0.0f);
            u = __fmaf_rn(both ? ge1 : 0.0f, xe, u);
            u = __fmaf_rn(both ? gs1 : 0.0f, x10, u);
            u = __fmaf_rn(both ? gn1 : 0.0f, xn, u);
            v = __fadd_rn(v, u);
            if (q0 == q && J0 + rl < C.ny) {
                const int b = C.b + l * cpl + at;
                if (far)
                    send(far + 4u * (unsigned)(b + J0 * RC), v, far_bar);
                else
                    sm[b] = v;
            }
        }
    }
}

// Columns of colour `color` in row j of a level of nx columns.
__device__ __forceinline__ int row_columns(int nx, int j, int color) { return (nx - ((j + color) & 1) + 1) >> 1; }

template <int MZ>
__global__ void __launch_bounds__(32 * (MZ < 4 ? 4 : MZ > kTailWarps ? kTailWarps : MZ), 1)
    k_tail(const __grid_constant__ TailPlan P, const __grid_constant__ TailMaps maps, const int* __restrict__ table,
           Ctl* ctl, Cond cond) {
    float* const sm = tail_smem();
    // the first sweep's factors and the tables; everything else of the operator;
    // the first level's b; the bottom's b (from the distributed levels); the
    // bottom's x (to them); and one a distributed level and sweep (red from
    // zero, black, black with the correction, red)
    __shared__ uint64_t bars[5 + 4 * kTailSpread];
    uint64_t *const bar0 = bars, *const bar1 = bars + 1, *const barb = bars + 2, *const bard = bars + 3,
                    *const baru = bars + 4, *const barh = bars + 5;
    const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = (int)blockDim.x >> 5;
    const int rank = (int)cluster_rank(), n = P.n, nd = P.nd, nz = P.nz;
    const bool dist = rank < P.dist, bottom = rank == P.bottom;
    const int k_lo = dist ? 0 : nd, k_hi = bottom ? n : nd;  // the levels held here
    for (int i = tid; i < 5 + 4 * nd; i += 32 * warps) tma::mbar_init(&bars[i], 1);
    tma::fence_barrier_init();
    __syncthreads();
    const unsigned base = tma::smem_addr(sm), bar_base = tma::smem_addr(barh);
    const unsigned far = remote(base, (unsigned)P.bottom), far_bar = remote(tma::smem_addr(bard), (unsigned)P.bottom);
    Halo halo{0u, 0u, 0u, 0u};
    if (dist && rank > 0) {
        halo.south = remote(base, (unsigned)rank - 1u);
        halo.south_bar = remote(bar_base, (unsigned)rank - 1u);
    }
    if (rank + 1 < P.dist) {
        halo.north = remote(base, (unsigned)rank + 1u);
        halo.north_bar = remote(bar_base, (unsigned)rank + 1u);
    }
    // The operator and factors do not change during a solve: their
    // copies are issued before the wait for the preceding kernel, those of the
    // first sweep on a barrier of their own; a level split by rows by tensor
    // copies (rows outside it come as zeros), a whole one by plain ones.
    if (tid == 0) {
        const unsigned b0 = (dist ? P.first_bytes : P.bottom_first_bytes) + (unsigned)P.table_bytes;
        const unsigned b1 = (dist ? P.dist_bytes : 0u) + (bottom ? P.bottom_bytes : 0u) + (unsigned)P.table_bytes - b0;
        tma::mbar_arrive_expect_tx(bar0, b0);
        tma::mbar_arrive_expect_tx(bar1, b1);
        tma::bulk_load(sm + P.tab, table, (unsigned)P.table_bytes, bar0);
    }
    __syncwarp();
    if (lane == 0)
        for (int a = warp; a < 4 * (k_hi - k_lo); a += warps) {
            const int kk = a >> 2, arr = a & 3, k = k_lo + kk;
            const TailLevel& L = P.L[k];
            const int dst = arr == 0 ? L.fi : arr == 1 ? L.gu : arr == 2 ? L.ge : L.gn;
            uint64_t* const bar = arr < 2 && k == k_lo ? bar0 : bar1;
            const int j0 = rank * L.rows;
            if (k < nd)
                tma::load_3d(sm + dst, &maps.m[k][arr], 0, arr == 3 ? j0 - 1 : j0, 0, bar);
            else
                tma::bulk_load(sm + dst, maps.whole[k][arr], (unsigned)(L.rows * 2 * L.hx * nz) * 4u, bar);
        }
    // what the peers will send: halo rows a sweep, the bottom's b and x
    if (warp == warps - 1 && nd > 0) {
        if (dist && lane < 4 * nd) {
            const int k = lane >> 2, color = (lane & 3) == 1 || (lane & 3) == 2 ? 1 : 0, j0 = rank * P.L[k].rows;
            int cols = 0;
            if (halo.south) cols += row_columns(P.L[k].nx, j0 - 1, color);
            if (halo.north) cols += row_columns(P.L[k].nx, j0 + P.L[k].rows, color);
            tma::mbar_arrive_expect_tx(&barh[lane], (unsigned)(cols * nz) * 4u);
        }
        if (lane == 0) {
            const TailLevel& B = P.L[nd];
            if (bottom) tma::mbar_arrive_expect_tx(bard, (unsigned)(B.nx * B.ny * nz) * 4u);
            const int r0 = max(rank * P.rd - 1, 0), r1 = min(rank * P.rd + P.rd, B.ny - 1);
            if (dist) tma::mbar_arrive_expect_tx(baru, (unsigned)((r1 - r0 + 1) * 2 * B.hx * nz) * 4u);
        }
    }
    // x starts at zero, halos and padding included (those are never written:
    // zeros beside the zero weights, and they go back out with x)
    for (int i = tid; i < P.x4; i += 32 * warps) reinterpret_cast<float4*>(sm + P.x)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    cluster_arrive();  // this CTA's shared memory may be written by its peers after this
    const bool first = k_lo == 0 && k_hi > 0;  // holds rows of the first level
    pdl_enter();
    pdl_trigger();  // the dependent's blocks load what this kernel does not write
    if (tid == 0 && first) {
        tma::mbar_arrive_expect_tx(barb, (unsigned)(P.L[0].rows * 2 * P.L[0].hx * nz) * 4u);
        tma::load_3d(sm + P.L[0].b, &maps.m[0][4], 0, nd > 0 ? rank * P.L[0].rows : 0, 0, barb);
    }
    const bool closed = loop_done(ctl, cond);  // the same in every thread of the cluster
    // A thread whose wait for the tables (the level descriptors come with them) runs
    // out does no work below: it would take offsets from what never landed. It keeps
    // to the barriers, whose number the parameters give.
    const bool landed = tma::mbar_wait(bar0, 0u, P.polls);
    bool ok = landed;
    if (landed && tid == 0 && nd > 0 && ((rank * P.rd) & 1)) {  // the coarse offsets for an odd first coarse row
        TailLevel& L = const_cast<TailLevel&>(tail_level(nd - 1));
        L.tpar += 2 * L.ncol;
        L.tcell += 2 * L.ncell;
    }
    Cta c;
    c.nz = landed ? nz : 0;
    c.tid = landed ? tid : INT_MAX;
    c.lane = lane;
    c.rank = rank;
    c.nd = nd;
    c.warp = warp;
    c.warps = warps;
    auto rows_of = [&](int k) { return k < nd ? min(tail_level(k).rows, tail_level(k).ny - c.row0(k)) : tail_level(k).ny; };
    ok = ok && (!first || tma::mbar_wait(barb, 0u, P.polls));
    cluster_wait();
    if (!closed) {
        // down: red from x = 0, black, restriction
#pragma unroll 1
        for (int k = k_lo; k < k_hi; ++k) {
            const bool spread = k < nd;
            const TailLevel& L = tail_level(k);
            const int j0 = c.row0(k), nr = rows_of(k);
            if (k == nd && nd > 0) ok = ok && receive(bard, P.polls);
            tail_recur<MZ, true>(c, L, nr, 0, halo, spread, 4 * k);
            if (k == k_lo) ok = ok && tma::mbar_wait(bar1, 0u, P.polls);
            if (k == n - 1) break;
            __syncthreads();
            if (spread) ok = ok && receive(&barh[4 * k], P.polls);
            tail_gather<false>(c, L, nr, 1, 0, 0);
            __syncthreads();
            tail_recur<MZ, false>(c, L, nr, 1, halo, spread, 4 * k + 1);
            __syncthreads();
            if (spread) ok = ok && receive(&barh[4 * k + 1], P.polls);
            tail_restrict(c, L, tail_level(k + 1), j0, k == nd - 1 ? far : 0u, far_bar);
            __syncthreads();
        }
        __syncthreads();
        // up: black with the coarse correction, red
#pragma unroll 1
        for (int k = min(k_hi, n - 1) - 1; k >= (dist ? 0 : max(nd - 1, 0)); --k) {
            const bool spread = k < nd;
            const TailLevel& L = tail_level(k);
            const TailLevel& N = tail_level(k + 1);
            const int nr = rows_of(k);
            int xc = N.x, xcp = (N.rows + 2) * 2 * N.hx;
            if (k == nd - 1) {
                // the bottom's finest x goes to each CTA, the rows of its parents:
                // a warp a plane, two lanes a CTA
                if (bottom) {
                    const int RC = 2 * N.hx, xdpl = (P.rd + 2) * RC, d = lane & 15;
                    const int j = d * P.rd - 1, r0 = max(j, 0), n4 = (min(j + P.rd + 1, N.ny - 1) - r0 + 1) * RC / 4;
                    if (d < P.dist) {
                        const unsigned to = remote(base, (unsigned)d) + 4u * (unsigned)(P.xd + (r0 - j) * RC);
                        const unsigned tb = remote(tma::smem_addr(baru), (unsigned)d);
                        for (int l = warp; l < c.nz; l += warps) {
                            const float4* const from = reinterpret_cast<const float4*>(sm + N.x + l * xcp + (r0 + 1) * RC);
#pragma unroll 4
                            for (int s = lane >> 4; s < n4; s += 2) send4(to + 4u * (unsigned)(l * xdpl) + 16u * (unsigned)s, from[s], tb);
                        }
                    }
                }
                if (!dist) break;
                ok = ok && receive(baru, P.polls);
                xc = P.xd;
                xcp = (P.rd + 2) * 2 * N.hx;
            }
            tail_gather<true>(c, L, nr, 1, xc, xcp);
            __syncthreads();
            tail_recur<MZ, false>(c, L, nr, 1, halo, spread, 4 * k + 2);
            __syncthreads();
            if (spread) ok = ok && receive(&barh[4 * k + 2], P.polls);
            tail_gather<false>(c, L, nr, 0, 0, 0);
            __syncthreads();
            tail_recur<MZ, false>(c, L, nr, 0, halo, spread && k > 0, 4 * k + 3);
            __syncthreads();
            if (spread && k > 0) ok = ok && receive(&barh[4 * k + 3], P.polls);
        }
    } else {
        ok = ok && tma::mbar_wait(bar1, 0u, P.polls);
    }
    cluster_arrive();  // no CTA leaves before its peers have sent what they send
    if (!closed && first) {  // the first level's x, whole rows (padding is zero)
        const TailLevel& F = tail_level(0);
        const int RS = 2 * F.hx, j0 = c.row0(0), row4 = (nd > 0 ? min(F.rows, F.ny - j0) : F.ny) * RS / 4;
        const float4* const x4 = reinterpret_cast<const float4*>(sm + F.x + RS);
        const int xpl4 = (F.rows + 2) * RS / 4;
        for (int l = warp; l < c.nz; l += warps)
            for (int i = lane; i < row4; i += 32)
                reinterpret_cast<float4*>(P.x0 + (size_t)l * P.plane + (size_t)j0 * RS)[i] = x4[l * xpl4 + i];
    }
    cluster_wait();
    if (__syncthreads_or(ok ? 0 : 1) && tid == 0) {
        // A bounded wait ran out: the phases ran on whatever was there (every
        // access stays in bounds: without the tables there are none). Record it and
        // stop the solve, only now that every CTA of the cluster has read the stop
        // flag. Before this CTA's shared memory goes, what is in flight to it lands:
        // its copies, and what its peers sent (all of them are past their sends).
        atomicExch(&ctl->err, 1);
        ctl->breakdown = 1;
        stop_loop(ctl, cond);
        const unsigned polls = P.polls / 64u + 1u;
        tma::mbar_wait(bar0, 0u, polls);
        tma::mbar_wait(bar1, 0u, polls);
        if (first) tma::mbar_wait(barb, 0u, polls);
        if (!closed && nd > 0) {
            if (bottom) receive(bard, polls);
            if (dist) {
                receive(baru, polls);
                for (int i = 0; i < 4 * nd; ++i)
                    if (i != 3) receive(&barh[i], polls);  // (the first level's last sweep sends nothing)
            }
        }
    }
}

}  // namespace

bool plan_tail(const LevelView<float>* views, int n, int ctas, bool apart, size_t smem_max, TailPlan* out) {
    if (n < 1 || n > kTailLevels || views[0].g.nz > 32) return false;
    const int nz = views[0].g.nz;
    int nd = 0;
    while (nd < n - 1 && views[nd].g.nx * views[nd].g.ny * nz > kTailBottomCells) ++nd;
    if (nd == 0) apart = false;
    if (nd > kTailSpread) return false;
    TailPlan p;
    std::memset(&p, 0, sizeof p);
    p.n = n;
    p.nd = nd;
    p.nz = nz;
    p.polls = tma::kWaitLimit;
    p.x0 = views[0].x;
    p.plane = views[0].g.plane;
    const int most = apart ? ctas - 1 : ctas;
    p.rd = nd > 0 ? (views[nd].g.ny + most - 1) / most : 0;
    for (int k = 0; k < n; ++k) {
        TailLevel& L = p.L[k];
        L.nx = views[k].g.nx;
        L.ny = views[k].g.ny;
        L.hx = views[k].g.hx;
        L.rows = k < nd ? p.rd << (nd - k) : L.ny;
        L.ncol = L.rows * L.hx;
        L.ncell = (L.rows + 1) / 2 * ((L.nx + 1) / 2);
        // a tensor copy's box takes at most 256 elements a side, a table's entry
        // 14 bits of offset and 8 of row
        if (2 * L.hx > 256 || L.rows + 1 > 255 || 2 * L.ncol >= (1 << kOwnBits)) return false;
    }
    p.dist = nd > 0 ? (p.L[0].ny + p.L[0].rows - 1) / p.L[0].rows : 0;
    p.bottom = apart ? p.dist : 0;
    p.ctas = std::max(1, p.dist + (apart ? 1 : 0));
    if (p.ctas > ctas) return false;
    // Shared memory, in floats: the descriptors and tables, then every x (zeroed
    // as one piece), then the rest. A bottom CTA of its own starts its levels
    // where the others start theirs.
    p.tab = kTailDescriptors;
    int ints = (int)sizeof(TailLevel) / 4 * n;
    for (int k = 0; k < n; ++k) {
        TailLevel& L = p.L[k];
        const int sets = k == nd - 1 && (p.rd & 1) ? 2 : 1;  // of the coarse offsets: even and odd first coarse rows
        L.tcol = p.tab + ints;
        ints += 2 * L.ncol;
        L.tpar = p.tab + ints;
        ints += sets * 2 * L.ncol;
        L.tcell = p.tab + ints;
        ints += sets * 2 * L.ncell;
    }
    p.table_bytes = (ints * 4 + 15) & ~15;
    const size_t start = p.tab + (((size_t)p.table_bytes / 4 + 31) & ~size_t(31));
    size_t at[2] = {start, start};  // the distributed levels' end, the bottom's
    auto take = [&](int which, size_t floats) {
        const size_t o = at[which];
        at[which] += (floats + 31) & ~size_t(31);
        return (int)o;
    };
    auto part = [&](int k) { return k < nd || !apart ? 0 : 1; };
    for (int k = 0; k < n; ++k) {
        TailLevel& L = p.L[k];
        L.x = take(part(k), (size_t)(L.rows + 2) * 2 * L.hx * nz);
    }
    if (nd > 0) p.xd = take(0, (size_t)(p.rd + 2) * 2 * p.L[nd].hx * nz);
    at[0] = at[1] = std::max(at[0], at[1]);
    p.x4 = (int)((at[0] - start) / 4);
    p.x = (int)start;
    for (int k = 0; k < n; ++k) {
        TailLevel& L = p.L[k];
        const int w = part(k);
        const size_t pl = (size_t)L.rows * 2 * L.hx * nz;
        L.b = take(w, pl);
        L.fi = take(w, pl);
        L.gu = take(w, pl);
        L.ge = take(w, pl);
        L.gnh = k < nd ? 2 * L.hx : 0;  // (a whole level has no row to its south)
        L.gn = take(w, pl + (size_t)L.gnh * nz);
    }
    for (int k = 0; k < n; ++k) {
        const TailLevel& L = p.L[k];
        const unsigned one = (unsigned)(L.rows * 2 * L.hx * nz) * 4u;
        (k < nd ? p.dist_bytes : p.bottom_bytes) += 4 * one + (unsigned)(L.gnh * nz) * 4u;
        if (k == 0) p.first_bytes = 2 * one;
        if (k == nd) p.bottom_first_bytes = 2 * one;
    }
    p.smem = (int)((std::max(at[0], at[1]) + 32) * 4);
    if ((std::max(at[0], at[1]) + 32) * 4 > smem_max) return false;
    *out = p;
    return true;
}

void fill_tail_table(const TailPlan& p, int* table) {
    std::memset(table, 0, (size_t)p.table_bytes);
    std::memcpy(table, p.L, sizeof(TailLevel) * (size_t)p.n);
    for (int k = 0; k < p.n; ++k) {
        const TailLevel& L = p.L[k];
        const int hx = L.hx, RS = 2 * hx;
        int* const col = table + (L.tcol - p.tab);
        for (int color = 0; color < 2; ++color)
            for (int q = 0; q < L.ncol; ++q) {
                const int r = q / hx, t = q - r * hx, e = (r + color) & 1, i = 2 * t + e;
                const int own = r * RS + (color ? hx : 0) + t;
                col[color * L.ncol + q] = own | r << kOwnBits | e << (kOwnBits + kRowBits) |
                                          (i > 0) << (kOwnBits + kRowBits + 1) | (i < L.nx) << (kOwnBits + kRowBits + 2);
            }
        if (k + 1 >= p.n) continue;
        const TailLevel& C = p.L[k + 1];
        const int hxc = C.hx, RC = 2 * hxc, cnx = C.nx;
        for (int set = 0; set < (k == p.nd - 1 && (p.rd & 1) ? 2 : 1); ++set) {
            // offset of coarse column (I, J), J counted from this CTA's first
            // coarse row, whose parity is `set`
            auto slot = [&](int I, int J, int row) { return row * RC + (((I + J + set) & 1) ? hxc : 0) + (I >> 1); };
            int* const par = table + (L.tpar - p.tab) + set * 2 * L.ncol;
            for (int q = 0; q < L.ncol; ++q) {  // black columns, rows of x with the halo row below
                const int r = q / hx, t = q - r * hx, e = (r + 1) & 1;
                const int I = std::min(t, cnx - 1), J = r >> 1, H = std::min(std::max(e ? t + 1 : t - 1, 0), cnx - 1);
                const int V = e ? J - 1 : J + 1;
                par[2 * q] = slot(I, J, J + 1) | slot(H, J, J + 1) << 16;
                par[2 * q + 1] = slot(I, V, V + 1);
            }
            int* const cell = table + (L.tcell - p.tab) + set * 2 * L.ncell;
            for (int q = 0; q < L.ncell; ++q) {
                const int rl = q / cnx, I = q - rl * cnx;
                cell[2 * q] = (2 * rl * RS + I) | rl << kOwnBits | (2 * I + 1 < L.nx) << (kOwnBits + kRowBits) |
                              (I > 0) << (kOwnBits + kRowBits + 1);
                cell[2 * q + 1] = slot(I, rl, rl);
            }
        }
    }
}

bool make_tail_maps(const TailPlan& p, const LevelView<float>* views, TailMaps* maps) {
    std::memset(maps, 0, sizeof *maps);
    for (int k = 0; k < p.n; ++k) {
        const LevelView<float>& v = views[k];
        const unsigned RS = 2u * (unsigned)v.g.hx, rows = (unsigned)p.L[k].rows, nz = (unsigned)p.nz;
        const float* src[5] = {v.finv, v.gU, v.gE, v.gN, v.b};
        for (int a = 0; a < 4; ++a) maps->whole[k][a] = src[a];
        if (k >= p.nd && k > 0) continue;  // (the first level's b is always a tensor copy)
        for (int a = 0; a < 5; ++a)
            if (!encode_tail_map(&maps->m[k][a], src[a], v.g, RS, a == 3 ? rows + 1u : rows, nz)) return false;
    }
    return true;
}

namespace {
// Calls f with the kernel for nz planes.
template <class F>
cudaError_t with_tail_kernel(int nz, F&& f) {
    if (nz <= 4) return f(k_tail<4>);
    if (nz <= 8) return f(k_tail<8>);
    if (nz <= 10) return f(k_tail<10>);
    if (nz <= 12) return f(k_tail<12>);
    if (nz <= 14) return f(k_tail<14>);
    if (nz <= 16) return f(k_tail<16>);
    if (nz <= 24) return f(k_tail<24>);
    return f(k_tail<32>);
}

template <class K>
cudaError_t tail_config(K kern, const TailPlan& p, cudaStream_t st, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at) {
    std::memset(cfg, 0, sizeof *cfg);
    cfg->gridDim = dim3((unsigned)p.ctas);
    cfg->blockDim = dim3(32u * (unsigned)std::min(std::max(p.nz, 4), kTailWarps));
    cfg->dynamicSmemBytes = (size_t)p.smem;
    cfg->stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)p.ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg->attrs = at;
    cfg->numAttrs = pdl_enabled() ? 2 : 1;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}
}  // namespace

bool tail_fits_device(const TailPlan& p) {
    int clusters = 0;
    const cudaError_t e = with_tail_kernel(p.nz, [&](auto kern) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[2];
        const cudaError_t r = tail_config(kern, p, nullptr, &cfg, at);
        cfg.numAttrs = 1;
        return r == cudaSuccess ? cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) : r;
    });
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess && clusters > 0;
}

cudaError_t launch_tail(cudaStream_t st, const TailPlan& p, const TailMaps& maps, const int* table, Ctl* ctl,
                        Cond cond) {
    return with_tail_kernel(p.nz, [&](auto kern) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[2];
        const cudaError_t r = tail_config(kern, p, st, &cfg, at);
        return r == cudaSuccess ? cudaLaunchKernelEx(&cfg, kern, p, maps, table, ctl, cond) : r;
    });
}

}  // namespace ct
