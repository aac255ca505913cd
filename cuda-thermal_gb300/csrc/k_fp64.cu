// k_fp64.cu - the FP64 outer PCG of the multigrid modes (CT_MG_FP32_FLEX,
// CT_MG_FP32, CT_MG_FP64): residual, A z with the dot products, the step of p,
// Ap and r, and the x update, all in IEEE double arithmetic as the reference's
// outer iteration is (Real = double, src/pcg3d.h:18-22; k_residual,
// k_apply, k_update_xr, k_mg_dot, k_update_p_mg, src/pcg3d_gpu.cu:159-256).
//
// On GB300 FP64 arithmetic is scarce: a DFMA issues at ~1/70 of the FFMA rate
// (0.53 T/s on 152 SMs), so at 800 x 800 x 10 every FP64 instruction per cell
// costs ~12 us while an 8-byte stream costs ~7.5 us at the measured copy
// bandwidth. So each kernel does the fewest FP64 instructions the algorithm
// needs, and few kernels touch each vector: the V-cycle's float faces and values
// are widened, and the residual narrowed to the V-cycle's float, with exact
// integer conversions (f64_dev.cuh) instead of the FP64-rate hardware
// conversions; the operator acts on the V-cycle's float z, whose products it
// adds up on the FP32 and integer pipes (sum6), in the same pass as the dot
// products (k_az64); and p, Ap and r follow in one more (k_step64). Per cell 4
// FP64 instructions each.
// The row kernels run one warp per row of one colour and plane (no index
// division per cell), the streaming kernels keep several items in flight per
// thread, and every kernel is launched with programmatic dependent launch.
#include <algorithm>
#include <cmath>

#include "f64_dev.cuh"
#include "kernels.h"
#include "reduce.cuh"

namespace ct {

using namespace f64dev;

namespace {

constexpr int kRowU = 2;  // cells a lane and step of the rows of A p

// w = (A + C/dt) z, r.z, z.Ap (the Ap of the iteration before), z.w; then beta,
// p.Ap and alpha. One warp per row of one colour and plane, a cell a lane; with
// the FP64 V-cycle, whose sums leave the integer pipe free, a thread takes two
// neighbouring slots with loads of two values (400 x 400 x 10: 42.7 us a launch
// against 53; the float form is no faster in pairs at 800 x 800 and 1 % of an
// iteration slower at 64 x 64 and 237 x 181, where half the threads wait twice as
// long).
//
// The operator acts on z, not on p: the V-cycle's z is a float, so its products
// with the float faces are exact in two floats and their sum runs on the FP32
// and integer pipes (sum6), where A p of the double p took seven DFMA a cell;
// p = z + beta p and Ap = w + beta Ap follow together in k_step64. Per cell 4
// FP64 instructions and 48 B (with the FP64 V-cycle 10 and 52), in place of the
// 8 of A p and 2 of the dots and 56 B, and no launch, grid
// reduction and second pass over r and Ap between them. 800 x 800 x 10:
// 82 us a launch (105 compiled for two cells a lane
// and the compiler's 101 registers, 94 / 82 / 87 for one cell at 2 / 5 / 6 blocks
// per SM against 4; the next cells' loads ahead of this one's arithmetic 84 to
// 98), against 107 + 37 for A p and the dots; the FP64 pipe is 62 % busy, memory
// 43 %, issue 64 %, each warp going from one to the other.
template <class T, bool FLEX>
__global__ void __launch_bounds__(NT, sizeof(T) == 8 ? 3 : 4)
    k_az64(OpView o, const double* __restrict__ diag, const T* __restrict__ z, const double* __restrict__ r,
           const double* __restrict__ Ap, double* __restrict__ w, Ctl* ctl, double* part, int maxb, Cond cond) {
    pdl_enter();
    if (loop_done(ctl, cond)) return;
    const bool first = ctl->iter == 0;  // no Ap yet
    double v[3] = {0.0, 0.0, 0.0};
    if constexpr (sizeof(T) == 8) {
        const unsigned n2 = o.g.plane * (unsigned)o.g.nz / 2u;
        for (unsigned q = blockIdx.x * NT + threadIdx.x; q < n2; q += gridDim.x * NT) {
            PairZ<T, double> a;
            if (!load_pair(o, diag, z, q, a)) continue;
            const double2 rv = load_two(r, a.k), av = first ? make_double2(0.0, 0.0) : load_two(Ap, a.k);
            dots64(v, a, rv, av, w);
        }
    } else {
        const unsigned rows = 2u * (unsigned)o.g.ny * (unsigned)o.g.nz;
        const int lane = (int)(threadIdx.x & 31u);
        struct More {
            double r, ap;
        };
        for (unsigned R = blockIdx.x * (NT / 32) + (threadIdx.x >> 5); R < rows; R += gridDim.x * (NT / 32))
            row_z(
                o, diag, z, R, lane, [&](unsigned k) { return More{r[k], first ? 0.0 : Ap[k]}; },
                [&](unsigned k, const More& m, const CellZ<T, double>& a) {
                    const double az = az64(a), zc = to_d(a.zc);
                    w[k] = az;
                    v[0] = __fma_rn(m.r, zc, v[0]);
                    v[1] = __fma_rn(zc, m.ap, v[1]);
                    v[2] = __fma_rn(zc, az, v[2]);
                });
    }
    pdl_trigger();
    if (publish_sums<3>(v, part, maxb, blockIdx.x, &ctl->ticket[SL_APPLY], gridDim.x)) {
        double t[3];
        gather_sums<3>(part, maxb, 0u, gridDim.x, &ctl->ticket[SL_APPLY], t);
        if (threadIdx.x == 0) {
            Scalars s;
            const bool ok = next_scalars(FLEX, first, t[0], t[1], t[2], ctl->rz, ctl->pAp, s);
            ctl->rz = t[0];
            ctl->zAp = t[1];
            ctl->beta = s.beta;
            ctl->pAp = s.pAp;
            ctl->alpha = s.alpha;
            if (!ok) {
                ctl->breakdown = 1;
                stop_loop(ctl, cond);
            }
        }
    }
}

// Ap = (A + C/dt) p, p.Ap and alpha = rz / p.Ap (the Jacobi form).
__global__ void __launch_bounds__(NT)
    k_apply64(OpView o, const double* __restrict__ diag, const double* __restrict__ p,
              double* __restrict__ Ap, Ctl* ctl, double* part, int maxb, Cond cond) {
    pdl_enter();
    if (loop_done(ctl, cond)) return;
    const Geo& g = o.g;
    const unsigned rows = 2u * (unsigned)g.ny * (unsigned)g.nz;
    const int lane = (int)(threadIdx.x & 31u);
    double pap = 0.0, unused = 0.0;
    for (unsigned R = blockIdx.x * (NT / 32) + (threadIdx.x >> 5); R < rows; R += gridDim.x * (NT / 32))
        row64<kRowU>(o, diag, p, R, lane, [&](unsigned k, bool valid, double av, double pc) {
            Ap[k] = av;
            if (valid) pap = __fma_rn(pc, av, pap);
        });
    pdl_trigger();
    block_sum2(pap, unused);
    if (publish2(pap, unused, part, maxb, &ctl->ticket[SL_APPLY])) {
        double PAP, U;
        gather2(part, maxb, &ctl->ticket[SL_APPLY], PAP, U);
        if (threadIdx.x == 0) {
            ctl->pAp = PAP;
            if (!(PAP > 0.0) || !isfinite(PAP)) {  // A is SPD: p.Ap > 0 unless p = 0
                ctl->breakdown = 1;
                ctl->alpha = 0.0;
                stop_loop(ctl, cond);
            } else {
                ctl->alpha = ctl->rz / PAP;
            }
        }
    }
}

// The start test of a solve from its residual sums (src/pcg3d_cpu.cpp:142-150).
__device__ __forceinline__ void start_test(Ctl* ctl, Cond cond, double RR, double BB) {
    ctl->rr = RR;
    ctl->bb = BB;
    if (BB == 0.0) {  // no heat in: x = 0 (src/pcg3d_cpu.cpp:146)
        ctl->bb_zero = 1;
        ctl->converged = 1;
        ctl->relres = 0.0;
        stop_loop(ctl, cond);
        return;
    }
    const double rel = sqrt(RR / BB);
    ctl->relres = rel;
    if (rel < ctl->tol) {
        ctl->converged = 1;
        stop_loop(ctl, cond);
    } else if (!isfinite(rel)) {
        ctl->breakdown = 1;
        stop_loop(ctl, cond);
    } else if (ctl->maxit <= 0) {
        stop_loop(ctl, cond);
    }
}

// ---- streaming kernels ---------------------------------------------------------

// Block b streams the contiguous items [begin, end), NT apart, in chunks of
// NT * U items.
struct Range {
    unsigned begin, end;
};
template <int U>
__device__ __forceinline__ Range block_range(unsigned n) {
    const unsigned per = ((n + gridDim.x - 1) / gridDim.x + NT * U - 1) / (NT * U) * (NT * U);
    const unsigned b = blockIdx.x * per;
    return Range{b + threadIdx.x, b + per < n ? b + per : n};
}

__device__ __forceinline__ void store_pair(float* b0, unsigned k, double a, double b) {
    reinterpret_cast<float2*>(b0)[k] = make_float2(narrow(a), narrow(b));
}
__device__ __forceinline__ void store_pair(double* b0, unsigned k, double a, double b) {
    reinterpret_cast<double2*>(b0)[k] = make_double2(a, b);
}

// r = b - (A + C/dt) x, b0 = r in the V-cycle precision, ||r||^2, ||b||^2 and
// the start test. A solve that starts from x = 0 (every steady solve) has
// r = b exactly and streams b once.
template <class T>
__global__ void __launch_bounds__(NT)
    k_residual64(OpView o, unsigned n, const double* __restrict__ diag, const double* __restrict__ b,
                 const double* __restrict__ x, double* __restrict__ r, T* __restrict__ b0, Ctl* ctl,
                 double* part, int maxb, Cond cond) {
    pdl_enter();
    const Geo& g = o.g;
    double rr = 0.0, bb = 0.0;
    if (ctl->x_zero) {
        // r = b, streamed in pairs with the next items' loads issued before
        // the current ones are stored (n is even: whole rows of both colours)
        const double2* b2 = reinterpret_cast<const double2*>(b);
        double2* r2 = reinterpret_cast<double2*>(r);
        stream_pipelined<2, double2>(
            blockIdx.x * NT + threadIdx.x, n / 2, gridDim.x * NT, [&](unsigned k) { return b2[k]; },
            [&](unsigned k, const double2& v) {
                r2[k] = v;
                store_pair(b0, k, v.x, v.y);
                bb = __fma_rn(v.x, v.x, bb);
                bb = __fma_rn(v.y, v.y, bb);
            });
        rr = bb;
    } else {
        const unsigned rows = 2u * (unsigned)g.ny * (unsigned)g.nz;
        const int lane = (int)(threadIdx.x & 31u);
        for (unsigned R = blockIdx.x * (NT / 32) + (threadIdx.x >> 5); R < rows;
             R += gridDim.x * (NT / 32))
            row64<kRowU>(o, diag, x, R, lane, [&](unsigned k, bool valid, double ax, double) {
                if (!valid) {
                    r[k] = 0.0;
                    b0[k] = T(0);
                    return;
                }
                const double bi = b[k];
                const double ri = bi - ax;
                r[k] = ri;
                b0[k] = from_d<T>(ri);
                rr = __fma_rn(ri, ri, rr);
                bb = __fma_rn(bi, bi, bb);
            });
    }
    block_sum2(rr, bb);
    if (publish2(rr, bb, part, maxb, &ctl->ticket[SL_INIT])) {
        double RR, BB;
        gather2(part, maxb, &ctl->ticket[SL_INIT], RR, BB);
        if (threadIdx.x == 0) start_test(ctl, cond, RR, BB);
    }
}

// p = z + beta p, Ap = w + beta Ap (p = z and Ap = w on the first iteration),
// r -= alpha Ap, b0 = r in the V-cycle precision, ||r||^2 and the convergence
// test (src/pcg3d_gpu.cu:218-256). Pairs of values (double2), each block a
// contiguous range.
// WX = false: x is left to k_update_x64 (x += alpha p off the critical path,
// beside the next V-cycle); alpha is kept in ctl->alpha_x for it. The x update
// that was pending at entry has run by then: none is pending when the loop has
// ended.
// 4 FP64 instructions and 64 B a cell. 800 x 800 x 10: 73 us (5.6 TB/s), against
// 22 + 37 for the p update and the update of r alone.
template <class T>
struct Pair;
template <>
struct Pair<float> {
    typedef float2 type;
};
template <>
struct Pair<double> {
    typedef double2 type;
};
__device__ __forceinline__ double2 to_d(float2 v) { return make_double2(widen(v.x), widen(v.y)); }
__device__ __forceinline__ double2 to_d(double2 v) { return v; }

constexpr int kStepU = 2;
template <class T, bool WX>
__global__ void __launch_bounds__(NT)
    k_step64(unsigned n2, const T* __restrict__ z, const double2* __restrict__ w, double2* __restrict__ p,
             double2* __restrict__ Ap, double2* __restrict__ x, double2* __restrict__ r, T* __restrict__ b0, Ctl* ctl,
             double* part, int maxb, Cond cond) {
    typedef typename Pair<T>::type Z2;
    pdl_enter();
    const bool done = loop_done(ctl, cond);
    const double alpha = ctl->alpha, malpha = -alpha, beta = ctl->beta;
    if (!WX && blockIdx.x == 0 && threadIdx.x == 0) ctl->alpha_x = done ? 0.0 : alpha;
    if (done) return;
    const bool first = ctl->iter == 0;
    const Z2* const z2 = reinterpret_cast<const Z2*>(z);
    double v[1] = {0.0};
    const Range br = block_range<kStepU>(n2);
    struct Item {
        Z2 z;
        double2 w, p, a, r;
    };
    stream_pipelined<kStepU, Item>(
        br.begin, br.end, NT,
        [&](unsigned k) {
            const double2 none = make_double2(0.0, 0.0);
            return Item{z2[k], w[k], first ? none : p[k], first ? none : Ap[k], r[k]};
        },
        [&](unsigned k, Item it) {
            const double2 zd = to_d(it.z);
            it.p.x = __fma_rn(beta, it.p.x, zd.x);
            it.p.y = __fma_rn(beta, it.p.y, zd.y);
            it.a.x = __fma_rn(beta, it.a.x, it.w.x);
            it.a.y = __fma_rn(beta, it.a.y, it.w.y);
            it.r.x = __fma_rn(malpha, it.a.x, it.r.x);
            it.r.y = __fma_rn(malpha, it.a.y, it.r.y);
            p[k] = it.p;
            Ap[k] = it.a;
            r[k] = it.r;
            store_pair(b0, k, it.r.x, it.r.y);
            if (WX) {
                const double2 xv = x[k];
                x[k] = make_double2(__fma_rn(alpha, it.p.x, xv.x), __fma_rn(alpha, it.p.y, xv.y));
            }
            v[0] = __fma_rn(it.r.x, it.r.x, v[0]);
            v[0] = __fma_rn(it.r.y, it.r.y, v[0]);
        });
    pdl_trigger();
    if (publish_sums<1>(v, part, maxb, blockIdx.x, &ctl->ticket[SL_UPDATE], gridDim.x)) {
        double t[1];
        gather_sums<1>(part, maxb, 0u, gridDim.x, &ctl->ticket[SL_UPDATE], t);
        if (threadIdx.x == 0) {
            ctl->rr = t[0];
            ctl->iter += 1;
            const double rel = sqrt(t[0] / ctl->bb);
            ctl->relres = rel;
            if (rel < ctl->tol) {
                ctl->converged = 1;
                stop_loop(ctl, cond);
            } else if (!isfinite(rel)) {
                ctl->breakdown = 1;
                stop_loop(ctl, cond);
            } else if (ctl->iter >= ctl->maxit) {
                stop_loop(ctl, cond);
            }
        }
    }
}

// x += alpha p with the alpha k_step64<T, false> left in ctl->alpha_x (0:
// nothing pending), the same rounding as the fused update. It runs beside the
// V-cycle of the next iteration (or after the loop for the last one) and
// before that iteration's k_step64, which writes the next p and alpha_x.
struct XItem {
    double2 p, x;
};
__global__ void __launch_bounds__(NT)
    k_update_x64(unsigned n2, const double2* __restrict__ p, double2* __restrict__ x, const Ctl* ctl) {
    const double alpha = *(volatile const double*)&ctl->alpha_x;
    if (alpha == 0.0) return;
    stream_pipelined<4, XItem>(
        blockIdx.x * NT + threadIdx.x, n2, gridDim.x * NT, [&](unsigned k) { return XItem{p[k], x[k]}; },
        [&](unsigned k, const XItem& it) {
            x[k] = make_double2(__fma_rn(alpha, it.p.x, it.x.x), __fma_rn(alpha, it.p.y, it.x.y));
        });
}

// ---- self-test of the integer conversions -----------------------------------

__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}

// Item q tests widen() on a float bit pattern and narrow() on a double bit
// pattern against the hardware conversions; the first 2^18 items sweep every
// float exponent and every double exponent near the float range (with
// mantissas at, just below and just above the rounding tie), the rest are
// hashed. NaN results compare by NaN-ness.
__global__ void k_conv_selftest(unsigned long long n, unsigned long long seed,
                                unsigned long long* mismatches) {
    unsigned long long bad = 0;
    for (unsigned long long q = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; q < n;
         q += (unsigned long long)gridDim.x * blockDim.x) {
        const unsigned long long h = mix64(q ^ seed);
        unsigned fb;
        unsigned long long db;
        if (q < (1ull << 18)) {
            const unsigned sel = (unsigned)(q & 15u), ex = (unsigned)(q >> 4) & 0x7ffu;
            fb = ((unsigned)(h >> 32) & 0x807fffffu) | ((ex & 0xffu) << 23);
            const unsigned long long tie = 1ull << 28, low = (h & 0xffffffe0000000ull);
            const unsigned long long tail = sel < 4 ? tie : sel < 8 ? tie - 1 : sel < 12 ? tie + 1 : (h & 0x1fffffffull);
            db = (h & 0x8000000000000000ull) | ((unsigned long long)ex << 52) | (low & 0xfffffe0000000ull) | tail;
        } else {
            fb = (unsigned)h;
            db = mix64(h);
        }
        const float f = __uint_as_float(fb);
        const double wd = widen(f), hd = (double)f;
        const bool wok = (isnan(hd) && isnan(wd)) || __double_as_longlong(wd) == __double_as_longlong(hd);
        const double d = __longlong_as_double((long long)db);
        const float nf = narrow(d), hf = (float)d;
        const bool nok = (isnan(hf) && isnan(nf)) || __float_as_uint(nf) == __float_as_uint(hf);
        bad += (wok ? 0u : 1u) + (nok ? 0u : 1u);
    }
    if (bad) atomicAdd(mismatches, bad);
}

// FP64-pipe peak probe: kDfmaChains independent DFMA chains per thread, kDfmaSteps
// steps each (no memory traffic but one store per thread).
constexpr int kDfmaChains = 8, kDfmaSteps = 2048;
__global__ void k_dfma_probe(double a, double* out) {
    double v[kDfmaChains];
#pragma unroll
    for (int c = 0; c < kDfmaChains; ++c) v[c] = threadIdx.x * 1e-3 + c;
    for (int k = 0; k < kDfmaSteps; ++k)
#pragma unroll
        for (int c = 0; c < kDfmaChains; ++c) v[c] = __fma_rn(v[c], a, 1e-9);
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < kDfmaChains; ++c) s += v[c];
    out[blockIdx.x * (size_t)blockDim.x + threadIdx.x] = s;
}

}  // namespace

// ---- launchers ------------------------------------------------------------------

void launch_apply64(cudaStream_t st, const OpView& o, const double* diag, const double* p,
                    double* Ap, Ctl* ctl, const Red& red, Cond cond) {
    static const int wb = wave_blocks(k_apply64, 1 << 30);
    launch_pdl(k_apply64, std::min(red.maxb, wb), NT, 0, st, o, diag, p, Ap, ctl, red.part, red.maxb, cond);
}

void launch_az64(cudaStream_t st, MgType mt, bool flexible, const OpView& o, const double* diag, const void* z,
                 const double* r, const double* Ap, double* w, Ctl* ctl, const Red& red, Cond cond) {
    const int rows = 2 * o.g.ny * o.g.nz;
    const int want = mt == MG_F64 ? (int)((o.g.plane * (unsigned)o.g.nz / 2u + NT - 1) / NT)
                                  : std::max(1, (rows + NT / 32 - 1) / (NT / 32));
    auto go = [&](auto kern, int wb, auto* zt) {
        launch_pdl(kern, std::min(std::min(red.maxb, wb), want), NT, 0, st, o, diag, zt, r, Ap, w, ctl, red.part,
                   red.maxb, cond);
    };
    if (mt == MG_F64) {
        static const int wb = wave_blocks(k_az64<double, false>, 1 << 30);
        go(k_az64<double, false>, wb, (const double*)z);
    } else if (flexible) {
        static const int wb = wave_blocks(k_az64<float, true>, 1 << 30);
        go(k_az64<float, true>, wb, (const float*)z);
    } else {
        static const int wb = wave_blocks(k_az64<float, false>, 1 << 30);
        go(k_az64<float, false>, wb, (const float*)z);
    }
}

void launch_residual64(cudaStream_t st, MgType mt, const OpView& o, unsigned n, const double* diag,
                       const double* b, const double* x, double* r, void* b0, Ctl* ctl, const Red& red,
                       Cond cond) {
    if (mt == MG_F64) {
        static const int wb = wave_blocks(k_residual64<double>, 1 << 30);
        launch_pdl(k_residual64<double>, std::min(red.maxb, wb), NT, 0, st, o, n, diag, b, x, r, (double*)b0,
                   ctl, red.part, red.maxb, cond);
    } else {
        static const int wb = wave_blocks(k_residual64<float>, 1 << 30);
        launch_pdl(k_residual64<float>, std::min(red.maxb, wb), NT, 0, st, o, n, diag, b, x, r, (float*)b0,
                   ctl, red.part, red.maxb, cond);
    }
}

void launch_step64(cudaStream_t st, MgType mt, unsigned n, const void* z, const double* w, double* p, double* Ap,
                   double* x, double* r, void* b0, Ctl* ctl, const Red& red, Cond cond, bool write_x) {
    const unsigned n2 = n / 2;
    auto d2 = [](auto* q) { return reinterpret_cast<double2*>(q); };
    // (wave_blocks once per kernel: the four have their own occupancies)
    auto go = [&](auto kern, int wb, auto* zt, auto* b) {
        launch_pdl(kern, std::min(red.blocks, wb), NT, 0, st, n2, zt, reinterpret_cast<const double2*>(w), d2(p), d2(Ap),
                   d2(x), d2(r), b, ctl, red.part, red.maxb, cond);
    };
    if (mt == MG_F64) {
        static const int wb1 = wave_blocks(k_step64<double, true>, 1 << 30);
        static const int wb0 = wave_blocks(k_step64<double, false>, 1 << 30);
        if (write_x) go(k_step64<double, true>, wb1, (const double*)z, (double*)b0);
        else go(k_step64<double, false>, wb0, (const double*)z, (double*)b0);
    } else {
        static const int wb1 = wave_blocks(k_step64<float, true>, 1 << 30);
        static const int wb0 = wave_blocks(k_step64<float, false>, 1 << 30);
        if (write_x) go(k_step64<float, true>, wb1, (const float*)z, (float*)b0);
        else go(k_step64<float, false>, wb0, (const float*)z, (float*)b0);
    }
}

void launch_update_x(cudaStream_t st, unsigned n, const double* p, double* x, const Ctl* ctl, int blocks) {
    static const int wb = wave_blocks(k_update_x64, 1 << 30);
    const unsigned n2 = n / 2;
    unsigned want = std::max(1u, (n2 + NT * 4 - 1) / (NT * 4));
    if (blocks > 0) want = std::min(want, (unsigned)blocks);
    k_update_x64<<<(int)std::min(want, (unsigned)wb), NT, 0, st>>>(n2, reinterpret_cast<const double2*>(p),
                                                                    reinterpret_cast<double2*>(x), ctl);
}

cudaError_t measure_dfma_rate(double* per_s) {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    const int blocks = std::max(1, sms) * 8;
    double* out = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    e = cudaMalloc(&out, (size_t)blocks * NT * sizeof(double));
    if (e == cudaSuccess) e = cudaEventCreate(&e0);
    if (e == cudaSuccess) e = cudaEventCreate(&e1);
    float ms = 0.0f;
    constexpr int kReps = 5;
    if (e == cudaSuccess) {
        for (int w = 0; w < 2; ++w) k_dfma_probe<<<blocks, NT>>>(0.999999, out);
        cudaEventRecord(e0);
        for (int r = 0; r < kReps; ++r) k_dfma_probe<<<blocks, NT>>>(0.999999, out);
        cudaEventRecord(e1);
        e = cudaEventSynchronize(e1);
        if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (out) cudaFree(out);
    if (e == cudaSuccess)
        *per_s = (double)blocks * NT * kDfmaChains * kDfmaSteps * kReps / (ms * 1e-3);
    return e;
}

cudaError_t launch_conv_selftest(cudaStream_t st, unsigned long long n, unsigned long long seed,
                                 unsigned long long* mismatches) {
    k_conv_selftest<<<1024, NT, 0, st>>>(n, seed, mismatches);
    return cudaGetLastError();
}

}  // namespace ct
