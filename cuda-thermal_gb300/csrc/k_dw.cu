// k_dw.cu - the outer PCG on the FP32 pipes: double-word (float-pair)
// arithmetic for CT_MG_FP32_FLEX_DW.
//
// On GB300 an FP64 instruction issues at ~1/70 of the FP32 rate (and float <->
// double conversions at the FP64 rate), so the FP64 outer kernels of the
// reference's algorithm are bound by the FP64 pipe, not by HBM. Here x, r, p,
// Ap and the diagonal are stored as float pairs (hi, lo) - the same 8 bytes
// per value as a double - and combined with error-free transformations
// (TwoSum, Fast2Sum, FMA-based TwoProd; Joldes, Muller and Popescu, "Tight
// and rigorous error bounds for basic building blocks of double-word
// arithmetic", 2017), which carry ~48 significant bits. Dot products are
// accumulated in double words per thread, per block and over the grid (on the
// FP32 pipe; only the grid's total is converted); alpha and beta stay FP64
// scalars on the device.
//
// Two limits of 48 bits, and how they are lifted:
//  - the recurrence residual drifts from the true residual by ~2^-48 times the
//    operator's cancellation (up to ~1e4 here). So the solve recomputes
//    r = b - A x once in FP64 (k_residual_x, "residual replacement") when the
//    recurrence first passes a threshold (1e-5 by default);
//  - a 48-bit x cannot hold T (~50 K) finely enough for ||P - A T|| / ||P|| to
//    reach 1e-10 where lateral conductances are large (the copper spreader).
//    So x is an FP64 base xb plus a double-word correction xw: the iteration
//    updates xw, and k_fold adds xw into xb (in FP64) before every FP64
//    residual - at the start and at the replacement - after which xw only
//    carries the small remaining correction.
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "dw_dev.cuh"
#include "f64_dev.cuh"
#include "kernels.h"
#include "reduce.cuh"

namespace ct {

using namespace dwdev;
using namespace f64dev;

namespace {

// ---- FP64 residual from a double-word x: start and replacement -------------

// r = b - (A + C/dt) x in FP64 from the folded base x, the stored FP64 diagonal;
// stores r as a double word and b0 = r (float, the V-cycle's input). `start`:
// the first residual of a solve (sets ||b||^2 and the start test); otherwise
// the residual replacement (phase 2 begins, or the solve ends if already
// converged). One warp per row of one colour of one plane, as k_residual64, with
// integer conversions: 640 x 640 x 10 from an x that is not zero 145 us, where a
// thread per column with the hardware's conversions took 222.
__global__ void __launch_bounds__(NT, 4)
    k_residual_x(OpView o, unsigned n, const double* __restrict__ diag, const double* __restrict__ b,
                 const double* __restrict__ x, float2* __restrict__ r, float* __restrict__ b0,
                 int start, Ctl* ctl, double* part, int maxb, Cond cond) {
    pdl_enter();
    // the pending x update went into the base before this residual
    if (!start && blockIdx.x == 0 && threadIdx.x == 0) ctl->alpha_xw = make_float2(0.0f, 0.0f);
    if (!start && *(volatile const int*)&ctl->done) {  // converged or stopped in phase 1
        if (cond.use && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(cond.h, 0u);
        return;
    }
    const Geo& g = o.g;
    double rr = 0.0, bb = 0.0;
    // A solve that starts from x = 0 (every steady solve) has r = b exactly.
    const bool zero = start && ctl->x_zero;
    if (zero) {
        const double2* b2 = reinterpret_cast<const double2*>(b);
        float4* r2 = reinterpret_cast<float4*>(r);
        float2* b02 = reinterpret_cast<float2*>(b0);
        stream_pipelined<2, double2>(
            blockIdx.x * NT + threadIdx.x, n / 2, gridDim.x * NT, [&](unsigned k) { return b2[k]; },
            [&](unsigned k, const double2& v) {
                const float2 u = split(v.x), w = split(v.y);
                r2[k] = make_float4(u.x, u.y, w.x, w.y);
                b02[k] = make_float2(u.x, w.x);
                bb = __fma_rn(v.x, v.x, bb);
                bb = __fma_rn(v.y, v.y, bb);
            });
    } else {
        const unsigned rows = 2u * (unsigned)g.ny * (unsigned)g.nz;
        const int lane = (int)(threadIdx.x & 31u);
        for (unsigned R = blockIdx.x * (NT / 32) + (threadIdx.x >> 5); R < rows; R += gridDim.x * (NT / 32))
            row64<1>(o, diag, x, R, lane, [&](unsigned k, bool valid, double ax, double) {
                if (!valid) {
                    r[k] = make_float2(0.0f, 0.0f);
                    b0[k] = 0.0f;
                    return;
                }
                const double bi = b[k], ri = bi - ax;
                const float2 rw = split(ri);
                r[k] = rw;
                b0[k] = rw.x;
                rr = __fma_rn(ri, ri, rr);
                bb = __fma_rn(bi, bi, bb);
            });
    }
    if (zero) rr = bb;
    block_sum2(rr, bb);
    if (publish2(rr, bb, part, maxb, &ctl->ticket[SL_INIT])) {
        double RR, BB;
        gather2(part, maxb, &ctl->ticket[SL_INIT], RR, BB);
        if (threadIdx.x == 0) {
            ctl->rr = RR;
            if (start) {
                ctl->bb = BB;
                if (BB == 0.0) {
                    ctl->bb_zero = 1;
                    ctl->converged = 1;
                    ctl->relres = 0.0;
                    stop_loop(ctl, cond);
                    return;
                }
            }
            const double rel = sqrt(RR / ctl->bb);
            ctl->relres = rel;
            ctl->phase_end = 0;
            if (!start) ctl->stop = ctl->tol;  // phase 2 runs to tol
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

// ---- the iteration ------------------------------------------------------------

constexpr int kStepU = 2;  // pairs a thread and step of k_step_dw

// w = (A + C/dt) z, r.z, z.Ap and z.w in one pass (two neighbouring slots of one
// colour a thread, half the loads and indexing of a cell a lane), then beta, p.Ap and alpha (next_scalars): the step below makes
// A p from w, so neither a dot pass nor an apply on p follows.
// 640 x 640 x 10: 44.8 us (4.4 TB/s; 48.8 a cell a lane, 52.8 at 3 blocks per SM),
// and the step 43.8 us (6.0 TB/s), where the
// dots, the p update, the apply on p and the update of x and r took 22.5 + 14.1 +
// 47.1 + 36.1 us; the x update (16.1 us alone) hides beside the V-cycle's bottom.
__global__ void __launch_bounds__(NT, 4)
    k_az_dw(OpView o, const float2* __restrict__ dgw, const float* __restrict__ z, const float2* __restrict__ r,
            const float2* __restrict__ Ap, float2* __restrict__ w, Ctl* ctl, double* part, int maxb, Cond cond) {
    pdl_enter();
    if (loop_done(ctl, cond)) return;
    const bool first = ctl->iter == 0;  // no Ap yet
    const unsigned n2 = o.g.plane * (unsigned)o.g.nz / 2u;
    DwAcc v[3] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
    for (unsigned q = blockIdx.x * NT + threadIdx.x; q < n2; q += gridDim.x * NT) {
        PairZ<float, float2> a;
        if (!load_pair(o, dgw, z, q, a)) continue;
        const float4 rv = load_two(r, a.k), av = first ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : load_two(Ap, a.k);
        dots_dw(v, a, rv, av, w);
    }
    pdl_trigger();
    if (publish_acc<3>(v, part, maxb, blockIdx.x, &ctl->ticket[SL_APPLY], gridDim.x)) {
        double t[3];
        gather_acc<3>(part, maxb, 0u, gridDim.x, &ctl->ticket[SL_APPLY], t);
        if (threadIdx.x == 0) {
            Scalars s;
            const bool ok = next_scalars(true, first, t[0], t[1], t[2], ctl->rz, ctl->pAp, s);
            ctl->rz = t[0];
            ctl->zAp = t[1];
            ctl->beta = s.beta;
            ctl->pAp = s.pAp;
            ctl->alpha = s.alpha;
            ctl->beta_w = dw_of(s.beta);
            ctl->alpha_w = dw_of(s.alpha);
            if (!ok) {
                ctl->breakdown = 1;
                stop_loop(ctl, cond);
            }
        }
    }
}

// p = z + beta p, Ap = w + beta Ap, r -= alpha Ap, b0 = r (hi word), ||r||^2,
// convergence test. Two values a thread and step (float4 = two double words),
// each block a contiguous range. WX = false: x is left to k_update_x_dw beside
// the next V-cycle, alpha in ctl->alpha_xw for it (k_step64 likewise).
template <bool WX>
__global__ void __launch_bounds__(NT)
    k_step_dw(unsigned n2, const float2* __restrict__ z, const float4* __restrict__ w, float4* __restrict__ p,
              float4* __restrict__ Ap, float4* __restrict__ x, float4* __restrict__ r, float2* __restrict__ b0,
              Ctl* ctl, double* part, int maxb, Cond cond) {
    pdl_enter();
    const bool done = loop_done(ctl, cond);
    const float2 alpha = ctl->alpha_w, beta = ctl->beta_w;
    if (!WX && blockIdx.x == 0 && threadIdx.x == 0) ctl->alpha_xw = done ? make_float2(0.0f, 0.0f) : alpha;
    if (done) return;
    const bool first = ctl->iter == 0;
    DwAcc v[1] = {{0.0f, 0.0f}};
    const unsigned per = ((n2 + gridDim.x - 1) / gridDim.x + NT * kStepU - 1) / (NT * kStepU) * (NT * kStepU);
    const unsigned begin = blockIdx.x * per, end = begin + per < n2 ? begin + per : n2;
    stream_pipelined<kStepU, StepItem>(
        begin + threadIdx.x, end, NT,
        [&](unsigned k) {
            const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            return StepItem{z[k], w[k], first ? none : p[k], first ? none : Ap[k], r[k]};
        },
        [&](unsigned k, StepItem it) {
            step_item(it, alpha, beta, v[0]);
            p[k] = it.p;
            Ap[k] = it.a;
            r[k] = it.r;
            b0[k] = make_float2(it.r.x, it.r.z);
            if (WX) x[k] = x_item(x[k], it.p, alpha);
        });
    pdl_trigger();
    if (publish_acc<1>(v, part, maxb, blockIdx.x, &ctl->ticket[SL_UPDATE], gridDim.x)) {
        double t[1];
        gather_acc<1>(part, maxb, 0u, gridDim.x, &ctl->ticket[SL_UPDATE], t);
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
            } else if (rel < ctl->stop) {
                // end of phase 1: the next step is the FP64 residual replacement
                ctl->phase_end = 1;
                if (cond.use) cudaGraphSetConditional(cond.h, 0u);
            }
        }
    }
}

// x += alpha p with the alpha k_step_dw<false> left in ctl->alpha_xw (zero:
// nothing pending), the same rounding as the fused update; ordered as
// k_update_x64 is.
struct XItemDw {
    float4 p, x;
};
__global__ void __launch_bounds__(NT)
    k_update_x_dw(unsigned n2, const float4* __restrict__ p, float4* __restrict__ x, const Ctl* ctl) {
    const float2 alpha = ctl->alpha_xw;
    if (alpha.x == 0.0f) return;
    stream_pipelined<4, XItemDw>(
        blockIdx.x * NT + threadIdx.x, n2, gridDim.x * NT, [&](unsigned k) { return XItemDw{p[k], x[k]}; },
        [&](unsigned k, const XItemDw& it) { x[k] = x_item(it.x, it.p, alpha); });
}

// xb += xw (in FP64), xw = 0: the double-word correction goes into the base.
// Skipped (all blocks) once the solve is done; runs before the residual
// replacement, which is what it serves.
__global__ void k_fold(unsigned n2, double2* __restrict__ xb, float4* __restrict__ xw,
                       const Ctl* ctl, int check_done) {
    pdl_enter();
    if (check_done && *(volatile const int*)&ctl->done) return;
    for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < n2; k += gridDim.x * blockDim.x) {
        const float4 w = xw[k];
        if (w.x != 0.0f || w.z != 0.0f) {
            double2 v = xb[k];
            v.x += dw_d(make_float2(w.x, w.y));
            v.y += dw_d(make_float2(w.z, w.w));
            xb[k] = v;
            xw[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
}

// ---- conversions at the boundary -------------------------------------------

// FP64 diagonal -> double word.
__global__ void k_to_dw(unsigned n, const double* __restrict__ in, float2* __restrict__ out) {
    for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
        out[k] = dw_of(in[k]);
}

unsigned blocks_of(size_t n) {
    size_t b = (n + NT - 1) / NT;
    if (b < 1) b = 1;
    if (b > 65535u * 16u) b = 65535u * 16u;
    return (unsigned)b;
}

}  // namespace

void launch_fold(cudaStream_t st, unsigned n, double* xb, float2* xw, const Ctl* ctl,
                 bool check_done) {
    static const int wb = wave_blocks(k_fold, 1 << 30);
    launch_pdl(k_fold, std::min((int)blocks_of(n / 2), wb), NT, 0, st, n / 2, (double2*)xb, (float4*)xw, ctl,
                                                               check_done ? 1 : 0);
}

void launch_residual_x(cudaStream_t st, const OpView& o, unsigned n, const double* diag, const double* b,
                       const double* x, float2* r, float* b0, bool start, Ctl* ctl,
                       const Red& red, Cond cond) {
    static const int wb = wave_blocks(k_residual_x, 1 << 30);
    launch_pdl(k_residual_x, std::min(red.blocks, wb), NT, 0, st, o, n, diag, b, x, r, b0, start ? 1 : 0, ctl, red.part,
                                            red.maxb, cond);
}

void launch_az_dw(cudaStream_t st, const OpView& o, const float2* dgw, const float* z, const float2* r,
                  const float2* Ap, float2* w, Ctl* ctl, const Red& red, Cond cond) {
    static const int wb = wave_blocks(k_az_dw, 1 << 30);
    const int want = (int)blocks_of(o.g.plane * (size_t)o.g.nz / 2);
    launch_pdl(k_az_dw, std::min(std::min(red.maxb, wb), want), NT, 0, st, o, dgw, z, r, Ap, w, ctl, red.part, red.maxb, cond);
}

void launch_step_dw(cudaStream_t st, unsigned n, const float* z, const float2* w, float2* p, float2* Ap, float2* x,
                    float2* r, float* b0, Ctl* ctl, const Red& red, Cond cond, bool write_x) {
    auto go = [&](auto kern, int wb) {
        launch_pdl(kern, std::min(red.blocks, wb), NT, 0, st, n / 2, (const float2*)z, (const float4*)w, (float4*)p,
                   (float4*)Ap, (float4*)x, (float4*)r, (float2*)b0, ctl, red.part, red.maxb, cond);
    };
    static const int wx = wave_blocks(k_step_dw<true>, 1 << 30), wr = wave_blocks(k_step_dw<false>, 1 << 30);
    if (write_x)
        go(k_step_dw<true>, wx);
    else
        go(k_step_dw<false>, wr);
}

void launch_update_x_dw(cudaStream_t st, unsigned n, const float2* p, float2* x, const Ctl* ctl, int blocks) {
    static const int wb = wave_blocks(k_update_x_dw, 1 << 30);
    const int want = std::min((int)blocks_of(n / 2), wb);
    k_update_x_dw<<<blocks > 0 ? std::min(blocks, want) : want, NT, 0, st>>>(n / 2, (const float4*)p, (float4*)x, ctl);
}

void launch_to_dw(cudaStream_t st, unsigned n, const double* in, float2* out) {
    k_to_dw<<<blocks_of(n), NT, 0, st>>>(n, in, out);
}

}  // namespace ct
