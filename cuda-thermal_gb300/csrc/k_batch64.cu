// k_batch64.cu - the batched solver's FP64 outer PCG (CT_MG_FP32_FLEX): the
// start residual, A z with the dot products, and the p, Ap, x, r update of every
// instance of a bucket, one launch each, in IEEE double arithmetic as the
// single solver's k_fp64.cu (same per-cell code, f64_dev.cuh).
// Block tables and per-instance reductions as in k_batch.cu (batch.h).
#include <cmath>

#include "batch.h"
#include "batch_dev.cuh"
#include "f64_dev.cuh"
#include "reduce.cuh"

namespace ct {

using namespace f64dev;

namespace {

// Cells per lane of a row pass: one. The batch's half-rows are 32 to 256
// slots, so a pass of 64 slots leaves lanes idle on most of them (the
// 256-instance batch: 48.5 ms of apply per solve against 59.7 ms with two).
constexpr int kRowU = 1;

// r = b - (A + C/dt) x, b0 = r (float), ||r||^2, ||b||^2 and the start test
// of every instance; items = rows of one colour and plane (a start from
// x = 0 copies b).
__global__ void __launch_bounds__(NT)
    kb_residual64(Plan p, const BInst* __restrict__ bi, Ctl* ctl, BRed red, BCtl* bc, Cond cond) {
    pdl_enter();
    const Task t = p.tasks[blockIdx.x];
    Ctl* c = &ctl[t.inst];
    if (inst_done(c)) return;
    const BInst I = bi[t.inst];
    const Geo& g = I.o.g;
    const bool zero = c->x_zero;
    const int lane = (int)(threadIdx.x & 31u);
    double rr = 0.0, bb = 0.0;
    for (unsigned R = t.begin + (threadIdx.x >> 5); R < t.end; R += NT / 32) {
        if (zero) {
            const unsigned rows = 2u * (unsigned)g.ny;
            const unsigned l = R / rows, row = l * g.plane + (R - l * rows) * (unsigned)g.hx;
            for (unsigned s = (unsigned)lane; s < (unsigned)g.hx; s += 32u) {
                const double bv = I.b[row + s];
                I.r64[row + s] = bv;
                I.b0[row + s] = narrow(bv);
                bb = __fma_rn(bv, bv, bb);
            }
        } else {
            row64<kRowU>(I.o, I.diag, I.x, R, lane, [&](unsigned k, bool valid, double ax, double) {
                if (!valid) {
                    I.r64[k] = 0.0;
                    I.b0[k] = 0.0f;
                    return;
                }
                const double bv = I.b[k];
                const double rv = bv - ax;
                I.r64[k] = rv;
                I.b0[k] = narrow(rv);
                rr = __fma_rn(rv, rv, rr);
                bb = __fma_rn(bv, bv, bb);
            });
        }
    }
    if (zero) rr = bb;
    block_sum2(rr, bb);
    if (publish_inst(rr, bb, red, p.ntasks, t.inst, p.inst_count[t.inst], (int)blockIdx.x)) {
        double RR, BB;
        gather_inst(red, p.ntasks, t.inst, p.inst_first[t.inst], p.inst_count[t.inst], RR, BB);
        if (threadIdx.x == 0) {
            c->rr = RR;
            c->bb = BB;
            if (BB == 0.0) {  // no heat in: x = 0 (src/pcg3d_cpu.cpp:146)
                c->bb_zero = 1;
                c->converged = 1;
                c->relres = 0.0;
                inst_stop(c, bc, cond);
                return;
            }
            const double rel = sqrt(RR / BB);
            c->relres = rel;
            if (rel < c->tol) {
                c->converged = 1;
                inst_stop(c, bc, cond);
            } else if (!isfinite(rel)) {
                c->breakdown = 1;
                inst_stop(c, bc, cond);
            } else if (c->maxit <= 0) {
                inst_stop(c, bc, cond);
            }
        }
    }
}

// w = (A + C/dt) z, r.z, z.Ap, z.w, then the instance's beta, p.Ap and alpha
// (k_az64); items = rows of one colour and plane.
__global__ void __launch_bounds__(NT, 4)
    kb_az64(Plan p, const BInst* __restrict__ bi, Ctl* ctl, BRed red, BCtl* bc, Cond cond) {
    pdl_enter();
    const Task t = p.tasks[blockIdx.x];
    Ctl* c = &ctl[t.inst];
    if (inst_done(c)) return;
    const BInst& I = bi[t.inst];
    const OpView o = I.o;
    const double *const r = I.r64, *const Ap = I.Ap64;
    double* const w = I.w64;
    const bool first = c->iter == 0;  // no Ap yet
    const int lane = (int)(threadIdx.x & 31u);
    double v[3] = {0.0, 0.0, 0.0};
    struct More {
        double r, ap;
    };
    for (unsigned R = t.begin + (threadIdx.x >> 5); R < t.end; R += NT / 32)
        row_z(
            o, I.diag, I.z, R, lane, [&](unsigned k) { return More{r[k], first ? 0.0 : Ap[k]}; },
            [&](unsigned k, const More& m, const CellZ<float, double>& a) {
                const double az = az64(a), zc = to_d(a.zc);
                w[k] = az;
                v[0] = __fma_rn(m.r, zc, v[0]);
                v[1] = __fma_rn(zc, m.ap, v[1]);
                v[2] = __fma_rn(zc, az, v[2]);
            });
    pdl_trigger();
    const unsigned count = (unsigned)p.inst_count[t.inst];
    if (publish_sums<3>(v, red.part, p.ntasks, blockIdx.x, &red.tickets[t.inst], count)) {
        double s3[3];
        gather_sums<3>(red.part, p.ntasks, (unsigned)p.inst_first[t.inst], count, &red.tickets[t.inst], s3);
        if (threadIdx.x == 0) {
            Scalars s;
            const bool ok = next_scalars(true, first, s3[0], s3[1], s3[2], c->rz, c->pAp, s);
            c->rz = s3[0];
            c->zAp = s3[1];
            c->beta = s.beta;
            c->pAp = s.pAp;
            c->alpha = s.alpha;
            if (!ok) {
                c->breakdown = 1;
                inst_stop(c, bc, cond);
            }
        }
    }
}

// p = z + beta p, Ap = w + beta Ap (p = z and Ap = w on the first iteration),
// x += alpha p, r -= alpha Ap, b0 = r (float), ||r||^2 and the instance's
// convergence test (k_step64); items = value pairs.
__global__ void __launch_bounds__(NT)
    kb_step64(Plan p, const BInst* __restrict__ bi, Ctl* ctl, BRed red, BCtl* bc, Cond cond) {
    pdl_enter();
    const Task t = p.tasks[blockIdx.x];
    Ctl* c = &ctl[t.inst];
    if (inst_done(c)) return;
    const BInst& I = bi[t.inst];
    const double alpha = c->alpha, malpha = -alpha, beta = c->beta;
    const bool first = c->iter == 0;
    const float2* __restrict__ z2 = reinterpret_cast<const float2*>(I.z);
    const double2* __restrict__ w2 = reinterpret_cast<const double2*>(I.w64);
    double2* __restrict__ p2 = reinterpret_cast<double2*>(I.p64);
    double2* __restrict__ a2 = reinterpret_cast<double2*>(I.Ap64);
    double2* __restrict__ x2 = reinterpret_cast<double2*>(I.x);
    double2* __restrict__ r2 = reinterpret_cast<double2*>(I.r64);
    float2* __restrict__ b02 = reinterpret_cast<float2*>(I.b0);
    double v[1] = {0.0};
    struct Item {
        float2 z;
        double2 w, p, a, x, r;
    };
    stream_pipelined<1, Item>(
        t.begin + threadIdx.x, t.end, NT,
        [&](unsigned k) {
            const double2 none = make_double2(0.0, 0.0);
            return Item{z2[k], w2[k], first ? none : p2[k], first ? none : a2[k], x2[k], r2[k]};
        },
        [&](unsigned k, Item it) {
            it.p.x = __fma_rn(beta, it.p.x, widen(it.z.x));
            it.p.y = __fma_rn(beta, it.p.y, widen(it.z.y));
            it.a.x = __fma_rn(beta, it.a.x, it.w.x);
            it.a.y = __fma_rn(beta, it.a.y, it.w.y);
            it.x.x = __fma_rn(alpha, it.p.x, it.x.x);
            it.x.y = __fma_rn(alpha, it.p.y, it.x.y);
            it.r.x = __fma_rn(malpha, it.a.x, it.r.x);
            it.r.y = __fma_rn(malpha, it.a.y, it.r.y);
            p2[k] = it.p;
            a2[k] = it.a;
            x2[k] = it.x;
            r2[k] = it.r;
            b02[k] = make_float2(narrow(it.r.x), narrow(it.r.y));
            v[0] = __fma_rn(it.r.x, it.r.x, v[0]);
            v[0] = __fma_rn(it.r.y, it.r.y, v[0]);
        });
    pdl_trigger();
    const unsigned count = (unsigned)p.inst_count[t.inst];
    if (publish_sums<1>(v, red.part, p.ntasks, blockIdx.x, &red.tickets[t.inst], count)) {
        double rr[1];
        gather_sums<1>(red.part, p.ntasks, (unsigned)p.inst_first[t.inst], count, &red.tickets[t.inst], rr);
        if (threadIdx.x == 0) {
            c->rr = rr[0];
            c->iter += 1;
            const double rel = sqrt(rr[0] / c->bb);
            c->relres = rel;
            if (rel < c->tol) {
                c->converged = 1;
                inst_stop(c, bc, cond);
            } else if (!isfinite(rel)) {
                c->breakdown = 1;
                inst_stop(c, bc, cond);
            } else if (c->iter >= c->maxit) {
                inst_stop(c, bc, cond);
            }
        }
    }
}

}  // namespace

void launch_b_residual64(cudaStream_t st, const Plan& p, const BInst* bi, Ctl* ctl, BRed red, BCtl* bc,
                         Cond cond) {
    launch_pdl(kb_residual64, p.ntasks, NT, 0, st, p, bi, ctl, red, bc, cond);
}

void launch_b_az64(cudaStream_t st, const Plan& p, const BInst* bi, Ctl* ctl, BRed red, BCtl* bc, Cond cond) {
    launch_pdl(kb_az64, p.ntasks, NT, 0, st, p, bi, ctl, red, bc, cond);
}

void launch_b_step64(cudaStream_t st, const Plan& p, const BInst* bi, Ctl* ctl, BRed red, BCtl* bc, Cond cond) {
    launch_pdl(kb_step64, p.ntasks, NT, 0, st, p, bi, ctl, red, bc, cond);
}

}  // namespace ct
