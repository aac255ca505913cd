// k_batch.cu - batched solver kernels: the double-word outer PCG and the
// FP32 V-cycle stages for many instances per launch (see batch.h for the
// block table and the per-instance reductions).
//
// Each kernel is the batched form of a single-solver kernel and uses the same
// per-column / per-cell device code (dw_dev.cuh, mg_dev.cuh), so one instance
// of a batch computes what a single solver computes for it.
#include <cstdlib>
#include <algorithm>
#include <cmath>

#include "batch.h"
#include "batch_dev.cuh"
#include "dw_dev.cuh"
#include "f64_dev.cuh"
#include "mg_dev.cuh"
#include "reduce.cuh"
#include "setup_dev.cuh"

namespace ct {

using namespace dwdev;
using namespace f64dev;
using namespace mgdev;

namespace {

// Start of every loop body: ends the loop once no instance is active, and
// bounds the number of bodies.
__global__ void kb_guard(BCtl* bc, Cond cond) {
    pdl_enter();
    pdl_trigger();
    if (threadIdx.x != 0) return;
    bc->body += 1;
    if (bc->active <= 0 || bc->body > bc->maxbody) {
        if (cond.use) cudaGraphSetConditional(cond.h, 0u);
    }
}

__global__ void __launch_bounds__(NT)
    kb_fold(Plan p, const BInst* __restrict__ bi, const Ctl* ctl, int only_phase_end) {
    pdl_enter();
    for (int task = (int)blockIdx.x; task < p.ntasks; task += (int)gridDim.x) {
        const Task t = p.tasks[task];
        const Ctl* c = &ctl[t.inst];
        if (only_phase_end && (inst_done(c) || !c->phase_end)) continue;
        double2* xb = reinterpret_cast<double2*>(bi[t.inst].x);
        float4* xw = reinterpret_cast<float4*>(bi[t.inst].xw);
        for (unsigned k = t.begin + threadIdx.x; k < t.end; k += NT) {
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
}

// r = b - A x in FP64 from the FP64 base x: the start of a solve, or (start
// = 0) the residual replacement of instances whose first phase ended. Items =
// rows of one colour and plane (k_residual_x; a start from x = 0 splits b).
__global__ void __launch_bounds__(NT, 4)
    kb_residual(Plan p, const BInst* __restrict__ bi, Ctl* ctl, BRed red, int start, BCtl* bc,
                Cond cond) {
    pdl_enter();
    for (int task = (int)blockIdx.x; task < p.ntasks; task += (int)gridDim.x) {
        const Task t = p.tasks[task];
        Ctl* c = &ctl[t.inst];
        if (inst_done(c) || (!start && !c->phase_end)) continue;
        const BInst& I = bi[t.inst];
        const OpView o = I.o;
        const double *const diag = I.diag, *const x = I.x, *const b = I.b;
        float2* const r = I.r;
        float* const b0 = I.b0;
        const bool zero = start && c->x_zero;
        const int lane = (int)(threadIdx.x & 31u);
        double rr = 0.0, bb = 0.0;
        for (unsigned R = t.begin + (threadIdx.x >> 5); R < t.end; R += NT / 32) {
            if (zero) {
                const unsigned s0 = R * (unsigned)o.g.hx;
                for (unsigned s = s0 + (unsigned)lane; s < s0 + (unsigned)o.g.hx; s += 32u) {
                    const double bv = b[s];
                    const float2 rw = split(bv);
                    r[s] = rw;
                    b0[s] = rw.x;
                    bb = __fma_rn(bv, bv, bb);
                }
            } else {
                row64<1>(o, diag, x, R, lane, [&](unsigned k, bool valid, double ax, double) {
                    if (!valid) {
                        r[k] = make_float2(0.0f, 0.0f);
                        b0[k] = 0.0f;
                        return;
                    }
                    const double bv = b[k], rv = bv - ax;
                    const float2 rw = split(rv);
                    r[k] = rw;
                    b0[k] = rw.x;
                    rr = __fma_rn(rv, rv, rr);
                    bb = __fma_rn(bv, bv, bb);
                });
            }
        }
        if (zero) rr = bb;
        block_sum2(rr, bb);
        if (publish_inst(rr, bb, red, p.ntasks, t.inst, p.inst_count[t.inst], task)) {
            double RR, BB;
            gather_inst(red, p.ntasks, t.inst, p.inst_first[t.inst], p.inst_count[t.inst], RR, BB);
            if (threadIdx.x == 0) {
                c->rr = RR;
                if (start) c->bb = BB;
                const bool none = start && BB == 0.0;  // no heat in
                const double rel = none ? 0.0 : sqrt(RR / c->bb);
                c->relres = rel;
                c->phase_end = 0;
                if (!start) c->stop = c->tol;
                if (none) {
                    c->bb_zero = 1;
                    c->converged = 1;
                    inst_stop(c, bc, cond);
                } else if (rel < c->tol) {
                    c->converged = 1;
                    inst_stop(c, bc, cond);
                } else if (!isfinite(rel)) {
                    c->breakdown = 1;
                    inst_stop(c, bc, cond);
                } else if (c->iter >= c->maxit) {
                    inst_stop(c, bc, cond);
                }
            }
            // block_sum2's shared arrays: warp 0 reads gather_inst's sums after that
            // sum's only barrier, and the next task's sums go to the same place
            __syncthreads();
        }
    }
}

// w = (A + C/dt) z, r.z, z.Ap, z.w, then the instance's beta, p.Ap and alpha
// (k_az_dw); items = rows of one colour and plane, walked in pairs of slots. 16
// stacks of 256 x 256 x 10: 115 us a launch, 127 compiled for 4 blocks per SM, 139
// a cell a lane.
__global__ void __launch_bounds__(NT, 3)
    kb_az_dw(Plan p, const BInst* __restrict__ bi, Ctl* ctl, BRed red, BCtl* bc, Cond cond) {
    pdl_enter();
    const Task t = p.tasks[blockIdx.x];
    Ctl* c = &ctl[t.inst];
    if (inst_done(c)) return;
    const BInst& I = bi[t.inst];
    const OpView o = I.o;
    const float2 *const r = I.r, *const Ap = I.Ap;
    float2* const w = I.w;
    const bool first = c->iter == 0;  // no Ap yet
    const float2* __restrict__ dgw = I.dgw;
    const float* __restrict__ z = I.z;
    const unsigned h = (unsigned)o.g.hx / 2u;  // pairs a row
    DwAcc v[3] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
    for (unsigned q = t.begin * h + threadIdx.x; q < t.end * h; q += NT) {
        PairZ<float, float2> a;
        if (!load_pair(o, dgw, z, q, a)) continue;
        const float4 rv = load_two(r, a.k), av = first ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : load_two(Ap, a.k);
        dots_dw(v, a, rv, av, w);
    }
    pdl_trigger();
    const unsigned count = (unsigned)p.inst_count[t.inst];
    if (publish_acc<3>(v, red.part, p.ntasks, blockIdx.x, &red.tickets[t.inst], count)) {
        double s3[3];
        gather_acc<3>(red.part, p.ntasks, (unsigned)p.inst_first[t.inst], count, &red.tickets[t.inst], s3);
        if (threadIdx.x == 0) {
            Scalars s;
            const bool ok = next_scalars(true, first, s3[0], s3[1], s3[2], c->rz, c->pAp, s);
            c->rz = s3[0];
            c->zAp = s3[1];
            c->beta = s.beta;
            c->pAp = s.pAp;
            c->alpha = s.alpha;
            c->beta_w = dw_of(s.beta);
            c->alpha_w = dw_of(s.alpha);
            if (!ok) {
                c->breakdown = 1;
                inst_stop(c, bc, cond);
            }
        }
    }
}

// p = z + beta p, Ap = w + beta Ap, x += alpha p, r -= alpha Ap, b0 = r, ||r||^2,
// the instance's convergence test (k_step_dw). Items are value pairs.
__global__ void __launch_bounds__(NT)
    kb_step_dw(Plan p, const BInst* __restrict__ bi, Ctl* ctl, BRed red, BCtl* bc, Cond cond) {
    pdl_enter();
    const Task t = p.tasks[blockIdx.x];
    Ctl* c = &ctl[t.inst];
    if (inst_done(c)) return;
    const BInst& I = bi[t.inst];
    const float2 alpha = c->alpha_w, beta = c->beta_w;
    const bool first = c->iter == 0;
    const float2* __restrict__ z2 = reinterpret_cast<const float2*>(I.z);
    const float4* __restrict__ w2 = reinterpret_cast<const float4*>(I.w);
    float4* __restrict__ p2 = reinterpret_cast<float4*>(I.p);
    float4* __restrict__ a2 = reinterpret_cast<float4*>(I.Ap);
    float4* __restrict__ x2 = reinterpret_cast<float4*>(I.xw);
    float4* __restrict__ r2 = reinterpret_cast<float4*>(I.r);
    float2* __restrict__ b02 = reinterpret_cast<float2*>(I.b0);
    DwAcc v[1] = {{0.0f, 0.0f}};
    struct Item {
        StepItem s;
        float4 x;
    };
    stream_pipelined<1, Item>(
        t.begin + threadIdx.x, t.end, NT,
        [&](unsigned k) {
            const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            return Item{StepItem{z2[k], w2[k], first ? none : p2[k], first ? none : a2[k], r2[k]}, x2[k]};
        },
        [&](unsigned k, Item it) {
            step_item(it.s, alpha, beta, v[0]);
            p2[k] = it.s.p;
            a2[k] = it.s.a;
            x2[k] = x_item(it.x, it.s.p, alpha);
            r2[k] = it.s.r;
            b02[k] = make_float2(it.s.r.x, it.s.r.z);
        });
    pdl_trigger();
    const unsigned count = (unsigned)p.inst_count[t.inst];
    if (publish_acc<1>(v, red.part, p.ntasks, blockIdx.x, &red.tickets[t.inst], count)) {
        double rr[1];
        gather_acc<1>(red.part, p.ntasks, (unsigned)p.inst_first[t.inst], count, &red.tickets[t.inst], rr);
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
            } else if (rel < c->stop) {
                c->phase_end = 1;  // the replacement at the end of this body
            }
        }
    }
}

// Pairs of values: b = P + C/dt x (x = FP64 base, folded), x_old = x; conversions
// on the integer pipe, as in set_dt (f64_dev.cuh).
__global__ void __launch_bounds__(NT)
    kb_rhs_transient(Plan p, const BInst* __restrict__ bi, const Ctl* ctl) {
    const Task t = p.tasks[blockIdx.x];
    const double inv_dt = ctl[t.inst].inv_dt;
    const BInst I = bi[t.inst];
    const double2* __restrict__ P = reinterpret_cast<const double2*>(I.P);
    const double2* __restrict__ x = reinterpret_cast<const double2*>(I.x);
    const float2* __restrict__ cap = reinterpret_cast<const float2*>(I.o.cap);
    double2* __restrict__ b = reinterpret_cast<double2*>(I.b);
    double2* __restrict__ xold = reinterpret_cast<double2*>(I.xold);
    for (unsigned k = t.begin + threadIdx.x; k < t.end; k += NT) {
        const double2 xv = x[k], pv = P[k];
        const float2 cv = cap[k];
        b[k] = make_double2(__dadd_rn(pv.x, __dmul_rn(__dmul_rn(widen(cv.x), inv_dt), xv.x)),
                            __dadd_rn(pv.y, __dmul_rn(__dmul_rn(widen(cv.y), inv_dt), xv.y)));
        xold[k] = xv;
    }
}

// Step records of every instance (items: fine column slots): T_max,
// heat_out = sum over the top and bottom faces of g x, and sum C (x - x_old)
// (src/stack3d.h:252-273), x the folded FP64 base; rec[3 i + 0..2].
__global__ void __launch_bounds__(NT)
    kb_step_record(Plan p, const BInst* __restrict__ bi, BRed red, double* __restrict__ mx,
                   double* __restrict__ rec) {
    const Task t = p.tasks[blockIdx.x];
    const BInst I = bi[t.inst];
    const Geo& g = I.o.g;
    double tmax = -INFINITY, qout = 0.0, qst = 0.0;
    for (unsigned s = t.begin + threadIdx.x; s < t.end; s += NT) {
        const Col c = col_of_slot(g, s);
        if (!c.valid) continue;
        for (int l = 0; l < g.nz; ++l) {
            const unsigned id = (unsigned)l * g.plane + s;
            const double xv = I.x[id];
            tmax = fmax(tmax, xv);
            qst += (double)I.o.cap[id] * (xv - I.xold[id]);
        }
        const unsigned top = (unsigned)(g.nz - 1) * g.plane + s;
        qout += (double)I.o.gU[top] * I.x[top];
        qout += (double)I.o.gB[s] * I.x[s];
    }
    __shared__ double sm[NT / 32];
    double m = tmax;
    for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, off));
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < NT / 32 ? sm[threadIdx.x] : -INFINITY;
        for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, off));
    }
    block_sum2(qout, qst);
    if (threadIdx.x == 0) mx[blockIdx.x] = m;
    const int first = p.inst_first[t.inst], count = p.inst_count[t.inst];
    if (publish_inst(qout, qst, red, p.ntasks, t.inst, count, (int)blockIdx.x)) {
        __threadfence();
        double mm = -INFINITY;
        for (int k = threadIdx.x; k < count; k += NT) mm = fmax(mm, __ldcg(mx + first + k));
        for (int off = 16; off > 0; off >>= 1) mm = fmax(mm, __shfl_down_sync(0xffffffffu, mm, off));
        __syncthreads();
        if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = mm;
        __syncthreads();
        if (threadIdx.x < 32) {
            mm = threadIdx.x < NT / 32 ? sm[threadIdx.x] : -INFINITY;
            for (int off = 16; off > 0; off >>= 1) mm = fmax(mm, __shfl_down_sync(0xffffffffu, mm, off));
        }
        double QO, QS;
        gather_inst(red, p.ntasks, t.inst, first, count, QO, QS);
        if (threadIdx.x == 0) {
            rec[3 * t.inst] = mm;
            rec[3 * t.inst + 1] = QO;
            rec[3 * t.inst + 2] = QS;
        }
    }
}

// set_dt of every instance: its FP64 (and double-word) diagonal, items =
// natural fine columns; 1/dt per instance from its control block.
__global__ void __launch_bounds__(NT) kb_diag(Plan p, const BInst* __restrict__ bi, const Ctl* ctl) {
    const Task t = p.tasks[blockIdx.x];
    const BInst& I = bi[t.inst];
    const double inv_dt = ctl[t.inst].inv_dt;
    for (unsigned q = t.begin + threadIdx.x; q < t.end; q += NT)
        setupdev::diag_column(I.o, I.dface, inv_dt, q, const_cast<double*>(I.diag), nullptr,
                              const_cast<float2*>(I.dgw));
}

// ... and the column factors of one level index of every instance that has it
// (items = natural columns of that level).
__global__ void __launch_bounds__(NT)
    kb_factor(Plan p, const LevelView<float>* __restrict__ views, const Ctl* ctl) {
    const Task t = p.tasks[blockIdx.x];
    const LevelView<float> L = views[t.inst];
    const float inv_dt = (float)ctl[t.inst].inv_dt;
    for (unsigned q = t.begin + threadIdx.x; q < t.end; q += NT) setupdev::factor_column<float>(L, inv_dt, q);
}

template <int MZ, bool ZERO, bool PRO>
__global__ void __launch_bounds__(NT)
    kb_sweep(Plan p, const LevelView<float>* __restrict__ views,
             const LevelView<float>* __restrict__ cviews, int color, const Ctl* ctl) {
    pdl_enter();
    const Task t = p.tasks[blockIdx.x];
    if (inst_done(&ctl[t.inst])) return;
    const LevelView<float> L = views[t.inst];
    const LevelView<float> C = PRO ? cviews[t.inst] : L;
    for (unsigned q = t.begin + threadIdx.x; q < t.end; q += NT)
        sweep_column<float, MZ, ZERO, PRO>(L, C, color, q);
}

// The same with one thread per column and plane (split_columns), 32 columns a block:
// the small levels, where a thread's nz planes of loads are the launch (48 stacks,
// the second to fifth level: 25, 15, 11, 8 us a launch against 32, 18, 17, 16 with a
// thread a column). The tuner times it beside the other forms. The dependent starts as
// the blocks leave: with several buckets at once, blocks that start early and wait hold
// room that the other buckets' kernels could use (signalled at entry 48 stacks took
// 27.4 ms against 27.2, 256 141.7 against 140.8).
template <int MZ, bool ZERO, bool PRO>
__global__ void __launch_bounds__(32 * MZ)
    kb_sweep_split(Plan p, const LevelView<float>* __restrict__ views, const LevelView<float>* __restrict__ cviews,
                   int color, const Ctl* ctl) {
    __shared__ SplitShared<float, MZ> S;
    const unsigned task = blockIdx.x / (unsigned)p.split;
    const Task t = p.tasks[task];
    const unsigned q = t.begin + (blockIdx.x - task * (unsigned)p.split) * 32u;
    if (q >= t.end) return;
    const LevelView<float> L = views[t.inst];
    const LevelView<float> C = PRO ? cviews[t.inst] : L;
    split_columns<float, MZ, ZERO, PRO>(
        L, C, color, q + threadIdx.x, t.end, S,
        [&] {
            pdl_enter();
            return *(volatile const int*)&ctl[t.inst].done;
        },
        [](int done) { return done != 0; });
}

// Coarse cells of one instance, kRestrictWide a thread; compiled for 4 blocks per SM
// (48 stacks, the finest level: 28.9 us a launch against 34.1 with the compiler's own
// choice).
__global__ void __launch_bounds__(NT, 4)
    kb_restrict(Plan p, const LevelView<float>* __restrict__ views,
                const LevelView<float>* __restrict__ cviews, const Ctl* ctl) {
    pdl_enter();
    const Task t = p.tasks[blockIdx.x];
    const Ctl* c = &ctl[t.inst];
    if (inst_done(c)) return;
    const LevelView<float> L = views[t.inst];
    const LevelView<float> C = cviews[t.inst];
    constexpr int W = kRestrictWide;
    const unsigned groups = ((unsigned)C.g.nx + W - 1u) / W;
    for (unsigned w = t.begin + threadIdx.x; w < t.end; w += NT) {
        const unsigned row = w / groups, l = row / (unsigned)C.g.ny;
        const int J = (int)(row - l * (unsigned)C.g.ny), I = (int)(w - row * groups) * (int)W;
        float s[W];
        restrict_wide<float, W>(L, wide_faces<float, W>(L, I, J, (int)l), I, J, (int)l, s);
        store_wide<float, W>(C, I, J, (int)l, s);
    }
}

template <int MZ>
__global__ void __launch_bounds__(kSmallThreads, 1)
    kb_small(const int* __restrict__ insts, const TailLevels<float>* __restrict__ small,
             Ctl* ctl, BCtl* bc, Cond cond) {
    const int i = insts[blockIdx.x];
    Ctl* c = &ctl[i];
    extern __shared__ __align__(16) unsigned char smem[];
    // the levels' operators and factors (not written inside the loop) are
    // copied before the dependent-launch wait, b and the done flag after it
    const auto wait = [] { pdl_enter(); };
    const auto go = [&] { return !inst_done(c); };
    if (vsmall_body<float, MZ>(small[i], smem, wait, go) == kSmallTimeout &&
        threadIdx.x == 0) {
        // a bounded wait ran out: record it and stop this instance
        atomicExch(&c->err, 1);
        c->breakdown = 1;
        inst_stop(c, bc, cond);
    }
}

}  // namespace

void launch_b_guard(cudaStream_t st, BCtl* bc, Cond cond) { launch_pdl(kb_guard, 1, 32, 0, st, bc, cond); }

// The blocks of the replacement's launches: in most bodies no instance's first phase
// has just ended, and a block per task is only there to find that out; one wave of
// blocks walks the tasks (a backward Euler step of 16 stacks of 256 x 256 x 10: 4.58
// ms against 4.70).
static int replacement_blocks(const Plan& p) {
    static const int wave = wave_blocks(kb_residual, 1 << 30);
    return std::min(p.ntasks, wave);
}

void launch_b_fold(cudaStream_t st, const Plan& p, const BInst* bi, Ctl* ctl, int only_phase_end) {
    launch_pdl(kb_fold, only_phase_end ? replacement_blocks(p) : p.ntasks, NT, 0, st, p, bi, ctl, only_phase_end);
}

void launch_b_residual(cudaStream_t st, const Plan& p, const BInst* bi, Ctl* ctl, BRed red,
                       int start, BCtl* bc, Cond cond) {
    launch_pdl(kb_residual, start ? p.ntasks : replacement_blocks(p), NT, 0, st, p, bi, ctl, red, start, bc, cond);
}

void launch_b_az_dw(cudaStream_t st, const Plan& p, const BInst* bi, Ctl* ctl, BRed red, BCtl* bc, Cond cond) {
    launch_pdl(kb_az_dw, p.ntasks, NT, 0, st, p, bi, ctl, red, bc, cond);
}

void launch_b_step_dw(cudaStream_t st, const Plan& p, const BInst* bi, Ctl* ctl, BRed red, BCtl* bc, Cond cond) {
    launch_pdl(kb_step_dw, p.ntasks, NT, 0, st, p, bi, ctl, red, bc, cond);
}

void launch_b_step_record(cudaStream_t st, const Plan& p, const BInst* bi, BRed red, double* mx,
                          double* rec) {
    if (p.ntasks > 0) kb_step_record<<<p.ntasks, NT, 0, st>>>(p, bi, red, mx, rec);
}

void launch_b_diag(cudaStream_t st, const Plan& p, const BInst* bi, const Ctl* ctl) {
    if (p.ntasks > 0) kb_diag<<<p.ntasks, NT, 0, st>>>(p, bi, ctl);
}

void launch_b_factor(cudaStream_t st, const Plan& p, const LevelView<float>* views, const Ctl* ctl) {
    if (p.ntasks > 0) kb_factor<<<p.ntasks, NT, 0, st>>>(p, views, ctl);
}

void launch_b_rhs_transient(cudaStream_t st, const Plan& p, const BInst* bi, const Ctl* ctl) {
    kb_rhs_transient<<<p.ntasks, NT, 0, st>>>(p, bi, ctl);
}

void launch_b_sweep(cudaStream_t st, const Plan& p, const LevelView<float>* views,
                    const LevelView<float>* cviews, int color, bool zero_x, bool prolong, int mz,
                    const Ctl* ctl) {
#define CT_BSPLIT(MZ)                                                                                        \
    do {                                                                                                     \
        const dim3 block(32, (unsigned)mz);                                                                  \
        if (zero_x)                                                                                          \
            launch_pdl(kb_sweep_split<MZ, true, false>, p.ntasks * p.split, block, 0, st, p, views, cviews, color, ctl);  \
        else if (prolong)                                                                                    \
            launch_pdl(kb_sweep_split<MZ, false, true>, p.ntasks * p.split, block, 0, st, p, views, cviews, color, ctl);  \
        else                                                                                                 \
            launch_pdl(kb_sweep_split<MZ, false, false>, p.ntasks * p.split, block, 0, st, p, views, cviews, color, ctl); \
    } while (0)
    if (p.split) {  // (at most 32 planes)
        if (mz <= 8)
            CT_BSPLIT(8);
        else if (mz <= 12)
            CT_BSPLIT(12);
        else if (mz <= 16)
            CT_BSPLIT(16);
        else
            CT_BSPLIT(32);
        return;
    }
#undef CT_BSPLIT
#define CT_BSWEEP(MZ)                                                                          \
    do {                                                                                       \
        if (zero_x)                                                                            \
            launch_pdl(kb_sweep<MZ, true, false>, p.ntasks, NT, 0, st, p, views, cviews, color, ctl);  \
        else if (prolong)                                                                      \
            launch_pdl(kb_sweep<MZ, false, true>, p.ntasks, NT, 0, st, p, views, cviews, color, ctl);  \
        else                                                                                   \
            launch_pdl(kb_sweep<MZ, false, false>, p.ntasks, NT, 0, st, p, views, cviews, color, ctl); \
    } while (0)
    if (mz <= 8)
        CT_BSWEEP(8);
    else if (mz <= 12)
        CT_BSWEEP(12);
    else if (mz <= 16)
        CT_BSWEEP(16);
    else if (mz <= 32)
        CT_BSWEEP(32);
    else
        CT_BSWEEP(0);
#undef CT_BSWEEP
}

void launch_b_restrict(cudaStream_t st, const Plan& p, const LevelView<float>* views,
                       const LevelView<float>* cviews, const Ctl* ctl) {
    launch_pdl(kb_restrict, p.ntasks, NT, 0, st, p, views, cviews, ctl);
}

cudaError_t launch_b_small(cudaStream_t st, const int* insts, int n,
                           const TailLevels<float>* small, size_t smem, int mz, Ctl* ctl, BCtl* bc,
                           Cond cond) {
    auto go = [&](auto kern) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             kSmallSmemMax);
        if (e != cudaSuccess) return e;
        launch_pdl(kern, n, kSmallThreads, smem, st, insts, small, ctl, bc, cond);
        return cudaGetLastError();
    };
    if (mz <= 8) return go(kb_small<8>);
    if (mz <= 12) return go(kb_small<12>);
    if (mz <= 16) return go(kb_small<16>);
    if (mz <= 32) return go(kb_small<32>);
    return go(kb_small<0>);
}

}  // namespace ct
