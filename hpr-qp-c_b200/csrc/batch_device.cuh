// What the batch kernels share: an instance's record, the kernels' arguments,
// the control state of a running solve and its workspace vectors.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace hpr {

struct BInst {
    long long q_nz, a_nz, at_nz;  // first entry of the instance's matrices
    int q_rp, a_rp, at_rp;        // first row pointer
    int var, row;                 // first variable / row in the packed vectors
    int n, m;
    int movable;                  // a cluster can go on with it (yield_now)
    int q_lg, a_lg, at_lg;        // log2 of the SpMV lane-group width of Q, A, A' (0..5)
    double obj_constant;
};

struct BResume;

struct BatchArgs {
    int K;
    const BInst *inst;
    const int *order;
    unsigned long long *counter;  // the work queue's two ends (take_instance)
    const int *q_rp, *q_ci, *a_rp, *a_ci, *at_rp, *at_ci;
    const double *q_v0, *a_v0, *at_v0, *c0, *l0, *u0, *AL0, *AU0;
    double *q_v, *a_v, *at_v;  // scaled copies
    double *ws;                // per-CTA workspace
    size_t ws_stride;
    int nmax, mmax;
    int vec_smem;              // 1: the gathered vectors live in shared memory
    // parameters
    double stoptol;
    long long max_iter;
    double time_limit;
    int check_iter;
    int print_frequency;
    int use_scaling;
    unsigned long long t_start;  // globaltimer at launch (ns), set by CTA 0
    // host-mapped flag set by hprqp_batch_request_abort (nonzero: stop);
    // read by thread 0 of each CTA when an instance starts and every
    // kAbortPoll iterations
    const int *abort_flag;
    // outputs (packed like the inputs)
    double *x, *y, *z, *w;
    int *status;
    long long *iters;
    double *pobj, *resid, *gap;
    int *restarts;
    unsigned long long *phase_clk;  // optional [grid x 8] clock64 totals per phase
    unsigned char *active_x;  // 1 = variable at a bound (for the adjoint)
    unsigned char *active_r;  // 1 = row at a bound
    double *col_norm_out, *row_norm_out;  // scaling of each instance (for the adjoint)
    // optional starting point in the caller's (unscaled) variables, packed
    // like the outputs; nullptr = start from zero as the reference does
    const double *x_start, *w_start, *y_start;
    const double *sigma_start;  // per instance, optional (<= 0: from the data)
    double *sigma_out;          // per instance: sigma at the end of the solve
    double *seconds_out;        // per instance: device time from its start to its end on its CTA
    // single-QP solves (solve_gpu of a small model runs as a batch of one):
    // the time limit counts from the start of the instance's iteration loop,
    // as the host loop's does (after setup); optional milestone, loop-time
    // and log outputs
    int time_from_loop;
    long long *iter4_out, *iter6_out;  // first checked iteration with KKT < 1e-4 / 1e-6 (-1: none)
    double *time4_out, *time6_out;     // loop seconds at those iterations
    double *loop_seconds_out;          // loop seconds at the end
    // Handing instances over (batch_launch): when at most yield_at of the
    // K_total instances are unfinished and this launch's queue is empty, the
    // running instances are saved (state in their workspace slots, control
    // state in resume_out) and their CTAs end, so that a next launch can give
    // each of them more SMs.  The next launch waits for all of a phase's, so
    // nothing is handed over while *hold > 0: it counts the unfinished
    // instances that no cluster takes and the parts of the call that are not
    // launched yet.  resume_in: the instances this launch goes on with (its
    // order then lists records).
    int K_total, yield_at;
    unsigned long long *hold;
    int slot0;                         // workspace slot of this launch's CTA (cluster) 0
    double *ws_all;                    // workspace slot 0
    unsigned long long *finished;      // instances finished so far, over all launches
    unsigned long long *resume_count;
    BResume *resume_out;
    const BResume *resume_in;
    double *log_buf;                   // kLogFields doubles per printed iteration (instance 0 only)
    int log_cap;
    int *log_count;
};

// optional per-CTA phase clocks: 0 load+scale, 1 setup norms/diag, 2 power
// iterations, 3 steps, 4 residuals, 5 m-norm, 6 sigma+restart, 7 total
#define PHASE_T0() long long _pt0 = clock64()
#define PHASE_ADD(k)                                                                       \
    do {                                                                                   \
        if (B.phase_clk && threadIdx.x == 0)                                               \
            B.phase_clk[blockIdx.x * 8 + (k)] += (unsigned long long)(clock64() - _pt0);   \
        _pt0 = clock64();                                                                  \
    } while (0)

static __device__ __forceinline__ unsigned long long globaltimer_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

constexpr int kAbortPoll = 16;  // iterations between reads of the host abort flag
// one log record: iter, errRp, errRd, primal obj, dual obj, gap, sigma, loop seconds
constexpr int kLogFields = 8;

// the host's abort request (a system-scope read of host-mapped memory)
__device__ __forceinline__ bool abort_requested(const int *flag)
{
    if (!flag) return false;
    int v;
    asm volatile("ld.relaxed.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    return v != 0;
}

__device__ __forceinline__ double clampd(double v, double lo, double hi)
{
    return v < lo ? lo : (v > hi ? hi : v);
}

// What both batch kernels compute from two products, rounded one way wherever
// it is compiled: an instance may start in k_batch_solve and go on in
// k_cluster_solve, at a moment that depends on the others, and must not show
// where it did.  (Left to the compiler, either product of a sum of two may be
// the fused one, and a product that is needed twice is not fused at all: sigma
// d was fused into 1 + sigma d in one kernel and shared with fact1 in the
// other.)
// p a + q b, the first product fused
__device__ __forceinline__ double two_products(double p, double a, double q, double b)
{
    return fma(p, a, __dmul_rn(q, b));
}
// the Halpern average h2 now + h1 anchor
__device__ __forceinline__ double average(double h2, double now, double h1, double anchor)
{
    return two_products(h2, now, h1, anchor);
}
__device__ __forceinline__ double diag_inverse(double sigma, double d) { return 1.0 / fma(sigma, d, 1.0); }
__device__ __forceinline__ double diag_fact1(double sigma, double d, double inv)
{
    return __dmul_rn(__dmul_rn(sigma, d), inv);
}
__device__ __forceinline__ double w_bar_of(double f1, double w, double f2, double x_hat)
{
    return two_products(f1, w, f2, x_hat);
}
// M-norm from its sums (reference control.cu:243-332); a: dx dx, dx Qdw,
// Qdw Qdw, dw Qdw; b: A'dy dx, dy dy; c: Qdw A'dy, A'dy QA'dy, A'dy M QA'dy
__device__ __forceinline__ double m_norm_of(double sigma, double lA, double lQ, bool rows, bool diag, const double *a,
                                            const double *b, const double *c)
{
    double m1 = 0.0, m3 = 0.0, m2 = two_products(1.0 / sigma, a[0], -2.0, a[1]);
    if (rows) {
        m1 = two_products(__dmul_rn(sigma, lA), b[1], -2.0 * sigma, c[0]);
        m2 += 2.0 * b[0];
        if (diag) {
            m3 = c[2];
            m1 = fma(sigma, a[2], m1);
        } else {
            m3 = (sigma * sigma) / fma(sigma, lQ, 1.0) * c[1];
            m1 = fma(__dmul_rn(sigma, lQ), a[3], m1);
        }
    } else if (!diag) {
        m1 = sigma * lQ * a[3];
    }
    m2 += m1 > 0.0 ? m1 : 0.0;
    return sqrt((m2 > 0.0 ? m2 : 0.0) + (m3 > 0.0 ? m3 : 0.0));
}
// the coefficient of sigma in the sigma estimate (reference control.cu:334-529)
__device__ __forceinline__ double sigma_slope(double lA, double lQ, bool rows, bool diag, double dy_dy, double dqw_atdy,
                                              double dqw_dqw, double dw_dqw)
{
    double a = rows ? two_products(lA, dy_dy, -2.0, dqw_atdy) : 0.0;
    a += diag ? dqw_dqw : __dmul_rn(lQ, dw_dqw);
    return fmax(a, 1e-12);
}

// CTA-shared control state of the instance being solved
struct CtaState {
    double sigma, lA, lQ;
    int q_is_diag, noC;
    int n, m;
    // restart (HPRQPRestart, include/shared/types.h:177-193)
    int restart_flag, first_restart;
    double last_gap, current_gap, save_gap, weighted_norm, best_gap, best_sigma;
    long long inner, times;
    // residuals (HPRQPResiduals)
    double rp, rd, kkt, pobj, dobj, gap;
    double norm_b_org, norm_c_org, obj_constant;
    int to_check, do_res, stop, final_status;
    int aborted;  // the host asked the batch to stop (sticky for the instance)
    int print_yes, got4, got6;
    int yield;    // the instance is to be handed over
    double red[16];
    double scal[8];
};

// a saved instance: its vectors are in workspace slot `slot`, its scaled
// matrices where the solve keeps them; it goes on at the top of iteration iter
struct BResume {
    int inst, slot;
    long long iter;
    unsigned long long t0;  // start of the instance (globaltimer)
    CtaState S;
};

// whether a running instance of a launch is to be handed over
static __device__ __forceinline__ bool yield_now(const BatchArgs &B, const BInst &I)
{
    if (B.yield_at <= 0 || !I.movable) return false;
    const unsigned long long taken = *(volatile unsigned long long *)B.counter;
    if ((taken & 0xffffffffull) + (taken >> 32) < (unsigned long long)B.K) return false;
    return (long long)B.K_total - (long long)*(volatile unsigned long long *)B.finished <= (long long)B.yield_at &&
           *(volatile unsigned long long *)B.hold == 0;
}

// instance I of k_batch_solve has ended (those of k_cluster_solve are movable)
static __device__ __forceinline__ void count_finished(const BatchArgs &B, const BInst &I)
{
    atomicAdd(B.finished, 1ull);
    if (!I.movable) atomicAdd(B.hold, ~0ull);
}

struct Vecs {
    double *c, *l, *u, *col_norm, *x, *x_bar, *x_hat, *w, *w_bar, *ATy, *ATy_bar, *ATdy, *Qw, *Qw_bar, *Qx,
        *dQw, *QATdy, *dx, *dw, *z_bar, *tempv, *diag_Q, *fact1, *fact2, *fact, *fact_M, *last_x, *last_Qw,
        *last_w, *last_ATy, *fac_c, *pn;
    double *AL, *AU, *row_norm, *y, *y_bar, *Ax, *dy, *s, *last_y, *fac_r, *pz, *pq;
};

constexpr int kBatchNVecs = 32, kBatchMVecs = 12;

static __device__ Vecs carve(double *base, int nmax, int mmax, double *smem_pool)
{
    Vecs V;
    double **nv[kBatchNVecs] = {&V.c,      &V.l,      &V.u,      &V.col_norm, &V.x,     &V.x_bar,  &V.x_hat,
                                &V.w,      &V.w_bar,  &V.ATy,    &V.ATy_bar,  &V.ATdy,  &V.Qw,     &V.Qw_bar,
                                &V.Qx,     &V.dQw,    &V.QATdy,  &V.dx,       &V.dw,    &V.z_bar,  &V.tempv,
                                &V.diag_Q, &V.fact1,  &V.fact2,  &V.fact,     &V.fact_M, &V.last_x, &V.last_Qw,
                                &V.last_w, &V.last_ATy, &V.fac_c, &V.pn};
    double **mv[kBatchMVecs] = {&V.AL, &V.AU, &V.row_norm, &V.y,     &V.y_bar, &V.Ax,
                                &V.dy, &V.s,  &V.last_y,   &V.fac_r, &V.pz,    &V.pq};
    const int na = (nmax + 31) & ~31, ma = (mmax + 31) & ~31;
    for (int k = 0; k < kBatchNVecs; ++k) *nv[k] = base + (size_t)k * na;
    for (int k = 0; k < kBatchMVecs; ++k) *mv[k] = base + (size_t)kBatchNVecs * na + (size_t)k * ma;
    if (smem_pool) {
        // the gather sources of the step, the residuals and the power iteration
        V.w = smem_pool;
        V.w_bar = smem_pool + na;
        V.tempv = smem_pool + 2 * na;
        V.x_bar = smem_pool + 3 * na;
        V.y_bar = smem_pool + 4 * na;
        V.y = smem_pool + 4 * na + ma;
    }
    return V;
}

static __device__ __forceinline__ size_t adaptive_step_d(long long iter)
{
    long long step = 10;
    if (iter == 0) return step;
    while (iter / step >= 100) step *= 10;
    return step;
}

// a % d == 0 for the iteration counters of thread 0, in 32-bit arithmetic
// while both fit (every practical count; 64-bit division is a long software
// sequence that the whole CTA would wait for at the next barrier)
static __device__ __forceinline__ bool divides(long long a, long long d)
{
    if (a >= 0 && d > 0 && a <= 0x7fffffffLL && d <= 0x7fffffffLL) return (unsigned)a % (unsigned)d == 0u;
    return a % d == 0;
}

// iter lies on the reference's adaptive print grid (src/shared/solver_backend.c
// print steps: every 10 below 1000, every 100 below 10000, ...)
static __device__ __forceinline__ bool on_print_grid(long long iter)
{
    if (iter >= 0 && iter <= 0x7fffffffLL) {
        const unsigned it = (unsigned)iter;
        unsigned step = 10;
        while (it / step >= 100u && step <= 100000000u) step *= 10;
        return it % step == 0u;
    }
    return iter % (long long)adaptive_step_d(iter) == 0;
}

}  // namespace hpr
