// One QP on a thread-block cluster: the same method as k_batch_solve
// (batch.cu), with the instance's rows split over the CTAs of a cluster and
// everything an iteration touches held in their shared memory.
//
// What bounds the one-CTA kernel is latency: an HPR step is four dependent
// products, and each waits for matrix quads, gathered entries and the
// operands of its epilogue from L1 or L2 (32 vectors and the matrices of an
// n = 1000 instance do not fit the L1 of one SM).  Here
//   * CTA r of C owns a contiguous range of the rows of Q, A and A'; their
//     entries (16-bit columns, values in two planes of 16-byte pairs so that
//     a quad is read without bank conflicts) and its slices of the iterates
//     live in its shared memory, matrices that do not fit stay in global
//     memory and are streamed;
//   * the vector a product gathers from has a full copy in every CTA; the
//     lane that owns a row sends its new entry to all C copies with
//     st.async, whose arrival is counted on the receiver's mbarrier: one
//     one-way trip is both the transfer and the barrier between two
//     products.  Measured per exchange of n = 1000 entries over 8 CTAs:
//     about 1150 cycles, against 1700 for remote stores followed by a
//     cluster barrier and 1220 for a bulk copy behind a CTA barrier.
//
// Measured, loop of one solve on the one-CTA kernel / on a cluster of 8 or
// 16: the plain QP of n = 1000 23.6 / 5.8 ms (19.7 / 4.8 us an iteration),
// n = 1999 65 / 8.0 ms, n = 120 (4 CTAs) 8.5 / 3.9 ms.  A product takes 0.4
// to 0.8 us, an exchange 0.15 to 0.6 us.  Per SM the one-CTA kernel does more
// work once there is an instance for every SM (n = 2000: 134 us an iteration
// on one SM, 230 SM-us on 8), so clusters serve the batches that leave SMs
// idle and the last instances of the others (choose_clusters, batch_launch).
// 256 threads: 512 are slower (128 registers spill, and a CTA's few rows on
// twice the warps cost issue slots: n = 1000 on 8 CTAs 7.0 against 13.5 ms),
// except where one CTA holds all of an instance's rows (cluster_threads).
//
// Results equal k_batch_solve's bit for bit.  A row's sum depends on the
// lane-group width only.  Reductions are folded in that kernel's order: the
// cluster's CTAs share its warps ("virtual" warps: vw of them, vw / C per
// CTA, each with the rows and the strided entries the one-CTA kernel gives
// that warp), products store their row sums, and the accumulations run over
// the virtual warps afterwards.
#pragma once

#include "batch_device.cuh"
#include "cluster_solve.h"
#include "rowblock.cuh"

#include <climits>

namespace hpr {

// places in an own row's record
enum { kX, kW, kLx, kLw, kAty, kLaty, kQw, kC, kL, kU, kXh };
enum { kY, kLy, kAL, kAU, kYb };
constexpr int kClHalpern = 128;  // Halpern weights held at a time
constexpr int kClSlots = 12;              // reduction slots
constexpr int kClMaxVw = 32;              // virtual warps
// waits on an mbarrier give up after this many polls (seconds; a peer answers within microseconds)
constexpr int kClMaxPolls = 1 << 22;

__device__ __forceinline__ unsigned cl_smem(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned cl_map(unsigned a, int rank)
{
    unsigned o;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(a), "r"(rank));
    return o;
}
__device__ __forceinline__ void cl_st(unsigned a, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void cl_st_async(unsigned a, double v, unsigned bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}

// one matrix of the instance, the CTA's rows of it
struct CMat {
    int lg, nloc, row0;            // lane-group width (log2), own rows, first own row
    int w0, nw;                    // this warp's rows: first, count
    int src;                       // lane that holds this lane's row sum after a pass
    bool single;                   // the warp's rows make one pass
    int rq;                        // first quad of each own row in shared memory (int index there)
    int va, vb, ci;                // planes and columns in shared memory (double2 / ushort4 index)
    bool res;                      // in shared memory
    int qb, qe;                    // this lane's quads in its warp's first pass (shared memory)
    int pad;                       // the gathered vectors' zero entry
    const int *rp;                 // row pointers of the own rows (global)
    const int4 *gci;
    double2 *gv;
};

template <int C, bool RES, int NT>
__global__ void __launch_bounds__(NT, 1) k_cluster_solve(const ClusterArgs P)
{
    constexpr int NW = NT / 32;
    constexpr bool MULTI = C > 1;
    extern __shared__ __align__(16) double sm[];
    __shared__ CtaState S;
    __shared__ double s_red[2][kClMaxVw][kClSlots];
    __shared__ double s_out[kClSlots], s_k[5], s_h[kClHalpern];
    __shared__ double s_mail[4];  // time-limit flag of each step (a warp without rows may be a step behind)
    __shared__ int s_inst, s_skip, s_dead;
    __shared__ __align__(8) unsigned long long s_bar[4];
    const BatchArgs &B = P.B;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int VW = P.vw, vwc = VW / C, VT = VW * 32;
    int rank = 0;
    if (MULTI) asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int cid = blockIdx.x / C;  // cluster index

    // distance in the cluster's shared window from this CTA's copy of an
    // address to CTA r's
    unsigned far[C];
#pragma unroll
    for (int r = 0; r < C; ++r) far[r] = MULTI ? cl_map(cl_smem(sm), r) - cl_smem(sm) : 0u;
    auto sync = [&]() {
        // (not the .aligned forms: they need a converged warp, which code before
        // a barrier does not promise; a diverged one would arrive in parts)
        __syncwarp();
        if (MULTI) asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
        else __syncthreads();
    };
    // store to the same shared address of every CTA of the cluster
    auto put_all = [&](double *p, double v) {
        if (MULTI) {
            const unsigned a = cl_smem(p);
#pragma unroll
            for (int r = 0; r < C; ++r) cl_st(a + far[r], v);
        } else {
            *p = v;
        }
    };
    // the same by a warp that holds one value: lane r serves CTA r
    auto put_all_warp = [&](double *p, double v) {
        if (MULTI) {
            if (lane < C) cl_st(cl_map(cl_smem(p), lane), v);
        } else if (lane == 0) {
            *p = v;
        }
    };
    // send to every CTA's copy, counted on barrier b there
    auto push = [&](double *p, double v, int b) {
        if (MULTI) {
            const unsigned a = cl_smem(p), ba = cl_smem(&s_bar[b]);
#pragma unroll
            for (int r = 0; r < C; ++r) cl_st_async(a + far[r], v, ba + far[r]);
        } else {
            *p = v;
        }
    };
    int bytes_n = 0, bytes_m = 0, mail_bar = 0;
    unsigned ph = 0;  // parity of the exchange barriers' current phase
    // arrive on the next phase of barrier b (every warp once; warp 0 announces the bytes)
    auto arm = [&](int b) {
        if (MULTI && lane == 0) {
            const unsigned a = cl_smem(&s_bar[b]);
            if (warp == 0) {
                const int bytes = (b == 3 ? bytes_m : bytes_n) + (b == mail_bar ? 8 : 0);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
            } else {
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
            }
        }
    };
    // wait until every entry of barrier b's vector has arrived here
    auto wait = [&](int b) {
        if (MULTI) {
            const unsigned a = cl_smem(&s_bar[b]);
            unsigned ok = 0;
            for (int i = 0; i < kClMaxPolls; ++i) {
                asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                             "selp.u32 %0, 1, 0, p;\n\t}"
                             : "=r"(ok)
                             : "r"(a), "r"(ph)
                             : "memory");
                if (ok) break;
                if (*(volatile int *)&s_dead) break;
            }
            if (!ok) *(volatile int *)&s_dead = 1;
            __syncwarp();
            arm(b);
        } else {
            __syncthreads();
        }
    };
    enum { kBarW = 0, kBarWb = 1, kBarT = 2, kBarY = 3 };

    const bool resume = B.resume_in != nullptr;
    int red_par = 0;
    // one virtual warp's values into slots slot .. slot + N - 1 of every CTA
    auto put = [&](int gv, int slot, double *v, int n_v, unsigned maxmask) {
        for (int k = 0; k < n_v; ++k) {
            const double r = (maxmask >> k) & 1 ? warp_max(v[k]) : warp_sum(v[k]);
            put_all_warp(&s_red[red_par][gv][slot + k], r);
        }
    };
    // fold the slots over the virtual warps, in their order; results in s_out
    auto finish = [&](int total, unsigned maxmask) {
        sync();
        if (tid < total) {
            const bool mx = (maxmask >> tid) & 1;
            double t = s_red[red_par][0][tid];
            for (int w = 1; w < VW; ++w) t = mx ? fmax(t, s_red[red_par][w][tid]) : t + s_red[red_par][w][tid];
            s_out[tid] = t;
        }
        __syncthreads();
        red_par ^= 1;
    };

    if (tid == 0) s_dead = 0;
    bool first_instance = true;
    sync();
    for (;;) {
        if (tid == 0 && rank == 0) {
            // (the rules of k_batch_solve)
            const bool back = cid & 1;
            const unsigned long long old = atomicAdd(B.counter, back ? (1ull << 32) : 1ull);
            const unsigned long long front_taken = old & 0xffffffffull, back_taken = old >> 32;
            const int inst = front_taken + back_taken >= (unsigned long long)B.K
                                 ? -1
                                 : B.order[back ? B.K - 1 - (int)back_taken : (int)front_taken];
            const int skip = inst >= 0 && !resume && (abort_requested(B.abort_flag) ||
                                           (!B.time_from_loop &&
                                            1e-9 * (double)(globaltimer_ns() - B.t_start) > B.time_limit));
            if (MULTI) {
                for (int r = 0; r < C; ++r) {
                    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cl_map(cl_smem(&s_inst), r)), "r"(inst) : "memory");
                    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cl_map(cl_smem(&s_skip), r)), "r"(skip) : "memory");
                }
            } else {
                s_inst = inst;
                s_skip = skip;
            }
        }
        sync();
        const int taken = s_inst;
        const bool skip = s_skip;
        sync();
        if (taken < 0 || s_dead) break;
        const BResume *const R = resume ? B.resume_in + taken : nullptr;
        const int k = resume ? R->inst : taken, slot = resume ? R->slot : B.slot0 + cid;
        const Vecs V = carve(B.ws_all + (size_t)slot * B.ws_stride, B.nmax, B.mmax, nullptr);
        const BInst I = B.inst[k];
        const int n = I.n, m = I.m;
        if (skip) {
            if (rank == 0) {
                for (int i = tid; i < n; i += NT) {
                    B.x[I.var + i] = B.w[I.var + i] = B.z[I.var + i] = 0.0;
                    if (B.active_x) B.active_x[I.var + i] = 0;
                    B.col_norm_out[I.var + i] = 1.0;
                }
                for (int i = tid; i < m; i += NT) {
                    B.y[I.row + i] = 0.0;
                    if (B.active_r) B.active_r[I.row + i] = 0;
                    B.row_norm_out[I.row + i] = 1.0;
                }
                if (tid == 0) {
                    B.status[k] = 5;
                    B.iters[k] = 0;
                    B.pobj[k] = 0.0;
                    B.resid[k] = INFINITY;
                    B.gap[k] = INFINITY;
                    B.restarts[k] = 0;
                    B.sigma_out[k] = 0.0;
                    B.seconds_out[k] = 0.0;
                    atomicAdd(B.finished, 1ull);  // (no instance here holds a hand-over up)
                }
            }
            continue;
        }
        const unsigned long long inst_t0 = resume ? R->t0 : globaltimer_ns();
        PHASE_T0();
        const long long _ptot = clock64();
        // ---- shared-memory layout -------------------------------------------
        const int per_n = (n + VW - 1) / VW, per_m = (m + VW - 1) / VW;
        const int nr0 = min(rank * vwc * per_n, n), nl = min((rank + 1) * vwc * per_n, n) - nr0;
        const int mr0 = min(rank * vwc * per_m, m), ml = min((rank + 1) * vwc * per_m, m) - mr0;
        const int nl_max = vwc * per_n, ml_max = vwc * per_m;
        // the gathered vectors end with a zero entry, which the padding of a
        // row's quads points to
        const int ne = (n + 2) & ~1, be = (max(n, m) + 2) & ~1, me = (m + 2) & ~1;
        double *const G1 = sm, *const G2 = sm + ne, *const G3 = sm + ne + be;  // gathered: w/tempv, w_bar, y_bar (noC: y)
        double *const own = sm + ne + be + me;
        double *const ownm = own + kClNOwn * nl_max;
        int next;  // next free 16-byte unit of shared memory
        int *const smi = reinterpret_cast<int *>(sm);
        // rows per warp: all warps, but at least the rows of one pass (Q and A'
        // alike, so that a row's epilogues run on one thread)
        auto per_warp = [](int nloc, int rpp) { return max((nloc + NW - 1) / NW, min(nloc, rpp)); };
        const int rpp_n = 32 >> max(I.q_lg, I.at_lg), rpp_m = 32 >> I.a_lg;
        CMat Q, A, AT;
        {
            const int d = (int)((ownm + kClMOwn * ml_max) - sm);
            int ints = 2 * ((d + 1) & ~1);
            auto mat = [&](CMat &M, const int *rp, const int *gci, double *gv, int lg, int nloc, int row0, int rpp, int pad) {
                M.lg = lg;
                M.nloc = nloc;
                M.row0 = row0;
                const int per = per_warp(nloc, rpp);
                M.w0 = min(warp * per, nloc);
                M.nw = min(per, nloc - M.w0);
                M.single = M.nw <= (32 >> lg);
                M.src = (lane & ((32 >> lg) - 1)) << lg;
                M.rq = ints;
                ints += nloc + 1;
                M.rp = rp + row0;
                M.gci = reinterpret_cast<const int4 *>(gci);
                M.gv = reinterpret_cast<double2 *>(gv);
                M.va = M.vb = M.ci = 0;
                M.res = false;
                M.pad = pad;
            };
            mat(Q, B.q_rp + I.q_rp, B.q_ci + I.q_nz, B.q_v + I.q_nz, I.q_lg, nl, nr0, rpp_n, n);
            mat(A, B.a_rp + I.a_rp, B.a_ci + I.a_nz, B.a_v + I.a_nz, I.a_lg, ml, mr0, rpp_m, n);
            mat(AT, B.at_rp + I.at_rp, B.at_ci + I.at_nz, B.at_v + I.at_nz, I.at_lg, nl, nr0, rpp_n, m);
            next = (ints + 3) >> 2;
        }
        // In shared memory every row has quads of its own: the aligned quads
        // that hold it in the packed arrays, with the entries outside the row
        // replaced by 0 times the zero entry (so a product needs no masks and
        // a lane still gets the same entries in the same order).
        auto scan = [&](const CMat &M) {  // one warp: first quad of each own row
            int base = 0;
            for (int r0 = 0; r0 < M.nloc; r0 += 32) {
                const int r = r0 + lane;
                int b = 0, e = 0;
                if (r < M.nloc) {
                    b = M.rp[r];
                    e = M.rp[r + 1];
                }
                const int len = e > b ? ((e + 3) >> 2) - (b >> 2) : 0;
                int incl = len;
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += u;
                }
                if (r < M.nloc) smi[M.rq + r] = base + incl - len;
                base += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) smi[M.rq + M.nloc] = base;
        };
        if (warp == 0) scan(Q);
        if (warp == 1) scan(A);
        if (warp == 2) scan(AT);
        if (tid == 0) G1[n] = G2[n] = G3[m] = 0.0;
        __syncthreads();
        // matrices into shared memory while they fit (Q first: an iteration
        // reads it twice), the others as a copy in global memory
        auto load = [&](CMat &M, const double *v0) {
            const int nq = smi[M.rq + M.nloc];
            const long long units = 2LL * nq + ((nq + 1) >> 1);
            // (columns are 16-bit byte offsets)
            M.res = RES || (next + units) * 16 <= P.smem_bytes;
            const int *ci = reinterpret_cast<const int *>(M.gci);
            if (!RES && !M.res) {
                double *d = reinterpret_cast<double *>(M.gv);
                if (v0 != d)
                    for (int e = M.rp[0] + tid; e < M.rp[M.nloc]; e += NT) d[e] = v0[e];
                return;
            }
            M.va = next;
            M.vb = next + nq;
            M.ci = 2 * (next + 2 * nq);
            next += (int)units;
            for (int r = warp; r < M.nloc; r += NW) {
                const int b = M.rp[r], e = M.rp[r + 1], q0 = smi[M.rq + r], nk = 4 * (smi[M.rq + r + 1] - q0);
                for (int t = lane; t < nk; t += 32) {
                    const int kk = (b & ~3) + t;
                    const bool in = kk >= b && kk < e;
                    reinterpret_cast<unsigned short *>(sm)[4 * (M.ci + q0) + t] = (unsigned short)(8 * (in ? ci[kk] : M.pad));
                    sm[2 * ((t & 2 ? M.vb : M.va) + q0 + (t >> 2)) + (t & 1)] = in ? v0[kk] : 0.0;
                }
            }
        };
        load(Q, (resume ? B.q_v : B.q_v0) + I.q_nz);
        load(A, (resume ? B.a_v : B.a_v0) + I.a_nz);
        load(AT, (resume ? B.at_v : B.at_v0) + I.at_nz);
        // entry kk (index in the instance) of own row r, whose entries start at b
        auto val = [&](const CMat &M, int r, int b, int kk) -> double & {
            const int t = kk - (b & ~3);
            if (RES || M.res) return sm[2 * ((t & 2 ? M.vb : M.va) + smi[M.rq + r] + (t >> 2)) + (t & 1)];
            return reinterpret_cast<double *>(M.gv)[kk];
        };
        auto col = [&](const CMat &M, int kk) -> int { return __ldg(reinterpret_cast<const int *>(M.gci) + kk); };
        if (resume) {
            // the saved iterates: own slices, and full copies of what the next
            // step gathers
            for (int i = tid; i < nl; i += NT) {
                const int gi = nr0 + i;
                double *o = own + kClNOwn * i;
                o[kX] = __ldcg(V.x + gi);
                o[kW] = __ldcg(V.w + gi);
                o[kLx] = __ldcg(V.last_x + gi);
                o[kLw] = __ldcg(V.last_w + gi);
                o[kAty] = __ldcg(V.ATy + gi);
                o[kLaty] = __ldcg(V.last_ATy + gi);
                o[kQw] = __ldcg(V.Qw + gi);
                o[kC] = __ldcg(V.c + gi);
                o[kL] = __ldcg(V.l + gi);
                o[kU] = __ldcg(V.u + gi);
                o[kXh] = 0.0;
            }
            for (int i = tid; i < ml; i += NT) {
                const int gi = mr0 + i;
                double *o = ownm + kClMOwn * i;
                o[kY] = __ldcg(V.y + gi);
                o[kLy] = __ldcg(V.last_y + gi);
                o[kAL] = __ldcg(V.AL + gi);
                o[kAU] = __ldcg(V.AU + gi);
                o[kYb] = __ldcg(V.y_bar + gi);
            }
            for (int i = tid; i < n; i += NT) {
                G1[i] = __ldcg(V.w + i);
                G2[i] = __ldcg(V.w_bar + i);
            }
            for (int i = tid; i < m; i += NT) G3[i] = __ldcg(V.y + i);
            if (tid == 0) {
                S = R->S;
                S.yield = 0;
            }
        } else {
            for (int i = tid; i < nl; i += NT) {
                own[kClNOwn * i + kC] = B.c0[I.var + nr0 + i];
                own[kClNOwn * i + kL] = B.l0[I.var + nr0 + i];
                own[kClNOwn * i + kU] = B.u0[I.var + nr0 + i];
                V.col_norm[nr0 + i] = 1.0;
            }
            for (int i = tid; i < ml; i += NT) {
                ownm[kClMOwn * i + kAL] = B.AL0[I.row + mr0 + i];
                ownm[kClMOwn * i + kAU] = B.AU0[I.row + mr0 + i];
                V.row_norm[mr0 + i] = 1.0;
            }
        }
        if (MULTI && tid == 0) {
            for (int b = 0; b < 4 && !first_instance; ++b)
                asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(cl_smem(&s_bar[b])) : "memory");
            for (int b = 0; b < 4; ++b)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(cl_smem(&s_bar[b])), "r"(NW) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        first_instance = false;
        __syncthreads();

        // this lane's quads [qb, qe) of row rr of a chunk that starts at c0
        auto lane_quads = [&](const CMat &M, int c0, int rr, int nr, int &qb, int &qe) {
            qb = qe = 0;
            if (rr >= nr) return;
            if (RES || M.res) {
                qb = smi[M.rq + c0 + rr];
                qe = smi[M.rq + c0 + rr + 1];
            } else if (M.rp[c0 + rr + 1] > M.rp[c0 + rr]) {
                qb = M.rp[c0 + rr] >> 2;
                qe = (M.rp[c0 + rr + 1] + 3) >> 2;
            }
            qb += lane & ((1 << M.lg) - 1);
        };
        auto first_pass = [&](CMat &M) { lane_quads(M, M.w0, lane >> M.lg, min(32, M.nw), M.qb, M.qe); };
        first_pass(Q);
        first_pass(A);
        first_pass(AT);

        // y = M x on the own rows: the lane layout and the order of
        // k_batch_solve's cta_spmv; f(own row, row sum) on the lane that owns
        // the row.  g(8 * column) reads the source.
        //
        // The time of a product is the instructions of its longest warp, one
        // after the other (a CTA's few warps have little to overlap with), so
        // what is the same in every product of a matrix (the first pass's
        // quads, the lane of a row's sum) is kept in registers, rows in
        // shared memory need no masks, and the next quad's columns and values
        // are loaded before the current quad's entries are added.
        auto lane_sum = [&](const CMat &M, int q, int qe, int b, int e, auto &&g) -> double {
            const int gw = 1 << M.lg;
            uint2 c;
            double2 va, vb;
            auto get = [&]() {
                if (RES || M.res) {
                    c = reinterpret_cast<const uint2 *>(sm)[M.ci + q];
                    va = reinterpret_cast<const double2 *>(sm)[M.va + q];
                    vb = reinterpret_cast<const double2 *>(sm)[M.vb + q];
                } else {
                    // the packed quad, entries outside the row as in the shared-memory form
                    const int4 ci = __ldg(M.gci + q);
                    va = M.gv[2 * q];
                    vb = M.gv[2 * q + 1];
                    const unsigned k0 = (unsigned)(4 * q - b), len = (unsigned)(e - b);
                    const bool i0 = k0 < len, i1 = k0 + 1 < len, i2 = k0 + 2 < len, i3 = k0 + 3 < len;
                    c.x = 8u * (i0 ? ci.x : M.pad) | (8u * (i1 ? ci.y : M.pad)) << 16;
                    c.y = 8u * (i2 ? ci.z : M.pad) | (8u * (i3 ? ci.w : M.pad)) << 16;
                    va.x = i0 ? va.x : 0.0;
                    va.y = i1 ? va.y : 0.0;
                    vb.x = i2 ? vb.x : 0.0;
                    vb.y = i3 ? vb.y : 0.0;
                }
            };
            double s = 0.0;
            if (q < qe) {
                get();
                for (;;) {
                    const double x0 = g((int)(c.x & 0xffffu)), x1 = g((int)(c.x >> 16));
                    const double x2 = g((int)(c.y & 0xffffu)), x3 = g((int)(c.y >> 16));
                    const double v0 = va.x, v1 = va.y, v2 = vb.x, v3 = vb.y;
                    q += gw;
                    const bool more = q < qe;
                    if (more) get();
                    s = fma(v0, x0, s);
                    s = fma(v1, x1, s);
                    s = fma(v2, x2, s);
                    s = fma(v3, x3, s);
                    if (!more) break;
                }
            }
            __syncwarp();
            for (int o = gw >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            return __shfl_sync(0xffffffffu, s, M.src);
        };
        auto bounds = [&](const CMat &M, int c0, int rr, int nr, int &b, int &e) {
            b = e = 0;
            if (!RES && !M.res && rr < nr) {
                b = M.rp[c0 + rr];
                e = M.rp[c0 + rr + 1];
            }
        };
        auto prod = [&](const CMat &M, auto &&g, auto &&f) {
            for (int c0 = 0; c0 < M.nw; c0 += 32) {
                const int r0 = M.w0 + c0, nr = min(32, M.nw - c0);
                double mine = 0.0;
                int b, e;
                if (M.single) {
                    bounds(M, r0, lane >> M.lg, nr, b, e);
                    mine = lane_sum(M, M.qb, M.qe, b, e, g);
                } else {
                    const int sh = 5 - M.lg;
                    for (int p = 0; (p << sh) < nr; ++p) {
                        const int rr = (p << sh) + (lane >> M.lg);
                        int qb, qe;
                        lane_quads(M, r0, rr, nr, qb, qe);
                        bounds(M, r0, rr, nr, b, e);
                        const double v = lane_sum(M, qb, qe, b, e, g);
                        if ((lane >> sh) == p) mine = v;
                    }
                }
                if (lane < nr) f(r0 + lane, mine);
            }
        };
        // sources: a vector in shared memory; one of len entries in global
        // memory, written by other CTAs (the zero entry is not there)
        auto from = [](const double *x) {
            return [x](int c) { return *reinterpret_cast<const double *>(reinterpret_cast<const char *>(x) + c); };
        };
        auto from_global = [](const double *x, int len) {
            return [x, len](int c) { return c < 8 * len ? __ldcg(x + (c >> 3)) : 0.0; };
        };
        // the owners' loop without a product (m = 0)
        auto rows_only = [&](const CMat &M, auto &&f) {
            for (int c0 = lane; c0 < M.nw; c0 += 32) f(M.w0 + c0, 0.0);
        };
        // accumulations in the one-CTA kernel's order: the rows of each
        // virtual warp (after a product), or its strided entries
        auto fold_rows = [&](int nrow, int per, int slot, int n_v, unsigned maxmask, auto &&f) {
            for (int v = warp; v < vwc; v += NW) {
                const int gv = rank * vwc + v, w0 = min(gv * per, nrow), w1 = min(w0 + per, nrow);
                double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                for (int r = w0 + lane; r < w1; r += 32) f(r, acc);
                put(gv, slot, acc, n_v, maxmask);
            }
        };
        auto fold_strided = [&](int len, int slot, int n_v, auto &&f) {
            for (int v = warp; v < vwc; v += NW) {
                const int gv = rank * vwc + v;
                double acc[4] = {0, 0, 0, 0};
                for (int i = gv * 32 + lane; i < len; i += VT) f(i, acc);
                put(gv, slot, acc, n_v, 0u);
            }
        };
        auto bound = [](double lo, double hi) {
            const double a = isinf(lo) ? 0.0 : fabs(lo), b = isinf(hi) ? 0.0 : fabs(hi);
            return a > b ? a : b;
        };

        if (!resume) {
        // norms of the original data
        fold_rows(m, per_m, 0, 1, 1u, [&](int r, double *a) { a[0] = fmax(a[0], bound(ownm[kClMOwn * (r - mr0) + kAL], ownm[kClMOwn * (r - mr0) + kAU])); });
        fold_rows(n, per_n, 1, 1, 1u, [&](int r, double *a) { a[0] = fmax(a[0], fabs(own[kClNOwn * (r - nr0) + kC])); });
        finish(2, 3u);
        if (tid == 0) {
            S.norm_b_org = s_out[0];
            S.norm_c_org = s_out[1];
        }
        // ---- scaling: Ruiz x10 + Pock-Chambolle (reference scale.cu:332-560) --
        if (B.use_scaling) {
            auto row_abs = [&](const CMat &M, int r, bool sum) -> double {
                double acc = 0.0;
                const int b = M.rp[r], e = M.rp[r + 1];
                for (int kk = b + lane; kk < e; kk += 32) {
                    const double a = fabs(val(M, r, b, kk));
                    acc = sum ? acc + a : fmax(acc, a);
                }
                return sum ? warp_sum(acc) : warp_max(acc);
            };
            auto scale_rows = [&](const CMat &M, const double *rs, const double *cs) {
                for (int r = warp; r < M.nloc; r += NW) {
                    const double inv = 1.0 / rs[M.row0 + r];
                    const int b = M.rp[r], e = M.rp[r + 1];
                    for (int kk = b + lane; kk < e; kk += 32) {
                        double v = val(M, r, b, kk) * inv;
                        v /= cs[col(M, kk)];
                        val(M, r, b, kk) = v;
                    }
                }
            };
            for (int pass = 0; pass < 11; ++pass) {
                const bool use_sum = pass == 10;
                for (int j = warp; j < nl; j += NW) {
                    double a = m > 0 ? row_abs(AT, j, use_sum) : 0.0;
                    const double b = row_abs(Q, j, use_sum);
                    a = use_sum ? a + b : fmax(a, b);
                    put_all_warp(G1 + nr0 + j, a > 0.0 ? sqrt(a) : 1.0);
                }
                for (int r = warp; r < ml; r += NW) {
                    const double a = row_abs(A, r, use_sum);
                    put_all_warp(G3 + mr0 + r, a > 0.0 ? sqrt(a) : 1.0);
                }
                sync();
                scale_rows(Q, G1, G1);
                if (m > 0) {
                    scale_rows(A, G3, G1);
                    scale_rows(AT, G1, G3);
                }
                for (int i = tid; i < nl; i += NT) {
                    const double f = G1[nr0 + i];
                    V.col_norm[nr0 + i] *= f;
                    own[kClNOwn * i + kC] /= f;
                    own[kClNOwn * i + kL] *= f;
                    own[kClNOwn * i + kU] *= f;
                }
                for (int i = tid; i < ml; i += NT) {
                    const double f = G3[mr0 + i];
                    V.row_norm[mr0 + i] *= f;
                    ownm[kClMOwn * i + kAL] /= f;
                    ownm[kClMOwn * i + kAU] /= f;
                }
                sync();
            }
        }
        // the scaled values for the adjoint; the scaled vectors for the strided folds
        auto write_back = [&](const CMat &M) {
            if (!RES && !M.res) return;
            double *d = reinterpret_cast<double *>(M.gv);
            for (int r = warp; r < M.nloc; r += NW) {
                const int b = M.rp[r], e = M.rp[r + 1];
                for (int kk = b + lane; kk < e; kk += 32) d[kk] = val(M, r, b, kk);
            }
        };
        write_back(Q);
        write_back(A);
        write_back(AT);
        for (int i = tid; i < nl; i += NT) {
            V.c[nr0 + i] = own[kClNOwn * i + kC];
            V.l[nr0 + i] = own[kClNOwn * i + kL];
            V.u[nr0 + i] = own[kClNOwn * i + kU];
        }
        for (int i = tid; i < ml; i += NT) {
            V.AL[mr0 + i] = ownm[kClMOwn * i + kAL];
            V.AU[mr0 + i] = ownm[kClMOwn * i + kAU];
        }
        sync();
        PHASE_ADD(0);
        // ---- setup: sigma0, noC, Q diagonal, eigenvalues (control.cu:156-241)
        {
            fold_strided(m, 0, 1, [&](int i, double *a) {
                const double bm = bound(__ldcg(V.AL + i), __ldcg(V.AU + i));
                a[0] += bm * bm;
            });
            fold_strided(n, 1, 2, [&](int i, double *a) {
                const double c = __ldcg(V.c + i);
                a[0] += c * c;
                if (isinf(__ldcg(V.l + i)) && isinf(__ldcg(V.u + i))) a[1] += 1.0;
            });
            for (int v = warp; v < vwc; v += NW) {
                const int gv = rank * vwc + v;
                double mx[2] = {0.0, 0.0};
                for (int r = min(gv * per_n, n), e = min(gv * per_n + per_n, n); r < e; ++r) {
                    double d = 0.0, off = 0.0;
                    const int b = Q.rp[r - nr0], k1 = Q.rp[r - nr0 + 1];
                    for (int kk = b + lane; kk < k1; kk += 32) {
                        const double v = val(Q, r - nr0, b, kk);
                        if (col(Q, kk) == r) d += v;
                        else off = fmax(off, fabs(v));
                    }
                    d = warp_sum(d);
                    if (lane == 0) V.diag_Q[r] = d;
                    mx[0] = fmax(mx[0], off);
                    mx[1] = fmax(mx[1], fabs(d));
                }
                put(gv, 3, mx, 2, 3u);
            }
            finish(5, 0x18u);
            if (tid == 0) {
                const double nb = sqrt(s_out[0]), nc = sqrt(s_out[1]);
                S.sigma = (nb > 1e-16 && nc > 1e-16 && nb < 1e16 && nc < 1e16) ? nb / nc : 1.0;
                if (B.sigma_start && B.sigma_start[k] > 0.0) S.sigma = clampd(B.sigma_start[k], 1e-12, 1e12);
                S.noC = n > 0 && 5.0 * s_out[2] > 4.0 * (double)n;
                S.q_is_diag = s_out[3] <= 1e-15;
                S.lQ = S.q_is_diag ? s_out[4] : 0.0;
                S.lA = 0.0;
                S.n = n;
                S.m = m;
                S.obj_constant = I.obj_constant;
            }
            __syncthreads();
        }
        PHASE_ADD(1);
        // power iteration (reference src/gpu/eigs.cu:185-383): q and z in full
        // in every CTA
        auto power = [&](bool is_a, int len, double *q, double *z) -> double {
            if (len == 0) return 0.0;
            auto probe = [&](int i) { return 1.0 + ((double)i + 1.0) / ((double)len + 1.0); };
            fold_strided(len, 0, 1, [&](int i, double *a) {
                const double t = probe(i);
                a[0] += t * t;
            });
            finish(1, 0u);
            double zz = s_out[0], lambda = 1.0;
            bool q_ready = false, first = true;
            for (int it = 0; it < 5000; ++it) {
                const double qn = sqrt(zz);
                if (qn <= 1e-16) {
                    lambda = 0.0;
                    break;
                }
                if (!q_ready) {
                    const double inv = 1.0 / qn;
                    for (int i = tid; i < len; i += NT) q[i] = (first ? probe(i) : z[i]) * inv;
                }
                first = false;
                __syncthreads();
                auto to_z = [&](int r, double s) { put_all(z + (is_a ? mr0 : nr0) + r, s); };
                if (is_a) {
                    prod(AT, from(q), [&](int r, double s) { put_all(G1 + nr0 + r, s); });
                    sync();
                    prod(A, from(G1), to_z);
                } else {
                    prod(Q, from(q), to_z);
                }
                __syncthreads();
                fold_rows(len, is_a ? per_m : per_n, 0, 2, 0u, [&](int r, double *a) {
                    const double s = z[r];
                    a[0] += q[r] * s;
                    a[1] += s * s;
                });
                finish(2, 0u);
                lambda = s_out[0];
                zz = s_out[1];
                const double zn = sqrt(zz);
                q_ready = zn > 1e-16;
                const double inv_next = q_ready ? 1.0 / zn : 0.0;
                fold_strided(len, 0, 1, [&](int i, double *a) {
                    const double r = z[i] - lambda * q[i];
                    a[0] += r * r;
                });
                __syncthreads();
                if (q_ready)
                    for (int i = tid; i < len; i += NT) q[i] = z[i] * inv_next;
                finish(1, 0u);
                if (sqrt(s_out[0]) / (zn + fabs(lambda) + 1e-16) < 1e-4) break;
            }
            __syncthreads();
            return lambda < 0.0 ? 0.0 : lambda;
        };
        if (!S.q_is_diag) {
            const int q_nnz = B.q_rp[I.q_rp + n];
            const double lq = q_nnz > 0 ? power(false, n, G1, G2) : 0.0;
            if (tid == 0) S.lQ = lq * 1.05;
        }
        {
            const double la = m > 0 ? power(true, m, G3, G2) : 0.0;
            if (tid == 0) S.lA = la * 1.05;
        }
        }
        sync();
        PHASE_ADD(2);
        // ---- starting iterates ----------------------------------------------
        const bool warm = B.x_start != nullptr;
        const bool noC = S.noC, diag = S.q_is_diag;
        auto diag_factors = [&]() {
            const double sg = S.sigma;
            for (int i = tid; i < nl; i += NT) {
                const double dq = V.diag_Q[nr0 + i], inv = diag_inverse(sg, dq);
                V.fact2[nr0 + i] = inv;
                V.fact[nr0 + i] = sg * inv;
                V.fact1[nr0 + i] = diag_fact1(sg, dq, inv);
                V.fact_M[nr0 + i] = sg * sg * inv;
            }
        };
        if (!resume) {
        for (int i = tid; i < nl; i += NT) {
            const int gi = nr0 + i;
            const double xs = warm ? B.x_start[I.var + gi] * V.col_norm[gi] : 0.0;
            const double ws = warm ? B.w_start[I.var + gi] * V.col_norm[gi] : 0.0;
            own[kClNOwn * i + kX] = own[kClNOwn * i + kLx] = V.x_bar[gi] = xs;
            own[kClNOwn * i + kW] = own[kClNOwn * i + kLw] = ws;
            own[kClNOwn * i + kAty] = own[kClNOwn * i + kLaty] = own[kClNOwn * i + kQw] = own[kClNOwn * i + kXh] = 0.0;
            V.last_Qw[gi] = 0.0;
            G2[gi] = ws;
            V.ATy_bar[gi] = V.Qw_bar[gi] = V.z_bar[gi] = 0.0;
            put_all(G1 + gi, ws);
        }
        if (tid == 0) G2[n] = 0.0;  // (an entry of the power iteration when m > n)
        if (diag) diag_factors();
        for (int i = tid; i < ml; i += NT) {
            const int gi = mr0 + i;
            const double ys = warm ? B.y_start[I.row + gi] * V.row_norm[gi] : 0.0;
            ownm[kClMOwn * i + kY] = ownm[kClMOwn * i + kLy] = ownm[kClMOwn * i + kYb] = ys;
            V.y_bar[gi] = ys;
            put_all(G3 + gi, ys);
        }
        sync();
        if (warm) {
            if (m > 0) prod(AT, from(G3), [&](int i, double s) { own[kClNOwn * i + kAty] = own[kClNOwn * i + kLaty] = V.ATy_bar[nr0 + i] = s; });
            if (noC) prod(Q, from(G1), [&](int i, double s) { own[kClNOwn * i + kQw] = V.last_Qw[nr0 + i] = V.Qw_bar[nr0 + i] = s; });
        }
        if (tid == 0) {
            S.restart_flag = 0;
            S.first_restart = 1;
            S.save_gap = S.current_gap = S.last_gap = S.best_gap = INFINITY;
            S.weighted_norm = INFINITY;
            S.best_sigma = S.sigma;
            S.inner = 0;
            S.times = 0;
            S.aborted = 0;
        }
        }
        bytes_n = 8 * n;
        bytes_m = 8 * m;
        // the time-limit flag travels with the last exchange of a step
        mail_bar = noC ? kBarY : kBarW;
        ph = 0;
        for (int b = 0; b < 4; ++b) arm(b);
        __syncthreads();

        auto save_w_bar = [&]() {
            for (int i = tid; i < nl; i += NT) V.w_bar[nr0 + i] = G2[nr0 + i];
        };
        // ---- residuals (reference residuals.cu:81-183) ------------------------
        // A'y_bar is at hand from a full step on the QP path (its last
        // product); x_bar goes to every CTA through w_bar's buffer, whose own
        // entries the event saved
        auto residuals = [&](long long iter, bool have_aty) {
            for (int i = tid; i < nl; i += NT) put_all(G2 + nr0 + i, V.x_bar[nr0 + i]);
            for (int i = tid; i < ml; i += NT) V.y_bar[mr0 + i] = ownm[kClMOwn * i + kYb];
            sync();
            if (!have_aty && m > 0) prod(AT, from_global(V.y_bar, m), [&](int r, double s) { V.ATdy[nr0 + r] = s; });
            if (m > 0) prod(A, from(G2), [&](int r, double s) { V.Ax[mr0 + r] = s; });
            prod(Q, from(G2), [&](int r, double s) { own[kClNOwn * r + kXh] = s; });  // (x_hat is not live between steps)
            __syncthreads();
            fold_rows(m, per_m, 0, 3, 3u, [&](int r, double *a) {
                const double ax = V.Ax[r];
                const double proj = clampd(ax, ownm[kClMOwn * (r - mr0) + kAL], ownm[kClMOwn * (r - mr0) + kAU]);
                const double sf = V.row_norm[r];
                a[0] = fmax(a[0], fabs((proj - ax) * sf));
                a[1] = fmax(a[1], fabs(ax * sf));
                a[2] += ownm[kClMOwn * (r - mr0) + kYb] * proj;
            });
            const double *a_ty = have_aty ? V.ATy_bar : V.ATdy;
            fold_rows(n, per_n, 3, 7, 0x47u, [&](int r, double *q) {
                const double qx = own[kClNOwn * (r - nr0) + kXh];
                const double sf = V.col_norm[r];
                const double xb = V.x_bar[r], aty = m > 0 ? a_ty[r] : 0.0, c = own[kClNOwn * (r - nr0) + kC], zb = V.z_bar[r];
                const double rd = (qx + c - aty - zb) * sf;
                q[0] = fmax(q[0], fabs(rd));
                q[1] = fmax(q[1], fabs(qx * sf));
                q[2] = fmax(q[2], fabs(aty * sf));
                q[3] += c * xb;
                q[4] += xb * qx;
                q[5] += zb * xb;
                if (iter == 0) {
                    const double lo = own[kClNOwn * (r - nr0) + kL] - xb, hi = xb - own[kClNOwn * (r - nr0) + kU];
                    double vv = 0.0;
                    if (lo > 0.0) vv += lo;
                    if (hi > 0.0) vv += hi;
                    q[6] = fmax(q[6], fabs(vv * (1.0 / sf)));
                }
            });
            finish(10, 3u | (0x47u << 3));
            if (tid == 0) {
                const double *a = s_out, *q = s_out + 3;
                S.pobj = (q[3] + 0.5 * q[4]) + S.obj_constant;
                S.dobj = (-0.5 * q[4] + q[5] + a[2]) + S.obj_constant;
                S.gap = fabs(S.pobj - S.dobj) / (1.0 + fmax(fabs(S.pobj), fabs(S.dobj)));
                S.rd = q[0] / (1.0 + fmax(S.norm_c_org, fmax(q[2], q[1])));
                S.rp = m > 0 ? a[0] / (1.0 + fmax(S.norm_b_org, a[1])) : 0.0;
                if (iter == 0 && q[6] > S.rp) S.rp = q[6];
                S.kkt = fmax(S.rp, fmax(S.rd, S.gap));
            }
            __syncthreads();
        };

        const long long iter0 = resume ? R->iter : 0;
        const unsigned long long loop_t0 = globaltimer_ns();  // used by rank 0
        // the cluster's clock and the abort flag, read by one thread; it polls
        // the flag every kAbortPoll iterations and keeps a request
        bool aborted = false;
        auto over_now = [&](long long it) -> double {
            if (((int)it & (kAbortPoll - 1)) == 0 && !aborted) aborted = abort_requested(B.abort_flag);
            const double el = 1e-9 * (double)(globaltimer_ns() - (B.time_from_loop ? loop_t0 : B.t_start));
            if (el > B.time_limit || aborted) return 1.0;
            return ((int)it & (kAbortPoll - 1)) == 0 && it > iter0 && yield_now(B, I) ? 2.0 : 0.0;
        };
        const bool timekeeper = rank == 0 && tid == (NW - 1) * 32;

        // ---- one HPR step (reference iteration.cu:1386-1442) ------------------
        // s_k: what a step needs of sigma, renewed with it
        auto step_constants = [&]() {
            if (tid == 0) {
                const double sigma = S.sigma, lA = S.lA, lQ = S.lQ;
                const double f2s = 1.0 / (1.0 + sigma * lQ), f1 = lA * sigma;
                s_k[0] = f2s;
                s_k[1] = 1.0 - f2s;
                s_k[2] = sigma / (1.0 + sigma * lQ);
                s_k[3] = f1;
                s_k[4] = 1.0 / f1;
            }
        };
        auto step = [&](bool full, int mail, long long next_iter, double h1) {
            const double sigma = S.sigma, h2 = 1.0 - h1;
            const double f2s = s_k[0], f1s = s_k[1];
            auto average = [&](double now, double anchor) { return hpr::average(h2, now, h1, anchor); };
            if (noC) {
                auto upd = [&](int i, double aty) {
                    const int gi = nr0 + i;
                    const double xi = own[kClNOwn * i + kX], wi = own[kClNOwn * i + kW];
                    own[kClNOwn * i + kAty] = aty;
                    const double z_raw = xi + sigma * (-own[kClNOwn * i + kQw] + aty - own[kClNOwn * i + kC]);
                    const double xb = clampd(z_raw, own[kClNOwn * i + kL], own[kClNOwn * i + kU]);
                    const double xh = 2.0 * xb - xi;
                    const double wb = diag ? w_bar_of(V.fact1[nr0 + i], wi, V.fact2[nr0 + i], xh) : w_bar_of(f1s, wi, f2s, xh);
                    push(G2 + gi, wb, kBarWb);
                    if (full) {
                        V.x_bar[gi] = xb;
                        V.z_bar[gi] = (xb - z_raw) / sigma;
                        V.dx[gi] = xb - xi;
                        V.dw[gi] = wb - wi;
                    }
                    own[kClNOwn * i + kXh] = xh;
                    own[kClNOwn * i + kX] = average(xh, own[kClNOwn * i + kLx]);
                    own[kClNOwn * i + kW] = average(2.0 * wb - wi, own[kClNOwn * i + kLw]);
                };
                if (m > 0) prod(AT, from(G3), upd);
                else rows_only(Q, upd);
                wait(kBarWb);
                if (timekeeper) push(&s_mail[mail], over_now(next_iter), kBarY);
                prod(Q, from(G2), [&](int i, double qwb) {
                    const double qw = own[kClNOwn * i + kQw];
                    push(G1 + nr0 + i, own[kClNOwn * i + kXh] + sigma * (qw - qwb), kBarT);
                    if (full) V.Qw_bar[nr0 + i] = qwb;
                    own[kClNOwn * i + kQw] = average(2.0 * qwb - qw, V.last_Qw[nr0 + i]);
                });
                wait(kBarT);
            } else {
                prod(Q, from(G1), [&](int i, double qw) {
                    const int gi = nr0 + i;
                    const double xi = own[kClNOwn * i + kX], wi = own[kClNOwn * i + kW];
                    const double z_raw = xi + sigma * (-qw + own[kClNOwn * i + kAty] - own[kClNOwn * i + kC]);
                    const double xb = clampd(z_raw, own[kClNOwn * i + kL], own[kClNOwn * i + kU]);
                    const double xh = 2.0 * xb - xi;
                    const double wb = diag ? w_bar_of(V.fact1[nr0 + i], wi, V.fact2[nr0 + i], xh) : w_bar_of(f1s, wi, f2s, xh);
                    push(G2 + gi, wb, kBarWb);
                    own[kClNOwn * i + kQw] = qw;
                    own[kClNOwn * i + kXh] = xh;
                    if (full) {
                        V.x_bar[gi] = xb;
                        V.z_bar[gi] = (xb - z_raw) / sigma;
                        V.dx[gi] = xb - xi;
                    }
                    own[kClNOwn * i + kX] = average(xh, own[kClNOwn * i + kLx]);
                });
                wait(kBarWb);
                // (only now has every CTA seen the end of the last step, so
                // that the flag counts for this one's last exchange)
                if (timekeeper) push(&s_mail[mail], over_now(next_iter), kBarW);
                if (m > 0) {
                    prod(Q, from(G2), [&](int i, double qwb) {
                        push(G1 + nr0 + i, own[kClNOwn * i + kXh] + sigma * (own[kClNOwn * i + kQw] - qwb), kBarT);
                    });
                    wait(kBarT);
                }
            }
            if (m > 0) {
                const double f1 = s_k[3], f2 = s_k[4];
                prod(A, from(G1), [&](int i, double ax) {
                    const double yi = ownm[kClMOwn * i + kY];
                    const double s_raw = ax - f1 * yi;
                    const double sp = clampd(s_raw, ownm[kClMOwn * i + kAL], ownm[kClMOwn * i + kAU]);
                    const double yb = f2 * (sp - s_raw);
                    const double yn = average(2.0 * yb - yi, ownm[kClMOwn * i + kLy]);
                    push(G3 + mr0 + i, noC ? yn : yb, kBarY);
                    ownm[kClMOwn * i + kYb] = yb;
                    if (full) V.dy[mr0 + i] = yb - yi;
                    ownm[kClMOwn * i + kY] = yn;
                });
            }
            if (m > 0 || noC) wait(kBarY);
            if (!noC) {
                const double fs = s_k[2];
                auto w2 = [&](int i, double atyb) {
                    const int gi = nr0 + i;
                    const double f = diag ? V.fact[nr0 + i] : fs;
                    const double aty = own[kClNOwn * i + kAty], wi = own[kClNOwn * i + kW];
                    const double wbn = G2[gi] + f * (atyb - aty);
                    const double wn = average(2.0 * wbn - wi, own[kClNOwn * i + kLw]);
                    push(G1 + gi, wn, kBarW);
                    if (full) {
                        V.dw[gi] = wbn - wi;
                        G2[gi] = wbn;
                        V.ATy_bar[gi] = atyb;
                    }
                    own[kClNOwn * i + kW] = wn;
                    own[kClNOwn * i + kAty] = average(2.0 * atyb - aty, own[kClNOwn * i + kLaty]);
                };
                if (m > 0) prod(AT, from(G3), w2);
                else rows_only(Q, w2);
                wait(kBarW);
            }
            ph ^= 1;
        };

        // ---- M-norm (reference control.cu:243-332) ---------------------------
        auto m_norm = [&]() -> double {
            sync();
            prod(Q, from_global(V.dw, n), [&](int i, double v) { V.dQw[nr0 + i] = v; });
            if (m > 0) prod(AT, from_global(V.dy, m), [&](int i, double v) { V.ATdy[nr0 + i] = v; });
            sync();
            if (m > 0) prod(Q, from_global(V.ATdy, n), [&](int i, double v) { V.QATdy[nr0 + i] = v; });
            __syncthreads();
            fold_rows(n, per_n, 0, 4, 0u, [&](int i, double *a) {
                const double v = V.dQw[i], dx = V.dx[i];
                a[0] += dx * dx;
                a[1] += v * dx;
                a[2] += v * v;
                a[3] += V.dw[i] * v;
            });
            if (m > 0) {
                fold_rows(n, per_n, 4, 1, 0u, [&](int i, double *b) { b[0] += V.ATdy[i] * V.dx[i]; });
                fold_strided(m, 5, 1, [&](int i, double *b) {
                    const double d = __ldcg(V.dy + i);
                    b[0] += d * d;
                });
                fold_rows(n, per_n, 6, 3, 0u, [&](int i, double *c) {
                    const double v = V.QATdy[i], at = V.ATdy[i];
                    c[0] += V.dQw[i] * at;
                    c[1] += at * v;
                    if (diag) c[2] += (at * V.fact_M[i]) * v;
                });
            }
            finish(m > 0 ? 9 : 4, 0u);
            const double *a = s_out, *b = s_out + 4, *c3 = s_out + 6;
            return m_norm_of(S.sigma, S.lA, S.lQ, m > 0, diag, a, b, c3);
        };

        // ---- sigma update (reference control.cu:334-529) ----------------------
        auto sigma_update = [&]() {
            const double sigma_old = S.sigma, lA = S.lA, lQ = S.lQ;
            for (int i = tid; i < nl; i += NT) {
                const int gi = nr0 + i;
                V.dx[gi] = V.x_bar[gi] - own[kClNOwn * i + kLx];
                V.dw[gi] = V.w_bar[gi] - own[kClNOwn * i + kLw];
                if (m > 0) V.ATdy[gi] = V.ATy_bar[gi] - own[kClNOwn * i + kLaty];
            }
            for (int i = tid; i < ml; i += NT) V.dy[mr0 + i] = ownm[kClMOwn * i + kYb] - ownm[kClMOwn * i + kLy];
            sync();
            fold_strided(n, 0, 1, [&](int i, double *d) {
                const double dx = __ldcg(V.dx + i);
                d[0] += dx * dx;
            });
            fold_strided(m, 1, 1, [&](int i, double *d) {
                const double dy = __ldcg(V.dy + i);
                d[0] += dy * dy;
            });
            prod(Q, from_global(V.dw, n), [&](int i, double v) { V.dQw[nr0 + i] = v; });
            if (m > 0) prod(Q, from_global(V.ATdy, n), [&](int i, double v) { V.QATdy[nr0 + i] = v; });
            __syncthreads();
            fold_rows(n, per_n, 2, 3, 0u, [&](int i, double *e) {
                const double v = V.dQw[i];
                if (m > 0) e[0] += v * V.ATdy[i];
                e[1] += v * v;
                e[2] += V.dw[i] * v;
            });
            fold_rows(m > 0 ? n : 0, per_n, 5, 1, 0u, [&](int i, double *e) { e[0] += V.ATdy[i] * V.QATdy[i]; });
            finish(6, 0u);
            const double e_dx = s_out[0], e_dy = s_out[1], e0 = s_out[2], e1 = s_out[3], e2 = s_out[4], e_f = s_out[5];
            const double a = sigma_slope(lA, lQ, m > 0, diag, e_dy, e0, e1, e2), b = fmax(e_dx, 1e-12);
            const double c_term = m > 0 ? e_f : 0.0, d_term = m > 0 ? lQ : 0.0;
            double est = 0.0;
            if (diag && m > 0) {
                // golden section with a cluster-wide sum per probe
                double left = 1e-12, right = 1e12;
                const double phi = (sqrt(5.0) - 1.0) / 2.0;
                auto f = [&](double xp) {
                    fold_strided(n, 0, 1, [&](int i, double *t) {
                        t[0] += __ldcg(V.ATdy + i) * (__ldcg(V.QATdy + i) / (1.0 + xp * __ldcg(V.diag_Q + i)));
                    });
                    finish(1, 0u);
                    return a * xp + b / xp + xp * xp * s_out[0];
                };
                double x1 = right - phi * (right - left), x2 = left + phi * (right - left);
                double fa = f(x1), fb = f(x2);
                for (int it = 0; it < 200; ++it) {
                    if (fabs(right - left) <= 1e-12 * fmax(1.0, fabs(left))) break;
                    if (fa > fb) {
                        left = x1;
                        x1 = x2;
                        fa = fb;
                        x2 = left + phi * (right - left);
                        fb = f(x2);
                    } else {
                        right = x2;
                        x2 = x1;
                        fb = fa;
                        x1 = right - phi * (right - left);
                        fa = f(x1);
                    }
                }
                est = fa < fb ? x1 : x2;
            } else if (!diag && m > 0) {
                if (tid == 0) {
                    const double cc = c_term > 0.0 ? c_term : 0.0, dd = d_term > 0.0 ? d_term : 0.0;
                    double left = 1e-12, right = 1e12;
                    const double ip = (sqrt(5.0) - 1.0) / 2.0, ip2 = (3.0 - sqrt(5.0)) / 2.0;
                    auto f = [&](double xp) { return a * xp + b / xp + cc * xp * xp / (1.0 + dd * xp); };
                    double x1 = left + ip2 * (right - left), x2 = left + ip * (right - left);
                    double fa = f(x1), fb = f(x2);
                    for (int it = 0; it < 256; ++it) {
                        if (fabs(right - left) <= 1e-13 * fmax(1.0, fmax(fabs(left), fabs(right)))) break;
                        if (fa > fb) {
                            left = x1;
                            x1 = x2;
                            fa = fb;
                            x2 = left + ip * (right - left);
                            fb = f(x2);
                        } else {
                            right = x2;
                            x2 = x1;
                            fb = fa;
                            x1 = left + ip2 * (right - left);
                            fa = f(x1);
                        }
                    }
                    est = 0.5 * (left + right);
                }
            } else {
                est = sqrt(b / a);
            }
            if (tid == 0) {
                est = clampd(est, 1e-12, 1e12);
                const double fact =
                    (S.best_gap > 0.0 && isfinite(S.best_gap)) ? exp(-0.05 * (S.current_gap / S.best_gap)) : 1.0;
                const double best = log(S.best_sigma > 0.0 ? S.best_sigma : sigma_old);
                const double cand = exp(two_products(1.0 - fact, best, fact, log(est)));
                double kappa = 1.0;
                const double t1 = fmax(fmin(S.rd, S.rp), fmin(S.gap, S.current_gap));
                if (t1 <= 9e-10 && S.rp > 0.0) {
                    const double ratio = S.rd / S.rp;
                    kappa = t1 > 5e-10 ? clampd(sqrt(ratio), 1e-2, 100.0) : clampd(ratio, 1e-2, 100.0);
                }
                S.sigma = clampd(kappa * cand, 1e-12, 1e12);
                S.scal[0] = sigma_old;
            }
            step_constants();
            __syncthreads();
            if (diag && fabs(S.sigma - S.scal[0]) > 1e-15) {
                diag_factors();
                __syncthreads();
            }
        };

        auto restart_apply = [&]() {
            for (int i = tid; i < nl; i += NT) {
                const int gi = nr0 + i;
                const double xb = V.x_bar[gi], wb = V.w_bar[gi];
                own[kClNOwn * i + kX] = own[kClNOwn * i + kLx] = xb;
                own[kClNOwn * i + kW] = own[kClNOwn * i + kLw] = wb;
                put_all(G1 + gi, wb);
                if (noC) own[kClNOwn * i + kQw] = V.last_Qw[nr0 + i] = V.Qw_bar[gi];
            }
            for (int i = tid; i < ml; i += NT) {
                const double yb = ownm[kClMOwn * i + kYb];
                ownm[kClMOwn * i + kY] = ownm[kClMOwn * i + kLy] = yb;
                if (noC) put_all(G3 + mr0 + i, yb);
            }
            if (m > 0)
                prod(AT, from_global(V.y_bar, m), [&](int i, double s) { V.ATy_bar[nr0 + i] = own[kClNOwn * i + kAty] = own[kClNOwn * i + kLaty] = s; });
            if (tid == 0) {
                S.last_gap = S.current_gap;
                S.save_gap = INFINITY;
                S.times += 1;
            }
            sync();
        };

        // ---- outer loop (reference solver_backend.c:432-513) ------------------
        auto log_record = [&](long long it) {
            if (!B.log_buf || k != 0 || rank != 0) return;
            const int slot = *B.log_count;
            if (slot >= B.log_cap) return;
            double *r = B.log_buf + (size_t)slot * kLogFields;
            r[0] = (double)it;
            r[1] = S.rp;
            r[2] = S.rd;
            r[3] = S.pobj;
            r[4] = S.dobj;
            r[5] = S.gap;
            r[6] = S.sigma;
            r[7] = 1e-9 * (double)(globaltimer_ns() - loop_t0);
            *B.log_count = slot + 1;
        };
        auto milestones = [&](long long it) {
            if (rank != 0) return;
            const double el = 1e-9 * (double)(globaltimer_ns() - loop_t0);
            if (!S.got4 && S.kkt < 1e-4) {
                S.got4 = 1;
                if (B.iter4_out) {
                    B.iter4_out[k] = it;
                    B.time4_out[k] = el;
                }
            }
            if (!S.got6 && S.kkt < 1e-6) {
                S.got6 = 1;
                if (B.iter6_out) {
                    B.iter6_out[k] = it;
                    B.time6_out[k] = el;
                }
            }
        };
        step_constants();
        if (!resume) {
            save_w_bar();
            residuals(0, false);
            if (tid == 0) {
                S.got4 = S.got6 = 0;
                if (B.iter4_out && rank == 0) B.iter4_out[k] = B.iter6_out[k] = -1;
                milestones(0);
                log_record(0);
            }
        }
        if (timekeeper) put_all(&s_mail[((int)iter0 + 3) & 3], over_now(iter0));
        sync();
        // the iterations after `it` that lie on the check or print grid
        const long long ci = B.check_iter, pf = B.print_frequency;
        auto next_mult = [](long long it, long long d) { return (it / d + 1) * d; };
        auto next_checked = [&](long long it) -> long long {
            long long nx = LLONG_MAX;
            if (ci > 0) nx = min(nx, next_mult(it, ci));
            if (pf == -1) nx = min(nx, next_mult(it, (long long)adaptive_step_d(it)));
            if (pf > 0) nx = min(nx, next_mult(it, pf));
            return nx;
        };
        long long iter = iter0, inner = resume ? S.inner : 0, checked = next_checked(iter0);
        long long at_ci = ci > 0 ? next_mult(iter0, ci) : LLONG_MAX;
        // iter lies on the check or print grid
        bool on_grid = iter0 > 0 && ((ci > 0 && divides(iter0, ci)) || (pf == -1 && on_print_grid(iter0)) ||
                                     (pf > 0 && divides(iter0, pf)));
        bool handed_over = false;
        // Between two events (a check, a print, the iteration limit) a step
        // is all there is: `left` steps to go, their Halpern weights
        // 1 / (inner + 2) in s_h (divided here, off the steps' path).
        int left = 0, h_at = 0;
        auto plan = [&]() {
            __syncthreads();
            for (int t = tid; t < kClHalpern; t += NT) s_h[t] = 1.0 / ((double)(inner + t) + 2.0);
            h_at = 0;
            const long long to = min(min(checked, B.max_iter > iter ? B.max_iter : LLONG_MAX) - iter, (long long)kClHalpern);
            left = (int)to;
            __syncthreads();
        };
        for (;; ++iter) {
            const double mail = s_mail[((int)iter + 3) & 3];
            const bool over = mail == 1.0;
            if (mail == 2.0) {
                handed_over = true;
                break;
            }
            int restart = 0;
            if (left == 0 || over) {
              if (iter == 0 || on_grid || over || iter == B.max_iter) {
                if (tid == 0) {
                    int print_yes = 0;
                    if (iter > 0) {
                        if (pf == -1 && (on_print_grid(iter) || iter == B.max_iter || over)) print_yes = 1;
                        if (pf > 0 && (divides(iter, pf) || iter == B.max_iter || over)) print_yes = 1;
                    }
                    S.do_res = iter > 0 && ((ci > 0 && divides(iter, ci)) || print_yes);
                    S.print_yes = print_yes;
                }
                __syncthreads();
                if (iter > 0) save_w_bar();  // (iteration 0's residuals have taken w_bar's buffer)
                PHASE_ADD(3);
                if (S.do_res) residuals(iter, on_grid && !noC);
                PHASE_ADD(4);
                if (tid == 0) {
                    if (S.do_res) milestones(iter);
                    int fs;
                    // (a warm start is not accepted before the first step)
                    if (S.kkt < B.stoptol && !(warm && iter == 0)) fs = 6;
                    else if (iter == B.max_iter) fs = 4;
                    else if (over) fs = 5;
                    else fs = 7;
                    S.final_status = fs;
                    // restart_check (src/cpu/control.c:231-282)
                    S.restart_flag = 0;
                    if (ci > 0) {
                        if (S.first_restart) {
                            if (iter == ci) {
                                S.first_restart = 0;
                                S.restart_flag = 1;
                                S.weighted_norm = S.current_gap;
                                S.best_gap = S.current_gap;
                                S.best_sigma = S.sigma;
                            }
                        } else if (divides(iter, ci)) {
                            if (S.current_gap < 0.0) S.current_gap = 1e-6;
                            if (S.current_gap <= 0.2 * S.last_gap) S.restart_flag = 1;
                            if (S.current_gap <= 0.8 * S.last_gap && S.current_gap > S.save_gap) S.restart_flag = 2;
                            const double f =
                                (S.weighted_norm > 0.0 && S.current_gap / S.weighted_norm > 1e-1) ? 0.5 : 0.2;
                            if ((double)inner >= f * (double)iter) S.restart_flag = 3;
                            if (S.best_gap > S.current_gap) {
                                S.best_gap = S.current_gap;
                                S.best_sigma = S.sigma;
                            }
                            S.save_gap = S.current_gap;
                        }
                    }
                }
                __syncthreads();
                restart = S.restart_flag;
                if (restart > 0) {
                    sigma_update();
                    restart_apply();
                    inner = 0;
                }
                PHASE_ADD(6);
                if (tid == 0 && (S.print_yes || S.final_status != 7)) log_record(iter);
                if (S.final_status != 7) break;
              }
              plan();
            }
            --left;
            on_grid = left == 0 && iter + 1 == checked;
            step(on_grid || restart > 0, (int)iter & 3, iter + 1, s_h[h_at++]);
            bool at_check = false;
            if (on_grid) {
                at_check = checked == at_ci;
                if (at_check) at_ci += ci;
                checked = next_checked(checked);
            }
            if (MULTI && *(volatile int *)&s_dead) break;
            if (restart > 0 || at_check) {
                PHASE_ADD(3);
                const double g = m_norm();
                if (tid == 0) {
                    if (restart > 0) S.last_gap = g;
                    if (at_check) S.current_gap = g;
                }
                PHASE_ADD(5);
                if (!isfinite(g)) {
                    if (tid == 0) S.final_status = 1;
                    save_w_bar();
                    break;
                }
            }
            ++inner;
        }
        __syncthreads();
        if (handed_over) {
            for (int i = tid; i < nl; i += NT) {
                const int gi = nr0 + i;
                const double *o = own + kClNOwn * i;
                V.x[gi] = o[kX];
                V.w[gi] = o[kW];
                V.last_x[gi] = o[kLx];
                V.last_w[gi] = o[kLw];
                V.ATy[gi] = o[kAty];
                V.last_ATy[gi] = o[kLaty];
                V.Qw[gi] = o[kQw];
                V.w_bar[gi] = G2[gi];
            }
            for (int i = tid; i < ml; i += NT) {
                const int gi = mr0 + i;
                const double *o = ownm + kClMOwn * i;
                V.y[gi] = o[kY];
                V.last_y[gi] = o[kLy];
                V.y_bar[gi] = o[kYb];
            }
            if (tid == 0 && rank == 0) {
                BResume *r = B.resume_out + atomicAdd(B.resume_count, 1ull);
                S.inner = inner;
                r->inst = k;
                r->slot = slot;
                r->iter = iter;
                r->t0 = inst_t0;
                r->S = S;
            }
            sync();
            break;
        }

        // ---- output (reference workspace.cu:427-511) ---------------------------
        for (int i = tid; i < nl; i += NT) {
            const int gi = nr0 + i;
            const double cn = V.col_norm[gi];
            B.x[I.var + gi] = V.x_bar[gi] / cn;
            B.w[I.var + gi] = V.w_bar[gi] / cn;
            B.z[I.var + gi] = V.z_bar[gi] * cn;
            if (B.active_x) B.active_x[I.var + gi] = V.z_bar[gi] != 0.0;
            B.col_norm_out[I.var + gi] = cn;
        }
        for (int i = tid; i < ml; i += NT) {
            const int gi = mr0 + i;
            const double yb = ownm[kClMOwn * i + kYb];
            B.y[I.row + gi] = yb / V.row_norm[gi];
            if (B.active_r) B.active_r[I.row + gi] = yb != 0.0;
            B.row_norm_out[I.row + gi] = V.row_norm[gi];
        }
        if (B.phase_clk && tid == 0) B.phase_clk[blockIdx.x * 8 + 7] += (unsigned long long)(clock64() - _ptot);
        if (tid == 0 && rank == 0) {
            B.status[k] = s_dead ? 3 : S.final_status;  // 3: a wait gave up (never expected)
            B.iters[k] = iter;
            B.pobj[k] = S.pobj;
            B.resid[k] = S.kkt;
            B.gap[k] = S.gap;
            B.restarts[k] = (int)S.times;
            B.sigma_out[k] = S.sigma;
            B.seconds_out[k] = 1e-9 * (double)(globaltimer_ns() - inst_t0);
            if (B.loop_seconds_out) B.loop_seconds_out[k] = 1e-9 * (double)(globaltimer_ns() - loop_t0);
            atomicAdd(B.finished, 1ull);
        }
        sync();
        if (MULTI && s_dead) break;
    }
    sync();
}

template <int C>
const void *cluster_kernel(bool resident)
{
    return resident ? (const void *)k_cluster_solve<C, true, cluster_threads(C, true)>
                    : (const void *)k_cluster_solve<C, false, cluster_threads(C, false)>;
}

template <int C>
cudaError_t cluster_launch(bool resident, const cudaLaunchConfig_t &cfg, const ClusterArgs &P)
{
    return resident ? cudaLaunchKernelEx(&cfg, k_cluster_solve<C, true, cluster_threads(C, true)>, P)
                    : cudaLaunchKernelEx(&cfg, k_cluster_solve<C, false, cluster_threads(C, false)>, P);
}

}  // namespace hpr
