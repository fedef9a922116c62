// ccd.cu -- the one-fit persistent CCD: a fit's whole coordinate loop, its
// convergence test included, in one launch (lr, pr, clr, cpr).
//
// CyclicCoordinateDescent::findMode (src/cyclops/CyclicCoordinateDescent.cpp
// :909-1216) is one serial chain of coordinate steps, so what bounds it is
// the latency of a step: the entries' row state, exp() and a division, a sum
// over the threads, the step's division, and the write of the row state.
// A step has no work for more than a few SMs, and a kernel boundary alone
// costs as much as a whole step (three launches a coordinate measured 9 us;
// here a step of a 100-entry column is well under 1 us).  So:
//  * a fit is one thread-block cluster of C CTAs that split the rows; C is 1
//    while a column has few entries per CTA, and the cluster's (gradient,
//    Hessian) sums cross CTAs through distributed shared memory by st.async,
//    which arrives on the receiver's mbarrier (see ccd_shape for the rule);
//  * the linear predictors of a CTA's rows live in shared memory for the
//    launch when they fit, else in global memory through L1 (every access is
//    to the CTA's own rows); exp(xb) is recomputed, never stored;
//  * a column's first kR entries per thread stay in registers from the
//    gradient to the update, and the next column's row ids and values load
//    while this one's sums cross the CTA;
//  * every thread computes the coordinate step from the same sums in the
//    same order, so nothing is broadcast and no second exchange is needed.
// Independent fits are independent clusters of one launch.
#include "ccd.cuh"

#include <cooperative_groups.h>
#include <math_constants.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <type_traits>

#include "mbar.cuh"
#include "row_terms.cuh"

namespace cg = cooperative_groups;

namespace cyc {

namespace {

constexpr int kR = 2;            // entries of a column a thread keeps in registers
constexpr int kU = 4;            // further entries a thread has in flight
constexpr int kCh = 128;         // coordinates staged at a time
constexpr int kWarps = kCcdThreads / 32;
constexpr int kRunRounds = 8;    // rounds of a warp over a column of a run

// the row's mean under the model; a logistic row whose exp(xb) overflows is NaN
// when `strict`, as exb / (1 + exb) is in the per-coordinate engine
template <class T, int MODEL>
__device__ __forceinline__ T fit_mean(T v, bool strict) {
    if constexpr (MODEL == CYC_LR && sizeof(T) == 8) {
        const double a = strict && v > 709.782712893384 ? CUDART_NAN : -v;
        return 1.0 / (1.0 + exp(a));
    } else {
        return row_mean<T, MODEL>(v);
    }
}

template <class T, int WM>
struct RowWeight {
    const T* w;
    const signed char* fold;
    int held;
    __device__ __forceinline__ T by_fold(int v) const { return v != held ? T(1) : T(0); }
    __device__ __forceinline__ T operator()(int k) const {
        if (WM == 0) return T(1);
        if (WM == 1) return by_fold((int)__ldg(fold + k));
        return __ldg(w + k);
    }
};

// a column of the current chunk, in this CTA's rows
struct ColMeta {
    const int* ci;       // row ids of its entries, null for dense columns (entry i is row r0 + i)
    const double* cv;    // values, null for indicators
    const int* es;       // strata of its entries (grouped models)
    const signed char* ef;   // fold ids of its entries (CV folds)
    int n;               // entries
    int pt;              // prior type
};

// what a column's step needs besides its sums, prepared when the chunk is
// staged so that selections and one division are left after the sums arrive
struct ColStep {
    double beta, bound, xjy;
    double pre, iv, lam;     // added to g, added to h, the Laplace rate (0: another prior)
    int s;                   // sign of beta (2: not a Laplace prior)
};

// a barrier of a team's threads, and one that only waits or only arrives
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// T: state type.  MODEL: cyc_model.  WM: row weights (0 ones, 1 CV folds, 2 a
// vector).  SM: the linear predictors of the CTA's rows are in shared memory.
//
// TEAMS = 2 (independent rows): two teams of NT threads take the columns in
// turn.  While one sums its column's terms, takes the step and writes the rows,
// the other loads the next column's rows and forms their terms from the
// predictors as they are; once the first team's rows are written it reads its
// predictors again and redoes the terms of those that changed.  Every sum thus
// sees exactly the state the serial loop would show it, and the loads, exp()
// and a division are off the chain except for rows that two columns in turn
// share: 10k rows x 1,000 columns of 100 entries 30.6 -> 26.9 ms, 100k rows with
// dense and Zipf columns 27.7 -> 25.2.  One team takes long columns better
// (twice the threads a column: 160 CV fits of 50k rows 19 ms, 28 with two), and
// grouped models always: a row there depends on its stratum's denominator,
// which the column before changes much more often (20k matched rows: 7.1 ms
// with one team, 9.2 with two).
//
// TEAMS = 0 (independent rows, one CTA): runs of short columns that share no row
// (ccd_runs) are taken at once, a warp a column: each sees the state that the
// serial loop would show it, and a run costs one barrier.  The other columns go
// as with one team.  63,000 columns of 3.5 entries over 3k rows: 0.16 us a column
// against 0.65; 25,000 of 162 over 705k rows 0.47 against 0.97.
//
// A column's entries are dealt to the team's threads in rounds of NT; up to kR
// rounds stay in registers from the gradient to the update.  The code of a
// round is straight-line (one round and kR rounds as separate instances): with
// one or two warps per scheduler the instructions of a step are latency too.
template <class T, int MODEL, int WM, bool SM, int TEAMS>
__global__ void __launch_bounds__(kCcdThreads, 1) k_ccd(const CcdArgs A) {
    constexpr bool kGrouped = (MODEL == CYC_CLR || MODEL == CYC_CPR);
    constexpr unsigned full = 0xffffffffu;
    cg::cluster_group cluster = cg::this_cluster();
    const int C = A.C;
    const int rank = C > 1 ? (int)cluster.block_rank() : 0;
    const int f = blockIdx.x / C;
    constexpr bool kRuns = TEAMS == 0;
    constexpr int kTeams = kRuns ? 1 : TEAMS;
    const int NT = blockDim.x / kTeams, NW = NT >> 5;
    const int lane = threadIdx.x & 31;
    const int team = threadIdx.x >= NT, tid = threadIdx.x - team * NT, warp = tid >> 5;
    if (A.active && !A.active[f]) {              // the whole cluster leaves
        if (rank == 0 && threadIdx.x == 0) { A.out_iter[f] = 0; A.out_flag[f] = CYC_SUCCESS; }
        return;
    }
    const int r0 = A.rpart[rank], r1 = A.rpart[rank + 1], nr = r1 - r0;
    // this CTA's rows; row ids are made relative to r0
    T* const xg = (T*)A.xb + (size_t)f * A.K + r0;
    const RowWeight<T, WM> weight{WM == 2 ? (const T*)A.w + (size_t)f * A.K + r0 : nullptr,
                                  WM == 1 ? A.fold + r0 : nullptr, WM == 1 ? A.fitfold[f] : 0};
    double* const dg = kGrouped ? A.denom + (size_t)f * A.S : nullptr;
    const double* const ng = kGrouped ? A.nw + (size_t)f * A.S : nullptr;
    const size_t fj = (size_t)f * A.J;
    const double var = A.variance[f];
    const double lam = sqrt(2.0 / var);          // LaplacePrior rate, CovariatePrior.h:282-292
    const double ivar = 1.0 / var;
    const bool strict = A.strict != 0;

    // by parity of the column (the two teams'): the warps' sums, the CTAs' sums
    // with their arrival, and the cluster's; [2] are the whole CTA's (the objective)
    __shared__ double2 s_part[3][kWarps];
    __shared__ __align__(16) double2 s_cl[3][kCcdCluster];
    __shared__ __align__(8) unsigned long long s_mb[3];
    __shared__ double2 s_all[3];
    __shared__ int s_dead;                       // a wait for the peers ran out
    __shared__ ColMeta c_m[kCh + 2];             // two empty columns after the last
    __shared__ ColStep c_s[kCh];
    __shared__ double c_ob[kCh], c_oh[kCh];
    __shared__ int c_j[kCh], c_up[kCh];
    __shared__ unsigned char c_len[kRuns ? kCh : 1];   // runs by place
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    T* const sx = reinterpret_cast<T*>(dyn_smem);
    auto get = [&](int k) -> T { return SM ? sx[k] : xg[k]; };
    auto put = [&](int k, T v) {
        if (SM) sx[k] = v;
        else xg[k] = v;
    };
    if (SM)
        for (int i = threadIdx.x; i < nr; i += blockDim.x) sx[i] = xg[i];
    if (threadIdx.x == 0) {
        s_dead = 0;
        for (int i = 0; i < 3; ++i) mbar_init(smem_addr(&s_mb[i]));
        mbar_init_fence();
    }
    if (C > 1) cluster.sync();
    else __syncthreads();

    // (a, b) summed over the cluster's threads of the column's team (which 0, 1)
    // or over all of them (which 2), the same in every one.  Warp sums by shuffles (a in the
    // lower half-warp, b in the upper), then over the warps, then over the CTAs,
    // in fixed orders.
    int phases = 0;                              // of the next exchange (bit `which`)
    bool gone = false;                           // this thread's wait for the peers ran out
    auto combine = [&](double& a, double& b, int which) {
        const int w = which == 2 ? (int)threadIdx.x >> 5 : warp, nw = which == 2 ? kTeams * NW : NW;
        auto sync = [&]() {
            if (which == 2) __syncthreads();
            else bar_sync(1 + team, NT);
        };
        {
            const bool up = (lane & 16) != 0;
            double v = up ? b : a;
            v += __shfl_xor_sync(full, up ? a : b, 16);
            v += __shfl_xor_sync(full, v, 8);
            v += __shfl_xor_sync(full, v, 4);
            v += __shfl_xor_sync(full, v, 2);
            v += __shfl_xor_sync(full, v, 1);
            if ((lane & 15) == 0) (&s_part[which][w].x)[lane >> 4] = v;
        }
        sync();
        auto total = [&](const double2* src, int n) {
            double2 t[4] = {};
            #pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i < n) t[i] = src[i];
            if (n > 4) {
                #pragma unroll
                for (int i = 4; i < kCcdCluster; ++i)
                    if (i < n) { t[i & 3].x += src[i].x; t[i & 3].y += src[i].y; }
            }
            a = (t[0].x + t[1].x) + (t[2].x + t[3].x);
            b = (t[0].y + t[1].y) + (t[2].y + t[3].y);
        };
        if (C == 1) {
            total(s_part[which], nw);
            return;
        }
        // a peer writes this slot again only after the exchange of the column
        // between, which needs this CTA's sums of that column, and those wait for
        // this column's update: after this reading
        if (w == 0) {
            const unsigned mb = smem_addr(&s_mb[which]);
            total(s_part[which], nw);
            // a warp whose wait ran out exchanges nothing more: its peers' next
            // waits run out too, and all leave at the end of the cycle (agree)
            if (!gone) {
                if (lane == 0) mbar_expect(mb, 16 * C);
                if (lane < C) push16(peer_addr(smem_addr(&s_cl[which][rank]), lane), peer_addr(mb, lane), a, b);
                if (!mbar_wait(mb, (phases >> which) & 1, A.wait.of(rank))) { s_dead = 1; gone = true; }
            }
            total(s_cl[which], C);
            if (lane == 0) s_all[which] = make_double2(a, b);
        }
        sync();
        a = s_all[which].x;
        b = s_all[which].y;
        phases ^= 1 << which;
    };

    // the convergence objective (getGradientObjective, getLogLikelihood, with
    // the log prior for Lange; 0 for ONE_STEP), or the Zhang-Oles criterion
    // (computeZhangOlesConvergenceCriterion, CyclicCoordinateDescent.cpp
    // :560-579, renewing xb_save), the same in every thread
    auto objective = [&]() -> double {
        if (A.conv == CYC_CONV_ONE_STEP) return 0.0;
        double a = 0.0, b = 0.0;
        if (A.conv == CYC_CONV_ZHANG_OLES) {
            T* save = (T*)A.xb_save + (size_t)f * A.K + r0;
            for (int k = threadIdx.x; k < nr; k += blockDim.x) {
                const double v = (double)get(k), w = (double)weight(k);
                a += fabs(v - (double)save[k]) * w;
                b += fabs(v) * w;
                save[k] = get(k);
            }
        } else {
            const bool use_ll = A.conv != CYC_CONV_GRADIENT;
            #pragma unroll 4
            for (int k = threadIdx.x; k < nr; k += blockDim.x) {
                const double v = (double)get(k), wt = (double)weight(k), yk = A.y[r0 + k];
                if (!use_ll) {
                    a += v * yk * wt;
                } else {
                    double c = (int)yk * v * wt;                    // logLikeNumeratorContrib(int, RealType)
                    if (MODEL == CYC_LR) c -= wt * log(1.0 + exp(v));
                    if (MODEL == CYC_PR) c -= wt * exp(v);
                    a += c;
                }
            }
            if (use_ll && kGrouped && nr > 0) {
                const int s0 = A.strat[r0], s1 = r1 >= A.K ? A.S : A.strat[r1];
                for (int s = s0 + threadIdx.x; s < s1; s += blockDim.x) a -= ng[s] * log(dg[s]);
            }
            if (A.conv == CYC_CONV_LANGE && rank == 0)
                for (int j = threadIdx.x; j < A.J; j += blockDim.x) b += log_density(A.ptype[j], var, A.beta[fj + j]);
        }
        combine(a, b, 2);
        if (A.conv == CYC_CONV_ZHANG_OLES) return a / (1.0 + b);
        if (A.conv != CYC_CONV_GRADIENT && (MODEL == CYC_PR || MODEL == CYC_CPR)) a += A.llfixed[f];
        return A.conv == CYC_CONV_LANGE ? a + b : a;
    };

    // ccdUpdateBeta (:1394-1413) with the priors' getDelta (as prior_delta_rate)
    auto step = [&](const ColStep& p, double g, double h) -> double {
        if (h < 0.0) { g = 0.0; h = 0.0; }                          // :1407-1410
        const double base = g + p.pre, up = base + p.lam, down = base - p.lam;
        const double zero = down > 0 ? down : (up < 0 ? up : 0.0);
        const double num = p.s == 0 ? zero : (p.s < 0 ? down : up);
        double delta = -num / (h + p.iv);
        if (p.s == 0) delta = (num != 0.0 && delta == delta) ? delta : 0.0;
        else if (p.s != 2 && sgn(p.beta + delta) != p.s) delta = -p.beta;
        if (delta < -p.bound) delta = -p.bound;                     // applyBounds :1503-1520
        else if (delta > p.bound) delta = p.bound;
        return delta;
    };
    // whether any CTA of the cluster lost the others, the same in every thread of
    // them all: they stop together, and none leaves while another may store to it
    auto agree = [&]() -> bool {
        if (C > 1) {
            if (threadIdx.x == 0 && *(volatile int*)&s_dead)
                for (int r = 0; r < C; ++r) *cluster.map_shared_rank(&s_dead, r) = 1;
            cluster.sync();
        }
        return *(volatile int*)&s_dead != 0;
    };
    auto next_bound = [](double bound, double delta) { return std_max(std_max(fabs(delta) * 2, bound / 2), 1E-3); };

    double last = A.conv == CYC_CONV_ZHANG_OLES ? 0.0 : objective();   // findMode :949-953
    const int* cols = A.cols + (size_t)f * A.cols_stride;
    const int ncols = A.ncols[(size_t)f * A.ncols_stride];
    int it = 0, flag = CYC_SUCCESS;
    int off = 0;                                 // parity of the chunk's first column (and its team)
    for (;;) {
        for (int base = 0; base < ncols; base += kCh) {
            const int jn = min(kCh, ncols - base);
            __syncthreads();                     // the last chunk's arrays have been read
            if (threadIdx.x < 2) c_m[jn + threadIdx.x] = ColMeta{A.idx, nullptr, A.strat, A.fold, 0, 0};
            for (int q = threadIdx.x; q < jn; q += blockDim.x) {
                const int j = cols[base + q];
                const int fm = A.fmt[j];
                const bool dn = (fm == CYC_DENSE || fm == CYC_INTERCEPT);
                const int e0 = dn ? r0 : A.split[j * (C + 1) + rank];
                const int e1 = dn ? r1 : A.split[j * (C + 1) + rank + 1];
                ColMeta m;
                m.ci = dn ? nullptr : A.idx + A.col_ptr[j] + e0;
                m.cv = (fm == CYC_SPARSE || fm == CYC_DENSE) ? A.val + A.val_ptr[j] + e0 : nullptr;
                m.es = !kGrouped ? nullptr : (dn ? A.strat + r0 : A.entry_strat + A.col_ptr[j] + e0);
                m.ef = WM != 1 ? nullptr : (dn ? A.fold + r0 : A.entry_fold + A.col_ptr[j] + e0);
                m.n = e1 - e0;
                m.pt = A.ptype[j];
                c_m[q] = m;
                c_j[q] = j;
                const double beta = A.beta[fj + j];
                ColStep p{beta, A.hdelta[fj + j], A.xjy[fj + j], 0.0, 0.0, 0.0, 2};
                if (m.pt == CYC_PRIOR_NORMAL) {
                    p.pre = beta / var;
                    p.iv = ivar;
                } else if (m.pt == CYC_PRIOR_LAPLACE) {
                    p.lam = lam;
                    p.s = sgn(beta);
                }
                c_s[q] = p;
                if (kRuns) c_len[q] = A.runs[base + q];
            }
            __syncthreads();
            // the team's next column and its first kR rounds, as loaded (nothing
            // here waits for a load): row ids (-1: no entry), values, fold ids,
            // and for grouped models the strata of the entry and of its
            // neighbours (-1: none)
            ColMeta nm = c_m[0];
            int nk[kR], nf[kR], ns[kR], np[kR], nn[kR];
            double nx[kR];
            auto fetch = [&](int r) {
                const int i = tid + r * NT;
                nk[r] = ns[r] = np[r] = nn[r] = -1;
                nx[r] = 1.0;
                nf[r] = 0;
                if (i < nm.n) {
                    if (WM == 1) nf[r] = (int)__ldg(nm.ef + i);
                    if (nm.ci) nk[r] = __ldg(nm.ci + i);
                    else nk[r] = r0 + i;
                    if (nm.cv) nx[r] = __ldg(nm.cv + i);
                    if (kGrouped) {
                        ns[r] = __ldg(nm.es + i);
                        if (i > 0) np[r] = __ldg(nm.es + i - 1);
                        if (i + 1 < nm.n) nn[r] = __ldg(nm.es + i + 1);
                    }
                }
            };
            int nq = -1;                         // the column loaded (runs)
            auto prefetch = [&](int q) {
                nm = c_m[q];
                nq = q;
                fetch(0);
                if (nm.n > NT) {
                    #pragma unroll
                    for (int r = 1; r < kR; ++r) fetch(r);
                }
            };
            // a run: this warp's column of it, as loaded
            int rk[kRunRounds], rf[kRunRounds], rq = -1;
            double rx[kRunRounds];
            auto load_run = [&](int q) {
                rq = q;
                const int L = q < jn ? c_len[kRuns ? q : 0] : 0;
                const bool mine = L > 1 && warp < L;
                const ColMeta m = c_m[mine ? q + warp : jn];
                #pragma unroll
                for (int r = 0; r < kRunRounds; ++r) {
                    const int i = lane + 32 * r;
                    rk[r] = -1;
                    rx[r] = 1.0;
                    rf[r] = 0;
                    if (i < m.n) {
                        rk[r] = __ldg(m.ci + i);
                        if (m.cv) rx[r] = __ldg(m.cv + i);
                        if (WM == 1) rf[r] = (int)__ldg(m.ef + i);
                    }
                }
            };
            auto run = [&](int q, int L) {
                if (rq != q) load_run(q);
                int kk[kRunRounds], ff[kRunRounds];
                double x8[kRunRounds];
                #pragma unroll
                for (int r = 0; r < kRunRounds; ++r) { kk[r] = rk[r] - r0; x8[r] = rx[r]; ff[r] = rf[r]; }
                load_run(q + L);
                auto column = [&](auto rounds) {
                    constexpr int R = decltype(rounds)::value;
                    const ColStep p = c_s[q + warp];
                    const bool ind = c_m[q + warp].cv == nullptr;
                    T vv[R], xx[R];
                    Kahan<T> ag, ah;
                    #pragma unroll
                    for (int r = 0; r < R; ++r) {
                        xx[r] = (T)x8[r];
                        vv[r] = kk[r] >= 0 ? get(kk[r]) : T(0);
                    }
                    #pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const T w = kk[r] < 0 ? T(0) : (WM == 1 ? weight.by_fold(ff[r]) : weight(kk[r]));
                        const bool on = WM == 2 && strict ? kk[r] >= 0 : w != T(0);
                        T gi, hi;
                        mean_terms<T, MODEL>(fit_mean<T, MODEL>(vv[r], strict), xx[r], WM == 2 ? w : T(1), ind, gi, hi);
                        ag.add(on ? gi : T(0));
                        ah.add(on ? hi : T(0));
                    }
                    const bool up = (lane & 16) != 0;
                    const double a = ag.value(), b = ah.value();
                    double v = up ? b : a;
                    v += __shfl_xor_sync(full, up ? a : b, 16);
                    v += __shfl_xor_sync(full, v, 8);
                    v += __shfl_xor_sync(full, v, 4);
                    v += __shfl_xor_sync(full, v, 2);
                    v += __shfl_xor_sync(full, v, 1);
                    const double g = __shfl_sync(full, v, 0), h = __shfl_sync(full, v, 16);
                    const double dl = step(p, g - p.xjy, h);
                    if (lane == 0) {
                        c_oh[q + warp] = next_bound(p.bound, dl);
                        c_ob[q + warp] = dl != 0.0 ? p.beta + dl : p.beta;
                        c_up[q + warp] = dl != 0.0;
                    }
                    if (dl != 0.0) {
                        #pragma unroll
                        for (int r = 0; r < R; ++r)
                            if (kk[r] >= 0) put(kk[r], vv[r] + (T)dl * xx[r]);
                    }
                };
                if (warp < L) {
                    const int n = c_m[q + warp].n;
                    if (n <= 32) column(std::integral_constant<int, 1>{});
                    else if (n <= 96) column(std::integral_constant<int, 3>{});
                    else column(std::integral_constant<int, kRunRounds>{});
                }
                __syncthreads();
            };
            const int first = kTeams == 2 ? team ^ off : 0;
            prefetch(min(first, jn));
            for (int q = first; q < jn; q += kTeams) {
                if constexpr (kRuns) {
                    const int L = c_len[q];
                    if (L > 1) {
                        run(q, L);
                        q += L - 1;
                        continue;
                    }
                    if (nq != q) prefetch(q);
                }
                const ColMeta m = nm;
                const bool ind = m.cv == nullptr;
                const ColStep p = c_s[q];
                double dl;
                // wait for the column before this one (the other team's)
                auto turn = [&]() {
                    if (kTeams == 2 && q > 0) bar_sync(4 - team, 2 * NT);
                };
                // the step from the sums, written down by one thread
                auto finish = [&](double g, double h) {
                    combine(g, h, (off + q) & 1);
                    dl = step(p, g - p.xjy, h);                             // :1181-1183
                    if (tid == 0) {
                        c_oh[q] = next_bound(p.bound, dl);
                        c_ob[q] = dl != 0.0 ? p.beta + dl : p.beta;
                        c_up[q] = dl != 0.0;
                    }
                };
                if constexpr (!kGrouped) {
                    auto column = [&](auto rounds) {
                        constexpr int R = decltype(rounds)::value;
                        int kk[R];
                        T xx[R], vv[R], ww[R], gi[R], hi[R];
                        bool on[R];                          // the entry enters the sums
                        auto terms = [&](int r) {
                            mean_terms<T, MODEL>(fit_mean<T, MODEL>(vv[r], strict), xx[r], WM == 2 ? ww[r] : T(1), ind,
                                                 gi[r], hi[r]);
                        };
                        #pragma unroll
                        for (int r = 0; r < R; ++r) {
                            kk[r] = nk[r] - r0;              // negative: no entry
                            xx[r] = (T)nx[r];
                            vv[r] = kk[r] >= 0 ? get(kk[r]) : T(0);
                            ww[r] = kk[r] < 0 ? T(0) : (WM == 1 ? weight.by_fold(nf[r]) : weight(kk[r]));
                            on[r] = WM == 2 && strict ? kk[r] >= 0 : ww[r] != T(0);
                        }
                        prefetch(q + kTeams);
                        // (lanes without an entry compute too: fewer branches are fewer cycles here)
                        #pragma unroll
                        for (int r = 0; r < R; ++r) terms(r);
                        turn();
                        #pragma unroll
                        for (int r = 0; r < R && kTeams == 2; ++r) {
                            const T v = kk[r] >= 0 ? get(kk[r]) : T(0);
                            if (v != vv[r]) {                // moved by the column before
                                vv[r] = v;
                                terms(r);
                            }
                        }
                        Kahan<T> ag, ah;
                        #pragma unroll
                        for (int r = 0; r < R; ++r) {
                            ag.add(on[r] ? gi[r] : T(0));
                            ah.add(on[r] ? hi[r] : T(0));
                        }
                        if (R == kR)
                            for (int b0 = kR * NT + tid; b0 < m.n; b0 += kU * NT) {
                                int k2[kU];
                                T x2[kU], v2[kU], w2[kU];
                                #pragma unroll
                                for (int u = 0; u < kU; ++u) {
                                    const int i = b0 + u * NT;
                                    k2[u] = i < m.n ? (m.ci ? __ldg(m.ci + i) - r0 : i) : -1;
                                    x2[u] = (i < m.n && m.cv) ? (T)__ldg(m.cv + i) : T(1);
                                }
                                #pragma unroll
                                for (int u = 0; u < kU; ++u) {
                                    v2[u] = k2[u] >= 0 ? get(k2[u]) : T(0);
                                    w2[u] = k2[u] < 0 ? T(0)
                                            : WM == 1 ? weight.by_fold((int)__ldg(m.ef + b0 + u * NT))
                                                      : weight(k2[u]);
                                }
                                #pragma unroll
                                for (int u = 0; u < kU; ++u) {
                                    T g1, h1;
                                    mean_terms<T, MODEL>(fit_mean<T, MODEL>(v2[u], strict), x2[u],
                                                         WM == 2 ? w2[u] : T(1), ind, g1, h1);
                                    const bool on = WM == 2 && strict ? k2[u] >= 0 : w2[u] != T(0);
                                    ag.add(on ? g1 : T(0));
                                    ah.add(on ? h1 : T(0));
                                }
                            }
                        finish(ag.value(), ah.value());
                        if (dl != 0.0) {                     // updateXBeta
                            const T d = (T)dl;
                            #pragma unroll
                            for (int r = 0; r < R; ++r)
                                if (kk[r] >= 0) put(kk[r], vv[r] + d * xx[r]);
                            if (R == kR)
                                for (int b0 = kR * NT + tid; b0 < m.n; b0 += kU * NT) {
                                    int k2[kU];
                                    T x2[kU], v2[kU];
                                    #pragma unroll
                                    for (int u = 0; u < kU; ++u) {
                                        const int i = b0 + u * NT;
                                        k2[u] = i < m.n ? (m.ci ? __ldg(m.ci + i) - r0 : i) : -1;
                                        x2[u] = (i < m.n && m.cv) ? (T)__ldg(m.cv + i) : T(1);
                                    }
                                    #pragma unroll
                                    for (int u = 0; u < kU; ++u) v2[u] = k2[u] >= 0 ? get(k2[u]) : T(0);
                                    #pragma unroll
                                    for (int u = 0; u < kU; ++u)
                                        if (k2[u] >= 0) put(k2[u], v2[u] + d * x2[u]);
                                }
                            if (kTeams == 1) __syncthreads();
                        }
                    };
                    if (m.n <= NT) column(std::integral_constant<int, 1>{});
                    else column(std::integral_constant<int, kR>{});
                } else {
                    // the first entry of each run of one stratum takes the run
                    // (ConditionalLogisticRegression::incrementGradientAndHessian,
                    // ModelSpecifics.h:820-837)
                    auto column = [&](auto rounds) {
                        constexpr int R = decltype(rounds)::value;
                        int kk[R], ss[R], bb[R];
                        T xx[R], vv[R], ex[R], gi[R], hi[R];
                        double dd[R], ev[R];
                        auto row = [&](int i) { return m.ci ? __ldg(m.ci + i) - r0 : i; };
                        auto rest = [&](int i, int s, T& n1, T& n2) {      // the run's further entries
                            for (++i; i < m.n && __ldg(m.es + i) == s; ++i) {
                                const T x = ind ? T(1) : (T)__ldg(m.cv + i);
                                const T e = fexp(get(row(i)));
                                n1 += e * x;
                                if (!ind) n2 += e * x * x;
                            }
                        };
                        auto run_terms = [&](T n1, T n2, double d, double nwk, T& g1, T& h1) {
                            const double t = (double)n1 / d;
                            const double gg = nwk * t;
                            g1 = (T)gg;
                            h1 = (T)(ind ? gg * (1.0 - t) : nwk * ((double)n2 / d - t * t));
                        };
                        auto terms = [&](int r) {
                            ex[r] = fexp(vv[r]);
                            T n1 = ex[r] * xx[r], n2 = ind ? T(0) : n1 * xx[r];
                            if ((bb[r] & 3) == 3) rest(tid + r * NT, ss[r], n1, n2);
                            run_terms(n1, n2, dd[r], ev[r], gi[r], hi[r]);
                        };
                        #pragma unroll
                        for (int r = 0; r < R; ++r) {
                            kk[r] = nk[r] - r0;              // negative: no entry
                            xx[r] = (T)nx[r];
                            ss[r] = ns[r];
                            // bit 0: the entry starts its stratum's run; bit 1: the run goes on
                            bb[r] = ss[r] >= 0 ? (np[r] != ss[r] ? 1 : 0) | (nn[r] == ss[r] ? 2 : 0) : 0;
                            vv[r] = kk[r] >= 0 ? get(kk[r]) : T(0);
                            dd[r] = (bb[r] & 1) ? dg[ss[r]] : 1.0;
                            ev[r] = (bb[r] & 1) ? __ldg(ng + ss[r]) : 0.0;
                        }
                        prefetch(q + kTeams);
                        #pragma unroll
                        for (int r = 0; r < R; ++r) terms(r);
                        // (the terms of an entry that starts no run mean nothing: without its
                        // stratum's denominator they overflow where exp(xb) alone is large)
                        Kahan<T> ag, ah;
                        #pragma unroll
                        for (int r = 0; r < R; ++r) {
                            ag.add((bb[r] & 1) ? gi[r] : T(0));
                            ah.add((bb[r] & 1) ? hi[r] : T(0));
                        }
                        if (R == kR)
                            for (int i = kR * NT + tid; i < m.n; i += NT) {
                                const int s = __ldg(m.es + i);
                                if (__ldg(m.es + i - 1) == s) continue;
                                const T x = ind ? T(1) : (T)__ldg(m.cv + i);
                                const T e = fexp(get(row(i)));
                                T n1 = e * x, n2 = ind ? T(0) : n1 * x, g1, h1;
                                rest(i, s, n1, n2);
                                run_terms(n1, n2, dg[s], ng[s], g1, h1);
                                ag.add(g1);
                                ah.add(h1);
                            }
                        finish(ag.value(), ah.value());
                        if (dl == 0.0) return;               // nothing moved: no write to order
                        const T d = (T)dl;                   // updateXBeta and the strata's denominators
                        auto move = [&](int i, int s, double& acc) {
                            for (; i < m.n && __ldg(m.es + i) == s; ++i) {
                                const T x = ind ? T(1) : (T)__ldg(m.cv + i);
                                const int k = row(i);
                                const T old = get(k), nv = old + d * x;
                                put(k, nv);
                                acc += (double)fexp(nv) - (double)fexp(old);
                            }
                        };
                        #pragma unroll
                        for (int r = 0; r < R; ++r)
                            if (bb[r] & 1) {
                                const T nv = vv[r] + d * xx[r];
                                put(kk[r], nv);
                                double acc = dd[r] + ((double)fexp(nv) - (double)ex[r]);
                                if (bb[r] & 2) move(tid + r * NT + 1, ss[r], acc);
                                dg[ss[r]] = acc;
                            }
                        if (R == kR)
                            for (int i = kR * NT + tid; i < m.n; i += NT) {
                                const int s = __ldg(m.es + i);
                                if (__ldg(m.es + i - 1) == s) continue;
                                double acc = dg[s];
                                move(i, s, acc);
                                dg[s] = acc;
                            }
                        __syncthreads();
                    };
                    if (m.n <= NT) column(std::integral_constant<int, 1>{});
                    else column(std::integral_constant<int, kR>{});
                }
                if (kTeams == 2 && q + 1 < jn) bar_arrive(3 + team, 2 * NT);     // this column's rows are written
            }
            off ^= jn & 1;
            __syncthreads();
            if (rank == 0)
                for (int q = threadIdx.x; q < jn; q += blockDim.x) {
                    const size_t o = fj + c_j[q];
                    A.beta[o] = c_ob[q];
                    A.hdelta[o] = c_oh[q];
                    if (c_up[q]) A.col_updates[o] += 1u;
                }
        }
        // ---- performCheckConvergence (:839-906)
        ++it;
        __syncthreads();
        // rank 0's coefficients are staged by every CTA in the next cycle
        if (C > 1) cluster.sync();
        const double o = objective();
        double conv;
        int ill = 0;
        if (A.conv == CYC_CONV_ZHANG_OLES) {
            conv = o;
        } else {
            if (o != o) { conv = 0.0; ill = 1; }
            else conv = fabs(o - last) / (fabs(o) + 1.0);
            last = o;
        }
        if (agree()) { flag = kTimedOut; break; }
        if (A.tol > 0 && conv < A.tol) { flag = ill ? CYC_ILLCONDITIONED : CYC_SUCCESS; break; }
        if (it == A.max_iter) { flag = CYC_MAX_ITERATIONS; break; }
    }
    if (SM) {
        __syncthreads();
        for (int i = threadIdx.x; i < nr; i += blockDim.x) xg[i] = sx[i];
    }
    if (flag == kTimedOut) stores_land();
    if (C > 1) cluster.sync();   // no CTA leaves while others may still write its shared memory
    if (rank == 0 && threadIdx.x == 0) {
        A.out_iter[f] = it;
        A.out_flag[f] = flag;
    }
}

// linear predictors of a CTA's rows in shared memory while they fit beside the
// static arrays; the rest of the 256 KB stays L1
constexpr size_t kRowBytes = 200 * 1024;

template <class T, int MODEL, int WM, bool SM, int TEAMS>
void launch_one(const CcdArgs& a, size_t dyn, cudaStream_t stream) {
    auto kern = k_ccd<T, MODEL, WM, SM, TEAMS>;
    if (SM) CYC_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowBytes));
    if (a.C > 8) CYC_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.F * a.C);
    cfg.blockDim = dim3(a.threads);
    cfg.dynamicSmemBytes = dyn;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = a.C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CYC_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
    count_launch();
}

template <class T, int MODEL, int WM>
void launch_rows(CcdArgs a, const std::vector<int>& rpart, cudaStream_t stream) {
    int rows = 0;
    for (int r = 0; r < a.C; ++r) rows = std::max(rows, rpart[r + 1] - rpart[r]);
    a.wait = wait_limit(rows);
    const size_t bytes = (size_t)rows * sizeof(T);
    const char* xs = std::getenv("CYC_BATCH_XB_SMEM");      // 0: global memory
    const bool fits = bytes <= kRowBytes && !(xs && std::atoi(xs) == 0);
    constexpr bool rows1 = MODEL == CYC_LR || MODEL == CYC_PR, two = sizeof(T) == 8 && rows1;
    auto with = [&](auto smem, size_t dyn) {
        constexpr bool SM = decltype(smem)::value;
        if constexpr (rows1) {
            if (a.runs) return launch_one<T, MODEL, WM, SM, 0>(a, dyn, stream);
        }
        if constexpr (two) {
            if (a.teams == 2) return launch_one<T, MODEL, WM, SM, 2>(a, dyn, stream);
        }
        launch_one<T, MODEL, WM, SM, 1>(a, dyn, stream);
    };
    if (fits) with(std::true_type{}, bytes);
    else with(std::false_type{}, 0);
}

template <class T, int MODEL>
void launch_weights(const CcdArgs& a, const std::vector<int>& rpart, cudaStream_t stream) {
    switch (a.weights) {
    case 0: launch_rows<T, MODEL, 0>(a, rpart, stream); break;
    case 1: launch_rows<T, MODEL, 1>(a, rpart, stream); break;
    default: launch_rows<T, MODEL, 2>(a, rpart, stream); break;
    }
}

__global__ void k_entry_folds(long long n, const int* __restrict__ idx, const signed char* __restrict__ fold,
                              signed char* __restrict__ out) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        out[e] = fold[idx[e]];
}

const KernelFile g_kernels((const void*)(&k_entry_folds));

}  // namespace

template <class T>
void launch_ccd(const CcdArgs& a, const std::vector<int>& rpart, cudaStream_t stream) {
    switch (a.model) {
    case CYC_LR: launch_weights<T, CYC_LR>(a, rpart, stream); break;
    case CYC_PR: launch_weights<T, CYC_PR>(a, rpart, stream); break;
    case CYC_CLR: launch_weights<T, CYC_CLR>(a, rpart, stream); break;
    case CYC_CPR: launch_weights<T, CYC_CPR>(a, rpart, stream); break;
    default: throw Error{CYC_ERR_UNSUPPORTED, "the persistent solver supports lr, pr, clr, cpr"};
    }
}
template void launch_ccd<double>(const CcdArgs&, const std::vector<int>&, cudaStream_t);
template void launch_ccd<float>(const CcdArgs&, const std::vector<int>&, cudaStream_t);

// clusters of this shape the device holds at once (as one representative of the
// kernel's instances is held: their register counts differ little)
static int resident_fits(int C, int threads, size_t dyn) {
    auto kern = k_ccd<double, CYC_LR, 1, true, 1>;
    CYC_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowBytes));
    CYC_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = dyn;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    CYC_CHECK_CUDA(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
    return n;
}

// The shape with the least modelled time of a cycle.  Measured here (us): a
// step, what its sums add when they cross a cluster, and every further round
// of a column's threads over a CTA's share of the column; fits whose clusters
// the device does not hold side by side wait their turn, and CTAs that share an
// SM slow one another (24 fits of 50k rows: 8 CTAs of 128 threads 6.6 ms, 4 of
// 256, one an SM, 5.6; 20 CV fits of 100k rows: 9.7 ms at 4 CTAs of 128, 7.2 at 6
// of 256; 40 fits: 14.6 at 2 CTAs, 12.7 at 3).  (10k rows, 1,000
// columns of 100 entries: 27 ms for 41 cycles with one CTA of two teams, 31.7
// of one team, 35 to 38 with clusters; 100k rows, 600 Zipf columns and 4 dense
// ones: 150 ms for 40 cycles with one CTA, 38 with four, 25 with sixteen; 80
// CV fits of 100k rows: 19 ms with one team, 29 with two.)
// Callers add the calls that share the device to F: 8 fits of 500k rows, one a
// call and all at once, take 214 ms with the 16 CTAs that are best alone (102 ms) and
// 150 with 8 (125 alone); 16 fits 346 and 315.
CcdShape ccd_shape(const Dataset& ds, int F, int only, bool varied) {
    only = std::min(only, kCcdCluster);
    struct { int C; double cross; } sizes[] = {{1, 0.0}, {2, 0.19}, {3, 0.2}, {4, 0.2}, {5, 0.25},
                                               {6, 0.25}, {8, 0.25}, {12, 0.26}, {16, 0.26}};
    struct { int teams, threads; double step, round; } kinds[] = {
        {2, 256, 0.67, 0.5}, {1, 256, 0.92, 0.5}, {1, 128, 0.80, 0.4}};
    CcdShape best{std::max(1, only), 128, 1, 1, 0.0};
    for (const auto& size : sizes) {
        if (only > 0 && (size.C < only || best.cycle_us > 0.0)) continue;
        const int C = only > 0 ? only : size.C;
        for (const auto& kind : kinds) {
            if (kind.teams == 2 && !model_independent(ds.model)) continue;
            const size_t bytes = ((size_t)ds.K + C - 1) / C * sizeof(double);
            const int slots = resident_fits(C, kind.threads, bytes <= kRowBytes ? bytes : 0);
            if (slots < 1) continue;
            // predictors of the fits in flight that neither shared memory nor
            // L2 holds come from HBM, a row at a time
            const bool far = bytes > kRowBytes && (double)std::min(F, slots) * ds.K * sizeof(double) > 100e6;
            const int deal = kind.threads / kind.teams;
            const double round = far ? 1.2 : kind.round;
            const double step = kind.step * (std::min(F, slots) * C > 148 ? 1.25 : 1.0) + (far ? 0.5 : 0.0) + size.cross;
            double us = 0.0;
            for (int j = 0; j < ds.J; ++j) {
                const double rounds = std::ceil((double)ds.col_len(j) / (C * deal));
                us += step + round * std::max(0.0, rounds - 1.0);
            }
            us *= ccd_turns(F, slots, varied);
            if (best.cycle_us == 0.0 || us < best.cycle_us) best = {C, kind.threads, kind.teams, slots, us};
        }
    }
    // CYC_BATCH_CLUSTER="CTAs[,threads[,teams]]" fixes the shape (teams 0: runs)
    if (const char* e = std::getenv("CYC_BATCH_CLUSTER")) {
        int c = best.C, t = best.threads, n = best.teams;
        std::sscanf(e, "%d,%d,%d", &c, &t, &n);
        best.C = std::max(1, std::min(kCcdCluster, c));
        best.teams = n == 2 && model_independent(ds.model) ? 2 : 1;
        best.threads = std::max(64, std::min(kCcdThreads, t / 64 * 64));
        best.runs = n == 0 && model_independent(ds.model);
        if (best.runs) { best.C = 1; best.threads = kCcdThreads; }       // a warp for each column of a run
    }
    return best;
}

CcdRuns ccd_runs(const Dataset& ds, const std::vector<int>& cols, bool local) {
    CcdRuns r{std::vector<unsigned char>(cols.size(), 1), 0.0};
    std::vector<int> seen(ds.K, -1);             // the last run with the row
    int start = 0, id = -1;
    auto close = [&](int end) {
        const int len = end - start;
        for (int i = start; i < end; ++i) r.len[i] = i == start ? (unsigned char)len : 0;
        long long n = 0;                         // the longest column
        for (int i = start; i < end; ++i) n = std::max(n, ds.col_len(cols[i]));
        if (len > 1) {
            r.cycle_us += n <= 32 ? (local ? 1.15 : 1.5) : n <= 96 ? (local ? 1.4 : 1.9) : (local ? 2.0 : 3.0);
        } else if (len == 1) {
            const double rounds = std::ceil((double)n / kCcdThreads);
            r.cycle_us += (local ? 1.05 : 1.35) + (local ? 0.5 : 0.7) * std::max(0.0, rounds - 1.0);
        }
        start = end;
    };
    for (int i = 0; i < (int)cols.size(); ++i) {
        const int j = cols[i], f = ds.fmt[j];
        const bool fits = (f == CYC_SPARSE || f == CYC_INDICATOR) && ds.col_len(j) <= 32 * kRunRounds;
        const int* rows = ds.h_idx.data() + ds.col_ptr[j];
        const int n = fits ? (int)ds.col_len(j) : 0;
        bool joins = fits && i > start && i % kCh != 0 && i - start < kWarps;
        for (int e = 0; joins && e < n; ++e) joins = seen[rows[e]] != id;
        if (!joins) {
            close(i);
            ++id;
        }
        for (int e = 0; e < n; ++e) seen[rows[e]] = id;
        if (!fits) {                             // a run by itself
            close(i + 1);
            ++id;
        }
    }
    close((int)cols.size());
    return r;
}

std::vector<int> ccd_rows(const Dataset& ds, int C) {
    std::vector<int> rpart(C + 1, ds.K);
    for (int r = 0; r < C; ++r) {
        int b = (int)((long long)ds.K * r / C);
        if (model_grouped(ds.model)) {
            auto it = std::lower_bound(ds.strat_ptr.begin(), ds.strat_ptr.end(), b);
            b = (it == ds.strat_ptr.end()) ? ds.K : *it;
        }
        rpart[r] = b;
    }
    for (int r = 1; r <= C; ++r) rpart[r] = std::max(rpart[r], rpart[r - 1]);
    return rpart;
}

void ccd_splits(const Dataset& ds, int C, const int* d_rpart, int* d_split, cudaStream_t stream) {
    launch(k_splits, (ds.J * (C + 1) + 255) / 256, 256, 0, stream, ds.J, C, ds.d_fmt.get(), ds.d_col_ptr.get(),
           ds.d_idx.get(), d_rpart, d_split);
}

void ccd_entry_folds(const Dataset& ds, const signed char* d_fold, signed char* d_out, cudaStream_t stream) {
    if (ds.nnz_idx)
        launch(k_entry_folds, grid_for(ds.nnz_idx, 4), kThreads, 0, stream, ds.nnz_idx, (const int*)ds.d_idx.get(),
               d_fold, d_out);
}

}  // namespace cyc
