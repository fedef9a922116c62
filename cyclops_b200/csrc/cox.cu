// cox.cu -- the persistent Breslow Cox CCD: a fit's whole coordinate loop in
// one launch.
//
// With n_e events and risk-set sum D_e at event group e, and A_e / B_e the sums
// of a column's w exp(xb) x / x^2 over the rows at risk at e, the reference
// walks every group for (ModelSpecifics.hpp:904-962)
//     g = sum_e n_e A_e / D_e,   h = sum_e n_e (B_e / D_e - (A_e / D_e)^2).
// A_e is a running sum of the column's entries, so the sums turn over:
//     g = sum_k v_k S1(e_k),  h = sum_k v_k x_k S1(e_k) - sum_k v_k (2 A'_k + v_k) S2(e_k)
// with v_k = w exp(xb) x of entry k, e_k its slot, A'_k the running sum before
// it, and S1, S2 the suffix sums (within the stratum) of n/D and n/D^2.  Every
// term of S1 and S2 has one sign and nothing is differenced, so FP64 sums in
// tree order carry no more error than D itself.  A column then costs a pass
// over its own entries; only a step that moves a coefficient renews the sums:
// one pass over the event groups (about a third of the rows here), not over
// every row, and nothing but S1 and S2 is written.  Groups of many rows are cut
// into slots (kSlotRows); a slot without events only passes the sums on.
//
// What bounds a step is latency at small sizes (block scans, two exchanges a
// cluster) and one division per event group at large ones, so a fit is one
// cluster of up to 16 CTAs that split the slots in order, with their rows; their
// carries cross by st.async on mbarriers.  The per-slot arrays stay in shared memory
// where they fit, S1 and S2 alone where only those do, else in L2.  (Before:
// seven launches a coordinate that rewrote nine arrays over all rows, 35 us a
// coordinate at 20k rows and 56 us at 500k.)
#include "cox.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <memory>
#include <set>

#include "ccd.cuh"
#include "engine.cuh"
#include "mbar.cuh"
#include "row_terms.cuh"

namespace cg = cooperative_groups;

namespace cyc {

namespace {

constexpr int kCh = 64;           // coordinates staged at a time
// slots of a thread taken at a time, without branches: every thread of a CTA
// runs the same number of blocks, past its last slot on zeros
constexpr int kB = 4;
constexpr int kMaxC = kCcdCluster;
// A slot's rows at most.  Rows between two events are one event group's, and a
// group can hold most of a cohort (everybody censored at the end of a fixed
// follow-up enters with the first event): groups are cut so that no thread walks
// a long run, and the CTAs' rows can be balanced.  100k rows, 87 % of them
// censored at one time, 100 indicator columns of 2,000 rows, 6 cycles: 441 ms
// uncut, 10.5 cut.
constexpr int kSlotRows = 32;
// in an entry's slot position: the slot's stratum goes on past the slots of its
// CTA (kTailBit), past those of its thread (kThreadBit)
constexpr int kTailBit = 1 << 30, kThreadBit = 1 << 29, kPosMask = kThreadBit - 1;
constexpr unsigned kFull = 0xffffffffu;
// relative bound on the rounding of a column's sums
constexpr double kZero = 0x1p-45;

// ---- the risk sets ------------------------------------------------------------

constexpr int kTileItems = 8;
constexpr int kTile = kThreads * kTileItems;

// inclusive scan over the rows in three launches: tile totals, their scan, the
// rows.  `item(k)` is the row's value, `op` max or plus.
struct OpMax {
    static constexpr int kZero = -1;
    __device__ int operator()(int a, int b) const { return max(a, b); }
};
struct OpSum {
    static constexpr int kZero = 0;
    __device__ int operator()(int a, int b) const { return a + b; }
};

template <class Op>
__device__ int block_scan(int v, int* s_w) {      // inclusive over the block's threads
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    Op op;
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(kFull, v, o);
        if (lane >= o) v = op(u, v);
    }
    if (lane == 31) s_w[w] = v;
    __syncthreads();
    int pre = Op::kZero;
    for (int q = 0; q < w; ++q) pre = op(pre, s_w[q]);
    __syncthreads();
    return op(pre, v);
}

template <class Op, class Item>
__global__ void k_rows_totals(int K, Item item, int* __restrict__ tiles) {
    __shared__ int s_w[kThreads / 32];
    const int k0 = blockIdx.x * kTile + threadIdx.x * kTileItems;
    Op op;
    int v = Op::kZero;
    for (int i = 0; i < kTileItems; ++i)
        if (k0 + i < K) v = op(v, item(k0 + i));
    v = block_scan<Op>(v, s_w);
    if (threadIdx.x == kThreads - 1) tiles[blockIdx.x] = v;
}

template <class Op>
__global__ void k_tiles_scan(int n, int* __restrict__ tiles) {       // one block: exclusive, in place
    __shared__ int s_w[kThreads / 32];
    __shared__ int s_carry;
    Op op;
    if (threadIdx.x == 0) s_carry = Op::kZero;
    __syncthreads();
    for (int b = 0; b < n; b += kThreads) {
        const int i = b + threadIdx.x;
        const int v = i < n ? tiles[i] : Op::kZero;
        const int inc = op(s_carry, block_scan<Op>(v, s_w));
        __syncthreads();
        int ex = __shfl_up_sync(kFull, inc, 1);
        if ((threadIdx.x & 31) == 31) s_w[threadIdx.x >> 5] = inc;
        __syncthreads();
        if ((threadIdx.x & 31) == 0) ex = threadIdx.x == 0 ? s_carry : s_w[(threadIdx.x >> 5) - 1];
        if (i < n) tiles[i] = ex;
        __syncthreads();
        if (threadIdx.x == kThreads - 1) s_carry = inc;
        __syncthreads();
    }
}

template <class Op, class Item>
__global__ void k_rows_scan(int K, Item item, const int* __restrict__ tiles, int* __restrict__ out) {
    __shared__ int s_w[kThreads / 32];
    const int k0 = blockIdx.x * kTile + threadIdx.x * kTileItems;
    Op op;
    int v[kTileItems];
    int t = Op::kZero;
    for (int i = 0; i < kTileItems; ++i) {
        t = op(t, k0 + i < K ? item(k0 + i) : Op::kZero);
        v[i] = t;
    }
    const int inc = block_scan<Op>(t, s_w);
    int pre = __shfl_up_sync(kFull, inc, 1);
    if ((threadIdx.x & 31) == 31) s_w[threadIdx.x >> 5] = inc;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) pre = threadIdx.x == 0 ? Op::kZero : s_w[(threadIdx.x >> 5) - 1];
    pre = op(tiles[blockIdx.x], pre);
    for (int i = 0; i < kTileItems; ++i)
        if (k0 + i < K) out[k0 + i] = op(pre, v[i]);
}

struct LastWeighted {                // the row itself where it has weight
    const double* w;
    __device__ int operator()(int k) const { return w[k] != 0.0 ? k : -1; }
};
// 1 where a row starts an event group (setPidForAccumulation's rule,
// ModelSpecifics.hpp:1809-1868: consecutive weighted rows share a group when
// both are events at one time of one stratum)
struct GroupStart {
    const double *w, *y, *time;
    const int *strat, *last;         // last weighted row up to each row (null: every row)
    __device__ int operator()(int k) const {
        if (y[k] == 0.0 || (w && w[k] == 0.0)) return 0;
        const int p = k == 0 ? -1 : (last ? last[k - 1] : k - 1);
        if (p < 0 || strat[p] != strat[k]) return 1;
        return !(y[p] == 1.0 && time[p] == time[k] && y[p] == y[k]);
    }
};

__global__ void k_slot_rows(int K, const double* __restrict__ w, const double* __restrict__ y,
                            const int* __restrict__ strat, const int* __restrict__ cnt, int* __restrict__ first,
                            int* __restrict__ end, int* __restrict__ sstr, int* __restrict__ total) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < K; k += gridDim.x * blockDim.x) {
        if (k == K - 1) *total = cnt[k];
        if (y[k] == 0.0 || (w && w[k] == 0.0)) continue;
        const int e = cnt[k] - 1;
        atomicMax(end + e, k);
        if (k == 0 || cnt[k - 1] == e) {
            first[e] = k;
            sstr[e] = strat[k];
        }
    }
}

// the first row of each event group's rows (those that enter the risk sets with it)
__global__ void k_group_rows(const int* __restrict__ groups, const int* __restrict__ gend, const int* __restrict__ gstr,
                             const int* __restrict__ strat_ptr, int* __restrict__ glo) {
    const int E = *groups;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < E; e += gridDim.x * blockDim.x)
        glo[e] = e == 0 || gstr[e - 1] != gstr[e] ? strat_ptr[gstr[e]] : gend[e - 1] + 1;
}

const KernelFile g_kernels((const void*)(&k_group_rows));
struct Pieces {                      // the slots of an event group
    const int *groups, *glo, *gend;
    __device__ int operator()(int e) const { return e < *groups ? (gend[e] - glo[e]) / kSlotRows + 1 : 0; }
};

// the event groups as the row kernels read them
struct Groups {
    const int *groups;               // their number
    const int *cnt;                  // by row: groups that start at it or before
    const int *glo, *gend, *gstr;    // rows and stratum of each
    const int *gcum;                 // slots up to and with each
    __device__ int first_slot(int e) const { return e > 0 ? gcum[e - 1] : 0; }
    // the group whose rows hold row k, or the next one
    __device__ int of(int k) const { const int c = cnt[k]; return c > 0 && gend[c - 1] >= k ? c - 1 : c; }
    // slots whose rows all precede row b; b itself goes down to the slot's
    // first row where it would cut one
    __device__ int before(int& b) const {
        if (b == 0) return 0;
        const int c = cnt[b - 1], e = c > 0 && gend[c - 1] >= b ? c - 1 : c;
        int s = first_slot(e);
        if (e < *groups && glo[e] < b) {
            const int q = (b - glo[e]) / kSlotRows;
            s += q;
            b = glo[e] + q * kSlotRows;
        }
        return s;
    }
};

// rows and stratum of every slot (a warp per group)
__global__ void k_slot_fill(Groups G, int* __restrict__ lo, int* __restrict__ end, int* __restrict__ sstr) {
    const int E = *G.groups, lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < E; e += nwarps) {
        const int s0 = G.first_slot(e), s1 = G.gcum[e];
        for (int s = s0 + lane; s < s1; s += 32) {
            const int k = G.glo[e] + (s - s0) * kSlotRows;
            lo[s] = k;
            end[s] = min(G.gend[e], k + kSlotRows - 1);
            sstr[s] = G.gstr[e];
        }
    }
}

// The split of rows and slots over the CTAs: each CTA's share of the rows and its
// share of the slots add up to 2 / C, and none has more than `room` slots.  (Slots
// are what a moving step renews, rows what the columns' entries follow: events
// may lie anywhere among the rows.)  Boundaries fall between slots.  A warp finds
// a boundary, 32 candidates at a time.
__global__ void k_slot_parts(int K, int C, int S, int room, Groups G, const int* __restrict__ end,
                             int* __restrict__ spart, int* __restrict__ rpart) {
    __shared__ int s_s[kMaxC + 1], s_b[kMaxC + 1];
    const int r = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (r < C) {
        const double want = 2.0 * r / C;
        int lo = 0, hi = K;                               // the share is below `want` at lo, not at hi
        while (hi - lo > 1) {
            const int b = lo + (int)((long long)(hi - lo) * (lane + 1) / 33);
            int at = b;
            const int s = G.before(at);
            const unsigned m = __ballot_sync(kFull, (double)b / K + (double)s / max(1, S) >= want);
            const int f = m ? __ffs(m) - 1 : 32;
            const int up = __shfl_sync(kFull, b, min(f, 31)), down = __shfl_sync(kFull, b, max(f - 1, 0));
            if (f < 32) hi = up;
            if (f > 0) lo = down;
        }
        if (lane == 0) {
            int b = r == 0 ? 0 : hi;
            s_s[r] = G.before(b);
            s_b[r] = b;
        }
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    s_s[C] = S;
    s_b[C] = K;
    for (int q = 1; q < C; ++q) {
        const int least = max(s_s[q - 1], S - (C - q) * room), most = s_s[q - 1] + room;
        const int s = min(max(s_s[q], least), most);
        if (s != s_s[q]) {
            s_s[q] = s;
            s_b[q] = end[s - 1] + 1;
        }
        s_b[q] = max(s_b[q], s_b[q - 1]);
    }
    for (int q = 0; q <= C; ++q) { spart[q] = s_s[q]; rpart[q] = s_b[q]; }
}

__device__ __forceinline__ int slot_position(int e, int C, int nt, const int* spart, int& r) {
    r = 0;
    while (r + 1 < C && e >= spart[r + 1]) ++r;
    const int s0 = spart[r], ns = spart[r + 1] - s0, m = (ns + nt - 1) / nt;
    const int q = e - s0;
    return (q % m) * nt + q / m;
}

// per event group (a warp each): its events, which its last slot has, and its slots' flags
__global__ void k_slots(int C, int nt, int per_cta, Groups G, const int* __restrict__ spart,
                        const int* __restrict__ first, const double* __restrict__ w, const double* __restrict__ y,
                        unsigned char* __restrict__ flag, double* __restrict__ n) {
    const int E = *G.groups, lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < E; e += nwarps) {
        double a = 0.0;
        for (int k = first[e] + lane; k <= G.gend[e]; k += 32) a += y[k] * (w ? w[k] : 1.0);
        for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(kFull, a, o);
        const int s0 = G.first_slot(e), s1 = G.gcum[e], str = G.gstr[e];
        const bool starts = e == 0 || G.gstr[e - 1] != str, ends = e + 1 == E || G.gstr[e + 1] != str;
        for (int s = s0 + lane; s < s1; s += 32) {
            int r;
            const int p = slot_position(s, C, nt, spart, r);
            n[(size_t)r * per_cta + p] = s == s1 - 1 ? a : 0.0;
            flag[(size_t)r * per_cta + p] = (unsigned char)((s == s0 && starts ? 1 : 0) | (s == s1 - 1 && ends ? 2 : 0));
        }
    }
}

// 1 / the sum of all events (one block)
__global__ void __launch_bounds__(1024) k_per_event(int np, const double* __restrict__ n, double* __restrict__ out) {
    __shared__ double s_w[32];
    double a = 0.0;
    #pragma unroll 4
    for (int p = threadIdx.x; p < np; p += 1024) a += n[p];
    for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(kFull, a, o);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < 32; ++w) a += s_w[w];
    *out = a > 0.0 ? 1.0 / a : 0.0;
}

// sums of w exp(xb) over each slot's rows (a warp each)
__global__ void k_slot_increments(int C, int nt, int per_cta, int S, const int* __restrict__ spart,
                                  const int* __restrict__ lo, const int* __restrict__ end,
                                  const double* __restrict__ w, const double* __restrict__ xb,
                                  double* __restrict__ d) {
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < S; e += nwarps) {
        double a = 0.0;
        for (int k = lo[e] + lane; k <= end[e]; k += 32) {
            const double wk = w ? w[k] : 1.0;
            if (wk != 0.0) a += wk * exp(xb[k]);
        }
        for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(kFull, a, o);
        if (lane == 0) {
            int r;
            const int p = slot_position(e, C, nt, spart, r);
            d[(size_t)r * per_cta + p] = a;
        }
    }
}

// every row's slot position in its CTA (-1: none), with kTailBit and kThreadBit.
// Rows of weight zero get the slot their
// place in the order gives (they add nothing), so a column's slots ascend.
__global__ void k_row_slots(int K, int C, int nt, int S, Groups G, const int* __restrict__ spart,
                            const int* __restrict__ sstr, const int* __restrict__ strat, int* __restrict__ out) {
    const int E = *G.groups;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < K; k += gridDim.x * blockDim.x) {
        int o = -1;
        const int g = G.of(k);
        if (g < E && G.gstr[g] == strat[k]) {
            const int s = G.first_slot(g) + (k - G.glo[g]) / kSlotRows;
            int r;
            o = slot_position(s, C, nt, spart, r);
            const int s0 = spart[r], next = spart[r + 1], m = (next - s0 + nt - 1) / nt;
            const int after = min(next, s0 + ((s - s0) / m + 1) * m);       // first slot past its thread's
            if (next < S && sstr[next] == sstr[s]) o |= kTailBit;
            if (after < S && sstr[after] == sstr[s]) o |= kThreadBit;
        }
        out[k] = o;
    }
}

__global__ void k_entry_slots(long long nnz, const int* __restrict__ idx, const int* __restrict__ rowslot,
                              int* __restrict__ out) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nnz; e += (long long)gridDim.x * blockDim.x)
        out[e] = rowslot[idx[e]];
}

// ---- the solver ------------------------------------------------------------------

struct ColMeta {
    const int* ci;       // row ids (null for dense columns: entry i is row r0 + i)
    const double* cv;    // values (null for indicators)
    const int* es;       // slot positions of the entries
    const int* st;       // strata of the entries (null: one stratum)
    int n;
    int before;          // the column has entries before this CTA's rows
};

// WHERE the per-slot arrays live: 0 all in shared memory, 1 S1 and S2 (and the
// flags), 2 global memory.  kNT threads: few while a thread has few slots (the
// scans cost every warp the same, so warps without work only take issue slots;
// 512 threads took 26 ms where 128 take 13 at 20k rows x 500 columns).  SEG:
// more than one stratum, so sums restart at their boundaries.
template <int WHERE, int kNT, bool SEG>
__global__ void __launch_bounds__(kNT, 1) k_cox(const CoxArgs* __restrict__ fits, int C) {
    constexpr int kNW = kNT / 32;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ CoxArgs A;
    static_assert(sizeof(CoxArgs) % 4 == 0, "copied by words");
    for (int i = threadIdx.x; i < (int)(sizeof(CoxArgs) / 4); i += kNT)
        reinterpret_cast<int*>(&A)[i] = reinterpret_cast<const int*>(fits + blockIdx.x / C)[i];
    __syncthreads();
    const int rank = C > 1 ? (int)cluster.block_rank() : 0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = A.rpart[rank], nr = A.rpart[rank + 1] - r0;
    const int ns = A.spart[rank + 1] - A.spart[rank];
    const int m = (ns + kNT - 1) / kNT;                   // slots of a thread
    const int mine = max(0, min(m, ns - tid * m));
    double* const xg = A.xb + r0;                         // this CTA's rows, relative to r0
    const double* const wg = A.weighted ? A.w + r0 : nullptr;
    const double var = A.variance;
    const double lam = sqrt(2.0 / var);                   // LaplacePrior rate, CovariatePrior.h:282-292
    const size_t base_slot = (size_t)rank * A.per_cta;

    extern __shared__ __align__(16) unsigned char dyn_smem[];
    double* const sm = reinterpret_cast<double*>(dyn_smem);
    const int nb = (m + kB - 1) / kB;                     // blocks of kB slots of a thread
    const int np = nb * kB * kNT;                         // positions in use
    double* const S1 = WHERE <= 1 ? sm : A.S1 + base_slot;
    double* const S2 = WHERE <= 1 ? sm + np : A.S2 + base_slot;
    double* const dd = WHERE == 0 ? sm + 2 * np : A.d + base_slot;
    double* const nn = WHERE == 0 ? sm + 3 * np : const_cast<double*>(A.n) + base_slot;
    // the sums before each block of kB slots of a thread
    double* const bp = WHERE <= 1 ? sm + (WHERE == 0 ? 4 : 2) * np : A.bp + base_slot / kB;
    unsigned char* const fl = WHERE <= 1 ? reinterpret_cast<unsigned char*>(bp + nb * kNT)
                                         : const_cast<unsigned char*>(A.flag) + base_slot;

    __shared__ double s_a[2][kNW], s_b[2][kNW];           // warp totals of a scan, by parity
    __shared__ int s_f[2][kNW];
    __shared__ double s_sum[5][kNW];                      // a column's sums by warp
    // exchanges: A (risk-set totals), B (a column's sums, three pieces), C (suffix totals)
    __shared__ __align__(16) double2 x_a[2][kMaxC], x_c[2][kMaxC], x_b[2][3][kMaxC];
    __shared__ __align__(8) unsigned long long s_mb[3][2];
    __shared__ double s_carry, s_c1, s_c2, s_dl;
    __shared__ double s_per_event;                        // 1 / the weight of the events
    __shared__ int s_dead;
    __shared__ int s_hasend[kMaxC];
    __shared__ ColMeta c_m[kCh + 1];
    __shared__ double c_beta[kCh], c_hd[kCh], c_xjy[kCh], c_ob[kCh], c_oh[kCh];
    __shared__ int c_j[kCh], c_pt[kCh], c_up[kCh];
    __shared__ double s_mv[kNT];                          // the entries' changes of their slots
    __shared__ int s_ms[kNT];                             // and the slots
    __shared__ double s_post1[kNT], s_post2[kNT];         // what follows each thread's slots in S1 and S2

    if (tid == 0) {
        s_dead = 0;
        s_carry = s_c1 = s_c2 = 0.0;
        s_per_event = *A.per_event;
        for (int i = 0; i < 6; ++i) mbar_init(smem_addr(&s_mb[i / 2][i % 2]));
        mbar_init_fence();
    }
    if (WHERE <= 1)
        for (int p = tid; p < np; p += kNT) {
            if (SEG) fl[p] = A.flag[base_slot + p];
            if (WHERE == 0) {
                dd[p] = A.d[base_slot + p];
                nn[p] = A.n[base_slot + p];
            }
        }
    __syncthreads();
    auto starts = [&](int p) { return SEG && (fl[p] & 1); };
    auto ends = [&](int p) { return SEG && (fl[p] & 2); };
    // this thread's first slot that starts a stratum, whether one ends in its
    // slots, and whether one ends in the CTA's
    int first_start = m, has_end = 0;
    if (SEG)
        for (int i = mine - 1; i >= 0; --i) {
            if (starts(i * kNT + tid)) first_start = i;
            has_end |= ends(i * kNT + tid);
        }
    const int my_end = __syncthreads_or(has_end);
    if (C > 1) {
        cluster.sync();                                   // mbarriers are ready, peers are here
        if (tid < C) *cluster.map_shared_rank(&s_hasend[rank], tid) = my_end;
        cluster.sync();
    }

    int use[3] = {0, 0, 0};                               // exchanges of each kind so far
    // warp 0 exchanges nothing more once its wait ran out; its peers' next waits
    // run out too, and all stop together (agree)
    bool gone = false;
    auto wait = [&](int kind) {                           // warp 0
        const int i = use[kind];
        if (!mbar_wait(smem_addr(&s_mb[kind][i & 1]), (i >> 1) & 1, A.wait.of(rank))) { s_dead = 1; gone = true; }
    };
    // whether any CTA of the cluster lost the others, the same in every thread of them all
    auto agree = [&]() -> bool {
        __syncthreads();
        if (C > 1) {
            if (tid == 0 && *(volatile int*)&s_dead)
                for (int r = 0; r < C; ++r) *cluster.map_shared_rank(&s_dead, r) = 1;
            cluster.sync();
        }
        return *(volatile int*)&s_dead != 0;
    };
    int par = 0;                                          // of the next block scan

    // exclusive segmented sum over the threads in order: (f, a) of this thread
    // becomes the sum since the last segment start before it (f: there is one);
    // the block's own total in (tf, ta).  One __syncthreads.
    auto warp_up = [&](int& f, double& a) {               // inclusive, within the warp
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int uf = SEG ? __shfl_up_sync(kFull, f, o) : 0;
            const double ua = __shfl_up_sync(kFull, a, o);
            if (lane >= o) {
                if (!SEG || !f) a = ua + a;
                f |= uf;
            }
        }
    };
    // sum of v over the lanes [lo, hi) of the warps' totals (hi <= kNW)
    auto among = [&](double v, int lo, int hi) {
        v = lane >= lo && lane < hi ? v : 0.0;
        #pragma unroll
        for (int o = kNW / 2; o; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
        return __shfl_sync(kFull, v, 0);
    };
    auto scan_up = [&](int& f, double& a, int& tf, double& ta) {
        warp_up(f, a);
        if (lane == 31) { s_f[par][warp] = f; s_a[par][warp] = a; }
        int ef = SEG ? __shfl_up_sync(kFull, f, 1) : 0;
        double ea = __shfl_up_sync(kFull, a, 1);
        if (lane == 0) { ef = 0; ea = 0.0; }
        __syncthreads();
        if constexpr (kNW <= 8) {                         // few totals: in order
            int pf = 0, qf = 0;
            double pa = 0.0, qa = 0.0;
            #pragma unroll
            for (int w = 0; w < kNW; ++w) {
                if (w == warp) { pf = qf; pa = qa; }
                const int wf = SEG ? s_f[par][w] : 0;
                qa = SEG && wf ? s_a[par][w] : qa + s_a[par][w];
                qf |= wf;
            }
            tf = qf;
            ta = qa;
            a = ef ? ea : pa + ea;
            f = ef | pf;
            par ^= 1;
            return;
        }
        const double wa = s_a[par][lane & (kNW - 1)];
        const unsigned fm = SEG ? __ballot_sync(kFull, lane < kNW && s_f[par][lane & (kNW - 1)]) : 0u;
        const unsigned before = fm & ((1u << warp) - 1u);
        const double pa = among(wa, before ? 31 - __clz(before) : 0, warp);
        if (C > 1 && warp == 0) {                         // the block's total, for the peers
            tf = fm != 0;
            ta = among(wa, fm ? 31 - __clz(fm) : 0, kNW);
        }
        a = ef ? ea : pa + ea;
        f = ef | (before != 0);
        par ^= 1;
    };
    // the same over the threads in reverse, for two sums (f: a segment ends)
    auto scan_down = [&](int f, double& a, double& b, double& ta, double& tb) {
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int uf = SEG ? __shfl_down_sync(kFull, f, o) : 0;
            const double ua = __shfl_down_sync(kFull, a, o), ub = __shfl_down_sync(kFull, b, o);
            if (lane + o < 32) {
                if (!SEG || !f) { a += ua; b += ub; }
                f |= uf;
            }
        }
        if (lane == 0) { s_f[par][warp] = f; s_a[par][warp] = a; s_b[par][warp] = b; }
        int ef = SEG ? __shfl_down_sync(kFull, f, 1) : 0;
        double ea = __shfl_down_sync(kFull, a, 1), eb = __shfl_down_sync(kFull, b, 1);
        if (lane == 31) { ef = 0; ea = eb = 0.0; }
        __syncthreads();
        if constexpr (kNW <= 8) {
            double pa = 0.0, pb = 0.0, qa = 0.0, qb = 0.0;
            #pragma unroll
            for (int w = kNW - 1; w >= 0; --w) {
                if (w == warp) { pa = qa; pb = qb; }
                const int wf = SEG ? s_f[par][w] : 0;
                qa = SEG && wf ? s_a[par][w] : qa + s_a[par][w];
                qb = SEG && wf ? s_b[par][w] : qb + s_b[par][w];
            }
            ta = qa;
            tb = qb;
            a = ef ? ea : ea + pa;
            b = ef ? eb : eb + pb;
            par ^= 1;
            return;
        }
        const double wa = s_a[par][lane & (kNW - 1)], wb = s_b[par][lane & (kNW - 1)];
        const unsigned fm = SEG ? __ballot_sync(kFull, lane < kNW && s_f[par][lane & (kNW - 1)]) : 0u;
        const unsigned after = fm & ~((2u << warp) - 1u);
        const int hi = after ? __ffs(after) : kNW;        // the first later warp with an end, included
        const double pa = among(wa, warp + 1, hi), pb = among(wb, warp + 1, hi);
        if (C > 1 && warp == 0) {
            const int h0 = fm ? __ffs(fm) : kNW;
            ta = among(wa, 0, h0);
            tb = among(wb, 0, h0);
        }
        a = ef ? ea : ea + pa;
        b = ef ? eb : eb + pb;
        par ^= 1;
    };

    // The risk-set sum before this thread's first slot (where no stratum starts
    // in between); leaves the sums before each block of its slots in `bp` and
    // the last block's increments in dv.
    double dv[kB];
    auto risk_prefix = [&]() -> double {
        double a = 0.0, nx[kB];
        #pragma unroll
        for (int u = 0; u < kB; ++u) nx[u] = nb > 0 ? dd[u * kNT + tid] : 0.0;
        for (int b = 0; b < nb; ++b) {
            #pragma unroll
            for (int u = 0; u < kB; ++u) dv[u] = nx[u];
            if (b + 1 < nb) {
                #pragma unroll
                for (int u = 0; u < kB; ++u) nx[u] = dd[((b + 1) * kB + u) * kNT + tid];
            }
            bp[b * kNT + tid] = a;
            #pragma unroll
            for (int u = 0; u < kB; ++u) a = starts((b * kB + u) * kNT + tid) ? dv[u] : a + dv[u];
        }
        int f = SEG && first_start < mine, tf = 0;
        double ta = 0.0;
        scan_up(f, a, tf, ta);
        if (C > 1) {
            if (warp == 0) {
                const int i = use[0] & 1;
                const unsigned mb = smem_addr(&s_mb[0][i]);
                if (!gone) {
                    if (lane == 0) mbar_expect(mb, 16 * C);
                    if (lane < C)
                        push16(peer_addr(smem_addr(&x_a[i][rank]), lane), peer_addr(mb, lane), ta, tf ? 1.0 : 0.0);
                    wait(0);
                }
                double c = 0.0;
                for (int r = 0; r < rank; ++r) {
                    const double2 t = x_a[i][r];
                    c = t.y != 0.0 ? t.x : c + t.x;
                }
                if (lane == 0) s_carry = c;
            }
            ++use[0];
            __syncthreads();
            if (!f) a = s_carry + a;
        }
        return a;
    };
    // the risk-set sums of block b's slots in `out` from the increments `in` (1
    // past the thread's last slot)
    auto risk_sums = [&](int b, double pre, const double (&in)[kB], double (&out)[kB]) {
        double run = bp[b * kNT + tid];
        #pragma unroll
        for (int u = 0; u < kB; ++u) {
            const int i = b * kB + u;
            run = starts(i * kNT + tid) ? in[u] : run + in[u];
            out[u] = i >= mine ? 1.0 : (!SEG || i < first_start ? pre + run : run);
        }
    };

    // S1, S2 from the risk-set increments (computeAccumlatedDenominator and the
    // n/D terms, ModelSpecifics.hpp:1670-1694), the thread's slots from the last
    // to the first; what follows them in the stratum is left in s_post1/2 (later
    // threads) and s_c1/2 (later CTAs) for the entries to add.
    auto renew = [&]() {
        const double pre = risk_prefix();
        double a1 = 0.0, a2 = 0.0;
        double nv[kB];
        #pragma unroll
        for (int u = 0; u < kB; ++u) nv[u] = nb > 0 ? nn[((nb - 1) * kB + u) * kNT + tid] : 0.0;
        for (int b = nb - 1; b >= 0; --b) {
            double D[kB], q1[kB], dx[kB], nx[kB];
            if (b > 0) {                                  // the next block's loads are in flight
                #pragma unroll
                for (int u = 0; u < kB; ++u) {
                    const int p = ((b - 1) * kB + u) * kNT + tid;
                    dx[u] = dd[p];
                    nx[u] = nn[p];
                }
            }
            risk_sums(b, pre, dv, D);
            #pragma unroll
            for (int u = 0; u < kB; ++u) {
                const double inv = 1.0 / D[u];            // one division for both terms
                D[u] = nv[u] != 0.0 ? inv : 0.0;          // (without events D may be anything)
                q1[u] = nv[u] * D[u];
            }
            #pragma unroll
            for (int u = kB - 1; u >= 0; --u) {
                const int p = (b * kB + u) * kNT + tid;
                const double q2 = q1[u] * D[u];
                const bool en = ends(p);
                a1 = en ? q1[u] : a1 + q1[u];
                a2 = en ? q2 : a2 + q2;
                S1[p] = a1;
                S2[p] = a2;
            }
            #pragma unroll
            for (int u = 0; u < kB; ++u) {
                dv[u] = dx[u];
                nv[u] = nx[u];
            }
        }
        double t1 = 0.0, t2 = 0.0;
        scan_down(has_end, a1, a2, t1, t2);
        s_post1[tid] = a1;
        s_post2[tid] = a2;
        if (C > 1 && warp == 0) {                         // what follows in the later CTAs
            const int ic = use[2] & 1;
            const unsigned mb = smem_addr(&s_mb[2][ic]);
            if (!gone) {
                if (lane == 0) mbar_expect(mb, 16 * C);
                if (lane < C) push16(peer_addr(smem_addr(&x_c[ic][rank]), lane), peer_addr(mb, lane), t1, t2);
                wait(2);
            }
            double c1 = 0.0, c2 = 0.0;
            for (int r = C - 1; r > rank; --r) {
                const double2 t = x_c[ic][r];
                if (SEG && s_hasend[r]) { c1 = t.x; c2 = t.y; }
                else { c1 += t.x; c2 += t.y; }
            }
            if (lane == 0) { s_c1 = c1; s_c2 = c2; }
        }
        ++use[2];
        __syncthreads();
    };

    // (a, b) summed over the cluster's threads, the same in every thread
    auto sum2 = [&](double& a, double& b) {
        for (int o = 16; o; o >>= 1) {
            a += __shfl_xor_sync(kFull, a, o);
            b += __shfl_xor_sync(kFull, b, o);
        }
        __syncthreads();
        if (lane == 0) { s_sum[0][warp] = a; s_sum[1][warp] = b; }
        __syncthreads();
        a = b = 0.0;
        for (int q = 0; q < kNW; ++q) { a += s_sum[0][q]; b += s_sum[1][q]; }
        if (C > 1) {
            const int i = use[0] & 1;
            if (warp == 0) {
                const unsigned mb = smem_addr(&s_mb[0][i]);
                if (!gone) {
                    if (lane == 0) mbar_expect(mb, 16 * C);
                    if (lane < C) push16(peer_addr(smem_addr(&x_a[i][rank]), lane), peer_addr(mb, lane), a, b);
                    wait(0);
                }
            }
            ++use[0];
            __syncthreads();
            a = b = 0.0;
            for (int r = 0; r < C; ++r) { a += x_a[i][r].x; b += x_a[i][r].y; }
        }
        __syncthreads();
    };

    // getLogLikelihood (ModelSpecifics.hpp:605-650)
    auto log_likelihood = [&]() -> double {
        const double pre = risk_prefix();
        double a = 0.0, b = 0.0;
        for (int g = 0; g < nb; ++g) {
            double D[kB];
            #pragma unroll
            for (int u = 0; u < kB; ++u) dv[u] = dd[(g * kB + u) * kNT + tid];
            risk_sums(g, pre, dv, D);
            #pragma unroll
            for (int u = 0; u < kB; ++u) {
                const double n = nn[(g * kB + u) * kNT + tid], l = n * log(D[u]);
                if (n != 0.0) b += l;
            }
        }
        for (int k = tid; k < nr; k += kNT) {
            if (A.predict) {
                const double w = wg ? wg[k] : 1.0;
                if (w != 0.0) a += A.y[r0 + k] * w * xg[k];
            } else if ((int)A.y[r0 + k] == 1) {
                a += wg ? xg[k] * wg[k] : xg[k];
            }
        }
        sum2(a, b);
        return a - b;
    };
    auto objective = [&]() -> double {
        double a = 0.0, b = 0.0;
        switch (A.conv) {
        case CYC_CONV_GRADIENT:
            for (int k = tid; k < nr; k += kNT) a += xg[k] * A.y[r0 + k] * (wg ? wg[k] : 1.0);
            sum2(a, b);
            return a;
        case CYC_CONV_MITTAL: return log_likelihood();
        case CYC_CONV_LANGE:
            a = log_likelihood();
            {
                double p = 0.0, u = 0.0;
                if (rank == 0)
                    for (int j = tid; j < A.J; j += kNT) p += log_density(A.ptype[j], var, A.beta[j]);
                sum2(p, u);
                return a + p;
            }
        case CYC_CONV_ZHANG_OLES:                         // renews xb_save
            for (int k = tid; k < nr; k += kNT) {
                const double w = wg ? wg[k] : 1.0, v = xg[k];
                a += fabs(v - A.xb_save[r0 + k]) * w;
                b += fabs(v) * w;
                A.xb_save[r0 + k] = v;
            }
            sum2(a, b);
            return a / (1.0 + b);
        default: return 0.0;                              // ONE_STEP
        }
    };

    if (A.max_iter == 0 && !A.score) {
        const double ll = log_likelihood();
        const bool dead = agree();
        if (rank == 0 && tid == 0) {
            *A.out_ll = ll;
            *A.out_iter = 0;
            *A.out_flag = dead ? kTimedOut : CYC_SUCCESS;
        }
        if (dead) stores_land();
        if (C > 1) cluster.sync();
        return;
    }
    // The increments formed again from the predictors, once a cycle: a step adds
    // its change of a slot to them, and the rounding adds up.  A warp takes 32
    // rows; the last of a slot's rows in it adds their sum.  A slot's rows lie in
    // two warps at most, so the order of the two does not matter.  (A thread
    // walking its slots' rows took 65 us a cycle at 20k rows and 350 at 500k;
    // 15 and 54 this way.)
    auto reform = [&]() {
        for (int p = tid; p < np; p += kNT) dd[p] = 0.0;
        __syncthreads();
        constexpr int kU = 4;
        for (int k0 = warp * 32; k0 < nr; k0 += kU * kNT) {
            int slot[kU];
            double v[kU], w[kU];
            #pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int k = k0 + u * kNT + lane;
                slot[u] = k < nr ? __ldg(A.rowslot + r0 + k) : -1;
                v[u] = k < nr ? xg[k] : 0.0;
                w[u] = k < nr && wg ? __ldg(wg + k) : 1.0;
            }
            #pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int p = slot[u] >= 0 ? slot[u] & kPosMask : -1 - lane;
                double a = slot[u] >= 0 && w[u] != 0.0 ? w[u] * exp(v[u]) : 0.0;
                #pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int up = __shfl_up_sync(kFull, p, o);
                    const double ua = __shfl_up_sync(kFull, a, o);
                    if (lane >= o && up == p) a += ua;
                }
                const int next = __shfl_down_sync(kFull, p, 1);
                if (p >= 0 && (lane == 31 || next != p)) atomicAdd(dd + p, a);
            }
        }
        __syncthreads();
    };
    double last = A.conv == CYC_CONV_ZHANG_OLES || A.score ? 0.0 : objective();
    renew();
    const int ncols = *A.ncols;
    int it = 0, flag = CYC_SUCCESS;
    for (;;) {
        for (int base = 0; base < ncols; base += kCh) {
            const int jn = min(kCh, ncols - base);
            __syncthreads();
            if (tid == 0) c_m[jn] = ColMeta{A.idx, nullptr, A.rowslot, nullptr, 0, 0};
            for (int q = tid; q < jn; q += kNT) {
                const int j = A.cols[base + q];
                const int fm = A.fmt[j];
                const bool dn = (fm == CYC_DENSE || fm == CYC_INTERCEPT);
                const int e0 = dn ? r0 : A.split[j * (C + 1) + rank];
                const int e1 = dn ? r0 + nr : A.split[j * (C + 1) + rank + 1];
                ColMeta c;
                c.ci = dn ? nullptr : A.idx + A.col_ptr[j] + e0;
                c.cv = (fm == CYC_SPARSE || fm == CYC_DENSE) ? A.val + A.val_ptr[j] + e0 : nullptr;
                c.es = dn ? A.rowslot + r0 : A.entry + A.col_ptr[j] + e0;
                c.st = !A.entry_strat ? nullptr : (dn ? A.strat + r0 : A.entry_strat + A.col_ptr[j] + e0);
                c.n = e1 - e0;
                c.before = e0 > 0;
                c_m[q] = c;
                c_j[q] = j;
                c_pt[q] = A.ptype[j];
                c_beta[q] = A.beta[j];
                c_hd[q] = A.hdelta[j];
                c_xjy[q] = A.xjy[j];
            }
            __syncthreads();
            // Columns of at most kNT - 32 entries in this CTA have one entry a
            // thread, from the second warp on: the first combines the sums and
            // takes the step while the others load the next column: its entry's
            // row, value, slot (and the one before), whether it starts a
            // stratum's entries; then the row's state.
            const int te = tid - 32;
            ColMeta nm = c_m[0];
            int nk = -1, nslot = -1, npslot = -1, nst = -1, npst = -1;
            double nx = 1.0, nxb = 0.0, nw = 1.0;
            auto load_ids = [&](int q) {
                nm = c_m[q];
                nk = nslot = npslot = nst = npst = -1;
                nx = 1.0;
                if (nm.n <= kNT - 32 && te >= 0 && te < nm.n) {
                    if (nm.ci) nk = __ldg(nm.ci + te);
                    else nk = r0 + te;
                    if (nm.cv) nx = __ldg(nm.cv + te);
                    nslot = __ldg(nm.es + te);
                    if (te > 0) npslot = __ldg(nm.es + te - 1);
                    if (SEG) {
                        nst = __ldg(nm.st + te);
                        if (te > 0 || nm.before) npst = __ldg(nm.st + te - 1);
                    }
                }
            };
            auto load_rows = [&]() {
                if (nk >= 0) {
                    nxb = xg[nk - r0];
                    if (wg) nw = __ldg(wg + nk - r0);
                }
            };
            load_ids(0);
            load_rows();
            for (int q = 0; q < jn; ++q) {
                const ColMeta c = nm;
                const bool one = c.n <= kNT - 32;         // one entry a thread at most
                const int per = (c.n + kNT - 1) / kNT;    // entries a thread otherwise, in order
                const int i0 = tid * per, i1 = min(c.n, i0 + per);
                const int k1 = nk - r0, slot1 = nslot, pslot1 = npslot;
                const double x1 = nx, xb1 = nxb, w1 = nw;
                const bool start1 = SEG && nst != npst;
                const bool ind = c.cv == nullptr;
                const double c1 = s_c1, c2 = s_c2;
                // ---- the column's sums
                double g = 0.0, h = 0.0, a = 0.0, vh2 = 0.0, ex1 = 0.0;
                int f = 0;
                auto entry = [&](double v, double x, int slot, bool start) {
                    if (SEG && start) { f = 1; a = 0.0; }
                    if (slot >= 0) {
                        const int p = slot & kPosMask;
                        const int t = p & (kNT - 1);      // the slot's thread
                        const double o1 = (slot & kThreadBit ? s_post1[t] : 0.0) + (slot & kTailBit ? c1 : 0.0);
                        const double o2 = (slot & kThreadBit ? s_post2[t] : 0.0) + (slot & kTailBit ? c2 : 0.0);
                        const double t1 = S1[p] + o1, t2 = S2[p] + o2;
                        g += v * t1;
                        h += v * x * t1 - v * (2.0 * a + v) * t2;
                        if (!SEG || !f) vh2 += v * t2;
                        a += v;
                    }
                };
                if (one) {
                    if (k1 >= 0) {
                        ex1 = exp(xb1);
                        const double w = wg ? w1 : 1.0;
                        entry(w != 0.0 ? w * ex1 * x1 : 0.0, x1, slot1, start1);
                    }
                } else {
                    for (int i = i0; i < i1; ++i) {
                        const int k = (c.ci ? __ldg(c.ci + i) - r0 : i);
                        const double x = ind ? 1.0 : __ldg(c.cv + i);
                        const bool st = SEG && ((i == 0 && !c.before) || __ldg(c.st + i) != __ldg(c.st + i - 1));
                        const int slot = __ldg(c.es + i);
                        const double w = wg ? __ldg(wg + k) : 1.0;
                        entry(slot >= 0 && w != 0.0 ? w * exp(xg[k]) * x : 0.0, x, slot, st);
                    }
                }
                // the threads' sums to the warp's: what precedes a thread in its
                // warp enters through the running sum, as what precedes a warp in
                // its CTA and a CTA in the cluster does below
                {
                    int wf = f;
                    double wa = a;
                    warp_up(wf, wa);
                    int ef = SEG ? __shfl_up_sync(kFull, wf, 1) : 0;
                    double ea = __shfl_up_sync(kFull, wa, 1);
                    if (lane == 0) { ef = 0; ea = 0.0; }
                    h -= 2.0 * ea * vh2;
                    if (SEG && ef) vh2 = 0.0;             // not reached by what precedes the warp
                    if (lane == 31) { s_sum[3][warp] = wa; s_sum[4][warp] = wf ? 1.0 : 0.0; }
                    // three sums at once: lanes keep (g, vh2) or h, then one value
                    const bool up = (lane & 16) != 0;
                    double u0 = up ? h : g, u1 = up ? 0.0 : vh2;
                    u0 += __shfl_xor_sync(kFull, up ? g : h, 16);
                    u1 += __shfl_xor_sync(kFull, up ? vh2 : 0.0, 16);
                    const bool up8 = (lane & 8) != 0;
                    double u = up8 ? u1 : u0;
                    u += __shfl_xor_sync(kFull, up8 ? u0 : u1, 8);
                    u += __shfl_xor_sync(kFull, u, 4);
                    u += __shfl_xor_sync(kFull, u, 2);
                    u += __shfl_xor_sync(kFull, u, 1);
                    if (lane == 0) s_sum[0][warp] = u;
                    if (lane == 16) s_sum[1][warp] = u;
                    if (lane == 8) s_sum[2][warp] = u;
                }
                __syncthreads();
                const int ib = use[1] & 1;
                if (warp == 0) {
                    g = h = vh2 = 0.0;
                    double pre = 0.0;                     // the running sum that reaches warp w
                    int tf = 0;
                    #pragma unroll
                    for (int w = 0; w < kNW; ++w) {
                        const double wa = s_sum[3][w], v2 = s_sum[2][w];
                        const bool wf = SEG && s_sum[4][w] != 0.0;
                        g += s_sum[0][w];
                        h += s_sum[1][w] - 2.0 * pre * v2;
                        if (!tf) vh2 += v2;
                        tf |= wf;
                        pre = wf ? wa : pre + wa;
                    }
                    if (C > 1) {
                        const unsigned mb = smem_addr(&s_mb[1][ib]);
                        if (!gone) {
                            if (lane == 0) mbar_expect(mb, 48 * C);
                            if (lane < C) {
                                const unsigned pm = peer_addr(mb, lane);
                                push16(peer_addr(smem_addr(&x_b[ib][0][rank]), lane), pm, g, h);
                                push16(peer_addr(smem_addr(&x_b[ib][1][rank]), lane), pm, vh2, pre);
                                push16(peer_addr(smem_addr(&x_b[ib][2][rank]), lane), pm, tf ? 1.0 : 0.0, 0.0);
                            }
                            wait(1);
                        }
                        g = h = pre = 0.0;
                        for (int r = 0; r < C; ++r) {
                            const double2 b0 = x_b[ib][0][r], b1 = x_b[ib][1][r];
                            g += b0.x;
                            h += b0.y - 2.0 * pre * b1.x;
                            pre = SEG && x_b[ib][2][r].x != 0.0 ? b1.y : pre + b1.y;
                        }
                    }
                    // ---- the coordinate step (ccdUpdateBeta :1394-1413, applyBounds :1503-1520)
                    // A column that is constant in every risk set has g = h = 0, which
                    // these sums give to their rounding only (A / D is x there where it is
                    // formed), and -g / h of two such numbers is any step.  Their scales:
                    // sum v S1, and sum v x S1 or, for values, its bound (sum v S1)^2 / events.
                    if (lane == 0) {
                        const double sum = g;
                        g -= c_xjy[q];                    // :1181-1183
                        const double near = kZero * (fabs(sum) + fabs(c_xjy[q]));
                        if (fabs(g) <= near && near <= 1e300 &&
                            h <= kZero * (c_m[q].cv ? sum * sum * s_per_event : fabs(sum)))
                            g = h = 0.0;
                        if (A.score) {
                            s_dl = 0.0;
                            if (rank == 0) A.score[base + q] = fabs(g);
                        } else {
                            if (h < 0.0) { g = 0.0; h = 0.0; }
                            const double b = c_beta[q];
                            double hd = c_hd[q];
                            double dl = prior_delta_rate(c_pt[q], var, lam, b, g, h);
                            dl = apply_bounds(&hd, dl);
                            s_dl = dl;
                            c_oh[q] = hd;
                            c_ob[q] = dl != 0.0 ? b + dl : b;
                            c_up[q] = dl != 0.0;
                        }
                    }
                }
                ++use[1];
                load_ids(q + 1);
                load_rows();                              // as they are if nothing moves
                __syncthreads();
                const double dl = s_dl;
                if (dl == 0.0) continue;
                // ---- updateXBeta: the first entry of each run of one slot takes the
                // run, with its change of the slot's increment
                auto move = [&](int i, int slot, double acc) {
                    for (; i < c.n && __ldg(c.es + i) == slot; ++i) {
                        const int k = c.ci ? __ldg(c.ci + i) - r0 : i;
                        const double x = ind ? 1.0 : __ldg(c.cv + i), w = wg ? __ldg(wg + k) : 1.0;
                        const double old = xg[k], v = add_mul_rn(old, dl, x);
                        xg[k] = v;
                        if (w != 0.0) acc += w * exp(v) - w * exp(old);
                    }
                    dd[slot & kPosMask] = acc;
                };
                if (one) {
                    if (k1 >= 0) {
                        const double v = add_mul_rn(xb1, dl, x1), w = wg ? w1 : 1.0;
                        xg[k1] = v;
                        s_mv[tid] = w != 0.0 ? w * exp(v) - w * ex1 : 0.0;
                        s_ms[tid] = slot1;
                    }
                    __syncthreads();
                    if (k1 >= 0 && slot1 >= 0 && slot1 != pslot1) {
                        double acc = dd[slot1 & kPosMask];
                        for (int i = tid; i < 32 + c.n && s_ms[i] == slot1; ++i) acc += s_mv[i];
                        dd[slot1 & kPosMask] = acc;
                    }
                } else {
                    for (int i = i0; i < i1; ++i) {
                        const int slot = __ldg(c.es + i);
                        if (slot < 0) {
                            const int k = c.ci ? __ldg(c.ci + i) - r0 : i;
                            xg[k] = add_mul_rn(xg[k], dl, ind ? 1.0 : __ldg(c.cv + i));
                        } else if (i == 0 || __ldg(c.es + i - 1) != slot) {
                            move(i, slot, dd[slot & kPosMask]);
                        }
                    }
                }
                __syncthreads();
                load_rows();                              // while the suffix sums are renewed
                renew();
            }
            __syncthreads();
            if (rank == 0 && !A.score)
                for (int q = tid; q < jn; q += kNT) {
                    const int j = c_j[q];
                    A.beta[j] = c_ob[q];
                    A.hdelta[j] = c_oh[q];
                    if (c_up[q]) A.col_updates[j] += 1u;
                }
        }
        if (A.score) break;
        // ---- performCheckConvergence (:839-906)
        ++it;
        __syncthreads();
        if (C > 1) cluster.sync();    // rank 0's coefficients are staged by every CTA in the next cycle
        reform();
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
        if (agree()) break;
        if (A.tol > 0 && conv < A.tol) { flag = ill ? CYC_ILLCONDITIONED : CYC_SUCCESS; break; }
        if (it == A.max_iter) { flag = CYC_MAX_ITERATIONS; break; }
    }
    const double ll = A.score ? 0.0 : log_likelihood();
    if (agree()) {
        flag = kTimedOut;
        stores_land();
    }
    if (C > 1) cluster.sync();       // no CTA leaves while others may still write its shared memory
    if (rank == 0 && tid == 0) {
        *A.out_ll = ll;
        *A.out_iter = it;
        *A.out_flag = flag;
    }
}

constexpr size_t kSmemBytes = 200 * 1024;

template <int WHERE, int kNT, bool SEG>
void launch_where(const CoxArgs* d_fits, int F, int C, size_t dyn, cudaStream_t stream) {
    auto kern = k_cox<WHERE, kNT, SEG>;
    CYC_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
    if (C > 8) CYC_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(F * C);
    cfg.blockDim = dim3(kNT);
    cfg.dynamicSmemBytes = dyn;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CYC_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, d_fits, C));
    count_launch();
}

}  // namespace

// shared bytes of a CTA of `threads` with room for `per_cta` slots: all per-slot
// arrays, or S1 and S2 alone, the block sums and the flags
static size_t cox_bytes(int threads, int per_cta, bool all) {
    const size_t m = (size_t)per_cta / threads;
    return threads * (m * (all ? 32 : 16) + m / kB * sizeof(double) + m);
}

// 0: all per-slot arrays in shared memory, 1: S1 and S2, 2: none
static int cox_where(CoxShape s) {
    if (cox_bytes(s.threads, s.per_cta, true) <= kSmemBytes) return 0;
    return s.threads == kCoxThreads && cox_bytes(s.threads, s.per_cta, false) <= kSmemBytes ? 1 : 2;
}

template <bool SEG>
static void launch_seg(const CoxArgs* d_fits, int F, CoxShape s, cudaStream_t stream) {
    const int where = cox_where(s), C = s.C;
    const size_t dyn = where == 2 ? 0 : cox_bytes(s.threads, s.per_cta, where == 0);
    if (s.threads == 128) launch_where<0, 128, SEG>(d_fits, F, C, dyn, stream);
    else if (s.threads == 256) launch_where<0, 256, SEG>(d_fits, F, C, dyn, stream);
    else if (where == 0) launch_where<0, 512, SEG>(d_fits, F, C, dyn, stream);
    else if (where == 1) launch_where<1, 512, SEG>(d_fits, F, C, dyn, stream);
    else launch_where<2, 512, SEG>(d_fits, F, C, dyn, stream);
}

void launch_cox(const CoxArgs* d_fits, int F, CoxShape shape, bool strata, cudaStream_t stream) {
    if (strata) launch_seg<true>(d_fits, F, shape, stream);
    else launch_seg<false>(d_fits, F, shape, stream);
}

// (the slots count rows as well as events: 2M rows with 1,000 events are 63,000
// slots and take 16 CTAs of 512 threads, 103 -> 32 ms for 4 cycles of 22 columns)
CoxShape cox_shape(int slots) {
    CoxShape s{1, 128};
    while (s.C < kMaxC && slots > 128 * 8 * s.C) s.C *= 2;
    while (s.threads < kCoxThreads && slots > s.threads * 12 * s.C) s.threads *= 2;
    // CYC_COX_CLUSTER="CTAs[,threads]" fixes the shape
    if (const char* e = std::getenv("CYC_COX_CLUSTER")) {
        int c = s.C, t = s.threads;
        std::sscanf(e, "%d,%d", &c, &t);
        s.C = std::max(1, std::min(kMaxC, c));
        s.threads = t <= 128 ? 128 : t <= 256 ? 256 : 512;
    }
    // 128 and 256 threads keep every per-slot array in shared memory
    const auto round_up = [&](int n) { return (n + kB * s.threads - 1) / (kB * s.threads) * (kB * s.threads); };
    const int even = std::max(1, (slots + s.C - 1) / s.C);
    while (s.threads < kCoxThreads && cox_bytes(s.threads, round_up(even), true) > kSmemBytes) s.threads *= 2;
    // room for up to twice the even share of the slots, as far as the arrays stay where the even share's are
    s.per_cta = round_up(2 * even);
    while (s.per_cta > round_up(even) && cox_where(s) != cox_where({s.C, s.threads, round_up(even)}))
        s.per_cta -= kB * s.threads;
    return s;
}

void CoxSlots::find(const double* d_w, cudaStream_t stream) {
    const int K = ds.K, nt = (K + kTile - 1) / kTile;
    const double* y = ds.d_y.get();
    const int* strat = ds.d_strat.get();
    const int events = std::max(1, ds.event_rows());
    cnt.alloc(K);
    tiles.alloc(nt);
    gend.alloc(events); first.alloc(events); glo.alloc(events); gstr.alloc(events); gcum.alloc(events);
    groups.alloc(1);
    const int* lastp = nullptr;
    if (d_w) {
        last.alloc(K);
        const LastWeighted item{d_w};
        launch(k_rows_totals<OpMax, LastWeighted>, nt, kThreads, 0, stream, K, item, tiles.get());
        launch(k_tiles_scan<OpMax>, 1, kThreads, 0, stream, nt, tiles.get());
        launch(k_rows_scan<OpMax, LastWeighted>, nt, kThreads, 0, stream, K, item, (const int*)tiles.get(), last.get());
        lastp = last.get();
    }
    const GroupStart item{d_w, y, ds.d_time.get(), strat, lastp};
    launch(k_rows_totals<OpSum, GroupStart>, nt, kThreads, 0, stream, K, item, tiles.get());
    launch(k_tiles_scan<OpSum>, 1, kThreads, 0, stream, nt, tiles.get());
    launch(k_rows_scan<OpSum, GroupStart>, nt, kThreads, 0, stream, K, item, (const int*)tiles.get(), cnt.get());
    CYC_CHECK_CUDA(cudaMemsetAsync(gend.get(), 0xff, events * sizeof(int), stream));
    launch(k_slot_rows, grid_for(K, 1), kThreads, 0, stream, K, d_w, y, strat, (const int*)cnt.get(), first.get(),
           gend.get(), gstr.get(), groups.get());
    // each group's rows, and the slots they are cut into
    launch(k_group_rows, grid_for(events, 1), kThreads, 0, stream, (const int*)groups.get(), (const int*)gend.get(),
           (const int*)gstr.get(), (const int*)ds.d_strat_ptr.get(), glo.get());
    const Pieces pieces{groups.get(), glo.get(), gend.get()};
    const int gt = (events + kTile - 1) / kTile;          // (no more tiles than the rows have)
    launch(k_rows_totals<OpSum, Pieces>, gt, kThreads, 0, stream, events, pieces, tiles.get());
    launch(k_tiles_scan<OpSum>, 1, kThreads, 0, stream, gt, tiles.get());
    launch(k_rows_scan<OpSum, Pieces>, gt, kThreads, 0, stream, events, pieces, (const int*)tiles.get(), gcum.get());
    CYC_CHECK_CUDA(cudaMemcpyAsync(&n_slots, gcum.get() + events - 1, sizeof(int), cudaMemcpyDeviceToHost, stream));
}

void CoxSlots::build(CoxShape s, const double* d_w, cudaStream_t stream) {
    shape = s;
    const int K = ds.K, C = shape.C, threads = shape.threads, room = std::max(1, n_slots);
    lo.alloc(room); end.alloc(room); sstr.alloc(room);
    rowslot.alloc(K); rpart.alloc(C + 1); spart.alloc(C + 1);
    split.alloc((size_t)ds.J * (C + 1));
    entry.alloc(std::max<long long>(1, ds.nnz_idx));
    flag.alloc(positions()); n.alloc(positions()); per_event.alloc(1);
    // positions past the slots read as empty
    CYC_CHECK_CUDA(cudaMemsetAsync(n.get(), 0, n.bytes(), stream));
    CYC_CHECK_CUDA(cudaMemsetAsync(flag.get(), 0, flag.bytes(), stream));
    const Groups G{groups.get(), cnt.get(), glo.get(), gend.get(), gstr.get(), gcum.get()};
    const int events = std::max(1, ds.event_rows());
    launch(k_slot_fill, grid_for(32ll * events, 1), kThreads, 0, stream, G, lo.get(), end.get(), sstr.get());
    launch(k_slot_parts, 1, 32 * kMaxC, 0, stream, K, C, n_slots, shape.per_cta, G, (const int*)end.get(), spart.get(),
           rpart.get());
    launch(k_slots, grid_for(32ll * events, 1), kThreads, 0, stream, C, threads, shape.per_cta, G,
           (const int*)spart.get(), (const int*)first.get(), d_w, (const double*)ds.d_y.get(), flag.get(), n.get());
    launch(k_per_event, 1, 1024, 0, stream, (int)positions(), (const double*)n.get(), per_event.get());
    launch(k_row_slots, grid_for(K, 1), kThreads, 0, stream, K, C, threads, n_slots, G, (const int*)spart.get(),
           (const int*)sstr.get(), (const int*)ds.d_strat.get(), rowslot.get());
    if (ds.nnz_idx)
        launch(k_entry_slots, grid_for(ds.nnz_idx, 4), kThreads, 0, stream, ds.nnz_idx, (const int*)ds.d_idx.get(),
               (const int*)rowslot.get(), entry.get());
    ccd_splits(ds, C, rpart.get(), split.get(), stream);
}

void CoxSlots::increments(const double* d_xb, const double* d_w, double* out, cudaStream_t stream) const {
    CYC_CHECK_CUDA(cudaMemsetAsync(out, 0, positions() * sizeof(double), stream));   // past the slots: empty
    launch(k_slot_increments, grid_for(32ll * std::max(1, n_slots), 1), kThreads, 0, stream, shape.C, shape.threads,
           shape.per_cta, n_slots, (const int*)spart.get(), (const int*)lo.get(), (const int*)end.get(), d_w, d_xb, out);
}

CoxState::CoxState(const CoxSlots& s, int F) : np(s.positions()) {
    const int where = cox_where(s.shape);
    d.alloc(F * np);
    if (where == 2) { S1.alloc(F * np); S2.alloc(F * np); bp.alloc(F * np / kB); }
}

void CoxState::set(CoxArgs& a, int f) const {
    a.d = d.get() + f * np;
    if (S1.get()) { a.S1 = S1.get() + f * np; a.S2 = S2.get() + f * np; a.bp = bp.get() + f * np / kB; }
}

CoxArgs CoxSlots::args() const {
    CoxArgs a{};
    a.K = ds.K; a.J = ds.J; a.per_cta = shape.per_cta;
    a.fmt = ds.d_fmt.get(); a.col_ptr = ds.d_col_ptr.get(); a.val_ptr = ds.d_val_ptr.get();
    a.idx = ds.d_idx.get(); a.val = ds.d_val.get();
    a.entry = entry.get(); a.rowslot = rowslot.get();
    if (ds.S > 1) {
        ds.ensure_entry_strata();
        a.entry_strat = ds.d_entry_strat.get();
    }
    a.strat = ds.d_strat.get();
    a.split = split.get(); a.rpart = rpart.get(); a.spart = spart.get();
    a.flag = flag.get();
    a.n = n.get(); a.per_event = per_event.get(); a.y = ds.d_y.get();
    a.wait = wait_limit(ds.K);
    return a;
}

// ---- many fits -------------------------------------------------------------------

// the fits of one launch: their risk sets, the fits, the scores of `held`
static void run_cox_fits(Dataset& ds, const std::vector<int>& pt, const cyc_fit_spec* specs, int F,
                         const cyc_control* ctl, cyc_fit_result* out, const double* const* held, double* pred,
                         cudaStream_t stream, cyc_run_stats& st) {
    const int K = ds.K, J = ds.J;

    // one set of risk sets per weight vector of this call
    struct Weighting {
        const double* host;
        DevBuf<double> w, xjy;
        std::unique_ptr<CoxSlots> slots;
    };
    std::vector<std::unique_ptr<Weighting>> sets;
    auto weighting = [&](const double* h, bool with_xjy) -> Weighting& {
        for (auto& s : sets)
            if (s->host == h && (!with_xjy || s->xjy.get())) return *s;
        sets.emplace_back(new Weighting{h});
        Weighting& s = *sets.back();
        if (h) {
            CYC_REQUIRE(std::any_of(h, h + K, [](double v) { return v != 0.0; }), CYC_ERR_ARGUMENT,
                        "all weights are zero");
            s.w.alloc(K);
            CYC_CHECK_CUDA(cudaMemcpyAsync(s.w.get(), h, K * sizeof(double), cudaMemcpyHostToDevice, stream));
        }
        s.slots.reset(new CoxSlots(ds));
        s.slots->find(s.w.get(), stream);
        if (with_xjy) {
            s.xjy.alloc(J);
            launch_xjy(ds, s.w.get(), s.xjy.get(), stream);
        }
        return s;
    };
    // the slots of the weightings from `first` on, for one launch
    auto build = [&](size_t first) -> CoxShape {
        CYC_CHECK_CUDA(cudaStreamSynchronize(stream));
        int slots = 0;
        for (size_t i = first; i < sets.size(); ++i) slots = std::max(slots, sets[i]->slots->n_slots);
        const CoxShape shape = cox_shape(slots);
        for (size_t i = first; i < sets.size(); ++i) sets[i]->slots->build(shape, sets[i]->w.get(), stream);
        return shape;
    };

    DevBuf<double> xb, xb_save, beta, hdelta, ll;
    DevBuf<int> ptype, cols, ncols, flags;
    DevBuf<unsigned> updates;
    DevBuf<CoxArgs> d_args;
    xb.alloc((size_t)F * K); beta.alloc((size_t)F * J); hdelta.alloc((size_t)F * J); ll.alloc(F);
    ptype.alloc(J); cols.alloc((size_t)F * J); ncols.alloc(F); flags.alloc(2 * F); updates.alloc((size_t)F * J);
    d_args.alloc(F);
    const bool zhang = ctl->convergence_type == CYC_CONV_ZHANG_OLES;
    if (zhang) xb_save.alloc((size_t)F * K);
    CYC_CHECK_CUDA(cudaMemcpyAsync(ptype.get(), pt.data(), J * sizeof(int), cudaMemcpyHostToDevice, stream));
    CYC_CHECK_CUDA(cudaMemsetAsync(updates.get(), 0, updates.bytes(), stream));
    std::vector<int> h_cols((size_t)F * J), h_n(F);
    std::vector<double> h_beta((size_t)F * J, 0.0);
    std::vector<CoxArgs> args(F);
    std::vector<Weighting*> of(F);
    for (int f = 0; f < F; ++f) {
        std::vector<char> fixed(J, 0);
        if (ds.has_offset) fixed[0] = 1;
        for (int i = 0; i < specs[f].n_fixed; ++i) fixed[specs[f].fixed[i]] = 1;
        for (int j = 0; j < J; ++j)
            if (!fixed[j]) h_cols[(size_t)f * J + h_n[f]++] = j;
        double* b = h_beta.data() + (size_t)f * J;
        if (specs[f].start_beta) std::copy(specs[f].start_beta, specs[f].start_beta + J, b);
        if (ds.has_offset) b[0] = 1.0;
        of[f] = &weighting(specs[f].weights, true);
    }
    CoxShape shape = build(0);
    std::unique_ptr<CoxState> state(new CoxState(*sets[0]->slots, F));
    CYC_CHECK_CUDA(cudaMemcpyAsync(cols.get(), h_cols.data(), cols.bytes(), cudaMemcpyHostToDevice, stream));
    CYC_CHECK_CUDA(cudaMemcpyAsync(ncols.get(), h_n.data(), F * sizeof(int), cudaMemcpyHostToDevice, stream));
    for (int f = 0; f < F; ++f) {
        CoxArgs a = of[f]->slots->args();
        a.weighted = of[f]->host != nullptr;
        a.w = of[f]->w.get();
        a.xb = xb.get() + (size_t)f * K;
        a.xb_save = zhang ? xb_save.get() + (size_t)f * K : nullptr;
        a.cols = cols.get() + (size_t)f * J;
        a.ncols = ncols.get() + f;
        a.ptype = ptype.get();
        a.variance = specs[f].variance;
        a.xjy = of[f]->xjy.get();
        a.beta = beta.get() + (size_t)f * J;
        a.hdelta = hdelta.get() + (size_t)f * J;
        a.col_updates = updates.get() + (size_t)f * J;
        a.conv = ctl->convergence_type;
        a.tol = ctl->tolerance;
        a.max_iter = ctl->max_iterations != 0 ? ctl->max_iterations : -1;
        a.out_iter = flags.get() + 2 * f;
        a.out_flag = flags.get() + 2 * f + 1;
        a.out_ll = ll.get() + f;
        state->set(a, f);
        args[f] = a;
    }
    const bool strata = ds.S > 1;
    // the fits of `run`: their increments, one launch, the flags read back
    std::vector<int> h_flags(2 * F);
    cudaEvent_t e0, e1;
    CYC_CHECK_CUDA(cudaEventCreate(&e0));
    CYC_CHECK_CUDA(cudaEventCreate(&e1));
    struct Events { cudaEvent_t a, b; ~Events() { cudaEventDestroy(a); cudaEventDestroy(b); } } events{e0, e1};
    auto pass = [&](const std::vector<int>& run, const std::vector<CoxArgs>& a, const std::vector<Weighting*>& w) {
        std::vector<CoxArgs> list;
        for (int f : run) {
            w[f]->slots->increments(a[f].xb, w[f]->w.get(), a[f].d, stream);
            list.push_back(a[f]);
        }
        CYC_CHECK_CUDA(cudaMemcpyAsync(d_args.get(), list.data(), list.size() * sizeof(CoxArgs), cudaMemcpyHostToDevice,
                                       stream));
        CYC_CHECK_CUDA(cudaEventRecord(e0, stream));
        launch_cox(d_args.get(), (int)run.size(), shape, strata, stream);
        CYC_CHECK_CUDA(cudaEventRecord(e1, stream));
        CYC_CHECK_CUDA(cudaMemcpyAsync(h_flags.data(), flags.get(), 2 * F * sizeof(int), cudaMemcpyDeviceToHost, stream));
        CYC_CHECK_CUDA(cudaStreamSynchronize(stream));
        float ms = 0.f;
        CYC_CHECK_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        for (int f : run)
            CYC_REQUIRE(h_flags[2 * f + 1] != kTimedOut, CYC_ERR_TIMEOUT, "a wait between the CTAs of a fit ran out");
        return ms;
    };
    // update (CyclicCoordinateDescent.cpp:586-615): fits that come back
    // ill-conditioned restart from beta 0 with a tenfold smaller trust region
    std::vector<int> run(F);
    for (int f = 0; f < F; ++f) run[f] = f;
    double bound = ctl->initial_bound;
    for (int count = 1; !run.empty(); ++count) {
        std::vector<double> hd((size_t)J, bound);
        for (int f : run) {
            const double* b = h_beta.data() + (size_t)f * J;
            CYC_CHECK_CUDA(cudaMemcpyAsync(args[f].beta, b, J * sizeof(double), cudaMemcpyHostToDevice, stream));
            CYC_CHECK_CUDA(cudaMemcpyAsync(args[f].hdelta, hd.data(), J * sizeof(double), cudaMemcpyHostToDevice, stream));
            if (std::all_of(b, b + J, [](double v) { return v == 0.0; }))
                CYC_CHECK_CUDA(cudaMemsetAsync(args[f].xb, 0, K * sizeof(double), stream));
            else
                launch_xbeta(ds, args[f].beta, args[f].xb, stream);
            if (zhang)
                CYC_CHECK_CUDA(cudaMemcpyAsync(args[f].xb_save, args[f].xb, K * sizeof(double), cudaMemcpyDeviceToDevice,
                                               stream));
        }
        CYC_CHECK_CUDA(cudaStreamSynchronize(stream));   // the host arrays go away
        st.kernel_ms += pass(run, args, of);
        st.launches += 1;
        std::vector<int> again;
        for (int f : run) {
            out[f].iterations = h_flags[2 * f];
            out[f].return_flag = h_flags[2 * f + 1];
            st.cycles += out[f].iterations;
            if (out[f].return_flag == CYC_ILLCONDITIONED && count < ctl->max_bound_count) {
                again.push_back(f);
                double* b = h_beta.data() + (size_t)f * J;
                std::fill(b, b + J, 0.0);
                if (ds.has_offset) b[0] = 1.0;
            }
        }
        run.swap(again);
        bound /= 10.0;
    }
    std::vector<double> h_ll(F);
    std::vector<unsigned> upd((size_t)F * J);
    CYC_CHECK_CUDA(cudaMemcpyAsync(h_beta.data(), beta.get(), beta.bytes(), cudaMemcpyDeviceToHost, stream));
    CYC_CHECK_CUDA(cudaMemcpyAsync(h_ll.data(), ll.get(), F * sizeof(double), cudaMemcpyDeviceToHost, stream));
    CYC_CHECK_CUDA(cudaMemcpyAsync(upd.data(), updates.get(), updates.bytes(), cudaMemcpyDeviceToHost, stream));
    CYC_CHECK_CUDA(cudaStreamSynchronize(stream));
    for (int f = 0; f < F; ++f) {
        const double* b = h_beta.data() + (size_t)f * J;
        std::copy(b, b + J, out[f].beta);
        out[f].log_likelihood = h_ll[f];
        double lp = 0.0;
        for (int j = 0; j < J; ++j) lp += log_density(pt[j], specs[f].variance, b[j]);
        out[f].log_prior = lp;
        for (int i = 0; i < h_n[f]; ++i) {
            const int j = h_cols[(size_t)f * J + i];
            const double n = (double)ds.col_len(j);
            st.gradient_entries += out[f].iterations * n;
            st.update_entries += upd[(size_t)f * J + j] * n;
            st.coordinate_steps += out[f].iterations;
        }
    }
    if (pred) {
        std::vector<CoxArgs> eval(F);
        std::vector<Weighting*> by(F);
        std::vector<int> good;
        state.reset();
        sets.clear();                                          // the training risk sets go
        for (int f = 0; f < F; ++f) {
            pred[f] = std::nan("");
            if (out[f].return_flag != CYC_SUCCESS) continue;   // AbstractCrossValidationDriver.cpp:236-240
            good.push_back(f);
            by[f] = &weighting(held[f], false);
        }
        if (!good.empty()) {
            shape = build(0);
            state.reset(new CoxState(*sets[0]->slots, F));
        }
        for (int f : good) {
            CoxArgs a = by[f]->slots->args();
            a.weighted = 1;
            a.w = by[f]->w.get();
            a.xb = args[f].xb;
            a.variance = args[f].variance;
            a.predict = 1;
            a.out_iter = args[f].out_iter;
            a.out_flag = args[f].out_flag;
            a.out_ll = args[f].out_ll;
            state->set(a, f);
            eval[f] = a;
        }
        if (!good.empty()) {
            pass(good, eval, by);
            CYC_CHECK_CUDA(cudaMemcpyAsync(h_ll.data(), ll.get(), F * sizeof(double), cudaMemcpyDeviceToHost, stream));
            CYC_CHECK_CUDA(cudaStreamSynchronize(stream));
            for (int f : good) pred[f] = h_ll[f];
        }
    }
}

// device bytes of a weighting's risk sets, and of a fit on them
static void cox_bytes_of(Dataset& ds, double* weighting, double* fit) {
    const double K = ds.K, J = ds.J, events = ds.event_rows();
    const CoxShape s = cox_shape((int)std::min(2e9, events + K / kSlotRows + 1));
    const double positions = (double)s.C * s.per_cta;
    *weighting = K * 20 + events * 20 + (events + K / kSlotRows) * 12 + J * (4 * (s.C + 1) + 8) +
                 (double)ds.nnz_idx * 4 + positions * 9;
    *fit = K * 16 + J * 24 + positions * (cox_where(s) == 2 ? 26 : 8);
}

void run_cox_batch(Dataset& ds, const cyc_prior* prior, const cyc_fit_spec* specs, int F, const cyc_control* ctl,
                   cyc_fit_result* out, const double* const* held, double* pred) {
    const int J = ds.J;
    CYC_REQUIRE(prior->prior_type >= CYC_PRIOR_NONE && prior->prior_type <= CYC_PRIOR_NORMAL, CYC_ERR_ARGUMENT,
                "Unknown prior type");
    CYC_REQUIRE(ctl->convergence_type >= CYC_CONV_GRADIENT && ctl->convergence_type <= CYC_CONV_ZHANG_OLES,
                CYC_ERR_ARGUMENT, "Unknown convergence criterion");
    std::vector<int> pt(J, prior->prior_type);
    for (int i = 0; i < prior->n_exclude; ++i) {
        CYC_REQUIRE(prior->exclude[i] >= 0 && prior->exclude[i] < J, CYC_ERR_ARGUMENT, "exclude index out of range");
        pt[prior->exclude[i]] = CYC_PRIOR_NONE;
    }
    for (int f = 0; f < F; ++f) {
        CYC_REQUIRE(out[f].beta, CYC_ERR_ARGUMENT, "null argument");
        CYC_REQUIRE(prior->prior_type == CYC_PRIOR_NONE || specs[f].variance > 0, CYC_ERR_ARGUMENT,
                    "prior variance must be positive");
        CYC_REQUIRE(specs[f].n_fixed >= 0 && (specs[f].n_fixed == 0 || specs[f].fixed), CYC_ERR_ARGUMENT,
                    "bad fixed-column list");
        for (int i = 0; i < specs[f].n_fixed; ++i)
            CYC_REQUIRE(specs[f].fixed[i] >= 0 && specs[f].fixed[i] < J, CYC_ERR_ARGUMENT, "fixed column out of range");
    }
    CYC_CHECK_CUDA(cudaSetDevice(ds.device));
    OwnedStream own;
    CYC_CHECK_CUDA(cudaStreamCreateWithFlags(&own.s, cudaStreamNonBlocking));
    StreamScope scope(own.s);
    // Fits run as many at a time as half of the device's free memory holds
    // (what the pool keeps counts as free): 1,000 bootstrap replicates of 2M rows
    // and 50M entries want 270 GB.  CYC_COX_BATCH_BYTES sets the bound.
    double per_weighting, per_fit;
    cox_bytes_of(ds, &per_weighting, &per_fit);
    double bound = 1e9;
    if (const char* e = std::getenv("CYC_COX_BATCH_BYTES")) {
        bound = std::atof(e);
    } else if (F * (per_weighting + per_fit) > bound) {
        size_t free_bytes = 0, total_bytes = 0;
        unsigned long long reserved = 0, used = 0;
        cudaMemPool_t pool;
        CYC_CHECK_CUDA(cudaMemGetInfo(&free_bytes, &total_bytes));
        CYC_CHECK_CUDA(cudaDeviceGetDefaultMemPool(&pool, ds.device));
        CYC_CHECK_CUDA(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved));
        CYC_CHECK_CUDA(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used));
        bound = 0.5 * ((double)free_bytes + (double)reserved - (double)used);
    }
    cyc_run_stats st{};
    for (int f0 = 0; f0 < F;) {
        std::set<const double*> weightings;
        int n = 0;
        for (; f0 + n < F; ++n) {
            weightings.insert(specs[f0 + n].weights);
            if (n > 0 && per_weighting * weightings.size() + per_fit * (n + 1) > bound) break;
        }
        run_cox_fits(ds, pt, specs + f0, n, ctl, out + f0, held ? held + f0 : nullptr, pred ? pred + f0 : nullptr, own.s,
                     st);
        f0 += n;
    }
    st.phases = 1;
    st.phase_ms[0] = st.kernel_ms;
    st.phase_state_bytes[0] = 8;
    set_last_stats(st);
}

}  // namespace cyc
