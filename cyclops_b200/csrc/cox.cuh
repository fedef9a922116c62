// cox.cuh -- the persistent Breslow Cox solver (cox.cu): the risk sets of one
// weighting and the kernel's launch.
#pragma once
#include "internal.cuh"

namespace cyc {

constexpr int kCoxThreads = 512;

// CTAs of a Cox fit and threads of a CTA
struct CoxShape {
    int C, threads;                // threads: 128, 256 or 512
};
CoxShape cox_shape(Dataset& ds);

// The risk sets of a weighting, reduced to the groups that hold events: slot e
// is an event group in row order (rows by stratum, then falling time; tied
// events of a stratum share one).  A row enters the risk sets from the first
// event group at or after it in its stratum on: that group is the row's slot,
// and a row after its stratum's last event has none.
// Slots are split over C CTAs in order; CTA r's slots are dealt to its threads
// in contiguous runs of `m` (slot t * m + i of the CTA at position i * threads
// + t), which is the order all per-slot arrays have.
struct CoxSlots {
    Dataset& ds;
    int C, threads;
    int cap;                       // at least the number of slots
    int per_cta;                   // positions a CTA has room for (a multiple of 4 `threads`)
    DevBuf<int> cnt, last, tiles;  // scans over the rows
    DevBuf<int> end, first, lo, sstr, rowslot, rpart, spart, total, split, entry;
    DevBuf<unsigned char> flag;    // [C][per_cta] bit 0: the slot starts its stratum, bit 1: it ends it
    DevBuf<double> n, d, S1, S2;   // [C][per_cta] events; risk-set increments; suffix sums of n/D, n/D^2
    DevBuf<double> bp;             // scratch of the solver

    CoxSlots(Dataset& ds, CoxShape shape);
    // for row weights d_w (K, device) or null
    void build(const double* d_w, cudaStream_t stream);
    // the risk-set increments (sums of w exp(xb) over each slot's rows)
    void increments(const double* d_xb, const double* d_w, cudaStream_t stream);
};

struct CoxArgs {
    int K, J, C, threads, per_cta;
    int weighted;                  // use `w`
    const int* fmt;
    const long long* col_ptr;
    const long long* val_ptr;
    const int* idx;
    const double* val;
    const int* entry;              // slot position of every entry of idx (-1: none; bit 30: see k_cox)
    const int* rowslot;            // the same by row (dense columns)
    const int* entry_strat;        // stratum of every entry (null: one stratum)
    const int* strat;              // by row
    const int* split;              // J x (C+1)
    const int* rpart;              // C+1 row boundaries
    const int* spart;              // C+1 slot boundaries
    const unsigned char* flag;
    const double* n;
    double *d, *S1, *S2, *bp;
    const double* y;
    const double* w;               // K
    double* xb;                    // K, current on entry and exit
    double* xb_save;               // K (Zhang-Oles)
    const int* cols;
    const int* ncols;
    const int* ptype;              // J
    double variance;
    const double* xjy;             // J
    double* beta;                  // J
    double* hdelta;                // J
    unsigned* col_updates;         // J, added to
    double* score;                 // not null: write |gradient| of the columns (in list order), step nothing
    int conv;
    double tol;
    int max_iter;                  // 0: evaluate the log likelihood only
    int* out_iter;
    int* out_flag;                 // kTimedOut (ccd.cuh): the CTAs lost one another
    double* out_ll;
};
void launch_cox(const CoxArgs& a, cudaStream_t stream);

}  // namespace cyc
