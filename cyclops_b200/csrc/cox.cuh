// cox.cuh -- the persistent Breslow Cox solver (cox.cu): the risk sets of one
// weighting and the kernel's launch.
#pragma once
#include "mbar.cuh"

namespace cyc {

constexpr int kCoxThreads = 512;

// CTAs of a Cox fit and threads of a CTA
struct CoxShape {
    int C, threads;                // threads: 128, 256 or 512
};
CoxShape cox_shape(Dataset& ds);

struct CoxArgs;

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
    DevBuf<double> n;              // [C][per_cta] events

    CoxSlots(Dataset& ds, CoxShape shape);
    // for row weights d_w (K, device) or null
    void build(const double* d_w, cudaStream_t stream);
    // the risk-set increments (sums of w exp(xb) over each slot's rows) in `out`
    void increments(const double* d_xb, const double* d_w, double* out, cudaStream_t stream) const;
    size_t positions() const { return (size_t)C * per_cta; }
    CoxShape shape() const { return {C, threads}; }
    // the arguments that follow from the dataset and the risk sets
    CoxArgs args() const;
};

// the solver's per-slot arrays of F fits: risk-set increments, and where shared
// memory does not hold them the suffix sums and block sums
struct CoxState {
    DevBuf<double> d, S1, S2, bp;
    size_t np;
    CoxState(const CoxSlots& s, int F);
    void set(CoxArgs& a, int f) const;
};

struct CoxArgs {
    int K, J, per_cta;
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
    int predict;                   // as getPredictiveLogLikelihood: every outcome at its value
    WaitLimit wait;
    int* out_iter;
    int* out_flag;                 // kTimedOut (ccd.cuh): the CTAs lost one another
    double* out_ll;
};
// one launch of F fits of one shape; `d_fits` is their arguments on the device
void launch_cox(const CoxArgs* d_fits, int F, CoxShape shape, int per_cta, bool strata, cudaStream_t stream);

// F Cox fits as one launch (each the one cyc_fit gives alone), weights per fit;
// with `held`, the predictive log likelihood of each fit's held-out rows under
// those weights in `pred` (NaN where the fit did not succeed)
void run_cox_batch(Dataset& ds, const cyc_prior* prior, const cyc_fit_spec* specs, int F, const cyc_control* ctl,
                   cyc_fit_result* out, const double* const* held, double* pred);

}  // namespace cyc
