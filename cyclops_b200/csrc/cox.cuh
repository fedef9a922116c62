// cox.cuh -- the persistent Breslow Cox solver (cox.cu): the risk sets of one
// weighting and the kernel's launch.
#pragma once
#include "mbar.cuh"

namespace cyc {

constexpr int kCoxThreads = 512;

// CTAs of a Cox fit, threads of a CTA, and the slots a CTA has room for (a
// multiple of 4 threads)
struct CoxShape {
    int C, threads;                // threads: 128, 256 or 512
    int per_cta = 0;
};
// for fits of at most `slots` slots each
CoxShape cox_shape(int slots);

struct CoxArgs;

// The risk sets of a weighting, reduced to slots of at most kSlotRows rows.  Rows
// are sorted by stratum, then falling time; tied events of a stratum are an event
// group, whose rows are those after the group before, to its last event: they
// enter the risk sets with it.  Rows after their stratum's last event have no
// group.  A group's rows are cut into slots, of which the last has its events.
// Slots are split over C CTAs in order; CTA r's slots are dealt to its threads
// in contiguous runs of `m` (slot t * m + i of the CTA at position i * threads
// + t), which is the order all per-slot arrays have.
struct CoxSlots {
    Dataset& ds;
    CoxShape shape{1, 128};
    int n_slots = 0;
    DevBuf<int> cnt, last, tiles;  // scans over the rows
    DevBuf<int> first, glo, gend, gstr, gcum, groups;      // the event groups
    DevBuf<int> lo, end, sstr, rowslot, rpart, spart, split, entry;
    DevBuf<unsigned char> flag;    // [C][per_cta] bit 0: the slot starts its stratum, bit 1: it ends it
    DevBuf<double> n, per_event;   // [C][per_cta] events; 1 / their sum

    explicit CoxSlots(Dataset& d) : ds(d) {}
    // the event groups and the number of slots for row weights d_w (K, device)
    // or null; n_slots is known once the stream is through
    void find(const double* d_w, cudaStream_t stream);
    // the slots, for a launch of this shape
    void build(CoxShape s, const double* d_w, cudaStream_t stream);
    // the risk-set increments (sums of w exp(xb) over each slot's rows) in `out`
    void increments(const double* d_xb, const double* d_w, double* out, cudaStream_t stream) const;
    size_t positions() const { return (size_t)shape.C * shape.per_cta; }
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
    const int* rowslot;            // the same by row
    const int* entry_strat;        // stratum of every entry (null: one stratum)
    const int* strat;              // by row
    const int* split;              // J x (C+1)
    const int* rpart;              // C+1 row boundaries
    const int* spart;              // C+1 slot boundaries
    const unsigned char* flag;
    const double* n;
    const double* per_event;
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
void launch_cox(const CoxArgs* d_fits, int F, CoxShape shape, bool strata, cudaStream_t stream);

// F Cox fits as one launch (each the one cyc_fit gives alone), weights per fit;
// with `held`, the predictive log likelihood of each fit's held-out rows under
// those weights in `pred` (NaN where the fit did not succeed)
void run_cox_batch(Dataset& ds, const cyc_prior* prior, const cyc_fit_spec* specs, int F, const cyc_control* ctl,
                   cyc_fit_result* out, const double* const* held, double* pred);

}  // namespace cyc
