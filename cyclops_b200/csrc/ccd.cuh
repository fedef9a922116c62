// ccd.cuh -- the one-fit persistent CCD kernel (ccd.cu): arguments, launch
// shape and launch.
#pragma once
#include "mbar.cuh"

namespace cyc {

constexpr int kCcdThreads = 256;   // most threads a CTA has
constexpr int kCcdCluster = 16;    // most CTAs a fit has (the non-portable cluster limit)
// out_flag of a fit whose CTAs lost one another (a bounded wait ran out)
constexpr int kTimedOut = -1;

// F fits over one dataset, each a thread-block cluster of C CTAs that split
// the rows.  Arrays marked [F] hold one element per fit.
struct CcdArgs {
    int model, K, J, S, F, C;
    int threads;                  // per CTA, a multiple of 64 up to kCcdThreads
    int teams;                    // 2: the CTA's threads take the columns in two teams (lr, pr)
    const unsigned char* runs;    // null, or by place in `cols`: columns of the run that starts there (ccd_runs; C 1, teams 1)
    int weights;                  // 0: all ones; 1: CV folds; 2: `w`
    int strict;                   // as the per-coordinate engine: a logistic row whose exb overflows is NaN,
                                  // and a row of weight zero that is NaN or infinite makes the sums NaN
    const int* fmt;
    const long long* col_ptr;
    const long long* val_ptr;
    const int* idx;
    const double* val;
    const int* entry_strat;       // stratum of every entry of idx (grouped models)
    const int* split;             // J x (C+1): first entry of rank r's rows, relative to the column
    const int* rpart;             // C+1 row boundaries
    const double* y;
    const int* strat;             // K (grouped)
    const int* cols;              // the columns a fit steps through, in order; fit f's at f * cols_stride
    const int* ncols;             // their number; fit f's at f * ncols_stride
    int cols_stride, ncols_stride;
    const int* ptype;             // J
    void* xb;                     // [F][K] T linear predictors, current on entry and exit
    void* xb_save;                // [F][K] T (Zhang-Oles convergence)
    const void* w;                // [F][K] T row weights (weights == 2)
    const signed char* fold;      // K fold id per row (weights == 1)
    const signed char* entry_fold;   // fold id of every entry of idx (weights == 1)
    const int* fitfold;           // [F] held-out fold
    double* denom;                // [F][S] (grouped), current on entry
    const double* nw;             // [F][S] (grouped)
    const double* xjy;            // [F][J]
    double* beta;                 // [F][J]
    double* hdelta;               // [F][J]
    const double* variance;       // [F]
    const double* llfixed;        // [F]
    const int* active;            // [F] 0: the fit is left alone; null: all run
    unsigned* col_updates;        // [F][J] steps that moved a coefficient, added to
    int conv;
    double tol;
    int max_iter;
    WaitLimit wait;               // set by launch_ccd
    int* out_iter;                // [F]
    int* out_flag;                // [F]
};

// CTAs a fit, threads and teams a CTA for F one-fit solves of a dataset, the
// clusters of that shape the device holds at once, and the modelled time of a
// cycle of the F fits.  `C` > 0 asks for that many CTAs; `varied`: the fits end
// after different numbers of cycles.
struct CcdShape {
    int C, threads, teams, slots;
    double cycle_us;
    bool runs = false;            // take the columns in runs (ccd_runs)
};
CcdShape ccd_shape(const Dataset& ds, int F, int C = 0, bool varied = false);
// cycles' worth of time that F fits take where `slots` run at a time: whole
// turns, or, when fits end at different times and the next take their places,
// their share
inline double ccd_turns(int F, int slots, bool varied) {
    if (F <= slots) return 1.0;
    return varied ? (double)F / slots : (double)((F + slots - 1) / slots);
}
// Runs of at most 8 columns, next to one another in `cols`, that share no row: by
// place, the length of the run that starts there (0 inside one).  `local`: the
// predictors are in shared memory.  Also the modelled time of a cycle: a run by its
// longest column, a column alone by its rounds, as measured on designs of 1k to
// 900k rows (3 to 200 entries a column: 0.16 to 0.7 us a column).
struct CcdRuns {
    std::vector<unsigned char> len;
    double cycle_us;
};
CcdRuns ccd_runs(const Dataset& ds, const std::vector<int>& cols, bool local);
// row boundaries of C CTAs, at stratum starts for grouped models
std::vector<int> ccd_rows(const Dataset& ds, int C);
// the split of every column's entries over those boundaries
void ccd_splits(const Dataset& ds, int C, const int* d_rpart, int* d_split, cudaStream_t stream);

// fold ids of the entries of idx (CV folds), so that a column's load beside its row ids
void ccd_entry_folds(const Dataset& ds, const signed char* d_fold, signed char* d_out, cudaStream_t stream);

// one launch of the F fits (T: double, or float with compensated sums)
template <class T>
void launch_ccd(const CcdArgs& a, const std::vector<int>& rpart, cudaStream_t stream);

}  // namespace cyc
