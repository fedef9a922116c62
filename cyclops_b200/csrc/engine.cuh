// engine.cuh -- the per-coordinate engine (one fit's device state + stream).
#pragma once
#include <memory>

#include "internal.cuh"

namespace cyc {

struct Engine {
    explicit Engine(Dataset* d);
    ~Engine();
    Engine(const Engine&) = delete;
    Engine& operator=(const Engine&) = delete;

    OwnedStream own;              // the engine's stream (declared first: destroyed last)
    Dataset* ds;                  // borrowed: the caller keeps the dataset alive
    int device = 0;
    cudaStream_t stream = nullptr;
    int model = 0;
    int N = 0;              // denominators: K (lr/pr), strata (clr/cpr), risk-set groups (cox)
    bool use_w = false;     // weights set with useCrossValidation
    bool stats_known = false;

    DevBuf<double> xb, xb_save, exb, kw, denom, nw, numer, numer2, xjy;
    DevBuf<double> weights_buf, beta_buf;
    DevBuf<double2> partial;
    DevBuf<unsigned> ticket;
    DevBuf<double> result, ll_fixed;
    PinnedBlock h_block;          // results (pinned, from the process-wide pool): kernels write them here
    double* h_result = h_block.as<double>();
    unsigned* h_word = h_block.as<unsigned>() + 8;      // past the results: the last signal's tag
    unsigned tag = 0;

    // cox
    DevBuf<int> group, grow_ptr, gstart, gend, glist;
    DevBuf<long long> glist_ptr;
    DevBuf<double> D, P1h, P1l, P2h, P2l;
    DevBuf<double> R1, R2;             // scan scratch: n/D and n/D^2 per group
    DevBuf<SegD> aggD;
    DevBuf<SegP> aggP;
    std::vector<long long> h_glist_ptr;
    std::vector<int> h_first_group;
    std::vector<double> h_weights;     // the weights the groups are to follow (empty: none)
    bool groups_current = false;

    void sync();
    HostSignal signal();
    void await(const HostSignal& sig);
    void alloc_denominators();
    const int* groups() const;
    const int* group_rows() const;
    void regroup(const double* w);
    void group_weights();
    void ensure_groups();

    void set_weights(const double* w, bool use_cv);
    void fixed_terms_ll(bool use_cv);
    void fixed_terms_gh(bool use_cv);
    void zero_xbeta();
    void axpy_xbeta(double beta, int j);
    void compute_xbeta(const double* beta_host);
    void compute_xbeta_device(const double* d_beta);
    void remaining_statistics(bool use_weights);
    void numerator_for_gradient(int j, bool use_weights);
    void launch_gradient(int j, bool use_weights, double* out, const HostSignal& sig);
    void gradient_hessian(int j, bool use_weights, double* g, double* h);
    void launch_update(int j, bool use_weights, double delta, const HostSignal& sig = HostSignal{},
                       const double* d_delta = nullptr);
    void update_xbeta(double delta, int j, bool use_weights);
    void cox_rescan(int lo);
    void launch_loglik(bool use_cv, double* out, const HostSignal& sig = HostSignal{});
    double log_likelihood(bool use_cv);
    void launch_gradient_objective(bool use_cv, double* out, const HostSignal& sig);
    double gradient_objective(bool use_cv);
    double predictive_log_likelihood(const double* w);
    void predictive_estimates(double* y, const double* w);
    void get_xbeta(double* out);
    void fisher_information(const int* cols, int n, double* out);
    void kkt_scores(const int* d_cols, int n, bool use_weights, double* d_out);
    void save_xbeta();
    void get_xbeta_save(double* out);
};

// XjY under row weights d_w (null: none), and the linear predictors of d_beta
void launch_xjy(const Dataset& ds, const double* d_w, double* d_xjy, cudaStream_t stream);
void launch_xbeta(Dataset& ds, const double* d_beta, double* d_xb, cudaStream_t stream);

}  // namespace cyc

struct cyc_engine {
    cyc_dataset* owner = nullptr;
    std::unique_ptr<cyc::Engine> eng;
};
