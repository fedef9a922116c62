// row_terms.cuh -- per-row terms of the device-resident solvers: the model
// means, gradient and Hessian terms, compensated sums, and the split of a
// column's entries over row ranges.  Shared by the 8-fit kernel (batch.cu)
// and the one-fit kernel (ccd.cu).
#pragma once
#include "solver_common.cuh"

namespace cyc {

template <class T>
struct Kahan {
    T s = 0, c = 0;
    __device__ __forceinline__ void add(T v) {
        const T yv = v - c;
        const T t = s + yv;
        c = (t - s) - yv;
        s = t;
    }
    __device__ __forceinline__ double value() const { return (double)s - (double)c; }
};

template <>
struct Kahan<double> {
    double s = 0;
    __device__ __forceinline__ void add(double v) { s += v; }
    __device__ __forceinline__ double value() const { return s; }
};

__device__ __forceinline__ float fexp(float x) { return __expf(x); }
__device__ __forceinline__ double fexp(double x) { return exp(x); }
__device__ __forceinline__ float flog(float x) { return __logf(x); }
__device__ __forceinline__ double flog(double x) { return log(x); }

// per-row contribution to (gradient, Hessian) of an independent-rows model
// (Logistic / PoissonRegression::incrementGradientAndHessian,
// ModelSpecifics.h:540-568, 1508-1543); the logistic probability is formed as
// 1 / (1 + exp(-xb)), which equals exb / (1 + exb) without overflowing
// the row's mean under the model: the logistic probability, or exp(xb)
template <class T, int MODEL>
__device__ __forceinline__ T row_mean(T v) {
    if (MODEL == CYC_LR) return T(1) / (T(1) + fexp(-v));
    return fexp(v);
}

// (gradient, Hessian) terms of one entry from its row's mean
template <class T, int MODEL>
__device__ __forceinline__ void mean_terms(T m, T x, T wt, bool ind, T& gi, T& hi) {
    if (MODEL == CYC_LR) {
        const T g1 = m * x;
        gi = wt * g1;
        hi = wt * (ind ? g1 * (T(1) - g1) : x * x * m * (T(1) - m));
    } else {
        const T n1 = m * x;
        gi = wt * n1;
        hi = wt * (ind ? n1 : n1 * x);
    }
}

template <class T, int MODEL>
__device__ __forceinline__ void row_terms(T v, T x, T wt, bool ind, T& gi, T& hi) {
    mean_terms<T, MODEL>(row_mean<T, MODEL>(v), x, wt, ind, gi, hi);
}

// (callers skip rows of weight zero: their terms are exactly zero, and the
// exp() they would cost is the FP64 pipe's largest load)
template <class T, int MODEL>
__device__ __forceinline__ void row_gh(T v, T x, T wt, bool ind, Kahan<T>& ag, Kahan<T>& ah) {
    T gi, hi;
    row_terms<T, MODEL>(v, x, wt, ind, gi, hi);
    ag.add(gi);
    ah.add(hi);
}

// xb + delta * x as one fused multiply-add, the same wherever a batch
// replays an update (the owning CTA and every CTA's copy of a shared row)
__device__ __forceinline__ float upd_fma(float d, float x, float v) { return __fmaf_rn(d, x, v); }
__device__ __forceinline__ double upd_fma(double d, double x, double v) { return __fma_rn(d, x, v); }

// first entry of column j whose row is >= rpart[r]
static __global__ void k_splits(int J, int C, const int* fmt, const long long* col_ptr, const int* idx,
                         const int* rpart, int* split) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= J * (C + 1)) return;
    const int j = t / (C + 1), r = t % (C + 1);
    const int f = fmt[j];
    if (f == CYC_DENSE || f == CYC_INTERCEPT) { split[t] = rpart[r]; return; }
    const int* c = idx + col_ptr[j];
    int lo = 0, hi = (int)(col_ptr[j + 1] - col_ptr[j]);
    const int key = rpart[r];
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (c[mid] < key) lo = mid + 1;
        else hi = mid;
    }
    split[t] = lo;
}

}  // namespace cyc
