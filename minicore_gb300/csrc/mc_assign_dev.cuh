// Device helpers shared by the assignment kernels: the running argmin, a pair's final value and
// the row-side transforms.
#pragma once
#include "mc_assign.cuh"

namespace mc {

// ------------------------------------------------------------------------------------
// argmin bookkeeping: lexicographic (value, index); NaN at center 0 wins (the reference's
// sequential scan then never moves off center 0), NaN elsewhere never wins.
// ------------------------------------------------------------------------------------
struct Best {
    float v;
    uint32_t j;
};

__device__ inline void best_init(Best &b) {
    b.v = __int_as_float(0x7f800000);
    b.j = 0xffffffffu;
}

__device__ inline void best_offer(Best &b, float v, uint32_t j) {
    if (v != v) {
        if (j != 0) return;
        v = __int_as_float(0xff800000);  // -inf marks "NaN at center 0"
    }
    if (v < b.v || (v == b.v && j < b.j)) {
        b.v = v;
        b.j = j;
    }
}

__device__ inline void best_merge_shfl(Best &b, int lanemask_xor) {
    const float ov = __shfl_xor_sync(0xffffffffu, b.v, lanemask_xor);
    const uint32_t oj = __shfl_xor_sync(0xffffffffu, b.j, lanemask_xor);
    if (ov < b.v || (ov == b.v && oj < b.j)) {
        b.v = ov;
        b.j = oj;
    }
}

// whether k_assign_few takes a list of nd rows: up to kFewRows, one resident wave of it
constexpr uint64_t kFewRows = 2048;
__host__ __device__ inline bool assign_few_takes(const AssignArgs &a, uint64_t nd) {
    return a.msr == SQRL2 && a.rows && !a.dmode && a.d <= 2048 && nd <= kFewRows;
}

// final value of a pair: compare key (float) and cost (double) per measure
template <int MSR>
__device__ inline float finish_key(float acc) {
    if (MSR == SQRL2) return acc;
    if (MSR == L1) return acc * 0.5f;
    if (MSR == HELLINGER) return sqrtf(acc);
    if (MSR == MKL) return post_divergence(acc);
    return post_divergence(acc * 0.5f);  // JSD
}

template <int MSR>
__device__ inline double key_to_cost(float key) {
    if (MSR == L1) return double(key) * 2.0;
    if (MSR == HELLINGER) return double(key) * kSqrt1_2;
    return double(key);
}

// row-side transform of a raw value x for the constant-prior path
template <int MSR>
__device__ inline void row_xform(float x, float pv, float rsi, float rinc, float &x0, float &x1) {
    if (MSR == SQRL2) { x0 = x; x1 = 0.f; }
    else if (MSR == L1) { x0 = x + pv; x1 = 0.f; }
    else if (MSR == HELLINGER) { x0 = sqrtf(x * rsi + rinc); x1 = 0.f; }
    else {
        const float b = x * rsi + rinc;
        if (MSR == MKL) { x0 = logf(b); x1 = 0.f; }
        else { x0 = b; x1 = b * logf(b); }
    }
}

// plain differences, by the rows' and the centers' bounds (l1_plain_bounds)
__device__ inline bool l1_plain(const AssignArgs &a) {
    const L1Stat &t = *a.l1;
    const double sums = __longlong_as_double((long long)t.xsum) + __longlong_as_double((long long)t.csum) +
                        2.0 * fabs(a.prior_sum);
    const float mn = fminf(__uint_as_float(t.xmin), __uint_as_float(t.cmin));
    return l1_plain_bounds(sums, a.prior, mn);
}

}  // namespace mc
