// Assignment kernel arguments and launchers (mc_assign.cu).
#pragma once
#include "mc_internal.cuh"

namespace mc {

// What decides whether L1 with a pair-dependent prior equals plain L1 (l1_plain in
// mc_assign_dev.cuh): the smallest nonzero magnitudes (float bits) and the largest sums (bits of
// doubles, not below 0) of the rows and the centers.
struct L1Stat {
    unsigned long long xsum, csum;
    unsigned xmin, cmin;
};

// L1 in pair mode adds the pair's pv to both values of a column: at most
// 7.0069e-42 (row sum + center sum), or the prior itself.  Where every nonzero magnitude exceeds
// 2^26 times that, v + pv rounds to v for v != 0, |pv - v| rounds to |v| and |pv - pv| is 0, so
// each term is exactly |c - x| of the raw values.  (A NaN sum or bound fails the comparison.)
__host__ __device__ inline bool l1_plain_bounds(double sums, double prior, float mn) {
    double pv = 7.0069e-42 * sums * 1.0001 + 1e-44;
    if (prior > pv) pv = prior;
    return double(mn) > pv * 67108864.0;
}

// Which dense L1 pair passes are offered to k_assign_dense: that launch, the bounds of the centers and
// the pair kernel's CTAs that leave cost some 17 us, and below 38,912 rows its 128-row tiles leave SMs
// idle.  Assignment in us, offered / the pair kernel alone, over the grid named at assign_dense_pays
// (n x d, k; work: n d times k rounded up to the pair kernel's 32): up to 16 centers, which that kernel
// pads to 32, it pays from a work of 1.2e8 (300,000 x 20, k = 10: 65 / 95), taken from 2.5e8, where a few
// passes make up for the 30 us that the rows' bounds take once per job; else from 4e8 and 32 columns
// (100,000 x 64, k = 50: 92 / 117), below which it loses (60,000 x 32, k = 64, 1.2e8: 64 / 54;
// 75,000 x 50, k = 32, 1.2e8: 63 / 54; 60,000 x 16, k = 1000, 9.8e8: 406 / 347)
inline bool l1_dense_pays(uint64_t n, uint64_t d, uint32_t k) {
    const double work = double(n) * double(d) * double((uint64_t(k) + 31) / 32 * 32);
    return n > 128 * 152 * 2 && (k <= 16 ? work >= 2.5e8 : d >= 32 && work >= 4e8);
}

struct AssignArgs {
    int msr = SQRL2;
    uint64_t n = 0, d = 0;
    uint32_t k = 0, kp = 0;           // centers, padded center count of CT0/CT1
    const float *X = nullptr;         // dense rows
    const uint32_t *rows = nullptr;   // dense only: optional row list (row r of the pass = X row rows[r])
    const unsigned long long *n_dev = nullptr;  // tiled kernel: row count read on the device (<= n)
    const float *vals = nullptr;      // CSR rows
    const uint32_t *idx = nullptr;
    const uint64_t *indptr = nullptr;
    uint64_t nnz = 0;                 // CSR nonzeros (autotuner shape bucket)
    const double *rowsum = nullptr;   // per row (pair mode, sparse HELL)
    const float *rsi = nullptr;       // per-row 1/rhsum (constant prior)
    const float *rinc = nullptr;      // per-row pv/rhsum (constant prior)
    const double *csum = nullptr;     // per-center sums
    float *CT0 = nullptr;             // [d][kp] center transform
    float *CT1 = nullptr;             // [d][kp] second center transform (MKL, JSD)
    double *consts = nullptr;         // [k][4] per-center FP64 constants (sparse-dot path)
    const uint32_t *grp = nullptr;    // JSD sparse-dot: per-row group of rows with equal rinc
    const double *ztab = nullptr;     // JSD sparse-dot: [group][k] zero-entry sums (k_jsd_ztable)
    float pv = 0.f;                   // constant-prior pv
    double prior = 0.0, prior_sum = 0.0;
    uint32_t *asn = nullptr;
    double *costs = nullptr;
    // optional distance output (cmp / pcmp): every pair's distance as float
    //   dmode 1: dmat[row * ldm + c]   2: dmat[c * ldm + row]
    //   dmode 3: condensed upper triangle, pairs c < row at c*ldm - c(c+1)/2 + row - c - 1
    float *dmat = nullptr;
    uint64_t ldm = 0;
    int dmode = 0;
    const L1Stat *l1 = nullptr;       // dense L1 in pair mode: set when the plain path may apply
};

__device__ __forceinline__ void write_dist(const AssignArgs &a, uint64_t row, uint32_t c, float v) {
    if (a.dmode == 1) {
        a.dmat[row * a.ldm + c] = v;
    } else if (a.dmode == 2) {
        a.dmat[uint64_t(c) * a.ldm + row] = v;
    } else if (a.dmode == 3 && uint64_t(c) < row) {
        const uint64_t cc = c;
        a.dmat[cc * a.ldm - cc * (cc + 1) / 2 + row - cc - 1] = v;
    }
}

int launch_prep_centers(const AssignArgs &a, const float *C, bool pair, bool sparse_consts, cudaStream_t st);
int launch_row_scalars(const double *rowsum, uint64_t n, uint64_t d, float pv, float *rsi, float *rinc,
                       cudaStream_t st);
// tune: the autotuner may time kernel variants on the first call for a shape (callers that
// must not synchronise or allocate pass false)
int launch_assign_tiled(const AssignArgs &a, bool csr, bool pair, cudaStream_t st, bool tune = true);
// dense rows in chunks of 64 centers (mc_assign_dense.cu): SQRL2, MKL with a constant prior, plain L1; and
// whether it rather than k_assign_tiled takes a pass
int launch_assign_dense(const AssignArgs &a, cudaStream_t st);
bool assign_dense_pays(const AssignArgs &a);
int launch_assign_sparse(const AssignArgs &a, cudaStream_t st, int sms, bool tune = true);
// L1 over CSR rows in pair mode (prior 0): a walk over the union of nonzero columns,
// bit-identical to the tiled kernel; work: l1_union_work_entries(k, d) floats
int launch_assign_l1_union(const AssignArgs &a, const float *C, float *work, int sms, cudaStream_t st,
                           bool tune = true);
uint64_t l1_union_work_entries(uint32_t k, uint64_t d);
// the largest work space (in entries) for which the union kernel is used
constexpr uint64_t kL1UnionMaxEntries = 1ull << 29;
// JSD sparse-dot table: ztab[g * k + c] = sum over all columns j of f(a_cj, gval[g]) with
// f(a, b) = a log a + b log b - (a + b) log((a + b) / 2) and a_cj the center transform; alog: 2 d
// jsd_log_centers() floats of work space (the transform and a log a of that many centers at a time), or
// null: every term forms its center's a log a itself, which pays for small tables (jsd_logs_pay)
uint32_t jsd_log_centers(uint32_t k, uint64_t d);
// 2,527 x 103, k = 10, 100 groups, an assignment: 47 us with the logarithms in a launch of their own, 42 without
inline bool jsd_logs_pay(uint64_t ngrp, uint64_t k, uint64_t d) { return ngrp * k * d >= 2000000; }
int launch_jsd_ztable(const float *C, uint32_t k, uint64_t d, const double *csum, float pv, const float *gval,
                      uint32_t ngrp, double *ztab, float *alog, cudaStream_t st);
// row / center part of an L1Stat (dense rows; csum: the centers' sums)
int launch_l1_row_stat(const float *X, uint64_t m, const double *rowsum, uint64_t n, L1Stat *stat, cudaStream_t st);
int launch_l1_center_stat(const float *C, uint64_t m, const double *csum, uint64_t k, L1Stat *stat, cudaStream_t st);
// JSD over CSR rows grouped by their zero-entry value (mc_assign_jsd.cu): bucket 0 holds the
// rows of groups too small for a table, the others one group each, largest first
struct JsdGroups {
    uint32_t nbucket = 0;
    const uint32_t *perm = nullptr;                     // [n] rows by bucket
    const uint64_t *start = nullptr, *count = nullptr;  // [nbucket] of perm
    const uint64_t *slab_start = nullptr;               // [nbucket + 1] slabs of rows before each bucket
    const double *bx = nullptr;                         // [n] row terms
};
struct JsdGroupWork;
// whether k_assign_jsd_groups takes a job's passes
bool jsd_groups_pay(uint64_t n, uint64_t d, uint32_t k, uint64_t nnz, uint32_t ngrp);
int launch_jsd_row_terms(const float *vals, const uint64_t *indptr, uint64_t n, const float *rsi, const float *rinc,
                         double *bx, int sms, cudaStream_t st);
// rows listed by bucket into w
int jsd_bucket_rows(const uint32_t *grp, uint64_t n, uint32_t ngrp, uint64_t nnz, uint64_t d, int sms, JsdGroupWork &w,
                    cudaStream_t st);
int launch_assign_jsd_groups(const AssignArgs &a, const JsdGroups &jg, cudaStream_t st);
uint32_t tiled_center_pad(uint32_t k, bool pair, int msr);
uint32_t sparse_center_pad(uint32_t k);

}  // namespace mc
