// JSD assignment of CSR rows grouped by their zero-entry value r (count data: equal row sums), many
// rows per group.
//
// A row's distance to center c is Z[g][c] (the zero-entry sum of its group, k_jsd_ztable) plus a
// row term plus, over the row's entries, m0 log(m0/2) - m1 log(m1/2) with m0 = a_cj + r and
// m1 = a_cj + b.  The m0 half depends on (group, column, center) only: where a group's rows have
// more entries than there are columns it is tabulated once per CTA instead of once per entry, which
// halves the logarithms, and they bound this pass: 50,000 rows of 1500 entries, 850 groups, 20,000
// columns, k = 50: 8.2 ms in k_assign_sparse, 7.1 here, instruction issue 88 % busy.  A CTA takes up
// to 96 rows of one group and walks the columns in bands of kJsdBand through shared memory: the
// center transform (double buffered by cp.async) and the band's table.  Rows of groups too small for
// a table share CTAs without one.  A warp visits its rows in turn in each band (sums and cursors
// wait in shared memory, so one copy of the code serves all rows: unrolled over eight rows in
// registers it ran out of the instruction cache: 97 ms), lane = two centers, the row's next 32
// entries one per lane.  Per (row, center) the terms and their order are those of k_assign_sparse,
// so the results are bit-identical to it.
#include "mc_assign_dev.cuh"
#include "mc_reduce.cuh"

namespace mc {

constexpr int kJsdBand = 256;  // columns: 128 KB of center transforms (two buffers), 64 KB of table
constexpr int kJsdRows = 3;    // rows per warp
constexpr int kJsdThreads = 1024, kJsdWarps = kJsdThreads / 32, kJsdSlab = kJsdWarps * kJsdRows;

struct JsdRow {  // a row's state between bands
    uint64_t begin;
    uint32_t pos, len;
    float rsi, r;
};
constexpr size_t kJsdSmem = 3ull * kJsdBand * 64 * sizeof(float) + kJsdSlab * (32 * sizeof(float2) + sizeof(JsdRow));

// per row: sum over its entries of b log b - r log r (k_assign_sparse's order: lanes strided over
// the entries, a butterfly), which depends on no center
__global__ void __launch_bounds__(256) k_jsd_row_terms(const float *__restrict__ vals,
                                                       const uint64_t *__restrict__ indptr, uint64_t n,
                                                       const float *__restrict__ rsi, const float *__restrict__ rinc,
                                                       double *bx) {
    const int lane = threadIdx.x & 31;
    const uint64_t nw = (gridDim.x * uint64_t(blockDim.x)) >> 5;
    for (uint64_t row = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5; row < n; row += nw) {
        const float si = rsi[row], r = rinc[row], rlr = r * logf(r);
        double s = 0.0;
        for (uint64_t p = indptr[row] + lane; p < indptr[row + 1]; p += 32) {
            const float b = vals[p] * si + r;
            s += double(b * logf(b) - rlr);
        }
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
        if (lane == 0) bx[row] = s;
    }
}

int launch_jsd_row_terms(const float *vals, const uint64_t *indptr, uint64_t n, const float *rsi, const float *rinc,
                         double *bx, int sms, cudaStream_t st) {
    k_jsd_row_terms<<<unsigned(umin64((n + 7) / 8, uint64_t(sms) * 16)), 256, 0, st>>>(vals, indptr, n, rsi, rinc, bx),
        note_launch();
    MC_CUDA_TRY(cudaGetLastError());
    return MC_OK;
}

// one entry: g = a row value's transform, c the centers', l0 = m0 log(m0/2)
__device__ __forceinline__ void jsd_entry(float2 &acc, float2 c, float2 l0, float g) {
    const float mx = c.x + g, my = c.y + g;
    acc.x = acc.x + (l0.x - mx * logf(mx * 0.5f));
    acc.y = acc.y + (l0.y - my * logf(my * 0.5f));
}
__device__ __forceinline__ float2 jsd_zero_half(float2 c, float r) {
    const float mx = c.x + r, my = c.y + r;
    return make_float2(mx * logf(mx * 0.5f), my * logf(my * 0.5f));
}

__global__ void __launch_bounds__(kJsdThreads, 1) k_assign_jsd_groups(const AssignArgs a, const JsdGroups jg) {
    extern __shared__ __align__(16) float jsd_sm[];  // [2][band][64] centers, [band][64] table, row states
    float *tab = jsd_sm + 2 * kJsdBand * 64;
    float2 *sums = reinterpret_cast<float2 *>(tab + kJsdBand * 64);
    JsdRow *state = reinterpret_cast<JsdRow *>(sums + kJsdSlab * 32);
    const int t = threadIdx.x, lane = t & 31, wib = t >> 5;
    const uint64_t q = blockIdx.x;
    if (q >= jg.slab_start[jg.nbucket]) return;
    const uint32_t bucket = find_bucket(jg.slab_start, jg.nbucket, q);
    const uint64_t first = (q - jg.slab_start[bucket]) * kJsdSlab;
    const int m = int(umin64(jg.count[bucket] - first, kJsdSlab));
    const uint32_t *rows = jg.perm + jg.start[bucket] + first;
    const bool table = bucket > 0;  // one group's rows; bucket 0 mixes small groups
    const float rt = a.rinc[rows[0]];
    const uint64_t nbands = (a.d + kJsdBand - 1) / kJsdBand;
    Best best[kJsdRows];
#pragma unroll
    for (int i = 0; i < kJsdRows; ++i) best_init(best[i]);
    for (uint32_t g0 = 0; g0 < a.k; g0 += 64) {
        const uint32_t kc = uint32_t(umin64(64, a.k - g0)), ke = (kc + 1) & ~1u;  // centers of this pass, even
        const bool lane_on = 2 * uint32_t(lane) < ke;
        // band b of CT0's columns from g0 into buffer buf
        auto stage = [&](uint64_t b, int buf) {
            const uint64_t b0 = b * kJsdBand, b1 = umin64(b0 + kJsdBand, a.d);
            const uint32_t items = uint32_t(b1 - b0) * 16;  // 16-byte items, 64 columns (kp is 64 or 128 m)
            float4 *dst = reinterpret_cast<float4 *>(jsd_sm + size_t(buf) * kJsdBand * 64);
            for (uint32_t e = t; e < items; e += kJsdThreads) {
                const float *src = a.CT0 + (b0 + (e >> 4)) * a.kp + g0 + 4 * (e & 15);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(uint32_t(__cvta_generic_to_shared(dst + e))),
                             "l"(src)
                             : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        __syncthreads();  // the buffers' readers of the pass before
        stage(0, 0);
        // rows are dealt round the warps: slot s belongs to warp s mod kJsdWarps
        for (int s = wib; s < m; s += kJsdWarps) {
            sums[s * 32 + lane] = make_float2(0.f, 0.f);
            if (lane == 0) {
                const uint32_t row = rows[s];
                JsdRow w;
                w.begin = a.indptr[row];
                w.pos = 0;
                w.len = uint32_t(a.indptr[row + 1] - w.begin);
                w.rsi = a.rsi[row];
                w.r = a.rinc[row];
                state[s] = w;
            }
        }
        __syncwarp();
        for (uint64_t b = 0; b < nbands; ++b) {
            const int buf = int(b & 1);
            const uint32_t b0 = uint32_t(b * kJsdBand), bend = uint32_t(umin64(b0 + kJsdBand, a.d));
            const float *cb = jsd_sm + size_t(buf) * kJsdBand * 64;
            // the first row's window, on its way while the band is staged
            JsdRow w{};
            uint32_t col = 0xffffffffu;
            float val = 0.f;
            auto window = [&](const JsdRow &r, uint32_t &c, float &v) {
                c = 0xffffffffu;
                v = 0.f;
                if (r.pos + lane < r.len) {
                    c = a.idx[r.begin + r.pos + lane];
                    v = a.vals[r.begin + r.pos + lane];
                }
            };
            if (wib < m) {
                w = state[wib];
                window(w, col, val);
            }
            if (b + 1 < nbands) {
                stage(b + 1, buf ^ 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
            if (table) {
                // (column j, center c < ke), packed over the threads
                const uint32_t items = (bend - b0) * ke, dj = kJsdThreads / ke, dc = kJsdThreads - dj * ke;
                uint32_t j = t / ke, c = t - j * ke;
                for (uint32_t e = t; e < items; e += kJsdThreads) {
                    const float m0 = cb[j * 64 + c] + rt;
                    tab[j * 64 + c] = m0 * logf(m0 * 0.5f);
                    j += dj;
                    c += dc;
                    if (c >= ke) {
                        c -= ke;
                        ++j;
                    }
                }
                __syncthreads();
            }
            const float2 *tb = reinterpret_cast<const float2 *>(cb) + lane;
            const float2 *tt = reinterpret_cast<const float2 *>(tab) + lane;
#pragma unroll 1
            for (int s = wib; s < m; s += kJsdWarps) {
                // the next row's window
                JsdRow wn{};
                uint32_t coln = 0xffffffffu;
                float valn = 0.f;
                if (s + kJsdWarps < m) {
                    wn = state[s + kJsdWarps];
                    window(wn, coln, valn);
                }
                float2 acc = sums[s * 32 + lane];
                for (;;) {
                    const float g = val * w.rsi + w.r;
                    // the window's entries before bend form a prefix (columns ascend)
                    const int mm = __popc(__ballot_sync(0xffffffffu, col < bend));
                    const uint32_t off = (col - b0) * 32;
                    int q0 = 0;
                    if (table) {
#pragma unroll 1
                        for (; q0 + 4 <= mm; q0 += 4) {
                            float2 cv[4], tv[4];
                            float gq[4];
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const uint32_t o = __shfl_sync(0xffffffffu, off, q0 + u);
                                gq[u] = __shfl_sync(0xffffffffu, g, q0 + u);
                                cv[u] = tb[o];
                                tv[u] = tt[o];
                            }
                            if (lane_on) {
#pragma unroll
                                for (int u = 0; u < 4; ++u) jsd_entry(acc, cv[u], tv[u], gq[u]);
                            }
                        }
                    }
#pragma unroll 1
                    for (; q0 < mm; ++q0) {
                        const uint32_t o = __shfl_sync(0xffffffffu, off, q0);
                        const float gq = __shfl_sync(0xffffffffu, g, q0);
                        const float2 cv = tb[o];
                        if (lane_on) jsd_entry(acc, cv, table ? tt[o] : jsd_zero_half(cv, w.r), gq);
                    }
                    w.pos += uint32_t(mm);
                    if (mm < 32) break;
                    window(w, col, val);  // the whole window lies in this band
                }
                sums[s * 32 + lane] = acc;
                __syncwarp();
                if (lane == 0) state[s].pos = w.pos;
                w = wn;
                col = coln;
                val = valn;
            }
            __syncthreads();  // every warp is done with the buffer and the table
        }
#pragma unroll
        for (int i = 0; i < kJsdRows; ++i) {
            const int s = i * kJsdWarps + wib;
            if (s >= m) continue;  // warp-uniform
            const uint32_t row = rows[s];
            const double *zrow = a.ztab + uint64_t(a.grp[row]) * a.k;
            const double bx = jg.bx[row];
            const float2 acc = sums[s * 32 + lane];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t c = g0 + 2 * lane + h;
                if (c < a.k) {
                    const float key = post_divergence(float((zrow[c] + bx + double(h ? acc.y : acc.x)) * 0.5));
                    best_offer(best[i], key, c);
                    if (a.dmode) write_dist(a, row, c, float(key_to_cost<JSD>(key)));
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < kJsdRows; ++i) {
        const int s = i * kJsdWarps + wib;
        if (s >= m) continue;
#pragma unroll
        for (int x = 16; x >= 1; x >>= 1) best_merge_shfl(best[i], x);
        if (lane == 0) {
            const bool nan0 = best[i].v == __int_as_float(0xff800000);
            const double cost = nan0 ? __longlong_as_double(0x7ff8000000000000ll) : key_to_cost<JSD>(best[i].v);
            a.asn[rows[s]] = best[i].j;
            a.costs[rows[s]] = double(float(cost));
        }
    }
}

// Groups of several rows over several bands (narrow matrices' centers stay in L1 for the gather); a row's entries at least 12 per band (below, its visits to bands with few
// entries cost more than the halved logarithms save: 200,000 rows, d = 2100, k = 50: 200 entries, 24
// per band, 3.3 ms against 4.4 of the gather kernel; 50 entries, 6 per band, 1.5 against 1.2); a last
// pass of centers that fills its lanes (k = 5: 3.5 against 3.0).  4096 groups bound the counting
// sort's scratch (32 bytes per row).
bool jsd_groups_pay(uint64_t n, uint64_t d, uint32_t k, uint64_t nnz, uint32_t ngrp) {
    return ngrp > 0 && ngrp <= 4096 && d >= 8 * kJsdBand && n >= 8 * uint64_t(ngrp) && (k - 1) % 64 >= 32 &&
           nnz / n * kJsdBand >= 12 * d;
}

int launch_assign_jsd_groups(const AssignArgs &a, const JsdGroups &jg, cudaStream_t st) {
    if (a.n == 0) return MC_OK;
    // a band's columns are staged 64 centers at a time, which CT0's padding has to hold
    if (a.kp % 64) return fail(MC_EINVAL, "JSD row groups: the centers are not padded to 64");
    MC_CUDA_TRY(cudaFuncSetAttribute(k_assign_jsd_groups, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kJsdSmem)));
    // slabs: at most one partial one per group
    const uint64_t slabs = a.n / kJsdSlab + jg.nbucket;
    k_assign_jsd_groups<<<unsigned(slabs), kJsdThreads, kJsdSmem, st>>>(a, jg), note_launch();
    MC_CUDA_TRY(cudaGetLastError());
    return MC_OK;
}

// rank of each group by row count, largest first: CTAs start in the order of the buckets, so the
// longest come first (in group order, the mixed rows last, a quarter of the SM time was idle)
__global__ void __launch_bounds__(256) k_jsd_group_ranks(const uint64_t *__restrict__ count, uint32_t ngrp,
                                                         uint32_t *rank) {
    const int lane = threadIdx.x & 31;
    const uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;  // a warp per group
    if (g >= ngrp) return;
    const uint64_t mine = count[g];
    uint32_t r = 0;
    for (uint32_t h = lane; h < ngrp; h += 32) r += count[h] > mine || (count[h] == mine && h < g);
    r = __reduce_add_sync(0xffffffffu, r);
    if (lane == 0) rank[g] = r;
}

// bucket of each row: its group's rank where the group's entries outnumber the columns, else 0
__global__ void k_jsd_buckets(const uint32_t *__restrict__ grp, const uint64_t *__restrict__ count,
                              const uint32_t *__restrict__ rank, uint64_t n, uint32_t ngrp, uint64_t avg, uint64_t d,
                              uint32_t *bucket) {
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += gridDim.x * uint64_t(blockDim.x)) {
        const uint32_t g = grp[i];
        bucket[i] = count[g] * avg > d ? rank[g] + 1 : 0;
    }
}

int jsd_bucket_rows(const uint32_t *grp, uint64_t n, uint32_t ngrp, uint64_t nnz, uint64_t d, int sms, JsdGroupWork &w,
                    cudaStream_t st) {
    DBuf<uint32_t> bucket, rank;
    MC_TRY(bucket.alloc(n, st));
    MC_TRY(rank.alloc(ngrp, st));
    MC_TRY(launch_sort_by_key(grp, nullptr, n, ngrp, w.sort, st));
    k_jsd_group_ranks<<<(ngrp + 7) / 8, 256, 0, st>>>(w.sort.bucket_count.p, ngrp, rank.p), note_launch();
    k_jsd_buckets<<<unsigned(umin64((n + 255) / 256, uint64_t(sms) * 8)), 256, 0, st>>>(
        grp, w.sort.bucket_count.p, rank.p, n, ngrp, nnz / n, d, bucket.p),
        note_launch();
    MC_TRY(launch_sort_by_key(bucket.p, nullptr, n, ngrp + 1, w.sort, st));
    MC_TRY(w.slabs.alloc(uint64_t(ngrp) + 2, st));
    return launch_scan_ceil_div(w.sort.bucket_count.p, w.slabs.p, uint64_t(ngrp) + 1, kJsdSlab, st);
}

}  // namespace mc
