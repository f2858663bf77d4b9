// Chunk partials of the centroid sums over CSR rows (set_centroids_full_mean,
// clustering/centroid.h:649-779): per chunk of a cluster's rows (ascending) and column, the
// compensated float sum (unweighted) or FP64 fma sum (weighted) of the stored values, rows in
// order.  Both kernels here give, per column, the additions of k_centroid_chunks_csr in the
// same order, so the partials are bit-identical to it; they differ in who waits for whom.
#include "mc_reduce.cuh"

#include <cstddef>

namespace mc {

// ------------------------------------------------------------------------------------
// Wide rows: one warp per (chunk, column band).
// ------------------------------------------------------------------------------------
// off[r][b] = number of entries of row r in bands below b (bands of 2^shift columns,
// b <= nb), so that a warp finds its band's part of a row without a search.  One warp per
// row; the indices are read once (coalesced).
__global__ void __launch_bounds__(256) k_csr_band_offsets(const uint32_t *__restrict__ idx,
                                                          const uint64_t *__restrict__ indptr, uint64_t n, int shift,
                                                          uint32_t nb, uint32_t *__restrict__ off) {
    const int lane = threadIdx.x & 31;
    const uint64_t nw = (gridDim.x * uint64_t(blockDim.x)) >> 5;
    for (uint64_t r = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5; r < n; r += nw) {
        const uint64_t pb = indptr[r], pe = indptr[r + 1];
        uint32_t *o = off + r * (uint64_t(nb) + 1);
        uint32_t next = 0;  // first band whose offset is not written yet (warp-uniform)
        for (uint64_t base = pb; base < pe; base += 32) {
            const uint64_t p = base + lane;
            const uint32_t b = p < pe ? idx[p] >> shift : nb;
            uint32_t from = __shfl_up_sync(0xffffffffu, b, 1) + 1;
            if (lane == 0) from = next;
            if (p < pe)
                for (uint32_t q = from; q <= b; ++q) o[q] = uint32_t(p - pb);
            const int last = int(umin64(32, pe - base)) - 1;
            next = __shfl_sync(0xffffffffu, b, last) + 1;
        }
        for (uint32_t q = next + lane; q <= nb; q += 32) o[q] = uint32_t(pe - pb);
    }
}

// Four warps per CTA, each with its own band of 2^shift columns in shared memory ((s, e)
// float pairs, or FP64 sums); no barrier anywhere.  A warp walks the chunk's rows in order:
// the rows' bounds in this band sit in shared memory, 64 rows at a time, and a row's entries
// (up to 32 kBandRounds of them, the rest straight from memory) are in registers kBandAhead
// rows before they are added.  The rows of a chunk are one dependent chain per column (a
// shared-memory read, a TwoSum, a write), and the instructions per (row, band) come second;
// bytes do not bound it.  200,000 x 20,000 rows of 1500 entries, k = 50, whole update: 1.2 ms
// (2.4 GB: 0.36 ms at the copy rate) against 6.1 ms with one CTA per chunk and all its columns
// (k_centroid_chunks_csr: two block barriers and a load latency per row, and a chunk per SM).
// Measured there: 4 rows ahead 1.48 ms; bands of 512 columns 1.30, of 1024 (three rounds) 1.6;
// the entries through a cp.async ring 1.4-2.1.
constexpr int kBandWarps = 4;
constexpr int kBandAhead = 8;
constexpr int kBandRounds = 2;
constexpr int kBandMeta = 64;
// per warp: row bounds and weights (64 rows), the band's sums, a spare slot per lane
constexpr size_t band_smem(int shift) { return kBandMeta * 24 + (size_t(8) << shift) + 256; }

template <bool WEIGHTED>
__global__ void __launch_bounds__(32 * kBandWarps) k_centroid_band_csr(
    const float *__restrict__ vals, const uint32_t *__restrict__ idx, const uint64_t *__restrict__ indptr, uint64_t d,
    int shift, uint32_t nb, const uint32_t *__restrict__ off, const uint32_t *__restrict__ perm,
    const uint64_t *__restrict__ bucket_start, const uint64_t *__restrict__ bucket_count,
    const uint64_t *__restrict__ chunk_start, uint32_t k, uint64_t ch, const double *__restrict__ w,
    double *__restrict__ partial, double *__restrict__ partial_w) {
    extern __shared__ __align__(16) unsigned char band_sm[];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const uint64_t q = blockIdx.x;
    if (q >= chunk_start[k]) return;
    const uint32_t b = blockIdx.y * kBandWarps + wp;
    if (b > nb || (b == nb && !WEIGHTED)) return;  // warps share nothing: no barrier below
    const uint32_t c = find_bucket(chunk_start, k, q);
    const uint64_t r0 = (q - chunk_start[c]) * ch;
    const int cnt = int(umin64(bucket_count[c] - r0, ch));
    const uint32_t *rows = perm + bucket_start[c] + r0;
    if (b == nb) {  // one warp more than bands: the chunk's weight, rows in order
        if (lane == 0) {
            double wq = 0.0;
            for (int r = 0; r < cnt; ++r) wq = wq + w[rows[r]];
            partial_w[q] = wq;
        }
        return;
    }
    const uint32_t bw = 1u << shift, j0 = b << shift;
    unsigned char *mine = band_sm + size_t(wp) * band_smem(shift);
    ulonglong2 *meta = reinterpret_cast<ulonglong2 *>(mine);  // (first entry, entries) of row r at r % 64
    double *wts = reinterpret_cast<double *>(meta + kBandMeta);
    double *acc = wts + kBandMeta;
    float2 *se = reinterpret_cast<float2 *>(acc);
    for (uint32_t j = lane; j < bw; j += 32) acc[j] = 0.0;  // the bits of (0.f, 0.f) too
    // bounds of row r of the chunk (row id `row`); no entries past the chunk's rows
    uint64_t st = 0;
    uint32_t len = 0;
    double wr = 0.0;
    auto fetch = [&](int r, uint32_t row) {
        st = 0;
        len = 0;
        if (r < cnt) {
            const uint32_t *o = off + uint64_t(row) * (uint64_t(nb) + 1) + b;
            const uint32_t a0 = o[0], a1 = o[1];
            st = indptr[row] + a0;
            len = a1 - a0;
            if (WEIGHTED) wr = w[row];
        }
    };
    auto put = [&](int at) {
        meta[at] = make_ulonglong2(st, len);
        if (WEIGHTED) wts[at] = wr;
    };
    auto row_id = [&](int r) { return r < cnt ? rows[r] : 0u; };
    auto add = [&](uint32_t col, float v, double wgt) {
        const uint32_t j = col - j0;
        if (j >= bw) return;
        if (WEIGHTED) {
            acc[j] = fma(wgt, double(v), acc[j]);
        } else {
            float2 t = se[j];
            two_sum_add(t.x, t.y, v);
            se[j] = t;
        }
    };
    // (a loaded column is touched only when its row is added: arithmetic beside the load would
    // wait for it)
    struct Slot {
        uint32_t len, c[kBandRounds];
        float v[kBandRounds];
    } S[kBandAhead];
    const uint32_t *idx_l = idx + lane;
    const float *vals_l = vals + lane;
    auto load = [&](int r, Slot &s) {
        const ulonglong2 m = meta[r & (kBandMeta - 1)];
        s.len = uint32_t(m.y);
#pragma unroll
        for (int i = 0; i < kBandRounds; ++i)
            if (i == 0 || s.len > 32 * i) {  // warp-uniform
                s.c[i] = 0xffffffffu;
                if (uint32_t(lane) + 32 * i < s.len) {
                    s.c[i] = __ldg(idx_l + m.x + 32 * i);
                    s.v[i] = __ldg(vals_l + m.x + 32 * i);
                }
            }
    };
    // lanes without an entry add into their own spare slot past the band
    auto slot_of = [&](uint32_t col) { return col - j0 < bw ? col - j0 : bw + lane; };
    fetch(lane, row_id(lane));
    put(lane);
    fetch(32 + lane, row_id(32 + lane));
    put(32 + lane);
    fetch(64 + lane, row_id(64 + lane));
    uint32_t next_row = row_id(96 + lane);
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kBandAhead; ++u) load(u, S[u]);
    for (int rb = 0; rb < cnt; rb += 32) {
        for (int t0 = rb; t0 < rb + 32; t0 += kBandAhead) {
#pragma unroll
            for (int u = 0; u < kBandAhead; ++u) {
                const int r = t0 + u;
                const uint32_t n = S[u].len;
                const double wgt = WEIGHTED ? wts[r & (kBandMeta - 1)] : 0.0;
                uint32_t j[kBandRounds];
                float2 t[kBandRounds];
                double td[kBandRounds];
#pragma unroll
                for (int i = 0; i < kBandRounds; ++i)
                    if (i == 0 || n > 32 * i) {
                        j[i] = slot_of(S[u].c[i]);
                        if (WEIGHTED) td[i] = acc[j[i]];
                        else t[i] = se[j[i]];
                    }
#pragma unroll
                for (int i = 0; i < kBandRounds; ++i)
                    if (i == 0 || n > 32 * i) {
                        if (WEIGHTED) {
                            acc[j[i]] = fma(wgt, double(S[u].v[i]), td[i]);
                        } else {
                            two_sum_add(t[i].x, t[i].y, S[u].v[i]);
                            se[j[i]] = t[i];
                        }
                    }
                if (n > 32 * kBandRounds) {
                    const uint64_t p0 = meta[r & (kBandMeta - 1)].x;
                    for (uint32_t p = uint32_t(lane) + 32 * kBandRounds; p < n; p += 32) add(idx[p0 + p], vals[p0 + p], wgt);
                }
                load(r + kBandAhead, S[u]);
                __syncwarp();  // this row's sums before the next row's
            }
        }
        // rows rb .. rb + 31 are done: their bounds make room for rows rb + 64 .. rb + 95
        __syncwarp();
        put((rb & 32) + lane);
        fetch(rb + 96 + lane, next_row);
        next_row = row_id(rb + 128 + lane);
        __syncwarp();
    }
    const uint32_t jn = uint32_t(umin64(bw, d - j0));
    for (uint32_t j = lane; j < jn; j += 32)
        partial[q * d + j0 + j] = WEIGHTED ? acc[j] : double(se[j].x) + double(se[j].y);
}

// ------------------------------------------------------------------------------------
// Short rows over narrow matrices (a few entries per row, d <= 2048): one CTA per (chunk,
// 512 columns), kShortRows rows at a time.
// ------------------------------------------------------------------------------------
// Thread t takes row t of the batch and marks it in every column it touches (mask[row / 32]
// [column], one bit per row); thread j then knows how many rows of the batch touch column j,
// a block scan gives every column its slots, and the rows write their values to slot
// start(column) + (marked rows before it).  Column j's values now lie side by side, rows in
// order, and thread j adds them.  Rows load concurrently, and a batch costs three dependent
// loads and five barriers whatever the number of entries; scattering 32 rows at a time into
// a dense tile and walking every column of it took four barriers and two dependent loads per
// 32 rows.  A batch with more entries than slots is ordered in halves or quarters of its rows (an update
// of 18,535 x 171 rows of 30 entries, k = 4: 1.34 ms without, 0.40), and a part that still has more is added 16 rows at a time through a dense [16][512] tile in the same
// memory (the masks say which cells are filled).
constexpr int kShortCols = 512, kShortRows = 512, kShortWords = kShortRows / 32;
constexpr int kShortSlots = 16 * kShortCols;

struct ShortSmem {
    uint32_t mask[kShortWords][kShortCols];
    uint32_t pre[kShortWords][kShortCols];  // slot of the first marked row of the word
    float slot[kShortSlots];
    uint32_t wsum[kShortCols / 32];
    // weighted only (not allocated otherwise: two CTAs per SM instead of one)
    double wt[kShortRows];
    uint32_t rowof[kShortSlots];  // the batch row of each slot
};

template <bool WEIGHTED>
__global__ void __launch_bounds__(kShortCols) k_centroid_short_csr(
    const float *__restrict__ vals, const uint32_t *__restrict__ idx, const uint64_t *__restrict__ indptr, uint64_t d,
    const uint32_t *__restrict__ perm, const uint64_t *__restrict__ bucket_start,
    const uint64_t *__restrict__ bucket_count, const uint64_t *__restrict__ chunk_start, uint32_t k, uint64_t ch,
    const double *__restrict__ w, double *__restrict__ partial, double *__restrict__ partial_w) {
    extern __shared__ __align__(16) unsigned char short_sm[];
    ShortSmem &sm = *reinterpret_cast<ShortSmem *>(short_sm);
    const uint64_t q = blockIdx.x;
    if (q >= chunk_start[k]) return;
    const uint32_t c = find_bucket(chunk_start, k, q);
    const uint64_t r0 = (q - chunk_start[c]) * ch;
    const int cnt = int(umin64(bucket_count[c] - r0, ch));
    const uint32_t *rows = perm + bucket_start[c] + r0;
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5;
    const uint32_t j0 = blockIdx.y * kShortCols;
    for (int i = 0; i < kShortWords; ++i) sm.mask[i][t] = 0u;
    float s = 0.f, e = 0.f;
    double acc = 0.0, wq = 0.0;
    // row t of the batch at b0
    uint64_t pb = 0, pe = 0;
    double wr = 0.0;
    auto bounds = [&](int b0) {
        pb = pe = 0;
        if (b0 + t < cnt) {
            const uint32_t row = rows[b0 + t];
            pb = indptr[row];
            pe = indptr[row + 1];
            if (WEIGHTED) wr = w[row];
        }
    };
    bounds(0);
    __syncthreads();
    for (int b0 = 0; b0 < cnt; b0 += kShortRows) {
        const int nrow = min(kShortRows, cnt - b0);
        if (WEIGHTED) sm.wt[t] = wr;
        const uint32_t bit = 1u << lane;
        for (uint64_t p = pb; p < pe; ++p) {
            const uint32_t j = idx[p] - j0;
            if (j < kShortCols) atomicOr(&sm.mask[wp][j], bit);
        }
        __syncthreads();
        // the batch's words (32 rows each) w0 .. w0 + words at a time: all of them, or as many as surely fit the
        // slots where they do not
        int words = kShortWords;
        for (int w0 = 0; w0 < kShortWords; w0 += words) {
            // slots of column t: the part's entries in the columns before it
            uint32_t mine = 0;
            if (words == kShortWords) {
#pragma unroll
                for (int i = 0; i < kShortWords; ++i) mine += __popc(sm.mask[i][t]);
            } else {
                for (int i = w0; i < w0 + words; ++i) mine += __popc(sm.mask[i][t]);
            }
            uint32_t inc = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            if (lane == 31) sm.wsum[wp] = inc;
            __syncthreads();
            uint32_t first = inc - mine, total = 0;
#pragma unroll
            for (int i = 0; i < kShortCols / 32; ++i) {
                const uint32_t v = sm.wsum[i];
                first += i < wp ? v : 0u;
                total += v;
            }
            // (all conditions here are the same for the block)
            if (total > uint32_t(kShortSlots) && words == kShortWords) {
                words = total <= uint32_t(kShortSlots) * 3 / 2 ? kShortWords / 2 : kShortWords / 4;
                w0 = -words;
                __syncthreads();  // the sums' readers
                continue;
            }
            if (w0 * 32 >= nrow) break;
            if (total <= uint32_t(kShortSlots)) {
                uint32_t at = first;
                if (words == kShortWords) {
#pragma unroll
                    for (int i = 0; i < kShortWords; ++i) {
                        sm.pre[i][t] = at;
                        at += __popc(sm.mask[i][t]);
                    }
                } else {
                    for (int i = w0; i < w0 + words; ++i) {
                        sm.pre[i][t] = at;
                        at += __popc(sm.mask[i][t]);
                    }
                }
                __syncthreads();
                if (wp >= w0 && wp < w0 + words)
                    for (uint64_t p = pb; p < pe; ++p) {
                        const uint32_t j = idx[p] - j0;
                        if (j < kShortCols) {
                            const uint32_t o = sm.pre[wp][j] + __popc(sm.mask[wp][j] & (bit - 1u));
                            sm.slot[o] = vals[p];
                            if (WEIGHTED) sm.rowof[o] = uint32_t(t);
                        }
                    }
                __syncthreads();
                for (uint32_t o = first; o < first + mine; ++o) {
                    if (WEIGHTED) acc = fma(sm.wt[sm.rowof[o]], double(sm.slot[o]), acc);
                    else two_sum_add(s, e, sm.slot[o]);
                }
            } else {
                for (int g = 32 * w0; g < min(nrow, 32 * (w0 + words)); g += 16) {
                    __syncthreads();
                    if (t >= g && t < g + 16)
                        for (uint64_t p = pb; p < pe; ++p) {
                            const uint32_t j = idx[p] - j0;
                            if (j < kShortCols) sm.slot[(t - g) * kShortCols + j] = vals[p];
                        }
                    __syncthreads();
                    uint32_t m = (sm.mask[g >> 5][t] >> (g & 31)) & 0xffffu;
                    while (m) {
                        const int r = __ffs(m) - 1;
                        m &= m - 1;
                        const float v = sm.slot[r * kShortCols + t];
                        if (WEIGHTED) acc = fma(sm.wt[g + r], double(v), acc);
                        else two_sum_add(s, e, v);
                    }
                }
            }
            if (words < kShortWords) __syncthreads();  // the part's slots and sums are read
        }
        if (WEIGHTED && t == 0 && blockIdx.y == 0)
            for (int r = 0; r < nrow; ++r) wq = wq + sm.wt[r];
        // column t's masks are read by this thread and, before the barrier above, by the rows
        for (int i = 0; i < kShortWords; ++i) sm.mask[i][t] = 0u;
        bounds(b0 + kShortRows);
        __syncthreads();
    }
    if (j0 + uint32_t(t) < d) partial[q * d + j0 + t] = WEIGHTED ? acc : double(s) + double(e);
    if (WEIGHTED && t == 0 && blockIdx.y == 0) partial_w[q] = wq;
}

// The band width for rows of avg entries over d columns, as a power of two (0: the bands
// would be too many for the row offsets to pay): about 24 entries of a row per band (a
// row's part mostly fills one warp load), at most
// 2048 columns (16 KB of sums per warp, 3 CTAs per SM), and at most avg / 4 offsets per row
// (an eighth of the rows' own bytes).
int csr_band_shift(uint64_t d, uint64_t avg) {
    if (avg < 16) return 0;
    int s = 7;
    while (s < 11 && (uint64_t(2) << s) * avg <= 24 * d) ++s;
    const uint64_t nb = (d + (uint64_t(1) << s) - 1) >> s;
    return (nb + 1) * 4 <= avg || nb <= 4 ? s : 0;
}

template <bool WEIGHTED>
static int band_launch(const CentroidArgs &a, SortWork &w, uint64_t max_chunks, uint64_t ch, int shift, uint32_t nb,
                       cudaStream_t st) {
    auto kern = k_centroid_band_csr<WEIGHTED>;
    const size_t smem = kBandWarps * band_smem(shift);
    // always the largest width's size: a smaller one could be set under another thread's launch
    MC_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     int(kBandWarps * band_smem(11))));
    const unsigned gy = (nb + (WEIGHTED ? 1u : 0u) + kBandWarps - 1) / kBandWarps;
    kern<<<dim3(unsigned(max_chunks), gy), 32 * kBandWarps, smem, st>>>(
        a.vals, a.idx, a.indptr, a.d, shift, nb, w.bands.p, w.perm.p, w.bucket_start.p, w.bucket_count.p,
        w.chunk_start.p, a.k, ch, a.w, w.partial.p, w.partial_w.p), note_launch();
    MC_CUDA_TRY(cudaGetLastError());
    return MC_OK;
}

// *done = false: neither kernel applies (very wide and sparse rows, or no memory for the band
// offsets: k_centroid_chunks_csr)
int launch_centroid_chunks_csr(const CentroidArgs &a, SortWork &w, uint64_t max_chunks, uint64_t ch, cudaStream_t st,
                               bool *done) {
    const uint64_t n = a.n, d = a.d;
    *done = true;
    if (a.nnz < 32 * n && d <= 4 * uint64_t(kShortCols)) {
        auto kern = a.w ? k_centroid_short_csr<true> : k_centroid_short_csr<false>;
        const size_t smem = a.w ? sizeof(ShortSmem) : offsetof(ShortSmem, wt);
        MC_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        kern<<<dim3(unsigned(max_chunks), unsigned((d + kShortCols - 1) / kShortCols)), kShortCols, smem, st>>>(a.vals, a.idx, a.indptr, d, w.perm.p, w.bucket_start.p, w.bucket_count.p, w.chunk_start.p, a.k,
                     ch, a.w, w.partial.p, w.partial_w.p), note_launch();
        MC_CUDA_TRY(cudaGetLastError());
        return MC_OK;
    }
    const int shift = n ? csr_band_shift(d, a.nnz / n) : 0;
    if (shift) {
        const uint32_t nb = uint32_t((d + (uint64_t(1) << shift) - 1) >> shift);
        if (!a.keep_bands || !w.bands_ready) {
            const uint64_t count = n * (uint64_t(nb) + 1);
            if (!w.bands_refused && count > w.bands.n)
                w.bands_refused = !device_room_to_spare(count * sizeof(uint32_t)) || w.bands.alloc(count, st) != MC_OK;
            if (w.bands_refused) {  // no room for the offsets, which no later update, maybe captured, asks for again
                cudaGetLastError();
                *done = false;
                return MC_OK;
            }
            k_csr_band_offsets<<<unsigned(umin64((n + 7) / 8, 152 * 8)), 256, 0, st>>>(a.idx, a.indptr, n, shift, nb,
                                                                                     w.bands.p), note_launch();
            MC_CUDA_TRY(cudaGetLastError());
            w.bands_ready = a.keep_bands;
        }
        return a.w ? band_launch<true>(a, w, max_chunks, ch, shift, nb, st)
                   : band_launch<false>(a, w, max_chunks, ch, shift, nb, st);
    }
    *done = false;
    return MC_OK;
}

}  // namespace mc
