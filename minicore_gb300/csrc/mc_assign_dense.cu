// Exact FP32 assignment of dense rows (SQRL2, MKL with a constant prior, plain L1): the
// argmin over centers of cmp::msr_with_prior (include/minicore/clustering/solve.h:234-285,
// include/minicore/dist/applicator.h:1632-1915), columns sequential per (row, center), so it is
// bit-identical to k_assign_tiled and the oracle's dense path.
//
// Every (row, center, column) costs two FP32 operations (a difference and its square or
// magnitude), so the FP32 lanes bound it: 128 lane-operations per SM and clock, 37.5e12 a second
// here (measured; packed f32x2 instructions run at the same rate per lane and half the issue
// slots, and a scalar sub + fma pair reaches 27e12).  Hence: two rows per packed instruction,
// rows in pairs and centers stored twice side by side, so that no operand needs a move; 8 rows x 8
// centers per thread, so that 6 shared-memory loads feed 64 packed operations; the row tile transformed
// and kept in shared memory for all centers (up to kDenseCols columns); center chunks of 64, 32 or
// 16, whatever the remainder of k needs, instead of padding k to 128.
// 300,001 x 100, k = 200, SQRL2: 700 -> 528 us (floor 320 us: 1.2e10 operations); fixed-latency
// stalls of three warps per scheduler and the row tile's load take the rest.  Row value duplicated
// by moves instead of the centers in shared memory: 630-660 us; the row tile by transposing 4-byte
// cp.async: 549 us; 96 or 64 columns held at a time for a fourth CTA per SM: 750-780 us.
#include "mc_assign_dev.cuh"

#include <type_traits>

namespace mc {

constexpr int kStep = 16;        // columns per center tile
constexpr int kDenseCols = 192;   // columns of the row tile held at a time
constexpr int kDenseRowsPerWarp = 32;

__device__ __forceinline__ void d2_unpack(unsigned long long v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long d2_sub(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long d2_add(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long d2_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// acc[p][j]: rows (2p, 2p + 1) of this lane's 8 against its center j, over the tile's columns.
// xs: the lane's 8 rows at the step's first column; cs0 / cs1: the lane's centers, duplicated
template <int MSR, int TN>
__device__ __forceinline__ void dense_step(const float *xs, int pitch, const float *cs0, const float *cs1,
                                           unsigned long long (&acc)[4][8]) {
    constexpr int CK = 2 * 8 * TN;  // floats per column of the duplicated center tile
#pragma unroll 16
    for (int kk = 0; kk < kStep; ++kk) {
        const ulonglong2 xa = *reinterpret_cast<const ulonglong2 *>(xs + kk * pitch);
        const ulonglong2 xb = *reinterpret_cast<const ulonglong2 *>(xs + kk * pitch + 4);
        const unsigned long long x[4] = {xa.x, xa.y, xb.x, xb.y};
#pragma unroll
        for (int q = 0; q < TN / 2; ++q) {
            const ulonglong2 ca = *reinterpret_cast<const ulonglong2 *>(cs0 + kk * CK + 32 * q);
            ulonglong2 cb = ca;
            if (MSR == MKL) cb = *reinterpret_cast<const ulonglong2 *>(cs1 + kk * CK + 32 * q);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const unsigned long long c0 = h ? ca.y : ca.x, c1 = h ? cb.y : cb.x;
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    unsigned long long &s = acc[p][2 * q + h];
                    if (MSR == MKL) {
                        s = d2_fma(c0, d2_sub(c1, x[p]), s);
                    } else {
                        const unsigned long long df = d2_sub(c0, x[p]);
                        if (MSR == L1) s = d2_add(s, df & 0x7fffffff7fffffffull);
                        else s = d2_fma(df, df, s);
                    }
                }
            }
        }
    }
}

template <int MSR>
struct DenseTile {
    static constexpr int CARR = (MSR == MKL) ? 2 : 1;                    // center arrays
    static constexpr int CARRF = kStep * 128;                            // floats of an array: 64 centers, twice
    static constexpr int CBUF = CARR * CARRF;                            // floats of one center buffer
};

template <int MSR, int WARPS>
struct DenseCta {
    static constexpr int BM = WARPS * kDenseRowsPerWarp, T = WARPS * 32;
    static constexpr int PITCH = BM + 4;  // a column's rows; rows of a warp's lanes in 16-byte groups
    const AssignArgs &a;
    float *Xs, *Cs;
    int kx, vec;
    uint64_t row0, nrows;

    // V consecutive columns per lane: a warp reads 32 / (16 / V) of its rows' 16-column pieces per
    // instruction and stores them transposed (two rows' lanes per bank at V = 4 and 2)
    template <int V>
    __device__ __forceinline__ void load_vec(uint64_t kb, int cols) const {
        using Vec = typename std::conditional<V == 4, float4, typename std::conditional<V == 2, float2, float>::type>::type;
        constexpr int Q = 16 / V, R = 32 / Q, I = 32 / R;  // lanes per row, rows per load, loads per piece
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, q = lane % Q, rl = w * 32 + lane / Q;
        const float *src[I];
#pragma unroll
        for (int i = 0; i < I; ++i) {
            const uint64_t row = row0 + rl + i * R;
            src[i] = row < nrows ? a.X + (a.rows ? uint64_t(a.rows[row]) : row) * a.d + kb + V * q : nullptr;
        }
        for (int c0 = 0; c0 < kx; c0 += 16) {
            Vec v[I];
#pragma unroll
            for (int i = 0; i < I; ++i) {
                v[i] = Vec{};
                if (src[i] && c0 + V * q < cols) v[i] = __ldg(reinterpret_cast<const Vec *>(src[i] + c0));
            }
#pragma unroll
            for (int i = 0; i < I; ++i) {
                float *dst = Xs + (c0 + V * q) * PITCH + rl + i * R;
                const float *f = reinterpret_cast<const float *>(&v[i]);
#pragma unroll
                for (int e = 0; e < V; ++e) dst[e * PITCH] = f[e];
            }
        }
    }

    // columns [kb, kb + kx) of the rows, transposed to [column][row], zeros past the rows and
    // columns, through the measure's row transform
    __device__ __forceinline__ void load_rows(uint64_t kb) const {
        const int t = threadIdx.x;
        const int cols = int(umin64(kx, a.d - kb));
        if (vec == 4) load_vec<4>(kb, cols);
        else if (vec == 2) load_vec<2>(kb, cols);
        else load_vec<1>(kb, cols);
        __syncthreads();
        if (MSR == SQRL2 || MSR == L1) return;  // raw values
        // thread t: row t % BM (BM divides T or T divides BM)
        for (int r = t % BM; r < BM; r += T) {
            const uint64_t row = row0 + r;
            if (row >= nrows) continue;
            const uint64_t g = a.rows ? uint64_t(a.rows[row]) : row;
            const float rsi = a.rsi[g], rinc = a.rinc[g];
#pragma unroll 8
            for (int c = 0; c < cols; ++c) {
                float x0, x1;
                row_xform<MSR>(Xs[c * PITCH + r], a.pv, rsi, rinc, x0, x1);
                Xs[c * PITCH + r] = x0;
            }
        }
        __syncthreads();
    }

    // the next center tile, two centers per load, in registers while the current one is used;
    // thread t loads center pair t % H of columns t / H, t / H + T / H, ...
    template <int TN>
    struct CenterRegs {
        static constexpr int H = 8 * TN / 2, COLS = T / H < kStep ? T / H : kStep, N = kStep / COLS;
        static_assert(N * COLS == kStep, "whole columns per pass");
        float2 v[DenseTile<MSR>::CARR][N];
    };
    template <int TN>
    __device__ __forceinline__ void fetch_centers(const float *c0, const float *c1, int left, CenterRegs<TN> &r) const {
        using R = CenterRegs<TN>;
        const int kk0 = int(threadIdx.x) / R::H;  // a CTA may have more threads than pairs in the tile
#pragma unroll
        for (int u = 0; u < R::N; ++u) {
            const bool ok = kk0 < R::COLS && kk0 + u * R::COLS < left;
            const uint32_t o = uint32_t(u * R::COLS) * a.kp;
            r.v[0][u] = ok ? *reinterpret_cast<const float2 *>(c0 + o) : make_float2(0.f, 0.f);
            if (MSR == MKL) r.v[DenseTile<MSR>::CARR - 1][u] = ok ? *reinterpret_cast<const float2 *>(c1 + o) : make_float2(0.f, 0.f);
        }
    }
    // (c0, c0, c1, c1) of pair q of lane tx at [column][q][tx]: every 16-byte read of a warp
    // covers 128 consecutive bytes
    template <int TN>
    __device__ __forceinline__ void store_centers(const CenterRegs<TN> &r, int buf) const {
        using R = CenterRegs<TN>;
        const int kk0 = int(threadIdx.x) / R::H, h = int(threadIdx.x) % R::H, tx = h / (TN / 2), q = h % (TN / 2);
        if (kk0 >= R::COLS) return;
        float *dst = Cs + buf * DenseTile<MSR>::CBUF + kk0 * 16 * TN + q * 32 + tx * 4;
#pragma unroll
        for (int arr = 0; arr < DenseTile<MSR>::CARR; ++arr)
#pragma unroll
            for (int u = 0; u < R::N; ++u) {
                const float2 v = r.v[arr][u];
                *reinterpret_cast<float4 *>(dst + arr * DenseTile<MSR>::CARRF + u * R::COLS * 16 * TN) =
                    make_float4(v.x, v.x, v.y, v.y);
            }
    }

    // 8 TN centers from cbase against the tile's rows; the row tile is loaded when it is not
    // there yet
    template <int TN>
    __device__ __forceinline__ void chunk(uint32_t cbase, bool &have_rows, Best &best) const {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, tx = lane & 7, ty = lane >> 3;
        unsigned long long acc[4][8];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
        const float *xs = Xs + w * kDenseRowsPerWarp + ty * 8;
        for (uint64_t kb = 0; kb < a.d; kb += kx) {
            const int steps = int((umin64(kx, a.d - kb) + kStep - 1) / kStep);
            CenterRegs<TN> cr;
            using R = CenterRegs<TN>;
            const uint64_t first = (kb + int(threadIdx.x) / R::H) * a.kp + cbase + 2 * (int(threadIdx.x) % R::H);
            const float *c0 = a.CT0 + first, *c1 = MSR == MKL ? a.CT1 + first : nullptr;
            const int left = int(umin64(a.d - kb, kDenseCols));  // columns from kb on
            fetch_centers<TN>(c0, c1, left, cr);
            __syncthreads();  // the last readers of the row tile and of center buffer 0
            if (!have_rows || uint64_t(kx) < a.d) {
                load_rows(kb);
                have_rows = true;
            }
            store_centers<TN>(cr, 0);
            for (int s = 0; s < steps; ++s) {
                if (s + 1 < steps) {
                    c0 += uint64_t(kStep) * a.kp;
                    if (MSR == MKL) c1 += uint64_t(kStep) * a.kp;
                    fetch_centers<TN>(c0, c1, left - (s + 1) * kStep, cr);
                }
                __syncthreads();  // buffer s & 1 is complete; the other's readers are done
                const float *cs = Cs + (s & 1) * DenseTile<MSR>::CBUF + tx * 4;
                dense_step<MSR, TN>(xs + s * kStep * PITCH, PITCH, cs, cs + DenseTile<MSR>::CARRF, acc);
                if (s + 1 < steps) store_centers<TN>(cr, (s + 1) & 1);
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint64_t row = row0 + w * kDenseRowsPerWarp + ty * 8 + i;
            Best b;
            best_init(b);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const uint32_t c = cbase + tx * TN + j;
                if (c < a.k) {
                    float lo, hi;
                    d2_unpack(acc[i >> 1][j], lo, hi);
                    const float key = finish_key<MSR>((i & 1) ? hi : lo);
                    best_offer(b, key, c);
                    if (a.dmode && row < nrows)
                        write_dist(a, a.rows ? uint64_t(a.rows[row]) : row, c, float(key_to_cost<MSR>(key)));
                }
            }
            // the eight lanes that share the row; lane tx == i keeps the row's running best
#pragma unroll
            for (int m = 4; m >= 1; m >>= 1) best_merge_shfl(b, m);
            if (tx == i && (b.v < best.v || (b.v == best.v && b.j < best.j))) best = b;
        }
    }
};

template <int MSR, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 12 / WARPS) k_assign_dense(const AssignArgs a, int kx, int vec) {
    extern __shared__ __align__(16) float dense_sm[];
    using Cta = DenseCta<MSR, WARPS>;
    if (MSR == L1 && !l1_plain(a)) return;
    uint64_t nrows = a.n;
    if (a.n_dev) {
        nrows = umin64(nrows, *a.n_dev);
        if (assign_few_takes(a, nrows)) return;
    }
    Cta cta{a, dense_sm, dense_sm + Cta::PITCH * kx, kx, vec, 0, nrows};
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, tx = lane & 7, ty = lane >> 3;
    for (uint64_t tile = blockIdx.x; tile * Cta::BM < nrows; tile += gridDim.x) {
        cta.row0 = tile * Cta::BM;
        Best best;  // of row 8 ty + tx of the warp's 32
        best_init(best);
        bool have_rows = false;
        uint32_t c = 0;
        // 64, 32 or 16 centers at a time; 33 to 48 go as 64, which takes less time than 32 and 16 (MKL
        // 100,000 x 160, k = 100: 376 us as 64 + 32 + 16, 315 as 64 + 64)
        while (c < a.k) {
            const uint32_t left = a.k - c;
            if (left > 32) {
                cta.template chunk<8>(c, have_rows, best);
                c += 64;
            } else if (left > 16) {
                cta.template chunk<4>(c, have_rows, best);
                c += 32;
            } else {
                cta.template chunk<2>(c, have_rows, best);
                c += 16;
            }
        }
        const uint64_t row = cta.row0 + w * kDenseRowsPerWarp + ty * 8 + tx;
        if (row < nrows) {
            const bool nan0 = best.v == __int_as_float(0xff800000);
            const uint64_t o = a.rows ? uint64_t(a.rows[row]) : row;
            a.asn[o] = best.j;
            a.costs[o] = nan0 ? __longlong_as_double(0x7ff8000000000000ll) : key_to_cost<MSR>(best.v);
        }
    }
}

// columns per load of a row
static int row_vec(const AssignArgs &a) {
    const uintptr_t xp = reinterpret_cast<uintptr_t>(a.X);
    return a.d % 4 == 0 && xp % 16 == 0 ? 4 : a.d % 2 == 0 && xp % 8 == 0 ? 2 : 1;
}

template <int MSR, int WARPS>
static int dense_launch_w(const AssignArgs &a, cudaStream_t st) {
    const int kx = int(umin64((a.d + kStep - 1) / kStep * kStep, kDenseCols));
    const int vec = row_vec(a);
    constexpr int BM = WARPS * kDenseRowsPerWarp;
    auto smem_of = [](int cols) { return (size_t(BM + 4) * cols + 2 * DenseTile<MSR>::CBUF) * sizeof(float); };
    auto kern = k_assign_dense<MSR, WARPS>;
    // always the widest tile's size: a smaller one could be set under another thread's launch
    MC_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem_of(kDenseCols))));
    const uint64_t tiles = (a.n + BM - 1) / BM;
    // a row count read on the device is usually far below a.n: a grid that fills the chip
    // walks what there is
    const uint64_t grid = a.n_dev ? umin64(tiles, 152 * 2) : tiles;
    kern<<<unsigned(umin64(grid, 0x7fffffffull)), 32 * WARPS, smem_of(kx), st>>>(a, kx, vec), note_launch();
    MC_CUDA_TRY(cudaGetLastError());
    return MC_OK;
}

// Which passes come here (n x d rows, k centers) and which go to k_assign_tiled, from both kernels' times
// (here / k_assign_tiled, us) over 17 row counts of 3,000 to 1,000,000, 21 column counts of 8 to 256 and
// 16 center counts of 8 to 1000; at the worst point of that grid the rule loses 4 %.  What decides:
//  * k_assign_tiled pads k to 64 (128 from 65 on), a chunk here to 16, 32 or 64: up to 32 centers this
//    kernel gains even where it runs less well (SQRL2 150,000 x 16, k = 8: 18 / 28; 100,000 x 64,
//    k = 32: 30 / 55);
//  * a chunk starts with a barrier and a fetch and ends with the argmin over its centers, which few
//    columns do not pay for (SQRL2 300,000 x 16, k = 64: 64 / 49; x 50, k = 128: 208 / 190);
//  * twelve warps per SM fit up to some 112 columns, eight up to 176 (MKL, whose center tile is twice as
//    large: 64 and 144), then four (SQRL2 300,000 x 192, k = 128: 758 / 671; MKL 39,500 x 256, k = 128:
//    264 / 247; at 144: 119 / 141); past kDenseCols the rows are also loaded, and MKL's logarithms taken, again for every
//    64 centers (SQRL2 300,000 x 256, k = 128: 1043 / 890);
//  * odd columns are loaded four bytes at a time (SQRL2 60,000 x 97, k = 100: 95 / 90; x 96: 82 / 86).
// Hellinger (a square root per row entry and CTA, k = 100: 120 / 111) and JSD (a logarithm per pair) do
// not come here, nor does MKL up to 64 centers.
bool assign_dense_pays(const AssignArgs &a) {
    const uint64_t n = a.n, d = a.d;
    const uint32_t k = a.k;
    const bool odd = row_vec(a) == 1;
    if (a.msr == MKL) return k > 64 && d >= (odd ? 112 : 64) && d <= (k > 128 ? 192 : 144);
    if (a.msr != SQRL2) return false;
    if (k <= 16) return d >= 16;
    if (k <= 32) return d >= 48 || (d >= 32 && n >= 12000);
    if (k > 64) return !odd && d >= 112 && d <= 176;
    if (odd) return d >= 112 && d <= 176;
    if (d > 176) return n > 128 * 152 * 2;
    return d >= 72 || (d >= 64 && n >= 75000);
}

int launch_assign_dense(const AssignArgs &a, cudaStream_t st) {
    // 128 rows per CTA; 64 where a tile of 128 rows leaves room for one CTA per SM (SQRL2 300,000 x 256,
    // k = 64: 457 / 559 us)
    switch (a.msr) {
        case SQRL2: return a.d <= 176 ? dense_launch_w<SQRL2, 4>(a, st) : dense_launch_w<SQRL2, 2>(a, st);
        case MKL: return dense_launch_w<MKL, 4>(a, st);
        // L1 in pair mode where its terms are plain differences (l1_plain); which sizes: l1_dense_pays
        case L1: return dense_launch_w<L1, 4>(a, st);
        default: return fail(MC_EUNSUPPORTED, "k_assign_dense does not cover this measure");
    }
}

}  // namespace mc
