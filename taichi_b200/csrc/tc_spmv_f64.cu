// tc_spmv_f64.cu -- the multiply in double precision: y = A x with FP64 x and
// y over the same resident plan (the reference's VALUE_TYPE=double build,
// TaiChi.h:62-64, which turns x, y and the kernels' accumulators into double;
// the pattern and the hybrid format are unchanged).
//
// A row belongs to a group of 2^lg lanes: its dense-diagonal terms in offset
// order, then its CSR words in stored order, each dealt out to the lanes in
// turn, three or four words of a lane in flight together, joined by a
// butterfly.  Plans of short rows run kBlock >> lg consecutive rows a CTA
// straight from the row pointers; plans with rows of more than kShortRow words
// run a CTA per tile of the plan's list (whose words are bounded), leaving a
// row that is long for its tile to a warp and a one-row tile to the whole CTA.
// The launch may overlap the end of the kernel before it, as in FP32: x is
// read and y written after griddepcontrol.wait only, with coherent loads.
//
// What bounds it: bytes (8 per x and y value), and the latency of row pointer
// -> word -> x.  Rows of a few words strided over a tile's CTA, one dependent
// word and gather after the other, which this replaces, ran at 35 % of the
// copy rate.  Measured per multiply (us, before -> now):
//   9-point mesh 1531^2 (hybrid, 6 words a row)      45.1 -> 27.8
//   banded 700,001 x 32                             107.5 -> 35.9
//   banded 65,536 x 18                                8.3 -> 4.9
//   banded 1,003,602 x 19                            39.7 -> 36.7
//   R-MAT scale 20 (0.6 words a row)                 22.9 -> 6.9
//   15 diagonals of 900,000 rows with holes          31.5 -> 14.4
//   power-law R-MAT scale 20 / 18 / 16          82 / 30 / 17 -> 73 / 23 / 12

#include <cuda_runtime.h>

#include "tc_internal.h"
#include "tc_tile.cuh"

namespace tc {
namespace {

constexpr int kF64Blocks = 8;     // resident CTAs per SM
constexpr int kShortRow = 128;    // plans with longer rows go by tiles
constexpr int kLaneWords = 8;     // in a tile: words of a lane on average, at most,
constexpr int kLaneMost = 32;     // and words of a lane past which its row is left to the warp
constexpr int kLongTile = 1024;   // a one-row tile of more words by the whole CTA
constexpr int kAheadWords = 1 << 14;   // most words of a later CTA prefetched into L2

__device__ __forceinline__ double ldx64(const double *p)
{
    double v;
    asm("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ void wait_prior64(const double *__restrict__ &x, double *__restrict__ &y)
{
    asm volatile("griddepcontrol.wait;" : "+l"(x), "+l"(y)::"memory");
}

// v of an addition word (c & 1), -v of a hole's.
__device__ __forceinline__ double signed_term64(double v, int c)
{
    return __hiloint2double(__double2hiint(v) ^ (int)((unsigned)~c << 31), __double2loint(v));
}

// Words j, j + by, ... (W of them, before e), and their terms added to acc.
template <int W>
__device__ __forceinline__ void load_words(const DevPlan &p, int j, int e, int by, int (&c)[W])
{
#pragma unroll
    for (int w = 0; w < W; ++w) c[w] = w * by < words_left(j, e) ? __ldg(p.cols + j + w * by) : 0;
}

template <bool SIGNED, int W>
__device__ __forceinline__ void add_words(const double *__restrict__ x, int j, int e, int by, const int (&c)[W],
                                          double &acc)
{
    double v[W];                  // a slot past the row loads x[0] and is not added
#pragma unroll
    for (int w = 0; w < W; ++w) v[w] = ldx64(x + (SIGNED ? c[w] >> 1 : c[w]));
#pragma unroll
    for (int w = 0; w < W; ++w)
        if (w * by < words_left(j, e)) acc += SIGNED ? signed_term64(v[w], c[w]) : v[w];
}

// The dense-diagonal terms of row r that lane `lane` of `lanes` owns
// (offsets lane, lane + lanes, ... of each shape holding the row).
__device__ __forceinline__ double diag_terms64(const DevPlan &p, const PlanDiags &q, const double *__restrict__ x,
                                               int r, int lane, int lanes)
{
    double acc = 0.0;
    if (q.n > 0) {                // offsets from the launch parameters
        if (r < q.rows.x || r >= q.rows.y) return acc;
        const bool inner = r >= q.in.x && r < q.in.y;          // every offset reaches the row
#pragma unroll 1
        for (int i = 0; i < q.n; i += 4) {
            double d[4];
            bool in[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                in[u] = i + u < q.n && (lanes == 1 || ((i + u) & (lanes - 1)) == lane);
                if (!inner) in[u] = in[u] && q.has(i + u, r);
                d[u] = ldx64(x + (in[u] ? r + q.col[i + u] : 0));
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (in[u]) acc += d[u];
        }
        return acc;
    }
    if (r < p.row_start || r >= p.row_stop) return acc;
    for (int s = 0; s < p.dia_shapes; ++s) {
        const int4 sh = __ldg(p.shapes + s);
        if (r < sh.x || r >= sh.y) continue;
        const int2 dr = __ldg(p.shape_dias + s);
        const int cb = r - sh.x + sh.z;
        for (int d = dr.x + lane; d < dr.y; d += 4 * lanes) {
            double v[4];
            bool in[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = d + u * lanes < dr.y ? cb + __ldg(p.offsets + d + u * lanes) : -1;
                in[u] = c >= sh.z && c < sh.z + sh.w;
                v[u] = ldx64(x + (in[u] ? c : 0));
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (in[u]) acc += v[u];
        }
    }
    return acc;
}

// Sum over the aligned group of `lanes` lanes (a power of two).
__device__ __forceinline__ double group_sum(double v, int lanes)
{
    for (int o = lanes >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Short rows: kBlock >> LG rows a CTA.
template <bool SIGNED, int LG>
__global__ void __launch_bounds__(kBlock, kF64Blocks)
    f64_rows_kernel(DevPlan p, const __grid_constant__ typename DiagsOf<SIGNED>::type q, int ahead,
                    const double *__restrict__ x, double *__restrict__ y)
{
    constexpr int G = 1 << LG, R = kBlock >> LG, W = LG ? 4 : 3;
    allow_next_grid();
    const int row0 = blockIdx.x * R, group = threadIdx.x >> LG, lane = threadIdx.x & (G - 1);
    const bool ok = group < p.M - row0;
    const int r = row0 + group;
    // one lane a row: most words are near the row, so the CTA's x goes to L2
    // while its row pointers and words are on the way (mesh 29.3 -> 27.8 us);
    // with lane groups the rows are few and their words far: 35.9 -> 37.5 on
    // the banded 700,001
    if (LG == 0 && threadIdx.x == 0) prefetch_x_window(x, p.N, row0, R);
    if (threadIdx.x == 0 && (long)row0 + (long)ahead * R < p.M) {
        const int ra = row0 + ahead * R, rb = ra + min(R, p.M - ra);
        const int za = __ldg(p.rowptr + ra), zb = __ldg(p.rowptr + rb);
        prefetch_rows_ahead(p, ra, rb, za, words_upto(za, zb, kAheadWords));
    }
    int j = words_from(ok ? __ldg(p.rowptr + r) : 0, lane);
    const int e = ok ? __ldg(p.rowptr + r + 1) : 0;
    int c[W];
    load_words(p, j, e, G, c);
    wait_prior64(x, y);
    double acc = 0.0;
    if constexpr (SIGNED) {
        if (ok) acc = diag_terms64(p, q, x, r, lane, G);
    }
    add_words<SIGNED>(x, j, e, G, c, acc);
    while (words_left(j, e) > W * G) {
        j += W * G;
        load_words(p, j, e, G, c);
        add_words<SIGNED>(x, j, e, G, c, acc);
    }
    acc = group_sum(acc, G);
    if (ok && lane == 0) y[r] = acc;
}

// A lane's share of the words [b, e): every by-th from word b + skipped on.
template <bool SIGNED>
__device__ __forceinline__ void sum_words64(const DevPlan &p, const double *__restrict__ x, int b, int e, int skipped,
                                            int by, double &acc)
{
    each_step(b, e, skipped, 4 * by, [&](int j, int) {
        int c[4];
        load_words(p, j, e, by, c);
        add_words<SIGNED>(x, j, e, by, c, acc);
    });
}

// Any plan: a CTA per tile.
template <bool SIGNED>
__global__ void __launch_bounds__(kBlock, kF64Blocks)
    f64_tiles_kernel(DevPlan p, const __grid_constant__ typename DiagsOf<SIGNED>::type q,
                     const double *__restrict__ x, double *__restrict__ y)
{
    __shared__ double red[kBlock / 32];
    allow_next_grid();
    const Tile t = p.tiles[blockIdx.x];
    const int nr = tile_nrows(t), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    wait_prior64(x, y);
    if (nr == 1 && t.nnz > kLongTile) {
        double acc = 0.0;
        if constexpr (SIGNED) {
            acc = diag_terms64(p, q, x, t.row0, threadIdx.x, kBlock);
        }
        sum_words64<SIGNED>(p, x, t.nz0, t.nz0 + t.nnz, threadIdx.x, kBlock, acc);
        acc = group_sum(acc, 32);
        if (lane == 0) red[warp] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int i = 1; i < kBlock / 32; ++i) acc += red[i];
            y[t.row0] = acc;
        }
        return;
    }
    int lg = 0;                   // lanes per row: about kLaneWords words each
    while (lg < 5 && t.nnz > (long)nr * (kLaneWords << lg)) ++lg;
    const int G = 1 << lg, gl = lane & (G - 1);
    for (int base = 0; base < nr; base += kBlock >> lg) {
        const int rl = base + (threadIdx.x >> lg), r = t.row0 + rl;
        const bool ok = rl < nr;
        const int b = ok ? __ldg(p.rowptr + r) : 0, e = ok ? __ldg(p.rowptr + r + 1) : 0;
        const bool own = e - b <= kLaneMost << lg;
        double acc = 0.0;
        if constexpr (SIGNED) {
            if (ok && own) acc = diag_terms64(p, q, x, r, gl, G);
        }
        if (own) sum_words64<SIGNED>(p, x, b, e, gl, G, acc);
        acc = group_sum(acc, G);
        if (ok && own && gl == 0) y[r] = acc;
        for (unsigned mid = __ballot_sync(0xffffffffu, !own && gl == 0); mid; mid &= mid - 1) {
            const int src = __ffs(mid) - 1;       // a row for the whole warp
            const int mr = __shfl_sync(0xffffffffu, r, src);
            const int mb = __shfl_sync(0xffffffffu, b, src), me = __shfl_sync(0xffffffffu, e, src);
            double a = 0.0;
            if constexpr (SIGNED) {
                a = diag_terms64(p, q, x, mr, lane, 32);
            }
            sum_words64<SIGNED>(p, x, mb, me, lane, 32, a);
            a = group_sum(a, 32);
            if (lane == 0) y[mr] = a;
        }
    }
}

template <bool SIGNED>
tc_status launch_f64(const DevPlan &dp, const PlanDiags &dg, int64_t nnz_csr, int max_row, const double *x, double *y,
                     cudaStream_t s)
{
    typename DiagsOf<SIGNED>::type q;
    if constexpr (SIGNED) q = dg;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kBlock);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = dp.pdl ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int ahead = dp.prefetch ? kF64Blocks * num_sms() : 1 << 30;
    auto grid = [&](int lg) { return dim3((unsigned)(((long)dp.M + (kBlock >> lg) - 1) / (kBlock >> lg))); };
    auto full = [&](int lg) { return kF64Blocks * (kBlock >> lg) * num_sms(); };    // rows of a wave
    if (max_row > kShortRow) {
        cfg.gridDim = dim3(dp.ntiles);
        TC_CUDA(cudaLaunchKernelEx(&cfg, f64_tiles_kernel<SIGNED>, dp, q, x, y));
    } else if (nnz_csr <= 8LL * dp.M) {
        // a thread a row while a warp's words of consecutive rows share lines;
        // above, more lanes the longer the rows (banded matrices, us at 1 / 2 /
        // 4 / 8 lanes: 2,000,000 x 9 43.5 / 42.2 / 48.8 / 77.2, 600,000 x 17
        // 14.8 / 13.7 / 16.4 / 20.8, 1,003,602 x 19 42.3 / 37.9 / 36.6 / 43.6,
        // 831,425 x 30 61.2 / 50.2 / 45.1 / 46.0, 363,335 x 32 62.5 / 32.4 /
        // 21.3 / 18.3), and more of them where these would not fill the GPU
        // (60,000 x 9 4.4 / 4.0 / 2.6 / 3.5, 31,935 x 18 4.0 at 4 and 2.6 at 8)
        cfg.gridDim = grid(0);
        TC_CUDA(cudaLaunchKernelEx(&cfg, f64_rows_kernel<SIGNED, 0>, dp, q, ahead, x, y));
    } else if (nnz_csr <= 17LL * dp.M && dp.M >= full(1)) {
        cfg.gridDim = grid(1);
        TC_CUDA(cudaLaunchKernelEx(&cfg, f64_rows_kernel<SIGNED, 1>, dp, q, ahead, x, y));
    } else if (nnz_csr <= 16LL * dp.M || (nnz_csr <= 28LL * dp.M && dp.M >= full(2))) {
        cfg.gridDim = grid(2);
        TC_CUDA(cudaLaunchKernelEx(&cfg, f64_rows_kernel<SIGNED, 2>, dp, q, ahead, x, y));
    } else {
        cfg.gridDim = grid(3);
        TC_CUDA(cudaLaunchKernelEx(&cfg, f64_rows_kernel<SIGNED, 3>, dp, q, ahead, x, y));
    }
    return TC_OK;
}

}  // namespace
}  // namespace tc

tc_status tc_spmv_f64(const tc_plan *p, const double *d_x, double *d_y, void *stream)
{
    using namespace tc;
    if (!p || (!d_x && p->N) || (!d_y && p->M)) return fail(TC_ERR_INVALID, "tc_spmv_f64: null argument");
    const DevPlan dp = p->dev_plan();
    if (dp.M == 0 || dp.ntiles == 0) return TC_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (dp.N == 0) {      // no terms, and no x for the unconditional loads
        TC_CUDA(cudaMemsetAsync(d_y, 0, sizeof(double) * (size_t)dp.M, s));
        return TC_OK;
    }
    return dp.hybrid ? launch_f64<true>(dp, p->diags, p->nnz_csr, p->max_row, d_x, d_y, s)
                     : launch_f64<false>(dp, p->diags, p->nnz_csr, p->max_row, d_x, d_y, s);
}
