// tc_spmm.cu -- Y = A X for up to 64 right-hand sides over a resident plan.
//
// No counterpart in the reference (one vector per taichi_SpMV call,
// TaiChi.cu:1331-1456).  Per row and right-hand side the terms are added in
// one fixed order: the row's CSR words in stored order (holes subtract,
// left-overs add), then its dense-diagonal terms, shapes and offsets in
// order.  In plans with a row of more than kSpmmMidRow words, such rows are
// summed in parts by a warp or a CTA.
//
// What bounds it: bytes at many right-hand sides (Y written, the X rows that
// occur read), instructions at few (a word's load, address and sign against
// one vector of columns).  So a row has only as many lanes as its columns
// need at four a lane, and what a lane does per word is shared by four
// columns.  A warp per four rows with two columns a lane, which this
// replaces, left lanes idle below 64 columns and walked the shapes per row.
// Measured per multiply (us, before -> now):
//   R-MAT scale 22, k = 64 (plain, 0.7 words a row)     479 -> 267
//   9-point mesh 1200^2, k = 8 (hybrid, 6 words a row)  505 -> 41
//   9-point mesh 800^2, k = 13 (no vector loads)        231 -> 49
//   banded 300,000 x 22, k = 32                         181 -> 55
//   15 diagonals of 400,000 rows with holes, k = 24     185 -> 49
//   power-law R-MAT scale 18, k = 16                   5800 -> 112

#include <cuda_runtime.h>

#include <algorithm>

#include "tc_internal.h"
#include "tc_tile.cuh"

namespace tc {
namespace {

// A row belongs to a group of 2^lg lanes; a lane holds V of its k columns:
// columns [V l, V l + V) moved as one vector (VEC: k, ldx, ldy multiples of V
// and X, Y aligned to it), or columns l + 2^lg i, i < V, moved singly.  A lane
// without columns (k not 2^lg V) loads column 0 and stores nothing, so no
// branch surrounds the loads.
template <int V, bool VEC>
struct Lane {
    int at, step, left;      // first column, column step, columns from `at` on (<= 0: none)
    __device__ __forceinline__ Lane(int lane, int lg, int k)
        : at(VEC ? lane * V : lane), step(1 << lg), left(k - at)
    {
        if (left <= 0) at = 0;
    }
};

template <int V, bool VEC>
struct Cols {
    float a[V];
    __device__ __forceinline__ void load(const float *__restrict__ x, const Lane<V, VEC> &l)
    {
        if (VEC && V == 4) {
            const float4 f = __ldg(reinterpret_cast<const float4 *>(x));
            a[0] = f.x;
            a[1 % V] = f.y;
            a[2 % V] = f.z;
            a[3 % V] = f.w;
        } else if (VEC && V == 2) {
            const float2 f = __ldg(reinterpret_cast<const float2 *>(x));
            a[0] = f.x;
            a[V - 1] = f.y;
        } else {
#pragma unroll
            for (int i = 0; i < V; ++i) a[i] = __ldg(x + (i * l.step < l.left ? i * l.step : 0));
        }
    }
    __device__ __forceinline__ void store(float *__restrict__ y, const Lane<V, VEC> &l) const
    {
        if (l.left <= 0) return;
        if (VEC && V == 4) {
            __stcs(reinterpret_cast<float4 *>(y), make_float4(a[0], a[1 % V], a[2 % V], a[3 % V]));
        } else if (VEC && V == 2) {
            __stcs(reinterpret_cast<float2 *>(y), make_float2(a[0], a[V - 1]));
        } else {
#pragma unroll
            for (int i = 0; i < V; ++i)
                if (i * l.step < l.left) __stcs(y + i * l.step, a[i]);
        }
    }
    __device__ __forceinline__ void add(const Cols &o)
    {
#pragma unroll
        for (int i = 0; i < V; ++i) a[i] += o.a[i];
    }
    // + or - o: s is 1 or -1, so the product is exact
    __device__ __forceinline__ void add(const Cols &o, float s)
    {
#pragma unroll
        for (int i = 0; i < V; ++i) a[i] = fmaf(s, o.a[i], a[i]);
    }
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int i = 0; i < V; ++i) a[i] = 0.f;
    }
};

template <bool SIGNED>
__device__ __forceinline__ int word_col(int c) { return SIGNED ? c >> 1 : c; }

template <bool SIGNED, int V, bool VEC>
__device__ __forceinline__ void add_word(Cols<V, VEC> &acc, const Cols<V, VEC> &v, int c)
{
    if (SIGNED) acc.add(v, (c & 1) ? 1.f : -1.f);
    else acc.add(v);
}

// The dense-diagonal terms of row r, added to acc in offset order, four loads
// in flight; Xc: the lane's first column of X.
template <int V, bool VEC>
__device__ __forceinline__ void diag_cols(const DevPlan &p, const PlanDiags &q, const float *__restrict__ Xc, int ldx,
                                          const Lane<V, VEC> &l, int r, Cols<V, VEC> &acc)
{
    if (q.n > 0) {                // offsets from the launch parameters
        if (r < q.rows.x || r >= q.rows.y) return;
        if (r >= q.in.x && r < q.in.y) {                       // every offset reaches the row
#pragma unroll 1
            for (int i = 0; i < q.n; i += 4) {
                Cols<V, VEC> d[4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (i + u < q.n) d[u].load(Xc + (long)(r + q.col[i + u]) * ldx, l);
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (i + u < q.n) acc.add(d[u]);
            }
            return;
        }
#pragma unroll 1
        for (int i = 0; i < q.n; i += 4) {
            Cols<V, VEC> d[4];
            bool in[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                in[u] = i + u < q.n && q.has(i + u, r);
                if (in[u]) d[u].load(Xc + (long)(r + q.col[i + u]) * ldx, l);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (in[u]) acc.add(d[u]);
        }
        return;
    }
    if (r < p.row_start || r >= p.row_stop) return;
    for (int s = 0; s < p.dia_shapes; ++s) {
        const int4 sh = __ldg(p.shapes + s);
        if (r < sh.x || r >= sh.y) continue;
        const int2 dr = __ldg(p.shape_dias + s);
        for (int n = dr.x; n < dr.y; n += 4) {
            Cols<V, VEC> d[4];
            bool in[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = n + u < dr.y ? r - sh.x + sh.z + __ldg(p.offsets + n + u) : -1;
                in[u] = c >= sh.z && c < sh.z + sh.w;
                d[u].load(Xc + (long)(in[u] ? c : 0) * ldx, l);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (in[u]) acc.add(d[u]);
        }
    }
}

constexpr int kAheadWords = 1 << 14;   // most words of a later CTA prefetched into L2
constexpr int kSpmmMidRow = 64;        // longer rows are summed by a whole warp,
constexpr int kSpmmLongRow = 1024;     // and one-row tiles longer than this by the whole CTA
// Resident CTAs per SM the kernels are compiled for: 8 at one or two columns
// a lane or three words in flight, 6 at four of both; 5 for the run kernel
// (4 words in flight; 4 CTAs with 8 words: 262 us in place of 266 at R-MAT
// scale 22, k = 64, but spills with single loads).
constexpr int kRunBlocks = 5;
constexpr int spmm_blocks(int V, int W) { return V < 4 || W < 4 ? 8 : 6; }

__device__ __forceinline__ void prefetch_later_rows(const DevPlan &p, long r0, int rows)
{
    if (r0 >= p.M) return;
    const int ra = (int)r0, rb = ra + min(rows, p.M - ra);
    const int za = __ldg(p.rowptr + ra), zb = __ldg(p.rowptr + rb);
    prefetch_rows_ahead(p, ra, rb, za, words_upto(za, zb, kAheadWords));
}

// Adds to acc the terms of every by-th of the words [b, e) from word b +
// skipped on, W of them in flight together (a slot past the end loads X's row
// 0 and is not added).
template <bool SIGNED, int V, bool VEC, int W>
__device__ __forceinline__ void sum_words(const DevPlan &p, const float *__restrict__ Xc, int ldx,
                                          const Lane<V, VEC> &l, int b, int e, int skipped, int by,
                                          Cols<V, VEC> &acc)
{
    auto round = [&](auto j, int left) {
        int c[W];
        Cols<V, VEC> v[W];
#pragma unroll
        for (int w = 0; w < W; ++w) c[w] = w * by < left ? __ldg(p.cols + j + w * by) : 0;
#pragma unroll
        for (int w = 0; w < W; ++w) v[w].load(Xc + (long)word_col<SIGNED>(c[w]) * ldx, l);
#pragma unroll
        for (int w = 0; w < W; ++w)
            if (w * by < left) add_word<SIGNED>(acc, v[w], c[w]);
    };
    // either walk stays inside the row; each is the faster one in its place
    // (meshes 64^2 to 256^2, k = 8, vectors: 4.2 to 5.9 us with Words, 4.4 to
    // 6.1 with each_step; power-law R-MAT scale 20, k = 3, single loads: 175
    // and 171)
    if constexpr (VEC) {
        for (Words a(b, e, skipped); a.left > 0; a.skip(W * by)) round(a.at, a.left);
    } else {
        each_step(b, e, skipped, W * by, round);
    }
}

// Rows [row0, row0 + nrow) of a CTA, nrow <= kBlock >> lg: one row per group
// of 2^lg lanes.  MID: a row of more than kSpmmMidRow words is left to its
// whole warp, whose groups sum every (32 >> lg)-th word each; a butterfly
// joins the parts.
template <bool SIGNED, int V, bool VEC, int W, bool MID>
__device__ __forceinline__ void spmm_rows(const DevPlan &p, const typename DiagsOf<SIGNED>::type &q,
                                          const float *__restrict__ Xc, int ldx, const Lane<V, VEC> &l, int lg,
                                           int row0, int nrow,
                                          float *__restrict__ Yc, int ldy)
{
    const int group = threadIdx.x >> lg, r = row0 + group;
    const int b = group < nrow ? __ldg(p.rowptr + r) : 0;
    const int e = group < nrow ? __ldg(p.rowptr + r + 1) : 0;
    if (group < nrow && (!MID || e - b <= kSpmmMidRow)) {
        Cols<V, VEC> acc;
        acc.zero();
        sum_words<SIGNED, V, VEC, W>(p, Xc, ldx, l, b, e, 0, 1, acc);
        if constexpr (SIGNED) diag_cols(p, q, Xc, ldx, l, r, acc);
        acc.store(Yc + (long)r * ldy, l);
    }
    if (!MID) return;
    const int gw = 32 >> lg, wg = (threadIdx.x & 31) >> lg;
    const bool lead = (threadIdx.x & ((1 << lg) - 1)) == 0;
    unsigned mid = __ballot_sync(0xffffffffu, lead && e - b > kSpmmMidRow);
    for (; mid; mid &= mid - 1) {
        const int src = __ffs(mid) - 1;
        const int mr = __shfl_sync(0xffffffffu, r, src), rb = __shfl_sync(0xffffffffu, b, src);
        const int re = __shfl_sync(0xffffffffu, e, src);
        Cols<V, VEC> acc;
        acc.zero();
        sum_words<SIGNED, V, VEC, W>(p, Xc, ldx, l, rb, re, wg, gw, acc);
#pragma unroll
        for (int u = 0; u < V; ++u)
            for (int o = 1 << lg; o < 32; o <<= 1) acc.a[u] += __shfl_xor_sync(0xffffffffu, acc.a[u], o);
        if (wg == 0) {
            if constexpr (SIGNED) diag_cols(p, q, Xc, ldx, l, mr, acc);
            acc.store(Yc + (long)mr * ldy, l);
        }
    }
}

// Plans whose longest row has at most kSpmmMidRow words: kBlock >> lg rows a
// CTA.
template <bool SIGNED, int V, bool VEC, int W>
__global__ void __launch_bounds__(kBlock, spmm_blocks(V, W))
    spmm_rows_kernel(DevPlan p, const __grid_constant__ typename DiagsOf<SIGNED>::type q,
                     const float *__restrict__ X, int ldx, int k, int lg, int ahead,
                     float *__restrict__ Y, int ldy)
{
    const int groups = kBlock >> lg, row0 = blockIdx.x * groups;
    const Lane<V, VEC> l(threadIdx.x & ((1 << lg) - 1), lg, k);
    if (threadIdx.x == 0) prefetch_later_rows(p, (long)row0 + (long)ahead * groups, groups);
    spmm_rows<SIGNED, V, VEC, W, false>(p, q, X + l.at, ldx, l, lg, row0, min(groups, p.M - row0), Y + l.at, ldy);
}

// Other plans: a CTA per tile of the plan's tile list, whose words are
// bounded, so that rows of many words do not gather in a few CTAs (they are
// neighbours in a power-law graph).  Tiles of short rows hold up to 4,096 of
// them, kBlock >> lg a pass; SPLIT deals the passes out to gridDim.y CTAs.  A
// row that is a tile of its own is summed by the whole CTA: each group adds
// every groups-th word, the first group joins the parts in group order.
template <bool SIGNED, int V, bool VEC, int W, bool SPLIT>
__global__ void __launch_bounds__(kBlock, spmm_blocks(V, W))
    spmm_tiles_kernel(DevPlan p, const __grid_constant__ typename DiagsOf<SIGNED>::type q,
                      const float *__restrict__ X, int ldx, int k, int lg, float *__restrict__ Y,
                      int ldy)
{
    __shared__ float part[kBlock * V];
    const int groups = kBlock >> lg, group = threadIdx.x >> lg;
    const Lane<V, VEC> l(threadIdx.x & ((1 << lg) - 1), lg, k);
    const float *__restrict__ Xc = X + l.at;
    const Tile t = p.tiles[blockIdx.x];
    const int nr = tile_nrows(t);
    if (nr > 1 || t.nnz <= kSpmmLongRow) {
        for (int i = SPLIT ? blockIdx.y * groups : 0; i < nr; i += SPLIT ? gridDim.y * groups : groups)
            spmm_rows<SIGNED, V, VEC, W, true>(p, q, Xc, ldx, l, lg, t.row0 + i, min(groups, nr - i), Y + l.at, ldy);
        return;
    }
    if (SPLIT && blockIdx.y) return;
    Cols<V, VEC> acc;
    acc.zero();
    sum_words<SIGNED, V, VEC, W>(p, Xc, ldx, l, t.nz0, t.nz0 + t.nnz, group, groups, acc);
#pragma unroll
    for (int u = 0; u < V; ++u) part[u * kBlock + threadIdx.x] = acc.a[u];
    __syncthreads();
    if (group == 0) {
        for (int g = 1; g < groups; ++g)
#pragma unroll
            for (int u = 0; u < V; ++u) acc.a[u] += part[u * kBlock + (g << lg) + threadIdx.x];
        if constexpr (SIGNED) diag_cols(p, q, Xc, ldx, l, t.row0, acc);
        acc.store(Y + (long)t.row0 * ldy + l.at, l);
    }
}

// Plain plans of few words a row: a warp takes 32 consecutive rows,
// its groups 2^lg consecutive ones each (lg >= 3), and a group walks its
// rows' words as one run, U words' X rows in flight, closing a row (one
// store) whenever the run passes its end.  So the loads in flight do not
// depend on how the words fall into rows (one row per group with two words
// in flight measured 460 us in place of 267 at R-MAT scale 22, k = 64: 240
// instructions per warp for 4 rows, and half the loads past short rows).
template <int V, bool VEC, int U>
__global__ void __launch_bounds__(kBlock, kRunBlocks)
    spmm_run_kernel(DevPlan p, const float *__restrict__ X, int ldx, int k, int lg, int ahead,
                    float *__restrict__ Y, int ldy)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gl = lane & ((1 << lg) - 1), first = lane - gl;     // lane of the group, its first lane
    const Lane<V, VEC> l(gl, lg, k);
    const float *__restrict__ Xc = X + l.at;
    if (threadIdx.x == 0) prefetch_later_rows(p, ((long)blockIdx.x + ahead) * kBlock, kBlock);
    const long start = (long)blockIdx.x * kBlock + warp * 32;
    if (start >= p.M) return;                                     // the whole warp
    const int r0 = (int)start;
    // lane i: the end of row r0 + i; the group's rows are r0 + first + [0, 2^lg)
    const int end = __ldg(p.rowptr + r0 + min(lane + 1, p.M - r0));
    const int z = __shfl_up_sync(0xffffffffu, end, 1);
    const int begin = lane ? z : __ldg(p.rowptr + r0);
    const unsigned mask = (lg == 5 ? 0xffffffffu : ((1u << (1 << lg)) - 1u)) << first;
    // positions of words: unsigned, as a step past the run's end may leave 2^31 - 1 behind
    const unsigned jb = __shfl_sync(mask, begin, first), je = __shfl_sync(mask, end, first + (1 << lg) - 1);
    int row = 0;                                                  // current row of the group
    unsigned re = __shfl_sync(mask, end, first);
    const int nrow = min(1 << lg, p.M - r0 - first);              // <= 0: no rows
    float *yr = Y + (long)(r0 + first) * ldy + l.at;
    Cols<V, VEC> acc;
    acc.zero();
    for (unsigned j0 = jb; j0 < je; j0 += 1 << lg) {
        // the next 2^lg words, one per lane of the group
        const int word = j0 + gl < je ? __ldg(p.cols + j0 + gl) : 0;
        const int n = min(1 << lg, (int)(je - j0));
        for (int t = 0; t < n; t += U) {
            int c[U];
            Cols<V, VEC> v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) c[u] = __shfl_sync(mask, word, first + t + u);
#pragma unroll
            for (int u = 0; u < U; ++u) v[u].load(Xc + (long)c[u] * ldx, l);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (t + u >= n) break;
                while (j0 + t + u >= re) {                        // the row before this word is done
                    acc.store(yr, l);
                    acc.zero();
                    yr += ldy;
                    ++row;
                    re = __shfl_sync(mask, end, first + row);
                }
                acc.add(v[u]);
            }
        }
    }
    for (; row < nrow; ++row) {                                   // the last row, and empty rows after it
        acc.store(yr, l);
        acc.zero();
        yr += ldy;
    }
}

template <bool SIGNED, int V, bool VEC>
tc_status launch(const DevPlan &dp, const PlanDiags &dg, int64_t nnz_csr, int max_row, const float *X, int ldx, int k,
                 float *Y, int ldy, cudaStream_t s)
{
    int lg = 0;
    while ((V << lg) < k) ++lg;
    typename DiagsOf<SIGNED>::type q;
    if constexpr (SIGNED) q = dg;
    // CTAs resident at once, whose operands later CTAs' prefetches run ahead by
    auto ahead = [&](int blocks) { return dp.prefetch ? blocks * num_sms() : 1 << 30; };
    // Runs: plain rows of at most two words on average, in groups of 8 lanes
    // or more (a run of 2^lg rows; smaller groups diverge more than they
    // save), and rows for two CTAs per SM, as a warp's 32 rows are a chain (k =
    // 64, R-MAT, us as runs and row by row: 8,192 rows 4.5 and 2.5, 32,768 5.0
    // and 3.8, 65,536 5.8 and 5.9, 131,072 8.2 and 9.9).  Longer rows keep a
    // group's loads in flight by themselves.
    if (!SIGNED && lg >= 3 && max_row <= kSpmmMidRow && nnz_csr <= 2LL * dp.M && dp.M >= 2 * kBlock * num_sms()) {
        const unsigned grid = (unsigned)((dp.M + (long)kBlock - 1) / kBlock);
        spmm_run_kernel<V, VEC, 4><<<grid, kBlock, 0, s>>>(dp, X, ldx, k, lg, ahead(kRunBlocks), Y, ldy);
    } else if (max_row > kSpmmMidRow) {
        // Two passes a CTA where the tiles hold more rows than stream tiles do
        // and more than four passes, on average (k = 64, one row of 65 words,
        // us with a CTA per tile and now: 65,536 rows of 0.6 words 33.0 and
        // 8.9, 1,048,576 190 and 119, 200,000 of one word and three diagonals
        // 78 and 58).  (Row by row whenever no row takes a CTA: the same for
        // these, but 400 neighbouring rows of 400 words 5 -> 76 at k = 2.)
        const int rows = dp.M / dp.ntiles, pass = kBlock >> lg;
        if (rows > std::max(kStreamRows, 4 * pass)) {
            const dim3 grid(dp.ntiles, (rows + 2 * pass - 1) / (2 * pass));
            spmm_tiles_kernel<SIGNED, V, VEC, 4, true><<<grid, kBlock, 0, s>>>(dp, q, X, ldx, k, lg, Y, ldy);
        } else {
            spmm_tiles_kernel<SIGNED, V, VEC, 4, false><<<dp.ntiles, kBlock, 0, s>>>(dp, q, X, ldx, k, lg, Y, ldy);
        }
    } else {
        // Rows of at most 8 words on average: three words in flight and two
        // more CTAs per SM (mesh 1200^2, k = 8: 41 us in place of 47);
        // longer ones four (power-law rows lose 15 % with three).
        constexpr int W = V == 4 ? 3 : 4;
        const int rows = kBlock >> lg;
        const unsigned grid = (unsigned)((dp.M + (long)rows - 1) / rows);
        if (nnz_csr <= 8LL * dp.M)
            spmm_rows_kernel<SIGNED, V, VEC, W><<<grid, kBlock, 0, s>>>(
                dp, q, X, ldx, k, lg, ahead(spmm_blocks(V, W)), Y, ldy);
        else
            spmm_rows_kernel<SIGNED, V, VEC, 4><<<grid, kBlock, 0, s>>>(
                dp, q, X, ldx, k, lg, ahead(spmm_blocks(V, 4)), Y, ldy);
    }
    TC_CUDA(cudaGetLastError());
    return TC_OK;
}

template <bool SIGNED>
tc_status launch_cols(const DevPlan &dp, const PlanDiags &dg, int64_t nnz_csr, int max_row, const float *X, int ldx,
                      int k, float *Y, int ldy, cudaStream_t s)
{
    const uintptr_t at = reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Y);
    const int all = ldx | ldy | k;
    // vectors of four or two columns where k, both leading dimensions and both
    // addresses allow them, else four single loads a lane 2^lg columns apart
    // (mesh 800^2, k = 13: 49 us in place of 100 with one column a lane)
    if (!(all & 3) && !(at & 15)) return launch<SIGNED, 4, true>(dp, dg, nnz_csr, max_row, X, ldx, k, Y, ldy, s);
    if (!(all & 1) && !(at & 7)) return launch<SIGNED, 2, true>(dp, dg, nnz_csr, max_row, X, ldx, k, Y, ldy, s);
    if (k <= 2) return launch<SIGNED, 1, false>(dp, dg, nnz_csr, max_row, X, ldx, k, Y, ldy, s);
    return launch<SIGNED, 4, false>(dp, dg, nnz_csr, max_row, X, ldx, k, Y, ldy, s);
}

}  // namespace

tc_status launch_spmm(const DevPlan &dp, const PlanDiags &dg, int64_t nnz_csr, int max_row, const float *X, int ldx,
                      int k, float *Y, int ldy, cudaStream_t s)
{
    if (dp.M == 0) return TC_OK;
    if (dp.N == 0) {      // no terms, and no X for the lanes' unconditional loads
        TC_CUDA(cudaMemset2DAsync(Y, sizeof(float) * (size_t)ldy, 0, sizeof(float) * (size_t)k, dp.M, s));
        return TC_OK;
    }
    return dp.hybrid ? launch_cols<true>(dp, dg, nnz_csr, max_row, X, ldx, k, Y, ldy, s)
                     : launch_cols<false>(dp, dg, nnz_csr, max_row, X, ldx, k, Y, ldy, s);
}

}  // namespace tc
