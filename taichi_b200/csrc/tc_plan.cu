// tc_plan.cu -- from a formatted matrix to a resident plan: the device
// format, the tile list and what the launches need to know about the rows.
//
// Replaces the upload part of taichi_SpMV (TaiChi.cu:1357-1385).  The format
// comes from host arrays or, after a partition, from device arrays; either
// way the row statistics and the tile list are computed on the GPU, so a
// partitioned matrix never crosses the host link.  What bounds a build is then
// the copies of the format (read and written once) and a few round trips of
// counts to the host.  Measured on the 9-point mesh 2048^2 (25.7 M words): 1 ms
// from device arrays in place of 85 ms for the copy to the host, the host's
// passes over the words and rows, and the copy back.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "tc_internal.h"
#include "tc_scan.cuh"

namespace tc {

int wide_tile_rows(int M, const tc_params &prm, int sms)
{
    if ((prm.flags & TC_FLAG_WIDE_FIXED) || sms <= 0) return kDirectWideRows;
    // two tiles per SM: every SM holds two CTAs of the same size
    const long per = ((long)M + 2L * sms - 1) / (2L * sms);
    return (int)std::min<long>(kDirectWideRows, std::max<long>(kDirectRows, (per + 3) & ~3L));
}

namespace {

// Rows are planned in strips of kStripRows, a CTA each; a tile never crosses a
// strip.  The last tile of a strip is what is left of it, so short strips make
// small tiles: strips of 2,048 rows gave banded plans of 17 to 30 words a row,
// whose tiles hold 136 to 240 rows, 5 to 10 % more tiles (220,000 rows of 24
// words: 1,397 in place of 1,298 and 24.9 us in place of 22.4).
constexpr int kStripRows = 16384;
constexpr int kMixedSpan = 2048;
constexpr int kPlanBlock = 1024;

struct RowStats {
    int max_row;                     // CSR words of the longest row
    int minus;                       // a word without the addition bit exists
    int hist[kStreamRowMax + 1];     // sampled rows by length
    int whist[kStreamRowMax + 1];    // groups of 32 rows by their longest row (at most kStreamRowMax words)
};

__global__ void row_stats(const int *__restrict__ rowptr, int M, int step, RowStats *__restrict__ st)
{
    __shared__ int hist[kStreamRowMax + 1], whist[kStreamRowMax + 1];
    for (int i = threadIdx.x; i <= kStreamRowMax; i += blockDim.x) hist[i] = whist[i] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    int most = 0;
    for (long r0 = (long)blockIdx.x * blockDim.x + threadIdx.x - lane; r0 < M; r0 += (long)gridDim.x * blockDim.x) {
        const long r = r0 + lane;                    // whole warps: 32 consecutive rows
        const int n = r < M ? __ldg(rowptr + r + 1) - __ldg(rowptr + r) : 0;
        if (r < M && n <= kStreamRowMax && r % step == 0) atomicAdd(hist + n, 1);
        const int longest = __reduce_max_sync(0xffffffffu, n);
        most = max(most, longest);
        if (lane == 0 && longest <= kStreamRowMax) atomicAdd(whist + longest, 1);
    }
    if (lane == 0) atomicMax(&st->max_row, most);
    __syncthreads();
    for (int i = threadIdx.x; i <= kStreamRowMax; i += blockDim.x) {
        if (hist[i]) atomicAdd(st->hist + i, hist[i]);
        if (whist[i]) atomicAdd(st->whist + i, whist[i]);
    }
}

__global__ void word_signs(const int *__restrict__ cols, long nnz, RowStats *__restrict__ st)
{
    int all = 1;
    for (long j = (long)blockIdx.x * blockDim.x + threadIdx.x; j < nnz; j += (long)gridDim.x * blockDim.x)
        all &= __ldg(cols + j);
    if (!__all_sync(0xffffffffu, all & 1) && (threadIdx.x & 31) == 0) st->minus = 1;
}

// The planner's parameters (see tc_params).
struct TilePrm {
    int mode, rows_cap, tile_nnz, long_len, spread, max_lanes, strided, no_direct;
};

// What the tiles of a plan come to, summed over its strips.
struct TileCounts {
    int vector, lng, stream, max_rows, max_nnz;   // max_*: tiles staged in shared memory
};

// Lanes per row from the mean row length of a run of rows: one lane per row
// until rows average more than 16 entries, then the smallest power of two
// giving each lane about 8 entries, capped at max_lanes.  (The CSR words come
// from shared memory, so a thread walking its own row costs no coalescing.)
__device__ __forceinline__ int lanes_for(double mean, int max_lanes)
{
    if (mean <= 16.0) return 1;
    int l = 1;
    while (l < max_lanes && 8.0 * l < mean) l <<= 1;
    return l;
}

// A strip in shared memory: its row pointers, and a bit per row for the rows
// of more than kStreamRowMax words and for those that get a CTA each.
struct Strip {
    const int *rp;
    const unsigned *mid, *lng;
    int n;                          // rows
    bool any_mid, any_long;         // in the whole matrix
};

// The first i in [0, limit) for which row r + i is marked, else limit; rows
// [r, r + limit) inside the strip.
__device__ __forceinline__ int first_marked(const unsigned *mask, int r, int limit)
{
    for (int w = r >> 5; 32 * w < r + limit; ++w) {
        unsigned v = mask[w];
        if (w == r >> 5) v &= ~0u << (r & 31);
        if (v) return min(limit, 32 * w + __ffs(v) - 1 - r);
    }
    return limit;
}

// The tile that starts at row r of a strip (tile_mode 2): its rows, and its
// kind from bit kTileRowBits on.
constexpr int kTileRowBits = 12;
static_assert(kMergeRows < 1 << kTileRowBits && TILE_MIXED < 1 << (16 - kTileRowBits), "packed in 16 bits");
__device__ __forceinline__ int tile_at(const Strip &s, const TilePrm &q, int r)
{
    if (s.any_long && (s.lng[r >> 5] >> (r & 31) & 1u)) return 1 | TILE_LONG << kTileRowBits;
    // stream tile: rows up to the row and entry caps.  A run that starts on a
    // multiple of 4 rows and holds many rows runs 4 consecutive rows per
    // thread: read directly from global memory when they average at most one
    // entry (TILE_DIRECT4), through shared memory when at most two
    // (TILE_STREAM4); otherwise one row per thread (TILE_STREAM; TILE_MIXED
    // when it holds a row of more than kStreamRowMax entries)
    const bool a4 = (r & 3) == 0 && !q.strided;
    const int cap_nnz = max(1, min(2 * min(q.tile_nnz, 1 << 24), q.spread));
    const int z = s.rp[r];
    // plans with long rows end tiles at every kMixedSpan rows as well: the
    // smaller tiles even out what the long rows make uneven (power-law R-MAT
    // scale 20 66.4 us, 67.9 without; in double precision at scale 16 12.0 and
    // 13.2)
    const int end = s.any_mid ? min(s.n, (r & ~(kMixedSpan - 1)) + kMixedSpan) : s.n;
    int m = 0;                    // most rows of at most cap_nnz words together
    for (int hi = min(min(q.rows_cap, a4 ? kDirectRows : kStreamRows), end - r); m < hi;) {
        const int half = (m + hi + 1) >> 1;
        if (s.rp[r + half] - z <= cap_nnz) m = half;
        else hi = half - 1;
    }
    if (s.any_long) m = first_marked(s.lng, r, m);
    if (m == 0) m = 1;            // a single row longer than cap_nnz
    const int small = s.any_mid ? first_marked(s.mid, r, m) : m;
    if (small >= 2 * kBlock) m = small;       // direct and four-row tiles hold short rows only
    const int ent = s.rp[r + m] - z;
    const bool direct = a4 && small >= 2 * kBlock && ent <= m && !q.no_direct;
    const bool four = !direct && a4 && small >= 2 * kBlock && ent <= 2 * m;
    if (!direct) m = min(m, four ? kStream4Rows : kStreamRows);
    if (r + m < end) {            // end on a multiple of 256 rows (whole row sweeps), else of 4
        const int cut = (r + m) & ~255;
        if (cut - r >= 256) m = cut - r;
        else if (m > 4) m -= (r + m) & 3;
    }
    return m | (direct ? TILE_DIRECT4 : four ? TILE_STREAM4 : small < m ? TILE_MIXED : TILE_STREAM) << kTileRowBits;
}

// The tile that starts at row r of a strip in tile_mode 0 or 1.
__device__ __forceinline__ int tile_at_lanes(const Strip &s, const TilePrm &q, int r)
{
    if (s.any_long && (s.lng[r >> 5] >> (r & 31) & 1u)) return 1 | TILE_LONG << kTileRowBits;
    // candidate run: up to 1024 rows (merge tiles: tile_rows), stopping
    // before a long row
    int m = min(q.mode == 0 ? min(q.rows_cap, kMergeRows) : 1024, s.n - r);
    if (s.any_long) m = first_marked(s.lng, r, m);
    const int z = s.rp[r];
    if (q.mode == 0) {            // merge tile: rows + entries split evenly
        while (m > 1 && s.rp[r + m] - z > kStageNnz) m = (m + 1) / 2;
        return m | TILE_MERGE << kTileRowBits;
    }
    int lanes = lanes_for((double)(s.rp[r + m] - z) / m, q.max_lanes);
    m = min(min(m, kBlock / lanes * 4), q.rows_cap);
    while (m > 1 && s.rp[r + m] - z > kStageNnz) m = (m + 1) / 2;   // fits a stage
    lanes = lanes_for((double)(s.rp[r + m] - z) / m, q.max_lanes);
    return m | (31 - __clz(lanes)) << kTileRowBits;
}

// Rows between the starts whose tiles are found ahead of the walk: tiles of
// stream plans start on multiples of 4 rows, but for a few.
constexpr int kAheadStep = 4;

size_t strip_smem(int rows)
{
    const size_t words = ((size_t)rows + 31) / 32;
    return sizeof(int) * ((size_t)rows + 1 + 2 * words) + sizeof(unsigned short) * (words * 32 / kAheadStep);
}

// The planner's parameters of a plan's own tiles and of those for batches
// (blockIdx.y).
struct PlanLists {
    TilePrm q[2];
};

// The tiles of one strip of one list: counted, and with WRITE written from
// tiles[first[strip]] on.  Which tile starts at a row depends on the rows
// alone, so the threads find the tile of every fourth row side by side, one
// thread follows the chain of starts (a shared-memory read a tile), and all
// write the tiles.  (A warp that looks through the rows tile by tile takes
// 20 us for such a strip.)
template <bool WRITE>
__global__ void __launch_bounds__(kPlanBlock)
    plan_strips(const int *__restrict__ rowptr, int M, const __grid_constant__ PlanLists lists,
                const RowStats *__restrict__ st, int *__restrict__ count, const int *__restrict__ first,
                Tile *__restrict__ tiles0, Tile *__restrict__ tiles1, TileCounts *__restrict__ sum)
{
    extern __shared__ int rp[];
    __shared__ int made_s;
    const TilePrm q = lists.q[blockIdx.y];
    const long row0 = (long)blockIdx.x * kStripRows;
    const int n = (int)min((long)kStripRows, (long)M - row0), words = (n + 31) >> 5;
    unsigned *const mid = reinterpret_cast<unsigned *>(rp + n + 1), *const lng = mid + words;
    unsigned short *const ahead = reinterpret_cast<unsigned short *>(lng + words);
#pragma unroll 4
    for (int i = threadIdx.x; i <= n; i += kPlanBlock) rp[i] = __ldg(rowptr + row0 + i);
    const Strip s{rp, mid, lng, n, st->max_row > kStreamRowMax, st->max_row > q.long_len};
    __syncthreads();
    if (s.any_mid || s.any_long) {
        for (int r = threadIdx.x; r < 32 * words; r += kPlanBlock) {        // whole warps
            const int len = r < n ? rp[r + 1] - rp[r] : 0;
            const unsigned m = __ballot_sync(0xffffffffu, len > kStreamRowMax);
            const unsigned l = __ballot_sync(0xffffffffu, len > q.long_len);
            if ((r & 31) == 0) {
                mid[r >> 5] = m;
                lng[r >> 5] = l;
            }
        }
        __syncthreads();
    }
    if (q.mode == 2) {
        for (int r = kAheadStep * threadIdx.x; r < n; r += kAheadStep * kPlanBlock)
            ahead[r / kAheadStep] = (unsigned short)tile_at(s, q, r);
        __syncthreads();
    }
    auto tile = [&](int r) {
        if (q.mode != 2) return tile_at_lanes(s, q, r);
        return r % kAheadStep ? tile_at(s, q, r) : (int)ahead[r / kAheadStep];
    };
    constexpr int kRows = (1 << kTileRowBits) - 1;
    const int at = (int)blockIdx.y * ((int)gridDim.x + 1) + (int)blockIdx.x;     // of the list's counts
    Tile *const out = WRITE ? (blockIdx.y ? tiles1 : tiles0) + first[at] : nullptr;
    if (threadIdx.x == 0) {
        TileCounts c{0, 0, 0, 1, 0};
        int made = 0;
        for (int r = 0; r < n; ++made) {
            const int t = tile(r), rows = t & kRows, kind = t >> kTileRowBits;
            if (WRITE) {
                out[made].row0 = r;
            } else {
                c.stream += kind == TILE_STREAM;
                c.lng += kind == TILE_LONG;
                c.vector += kind > TILE_L1 && kind <= TILE_L32;
                if (kind <= TILE_L32 || kind == TILE_MERGE) {
                    c.max_rows = max(c.max_rows, rows);
                    c.max_nnz = max(c.max_nnz, rp[r + rows] - rp[r]);
                }
            }
            r += rows;
        }
        made_s = made;
        if (!WRITE) {
            TileCounts *const total = sum + blockIdx.y;
            count[at] = made;
            if (c.vector) atomicAdd(&total->vector, c.vector);
            if (c.lng) atomicAdd(&total->lng, c.lng);
            if (c.stream) atomicAdd(&total->stream, c.stream);
            atomicMax(&total->max_rows, c.max_rows);
            atomicMax(&total->max_nnz, c.max_nnz);
        }
    }
    if (!WRITE) return;
    __syncthreads();
    for (int k = threadIdx.x; k < made_s; k += kPlanBlock) {
        const int r = out[k].row0, t = tile(r), rows = t & kRows;
        out[k] = Tile{(int)(row0 + r), rp[r], rp[r + rows] - rp[r], tile_word(rows, t >> kTileRowBits)};
    }
}

// Wide direct tiles: `rows` rows each, in row order.
__global__ void wide_tiles(const int *__restrict__ rowptr, int M, int rows, int ntiles, Tile *__restrict__ tiles)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ntiles) return;
    const int r = i * rows, n = min(rows, M - r), z = __ldg(rowptr + r);
    tiles[i] = Tile{r, z, __ldg(rowptr + r + n) - z, tile_word(n, TILE_DIRECT_WIDE)};
}

// Sets each tile's diagonal class (see kDiagGeneral / kDiagNone), a warp per
// tile: the multiply adds the dense-diagonal terms of a classed tile without
// searching the shapes per row, with the same terms in the same order.
__global__ void classify_tiles(Tile *__restrict__ tiles, int ntiles, const int4 *__restrict__ shapes,
                               const int2 *__restrict__ shape_dias, const int *__restrict__ offsets,
                               int dia_shapes, int row_start, int row_stop)
{
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= ntiles) return;
    const int r0 = tiles[i].row0, r1 = r0 + tile_nrows(tiles[i]);
    int dc = kDiagNone;
    if (r1 > row_start && r0 < row_stop) {
        int found = -1;
        bool two = false;                            // two shapes share rows of the tile
        for (int s = 0; s < dia_shapes && !two; ++s) {
            const int4 sh = shapes[s];
            if (r1 <= sh.x || r0 >= sh.y) continue;
            two = found >= 0;
            found = s;
        }
        if (two) dc = kDiagGeneral;
        else if (found >= 0) {
            const int4 sh = shapes[found];
            const int2 dr = shape_dias[found];
            bool in = r0 >= sh.x && r1 <= sh.y && r0 >= row_start && r1 <= row_stop && found + 1 < kDiagNone;
            for (int d = dr.x + lane; d < dr.y; d += 32)
                in = in && r0 - sh.x + offsets[d] >= 0 && r1 - 1 - sh.x + offsets[d] < sh.w;
            dc = __all_sync(0xffffffffu, in) ? found + 1 : kDiagGeneral;
        }
    }
    if (lane == 0) tiles[i].nrows_kind |= dc << kDiagShift;
}

size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

unsigned blocks_for(long n, int threads)
{
    return (unsigned)std::max(1L, std::min((n + threads - 1) / threads, 16L * num_sms()));
}

}  // namespace

tc_status plan_upload(tc_plan *p, const int *csrRow, const int *csrCol, int64_t nnz_csr, bool on_device,
                      cudaStream_t stream)
{
    const int M = p->M;
    const tc_params &prm = p->params;
    p->nnz_csr = nnz_csr;
    p->set_diags();
    // shape table {xStart, xStop, yStart, Msub} and offset ranges
    std::vector<int4> shapes(p->dia_shapes);
    std::vector<int2> sd(p->dia_shapes);
    for (int s = 0; s < p->dia_shapes; ++s) {
        shapes[s] = make_int4(p->h_xStart[s], p->h_xStop[s], p->h_yStart[s],
                              p->h_xStop[s] - p->h_xStart[s]);
        sd[s] = make_int2(p->h_nDiasPtr[s], p->h_nDiasPtr[s + 1]);
        if (sd[s].y <= sd[s].x) return fail(TC_ERR_FORMAT, "shape %d has no diagonals", s);
        for (int n = sd[s].x + 1; n < sd[s].y; ++n)
            if (p->h_offsets[n] <= p->h_offsets[n - 1])
                return fail(TC_ERR_FORMAT, "offsets of shape %d are not increasing", s);
    }

    // window plan: a second tile list for the window kernel (the batch and
    // served launches keep running `tiles`, with the same terms and order),
    // planned on the host
    std::vector<Tile> wtiles;
    p->nwtiles = 0;
    if (prm.flags & TC_FLAG_WINDOW) {
        std::vector<int> hr, hc;
        const int *wr = csrRow, *wc = csrCol;
        if (on_device) {
            hr.resize((size_t)M + 1);
            hc.resize((size_t)nnz_csr);
            TC_CUDA(cudaMemcpyAsync(hr.data(), csrRow, sizeof(int) * hr.size(), cudaMemcpyDeviceToHost, stream));
            if (nnz_csr)
                TC_CUDA(cudaMemcpyAsync(hc.data(), csrCol, sizeof(int) * hc.size(), cudaMemcpyDeviceToHost, stream));
            TC_CUDA(cudaStreamSynchronize(stream));
            wr = hr.data();
            wc = hc.data();
        }
        int wlo = 0, whi = 0, wrows = 0, wnnz = 0;
        if (plan_window(p, wr, wc, wtiles, &wlo, &whi, &wrows, &wnnz)) {
            const int w_rp = (wrows + 8 + 3) & ~3, w_cw = (wnnz + 8 + 3) & ~3;
            const int w_xw = (wrows + whi - wlo + 8 + 3) & ~3;
            const size_t stage = 4 * (size_t)(w_rp + w_cw + w_xw);
            const int S = (int)std::min<size_t>(kWinMaxStages, (kWinSmemBudget - 128) / stage);
            if (S >= 2) {
                p->nwtiles = (int)wtiles.size();
                p->wlo = wlo;
                p->whi = whi;
                p->w_rp = w_rp;
                p->w_cw = w_cw;
                p->w_xw = w_xw;
                p->w_stages = S;
                p->w_grid = std::min(p->nwtiles, num_sms());
            } else {
                wtiles.clear();
            }
        }
    }

    Scratch up_rp, up_col;                    // host arrays go through device scratch
    if (!on_device) {
        TC_CHECK(up_rp.alloc(sizeof(int) * ((size_t)M + 1), stream));
        TC_CHECK(up_col.alloc(sizeof(int) * (size_t)nnz_csr, stream));
        TC_CUDA(cudaMemcpyAsync(up_rp.p, csrRow, sizeof(int) * ((size_t)M + 1), cudaMemcpyHostToDevice, stream));
        if (nnz_csr)
            TC_CUDA(cudaMemcpyAsync(up_col.p, csrCol, sizeof(int) * (size_t)nnz_csr, cudaMemcpyHostToDevice, stream));
        csrRow = up_rp.as<int>();
        csrCol = up_col.as<int>();
    }

    // row statistics, and the tiles per strip unless the tiles are wide
    const int strips = (int)(((long)M + kStripRows - 1) / kStripRows);
    const size_t o_sum = align256(sizeof(RowStats)), o_cnt = align256(o_sum + 2 * sizeof(TileCounts));
    const size_t o_first = align256(o_cnt + sizeof(int) * 2 * ((size_t)strips + 1));
    const size_t o_tmp = align256(o_first + sizeof(int) * 2 * ((size_t)strips + 1));
    Scratch tmp;
    TC_CHECK(tmp.alloc(o_tmp + sizeof(int) * scan_tmp_ints(strips), stream));
    char *t = tmp.as<char>();
    RowStats *d_st = reinterpret_cast<RowStats *>(t);
    TileCounts *d_sum = reinterpret_cast<TileCounts *>(t + o_sum);
    int *d_cnt = reinterpret_cast<int *>(t + o_cnt), *d_first = reinterpret_cast<int *>(t + o_first);
    int *d_bcnt = d_cnt + strips + 1, *d_bfirst = d_first + strips + 1;
    int *d_tmp = reinterpret_cast<int *>(t + o_tmp);
    TC_CUDA(cudaMemsetAsync(t, 0, o_first, stream));
    const int step = std::max(1, M / 65536);
    if (M) row_stats<<<blocks_for(M, 256), 256, 0, stream>>>(csrRow, M, step, d_st);
    if (p->hybrid && nnz_csr)
        word_signs<<<blocks_for(nnz_csr, 256), 256, 0, stream>>>(csrCol, nnz_csr, d_st);
    const int min_tiles = 4 * num_sms();
    TilePrm q;
    q.mode = prm.tile_mode;
    q.rows_cap = std::max(1, std::min(prm.tile_rows, kMaxTileRows));
    q.tile_nnz = prm.tile_nnz;
    q.long_len = std::max(1, std::min(prm.tile_nnz, q.mode == 2 ? kStreamNnz : kStageNnz));
    // stream tiles hold at most nnz_csr / min_tiles entries (not below 512),
    // so a small matrix still spreads over the GPU
    q.spread = (int)std::min<int64_t>(kStreamNnz, std::max<int64_t>(512, nnz_csr / std::max(1, min_tiles)));
    q.max_lanes = prm.max_lanes;
    q.strided = (prm.flags & TC_FLAG_ROWS_STRIDED) != 0;
    const bool no_direct = (prm.flags & TC_FLAG_NO_DIRECT) || nnz_csr > kDirectMaxWords;
    q.no_direct = no_direct;
    TilePrm bq = q;                           // the tiles of batch and served launches
    bq.spread = kStreamNnz;
    const bool second = M > 0 && prm.tile_mode == 2 && q.spread < kStreamNnz;
    const size_t smem = strip_smem(std::min(M, kStripRows));
    const PlanLists lists{{q, bq}};
    if (M) {
        TC_CHECK(ensure_smem((const void *)plan_strips<false>, smem));
        TC_CHECK(ensure_smem((const void *)plan_strips<true>, smem));
        plan_strips<false><<<dim3(strips, second ? 2 : 1), kPlanBlock, smem, stream>>>(csrRow, M, lists, d_st, d_cnt, nullptr,
                                                                                     nullptr, nullptr, d_sum);
        TC_CUDA(cudaGetLastError());
        TC_CHECK(exclusive_scan(d_cnt, d_first, strips, d_tmp, stream));
        if (second) TC_CHECK(exclusive_scan(d_bcnt, d_bfirst, strips, d_tmp, stream));
    }
    RowStats st{};
    TileCounts sum{};
    int made = 0, bmade = 0;
    TC_CUDA(cudaMemcpyAsync(&st, d_st, sizeof st, cudaMemcpyDeviceToHost, stream));
    TC_CUDA(cudaMemcpyAsync(&sum, d_sum, sizeof sum, cudaMemcpyDeviceToHost, stream));
    if (M) TC_CUDA(cudaMemcpyAsync(&made, d_first + strips, sizeof made, cudaMemcpyDeviceToHost, stream));
    if (M && second) TC_CUDA(cudaMemcpyAsync(&bmade, d_bfirst + strips, sizeof bmade, cudaMemcpyDeviceToHost, stream));
    TC_CUDA(cudaStreamSynchronize(stream));
    p->max_row = st.max_row;
    p->all_pos = !st.minus;                   // a hybrid plan with no holes: every word adds its term
    // rows of at most one entry on average and none long, at most one dense
    // diagonal: the whole matrix as wide direct tiles (a 1024-thread CTA
    // each).  Several diagonals make a thread's four rows a long chain and its
    // loads of x four to a line; the rows kernel takes those plans.
    const bool wide = prm.tile_mode == 2 && prm.tile_rows >= kDirectRows &&
                      !no_direct && !(prm.flags & (TC_FLAG_NO_WIDE | TC_FLAG_ROWS_STRIDED)) &&
                      M >= kDirectWideRows && nnz_csr <= M && st.max_row <= kStreamRowMax && p->num_negs <= 1;
    p->wide_rows = wide ? wide_tile_rows(M, prm, num_sms()) : kDirectWideRows;
    p->ntiles = wide ? (int)(((long)M + p->wide_rows - 1) / p->wide_rows) : made;
    const bool own = wide || !second;         // batches run the plan's own tiles
    p->nbtiles = own ? p->ntiles : bmade;
    p->ntiles_wide = wide ? p->ntiles : 0;
    p->ntiles_vector = wide ? 0 : sum.vector;
    p->ntiles_long = wide ? 0 : sum.lng;
    p->ntiles_stream = wide ? 0 : sum.stream;
    // shared-memory stage sizes (ints, multiples of 4) from the largest tile
    p->stage_rp = (std::max(1, wide ? 1 : sum.max_rows) + 1 + 8 + 3) & ~3;
    p->stage_cw = ((wide ? 0 : sum.max_nnz) + 8 + 3) & ~3;
    {   // the most common length of the rows stream tiles hold: skewed slots
        // when it is a multiple of 8 (see vslot), sampled rows
        const int *h = st.hist;
        const int mode = (int)(std::max_element(h + 1, h + kStreamRowMax + 1) - h);
        p->stream_skew = h[mode] > 0 && mode % 8 == 0;
        // the rows kernel loads W words of a row together: the least of 2, 4,
        // 6, 8 that holds 90 % of the rows whole, 2 only where the longest
        // row takes four rounds (3 diagonals of 100,000 rows, 0.3 words each
        // and one row of 32: 4.8 us at 2, 3.2 at 4; of 1,000,000 rows and 1 %
        // of 16 words: 9.8 and 8.7; without the long ones 6.2 and 6.5)
        int64_t tot = 0, upto = 0, many = 0;
        for (int L = 0; L <= kStreamRowMax; ++L) tot += h[L];
        p->rows_w = 8;
        for (int L = 0, w = 2; L <= 8 && tot > 0; ++L) {
            upto += h[L];
            if (L == w) {
                if (upto * 10 >= tot * 9 && (w > 2 || st.max_row <= 8)) {
                    p->rows_w = w;
                    break;
                }
                w += 2;
            }
        }
        // whether the rows kernel also takes the plan's direct and four-row
        // tiles (hybrid plans).  A long row is one thread's there, and its
        // warp waits.  Up to a word a row it is in those tiles too, in runs of
        // four rows, and what counts is the number of rows: with few, a thread
        // a row keeps more loads in flight; over several waves of CTAs the
        // runs' wide accesses win (3 diagonals, 0.3 words a row, us in rows
        // and in tiles: 100,000 rows 1.9 and 3.3; 650,000 4.5 and 4.6;
        // 2,500,000 13.6 and 10.5; 7 diagonals 6.1 and 6.5 at 650,000, 8.5 and
        // 8.1 at 1,000,000; 2 diagonals 6.1 and 5.4 there).  Above a word a
        // row the tiles gather the words side by side, and the rows kernel is
        // the faster one while no row takes more than 8 rounds and at most a
        // seventh of the warps hold one of more than 4 (300,000 rows of 1.3
        // words, 3 diagonals: 3.0 and 5.4; with 0.1 % of 64 words 7.6 and 4.8,
        // with one row of 128 11.0 and 5.2; 1,000,000 rows with 1 % of 32 words
        // anywhere, 27 % of the warps, 12.6 and 11.5, with 0.1 % of 16 8.2 and
        // 10.0; 697,228 rows of 19 diagonals with 0.8 % of 19 words, all at the
        // end, 12.5 and 14.8)
        const int W = prm.rows_w ? prm.rows_w : p->rows_w;
        for (int L = std::min(4 * W, kStreamRowMax) + 1; L <= kStreamRowMax; ++L) many += st.whist[L];
        const int64_t wave = (int64_t)kRowsMinBlocks * num_sms() * kBlock;
        p->rows_any = nnz_csr <= M ? M <= (p->num_negs <= 2 ? 3 : 4) * wave
                                   : st.max_row <= 8 * W && many * 7 <= (M + 31L) / 32;
    }

    // the format: row pointers and words, each followed by at least 16 zero
    // bytes (the kernels' aligned loads run past the last element), the
    // shapes, the error word, the tiles
    const size_t rp_end = sizeof(int) * ((size_t)M + 1);
    const size_t o_cols = align256(rp_end + 16), cols_end = o_cols + sizeof(int) * (size_t)nnz_csr;
    const size_t o_sh = align256(cols_end + 16);
    const size_t o_sd = align256(o_sh + sizeof(int4) * shapes.size());
    const size_t o_off = align256(o_sd + sizeof(int2) * sd.size());
    const size_t o_err = align256(o_off + sizeof(int) * (size_t)p->num_negs + 16);
    const size_t o_tiles = align256(o_err + 16);
    const size_t o_bt = align256(o_tiles + sizeof(Tile) * (size_t)p->ntiles);
    const size_t o_wt = align256(o_bt + sizeof(Tile) * (size_t)(own ? 0 : p->nbtiles));
    const size_t total = align256(o_wt + sizeof(Tile) * wtiles.size());
    TC_CHECK(device_alloc(&p->dev, total, stream));
    char *const base = static_cast<char *>(p->dev);
    p->dev_bytes = total;
    p->d_rowptr = reinterpret_cast<int *>(base);
    p->d_cols = reinterpret_cast<int *>(base + o_cols);
    p->d_shapes = reinterpret_cast<int4 *>(base + o_sh);
    p->d_shape_dias = reinterpret_cast<int2 *>(base + o_sd);
    p->d_offsets = reinterpret_cast<int *>(base + o_off);
    p->d_err = reinterpret_cast<int *>(base + o_err);
    p->d_tiles = reinterpret_cast<Tile *>(base + o_tiles);
    p->d_btiles = own ? p->d_tiles : reinterpret_cast<Tile *>(base + o_bt);
    p->d_wtiles = p->nwtiles ? reinterpret_cast<Tile *>(base + o_wt) : nullptr;
    TC_CUDA(cudaMemsetAsync(base + rp_end, 0, o_cols - rp_end, stream));
    TC_CUDA(cudaMemsetAsync(base + cols_end, 0, o_sh - cols_end, stream));
    TC_CUDA(cudaMemsetAsync(base + o_off, 0, o_tiles - o_off, stream));
    TC_CUDA(cudaMemcpyAsync(p->d_rowptr, csrRow, rp_end, cudaMemcpyDeviceToDevice, stream));
    if (nnz_csr)
        TC_CUDA(cudaMemcpyAsync(p->d_cols, csrCol, sizeof(int) * (size_t)nnz_csr, cudaMemcpyDeviceToDevice, stream));
    if (!shapes.empty()) {
        TC_CUDA(cudaMemcpyAsync(p->d_shapes, shapes.data(), sizeof(int4) * shapes.size(),
                                cudaMemcpyHostToDevice, stream));
        TC_CUDA(cudaMemcpyAsync(p->d_shape_dias, sd.data(), sizeof(int2) * sd.size(),
                                cudaMemcpyHostToDevice, stream));
        TC_CUDA(cudaMemcpyAsync(p->d_offsets, p->h_offsets.data(), sizeof(int) * p->num_negs,
                                cudaMemcpyHostToDevice, stream));
    }
    if (p->nwtiles)
        TC_CUDA(cudaMemcpyAsync(p->d_wtiles, wtiles.data(), sizeof(Tile) * wtiles.size(),
                                cudaMemcpyHostToDevice, stream));

    if (wide)
        wide_tiles<<<(unsigned)((p->ntiles + 255) / 256), 256, 0, stream>>>(p->d_rowptr, M, p->wide_rows, p->ntiles,
                                                                          p->d_tiles);
    else if (M)
        plan_strips<true><<<dim3(strips, own ? 1 : 2), kPlanBlock, smem, stream>>>(p->d_rowptr, M, lists, d_st, nullptr, d_first,
                                                                                 p->d_tiles, p->d_btiles, nullptr);
    for (int k = 0; k < 3; ++k) {
        Tile *list = k == 0 ? p->d_tiles : k == 1 ? p->d_wtiles : p->d_btiles;
        const int n = k == 0 ? p->ntiles : k == 1 ? p->nwtiles : own ? 0 : p->nbtiles;
        if (n) classify_tiles<<<(unsigned)((n + 7L) / 8), 256, 0, stream>>>(
            list, n, p->d_shapes, p->d_shape_dias, p->d_offsets, p->dia_shapes, p->row_start, p->row_stop);
    }
    TC_CUDA(cudaGetLastError());
    // wide plans of few tiles: each tile's first word travels in the launch
    // parameters, for the word prefetch or the staged words
    const bool bounds = wide && p->ntiles <= kWideBoundTiles && M % kDirectWideRows == 0 &&
                        (prm.flags & TC_FLAG_WIDE_BOUNDS);
    const bool starts = wide && p->ntiles <= kWideParamTiles &&
                        !(prm.flags & (TC_FLAG_NO_PREFETCH | TC_FLAG_NO_PARAM_STARTS));
    p->h_wide_nz.clear();
    p->h_wide_z.clear();
    if (bounds || starts) {
        std::vector<Tile> ht(p->ntiles);
        TC_CUDA(cudaMemcpyAsync(ht.data(), p->d_tiles, sizeof(Tile) * ht.size(), cudaMemcpyDeviceToHost, stream));
        TC_CUDA(cudaStreamSynchronize(stream));
        std::vector<int> nz;
        for (const Tile &w : ht) nz.push_back(w.nz0);
        nz.push_back((int)nnz_csr);
        if (starts) p->h_wide_z = nz;
        if (bounds) p->h_wide_nz = nz;
    }
    p->grid = 1;
    if (prm.tile_mode != 2) {   // persistent grid: CTAs per SM from occupancy at this stage size
        DevPlan dp = p->dev_plan();
        TC_CHECK(tiles_grid(dp, prm.ctas_per_sm, &p->grid));
    }
    if (p->nwtiles) {
        DevPlan dp = p->dev_plan();
        TC_CHECK(window_prepare(dp));
    }
    if (prm.flags & TC_FLAG_KEEP_HOST) {
        p->h_rowptr.resize((size_t)M + 1);
        p->h_cols.resize((size_t)nnz_csr);
        TC_CUDA(cudaMemcpyAsync(p->h_rowptr.data(), p->d_rowptr, rp_end, cudaMemcpyDeviceToHost, stream));
        if (nnz_csr)
            TC_CUDA(cudaMemcpyAsync(p->h_cols.data(), p->d_cols, sizeof(int) * (size_t)nnz_csr,
                                    cudaMemcpyDeviceToHost, stream));
    }
    TC_CUDA(cudaStreamSynchronize(stream));
    return TC_OK;
}

}  // namespace tc
