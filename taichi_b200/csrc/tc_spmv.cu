// tc_spmv.cu -- the multiply: the value-free hybrid SpMV kernels for sm_100a
// and their launch.
//
// Replaces taichi_SpMV's dispatch and kernels (TaiChi.cu:965-1329).  The
// reference launches one of four CSR-vector kernels with a single vector
// width per matrix (TPV = sqrt of the mean row length) and a volatile
// shared-memory reduction.  Here the planner (tc_plan.cu) cuts the rows into tiles
// and gives each tile its own lanes-per-row from that tile's row lengths (a
// CTA per row above a length limit); the kernel walks the tile list, keeps
// kRPT rows' loads in flight per lane group, adds the dense-diagonal terms in
// registers and writes y once with warp-shuffle reductions.  Launches use
// programmatic dependent launch so the next multiply's index loads overlap
// the previous one's tail.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "tc_internal.h"
#include "tc_tile.cuh"
#include "tc_tma.cuh"

namespace tc {

// ------------------------------------------------------------------ kernels
namespace {

// Issues the copies of tile t into stage s (thread 0 only).
__device__ __forceinline__ void stage_tile(const DevPlan &p, int t, int *rp_buf, int *cw_buf,
                                           uint64_t *bar)
{
    if (t >= p.ntiles) return;
    const Tile tile = p.tiles[t];
    if (tile_kind(tile) == TILE_LONG || tile_kind(tile) >= TILE_STREAM) return;   // read from global
    const Window wr = window_of(tile.row0, (long)tile.row0 + tile_nrows(tile) + 1);
    const Window wc = window_of(tile.nz0, (long)tile.nz0 + tile.nnz);
    const unsigned br = (unsigned)(wr.b - wr.a), bc = tile.nnz ? (unsigned)(wc.b - wc.a) : 0u;
    mbar_expect_tx(bar, br + bc);
    bulk_load(rp_buf, reinterpret_cast<const char *>(p.rowptr) + wr.a, br, bar);
    if (bc) bulk_load(cw_buf, reinterpret_cast<const char *>(p.cols) + wc.a, bc, bar);
}

// The multiply: a persistent grid; each CTA walks tiles blockIdx.x,
// blockIdx.x + gridDim.x, ... with a two-stage pipeline: while one tile is
// processed from shared memory, the TMA engine brings in the row pointers
// and CSR words of the tile after next.  Rows longer than a stage are read
// straight from global memory (TILE_LONG).
template <bool SIGNED>
__global__ void __launch_bounds__(kBlock) spmv_tiles_kernel(DevPlan p, const float *__restrict__ x,
                                                            float *__restrict__ y)
{
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem);
    int *const buf = reinterpret_cast<int *>(smem + 16);
    const int stride = p.stage_rp + p.stage_cw;          // ints per stage
    allow_next_grid();
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        mbar_init(bar + 1, 1);
        mbar_fence_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        stage_tile(p, blockIdx.x, buf, buf + p.stage_rp, bar);
        stage_tile(p, blockIdx.x + gridDim.x, buf + stride, buf + stride + p.stage_rp, bar + 1);
    }
    unsigned phases = 0u;                                // bit s: parity of stage s
    bool waited = false;
    int i = 0;
    for (int t = blockIdx.x; t < p.ntiles; t += gridDim.x, ++i) {
        const int s = i & 1;
        int *const rp_s = buf + s * stride;
        int *const cw_s = rp_s + p.stage_rp;
        const Tile tile = p.tiles[t];
        if (tile_kind(tile) == TILE_LONG || tile_kind(tile) >= TILE_STREAM) {
            run_tile<SIGNED>(p, tile, x, y, !waited);
        } else {
            const bool ok = mbar_wait(bar + s, (phases >> s) & 1u);
            if (!__syncthreads_and(ok)) {          // every thread takes the same branch
                if (threadIdx.x == 0) atomicExch(p.err, 1);
                mbar_wait(bar + (s ^ 1), (phases >> (s ^ 1)) & 1u);   // copies in flight land
                return;
            }
            phases ^= 1u << s;
            const Window wr = window_of(tile.row0, 0), wc = window_of(tile.nz0, 0);
            const SharedSrc src{rp_s + wr.shift, cw_s + wc.shift, tile.nz0};
            run_tile_src<SIGNED>(p, tile, src, x, y, !waited);
        }
        waited = true;
        after_wait(x, y);                 // later tiles' x / y accesses follow the first tile's wait
        __syncthreads();                  // stage s is free again
        if (threadIdx.x == 0) {
            fence_async_shared();
            stage_tile(p, t + 2 * gridDim.x, rp_s, cw_s, bar + s);
        }
    }
    if (!waited) wait_prior_grid();
}

// The multiply of a plan of wide direct tiles: one 1024-thread CTA per 4096
// rows, one run of 4 rows per thread.  Few CTAs (the block scheduler's launch
// cost grows with the CTA count) that all fit at once (2 per SM at 32
// registers), each holding 1024 independent load chains.
// (A variant that read a per-run descriptor -- 4 packed row lengths and the
// run's words padded to an int4, loaded together instead of row pointers then
// words -- measured slower on R-MAT, 7.35 against 5.9 µs, and was dropped.)
// FULL: every tile is whole (M a multiple of kDirectWideRows, N >= M) and x
// and y are 16-byte aligned, so each run takes the edge-free path and the x
// window is one aligned 16 KB prefetch; the launch picks it from those facts.
// (One kernel holding both paths behind a per-tile branch ran the full tiles
// 0.8 µs slower per R-MAT scale 20 multiply than this split.)
// POS (with SIGNED and FULL): every word of the plan is an addition (no
// holes in its dense diagonals), so the gathers skip the sign.  The FULL
// body: z0 / z1, when z0 >= 0, are the tile's CSR word range as the launch
// parameters give it (the prefetch of the words then goes out at once),
// otherwise thread 0 reads the range from the tile record first.
template <bool SIGNED, bool POS>
__device__ __forceinline__ void wide_full(const DevPlan &p, const float *__restrict__ x, float *__restrict__ y,
                                          int z0, int z1)
{
    const int row0 = blockIdx.x * p.wide_rows;
    const int nr = min(p.wide_rows, p.M - row0);
    const int dc = SIGNED && p.dn != 1 ? tile_dclass(p.tiles[blockIdx.x]) : kDiagNone;
    if (threadIdx.x == 0) {
        prefetch_l2(x + row0, (unsigned)nr * sizeof(float));
        if (z0 >= 0) {
            prefetch_span(p.cols, z0, z1);
        } else if (p.prefetch) {
            // the tile's CSR words, so that the runs' word loads, which wait
            // for their row pointers, find them in L2
            const Tile t = p.tiles[blockIdx.x];
            prefetch_span(p.cols, t.nz0, t.nz0 + t.nnz);
        }
    }
    if (4 * (int)threadIdx.x >= nr) {
        wait_prior_grid(x, y);
        return;
    }
    direct_run_full<SIGNED, POS>(p, dc, x, y, row0 + 4 * threadIdx.x);
}

template <bool SIGNED, bool FULL, bool POS = false>
__global__ void __launch_bounds__(kDirectWideBlock, 2) spmv_wide_kernel(DevPlan p, const float *__restrict__ x,
                                                                     float *__restrict__ y)
{
    allow_next_grid();
    // wide tiles are laid out in order, p.wide_rows rows each (the last one
    // may be shorter), so the rows are known without waiting for the tile
    // record; only the diagonal class comes from it (a one-diagonal plan
    // needs no tile record: the parameters say which rows have the term)
    if (FULL) {
        wide_full<SIGNED, POS>(p, x, y, -1, -1);
    } else {
        // the edge path (direct_run) has no one-diagonal shortcut: every plan's
        // diagonal terms come from the tile's class
        const int row0 = blockIdx.x * p.wide_rows;
        const int nr = min(p.wide_rows, p.M - row0);
        const int dc = SIGNED ? tile_dclass(p.tiles[blockIdx.x]) : kDiagNone;
        if (threadIdx.x == 0) prefetch_x_window(x, p.N, row0, nr);
        direct_run<SIGNED>(p, row0, nr, dc, x, y, true, 4 * threadIdx.x);
    }
}

// The whole-tile wide kernel with each tile's first CSR word in the launch
// parameters (plans of at most kWideParamTiles tiles): the prefetch of a
// tile's words into L2 goes out when the CTA starts, together with its
// row-pointer loads, instead of after a read of the tile record.
template <bool SIGNED, bool POS>
__global__ void __launch_bounds__(kDirectWideBlock, 2)
    spmv_wide_starts_kernel(DevPlan p, const __grid_constant__ WideStarts ws, const float *__restrict__ x,
                            float *__restrict__ y)
{
    allow_next_grid();
    wide_full<SIGNED, POS>(p, x, y, ws.nz[blockIdx.x], ws.nz[blockIdx.x + 1]);
}

// The multiply of a stream plan of short rows, one row per thread, read
// straight from global memory: no tile records, shared memory or barriers.
// A CTA runs kBlock consecutive rows (coalesced row pointers and y
// stores).  Each thread loads its row's first W words together
// (immutable plan data, before griddepcontrol.wait), then their gathers and
// its dense-diagonal terms together, and adds the diagonal terms (offset
// order), then the words (stored order), then any further words W at a
// time: the terms and order of tile_rows_seq, so y is bit-identical to the
// stream tiles'.  Consecutive lanes hold consecutive rows, so a warp's load
// of word w of its 32 rows touches the few cache lines holding those rows,
// and its later words hit L1.  Against the stream tiles it spends no
// instructions on parking terms in shared memory and no barrier waits.
template <bool SIGNED, int W>
__global__ void __launch_bounds__(kBlock, kRowsMinBlocks)
    spmv_rows_kernel(DevPlan p, const __grid_constant__ typename DiagsOf<SIGNED>::type q,
                     const float *__restrict__ x, float *__restrict__ y)
{
    allow_next_grid();
    const int r = blockIdx.x * kBlock + threadIdx.x;
    const bool own = (unsigned)r < (unsigned)p.M;     // a last CTA's rows may lie past 2^31 - 1
    // warp 0 also brings into L2 the x window of the strip and the operands
    // of the strip a wave later (thread 0; the other warps skip it whole)
    const bool lead = threadIdx.x < 32;
    const bool ahead = lead && blockIdx.x + p.ahead < gridDim.x;
    int za = 0, zb = 0;
    if (lead && threadIdx.x == 0) prefetch_x_window(x, p.N, r, kBlock);
    const int b = own ? __ldg(p.rowptr + r) : 0;
    const int e = own ? __ldg(p.rowptr + r + 1) : 0;
    if (ahead) {
        const int ra = (blockIdx.x + p.ahead) * kBlock;
        za = __ldg(p.rowptr + ra);
        zb = __ldg(p.rowptr + ra + min(kBlock, p.M - ra));
    }
    const int n = e - b;
    int c[W];
#pragma unroll
    for (int w = 0; w < W; ++w) c[w] = w < n ? __ldg(p.cols + b + w) : 0;
    if (ahead && threadIdx.x == 0) {
        const int ra = (blockIdx.x + p.ahead) * kBlock;
        prefetch_rows_ahead(p, ra, ra + min(kBlock, p.M - ra), za, zb);
    }
    wait_prior_grid(x, y);
    // every slot is loaded (a slot past the row holds word 0, a load of x[0]
    // that is never added): no branch around the gathers
    float v[W];
#pragma unroll
    for (int w = 0; w < W; ++w) v[w] = gather<SIGNED>(x, c[w]);
    float acc = 0.f;
    if constexpr (SIGNED) {
        if (p.dn > 0 && r >= p.d_in.x && r < p.d_in.y) {
            // the plan's offsets in order, named by constant indices (operands
            // straight from the parameter bank)
            float d[kPlanDiags];
#pragma unroll
            for (int u = 0; u < kPlanDiags; ++u) d[u] = u < p.dn ? ldx(x + r + p.d_col[u]) : 0.f;
#pragma unroll
            for (int u = 0; u < kPlanDiags; ++u)
                if (u < p.dn) acc += d[u];
        } else if (q.n > 0) {
            acc = diag_plan_row(q, x, r);
        } else {
            acc = diag_row(p, x, r);
        }
    }
#pragma unroll
    for (int w = 0; w < W; ++w)
        if (w < n) acc += v[w];
#pragma unroll 1
    for (Words a(b, e, W); a.left > 0; a.skip(W)) {                 // longer rows, W words at a time
        int cc[W];
        float vv[W];
#pragma unroll
        for (int u = 0; u < W; ++u) cc[u] = u < a.left ? __ldg(p.cols + a.at + u) : 0;
#pragma unroll
        for (int u = 0; u < W; ++u) vv[u] = gather<SIGNED>(x, cc[u]);
#pragma unroll
        for (int u = 0; u < W; ++u)
            if (u < a.left) acc += vv[u];
    }
    if (own) y[r] = acc;
}

// The multiply of a stream plan (any of its tile kinds): one CTA per tile, no
// shared-memory stages (stream tiles read their CSR words as coalesced int4s;
// direct and long tiles read global memory directly).
template <bool SIGNED>
__global__ void __launch_bounds__(kBlock, kLeanMinBlocks)
    spmv_grid_kernel(DevPlan p, const float *__restrict__ x, float *__restrict__ y)
{
    allow_next_grid();
    const Tile t = p.tiles[blockIdx.x];
    if (threadIdx.x == 0) prefetch_x_window(x, p.N, t.row0, tile_nrows(t));
    run_lean_tile<SIGNED>(p, t, x, y, true);
}

// The whole-tile wide kernel with the tiles' word bounds in the launch
// parameters: each CTA reads its tile's CSR words into shared memory with
// coalesced int4 loads issued together with its row-pointer loads, so the
// chain before the gathers is one memory round trip instead of two (row
// pointers, then the words they point to).  Same runs, terms and order as
// spmv_wide_kernel<SIGNED, true>.
template <bool SIGNED>
__global__ void __launch_bounds__(kDirectWideBlock, 2)
    spmv_wide_bounds_kernel(DevPlan p, const __grid_constant__ WideBounds tb, const float *__restrict__ x,
                            float *__restrict__ y)
{
    __shared__ int4 sw[kWideWordQ];
    allow_next_grid();
    const int row0 = blockIdx.x * kDirectWideRows;
    const int dc = SIGNED ? tile_dclass(p.tiles[blockIdx.x]) : kDiagNone;
    if (threadIdx.x == 0) prefetch_l2(x + row0, kDirectWideRows * sizeof(float));
    const int nz0 = tb.nz[blockIdx.x], nz1 = tb.nz[blockIdx.x + 1];
    const int base = nz0 & ~3;
    const int nq = min((nz1 - base + 3) >> 2, kWideWordQ);
    const int4 *cq = reinterpret_cast<const int4 *>(p.cols + base);
    for (int i = threadIdx.x; i < nq; i += kDirectWideBlock) sw[i] = __ldg(cq + i);
    const int g = row0 + 4 * threadIdx.x;
    const int4 r4 = __ldg(reinterpret_cast<const int4 *>(p.rowptr + g));
    const int e4 = __ldg(p.rowptr + g + 4);
    __syncthreads();
    direct_run_staged<SIGNED>(p, dc, x, y, g, r4, e4, reinterpret_cast<const int *>(sw), base, 4 * nq);
}

// The multiply of a plan of stream tiles only (meshes, banded and other
// matrices of short, even rows): the grid kernel with no code for the other
// tile kinds, compiled for B CTAs per SM (see kStreamFewMinBlocks).
template <bool SIGNED, int B>
__global__ void __launch_bounds__(kBlock, B)
    spmv_stream_kernel(DevPlan p, const float *__restrict__ x, float *__restrict__ y)
{
    allow_next_grid();
    const Tile t = p.tiles[blockIdx.x];
    if (threadIdx.x == 0) {
        prefetch_x_window(x, p.N, t.row0, tile_nrows(t));
        if (B == kStreamManyMinBlocks && blockIdx.x + p.ahead < p.ntiles) {   // the tile a wave later
            const Tile a = p.tiles[blockIdx.x + p.ahead];
            prefetch_rows_ahead(p, a.row0, a.row0 + tile_nrows(a), a.nz0, a.nz0 + a.nnz);
        }
    }
    tile_stream<SIGNED>(p, t, x, y, true);
}

}  // namespace

static int g_num_sms = 0;

int num_sms()
{
    if (g_num_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_num_sms <= 0) g_num_sms = 148;
    }
    return g_num_sms;
}

size_t stream_smem_bytes(const DevPlan &dp)
{
    return 16 + 2 * sizeof(int) * (size_t)(dp.stage_rp + dp.stage_cw);
}

tc_status tiles_grid(const DevPlan &dp, int ctas_per_sm, int *grid)
{
    const size_t smem = stream_smem_bytes(dp);
    int per_sm = 0;
    TC_CHECK(ensure_smem((const void *)spmv_tiles_kernel<false>, smem));
    TC_CHECK(ensure_smem((const void *)spmv_tiles_kernel<true>, smem));
    TC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, spmv_tiles_kernel<true>, kBlock, smem));
    const int cps = std::max(1, std::min(per_sm, ctas_per_sm));
    *grid = std::max(1, std::min(dp.ntiles, cps * num_sms()));
    return TC_OK;
}

template <bool SIGNED>
static tc_status launch_tiles(const DevPlan &dp, const PlanDiags &dg, const WideBounds *wb, const WideStarts *ws,
                              const float *x, float *y, cudaStream_t s)
{
    if (dp.ntiles <= 0) return TC_OK;
    const size_t smem = dp.per_tile ? 0 : stream_smem_bytes(dp);
    if (!dp.per_tile) TC_CHECK(ensure_smem((const void *)spmv_tiles_kernel<SIGNED>, smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(dp.per_tile ? dp.ntiles : dp.grid);
    cfg.blockDim = dim3(dp.per_tile == 3 ? kDirectWideBlock : kBlock);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = dp.pdl ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const bool full = dp.M % 4 == 0 && dp.N >= dp.M &&
                      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0;
    if (dp.per_tile == 3 && full && wb && dp.wide_rows == kDirectWideRows && dp.M % kDirectWideRows == 0)
        TC_CUDA(cudaLaunchKernelEx(&cfg, spmv_wide_bounds_kernel<SIGNED>, dp, *wb, x, y));
    else if (dp.per_tile == 3 && full && ws && SIGNED && dp.pos)
        TC_CUDA(cudaLaunchKernelEx(&cfg, spmv_wide_starts_kernel<SIGNED, true>, dp, *ws, x, y));
    else if (dp.per_tile == 3 && full && ws)
        TC_CUDA(cudaLaunchKernelEx(&cfg, spmv_wide_starts_kernel<SIGNED, false>, dp, *ws, x, y));
    else if (dp.per_tile == 3 && full && SIGNED && dp.pos)
        TC_CUDA(cudaLaunchKernelEx(&cfg, spmv_wide_kernel<SIGNED, true, true>, dp, x, y));
    else if (dp.per_tile == 3 && full) TC_CUDA(cudaLaunchKernelEx(&cfg, spmv_wide_kernel<SIGNED, true>, dp, x, y));
    else if (dp.per_tile == 3) TC_CUDA(cudaLaunchKernelEx(&cfg, spmv_wide_kernel<SIGNED, false>, dp, x, y));
    else if (dp.rows) {
        cfg.gridDim = dim3((unsigned)(((long)dp.M + kBlock - 1) / kBlock));
        typename DiagsOf<SIGNED>::type q;
        if constexpr (SIGNED) q = dg;
        if (dp.rows_w <= 2) TC_CUDA(cudaLaunchKernelEx(&cfg, spmv_rows_kernel<SIGNED, 2>, dp, q, x, y));
        else if (dp.rows_w <= 4) TC_CUDA(cudaLaunchKernelEx(&cfg, spmv_rows_kernel<SIGNED, 4>, dp, q, x, y));
        else if (dp.rows_w <= 6) TC_CUDA(cudaLaunchKernelEx(&cfg, spmv_rows_kernel<SIGNED, 6>, dp, q, x, y));
        else TC_CUDA(cudaLaunchKernelEx(&cfg, spmv_rows_kernel<SIGNED, 8>, dp, q, x, y));
    }
    else if (dp.per_tile == 4 && dp.ntiles <= kStreamFewMinBlocks * num_sms())
        TC_CUDA(cudaLaunchKernelEx(&cfg, spmv_stream_kernel<SIGNED, kStreamFewMinBlocks>, dp, x, y));
    else if (dp.per_tile == 4 && dp.ntiles <= kStreamWaveMinBlocks * num_sms())
        TC_CUDA(cudaLaunchKernelEx(&cfg, spmv_stream_kernel<SIGNED, kStreamWaveMinBlocks>, dp, x, y));
    else if (dp.per_tile == 4)
        TC_CUDA(cudaLaunchKernelEx(&cfg, spmv_stream_kernel<SIGNED, kStreamManyMinBlocks>, dp, x, y));
    else if (dp.per_tile) TC_CUDA(cudaLaunchKernelEx(&cfg, spmv_grid_kernel<SIGNED>, dp, x, y));
    else TC_CUDA(cudaLaunchKernelEx(&cfg, spmv_tiles_kernel<SIGNED>, dp, x, y));
    return TC_OK;
}

tc_status launch_spmv(const DevPlan &dp, const PlanDiags &dg, const float *x, float *y, cudaStream_t s,
                      const WideBounds *wb, const WideStarts *ws)
{
    if (dp.M == 0) return TC_OK;
    // no columns: no terms, and the kernels' unconditional loads of x[0]
    // (slots past a row's words) would have no x to read
    if (dp.N == 0) {
        TC_CUDA(cudaMemsetAsync(y, 0, sizeof(float) * (size_t)dp.M, s));
        return TC_OK;
    }
    if (dp.nwtiles > 0) return launch_window(dp, x, y, s);
    return dp.hybrid ? launch_tiles<true>(dp, dg, wb, ws, x, y, s) : launch_tiles<false>(dp, dg, wb, ws, x, y, s);
}

tc_status launch_plan(const tc_plan *p, const float *x, float *y, cudaStream_t s)
{
    if (!p->h_wide_nz.empty()) {
        WideBounds wb;
        memcpy(wb.nz, p->h_wide_nz.data(), sizeof(int) * p->h_wide_nz.size());
        return launch_spmv(p->dev_plan(), p->diags, x, y, s, &wb, nullptr);
    }
    if (!p->h_wide_z.empty()) {
        WideStarts ws;
        memcpy(ws.nz, p->h_wide_z.data(), sizeof(int) * p->h_wide_z.size());
        return launch_spmv(p->dev_plan(), p->diags, x, y, s, nullptr, &ws);
    }
    return launch_spmv(p->dev_plan(), p->diags, x, y, s, nullptr, nullptr);
}

}  // namespace tc

tc::DevPlan tc_plan::dev_plan() const
{
    tc::DevPlan d{};
    d.rowptr = d_rowptr;
    d.cols = d_cols;
    d.tiles = d_tiles;
    d.shapes = d_shapes;
    d.shape_dias = d_shape_dias;
    d.offsets = d_offsets;
    d.M = M;
    d.N = N;
    d.ntiles = ntiles;
    d.dia_shapes = dia_shapes;
    d.row_start = row_start;
    d.row_stop = row_stop;
    d.hybrid = hybrid;
    d.pdl = (params.flags & TC_FLAG_NO_PDL) ? 0 : 1;
    d.stage_rp = stage_rp;
    d.stage_cw = stage_cw;
    d.grid = grid;
    d.per_tile = params.tile_mode != 2 ? 0
               : ntiles == 0 ? 2
               : ntiles_wide == ntiles ? 3
               : ntiles_stream == ntiles ? 4 : 2;
    d.err = d_err;
    d.wide_rows = wide_rows;
    d.skew = stream_skew;
    d.dn = 0;
    if (diags.n > 0 && diags.n <= tc::kPlanDiags) {
        d.dn = diags.n;
        d.d_in = diags.in;
        for (int i = 0; i < diags.n; ++i) {
            d.d_col[i] = diags.col[i];
            d.d_lo[i] = std::max(diags.rows.x, diags.cols.x - diags.col[i]);
            d.d_hi[i] = std::min(diags.rows.y, diags.cols.y - diags.col[i]);
        }
    }
    // the rows kernel: a stream plan (every row at most kStreamRowMax words)
    // of short rows, or any stream plan on request; hybrid plans that are not
    // wide run it whatever their tiles (direct and four-row tiles among them),
    // unless a row is a CTA's: the CTA adds its words in another order, and a
    // plan gives the same y alone, in a batch and served
    const bool any_tiles = d.dia_shapes > 0 && d.per_tile == 2 && max_row <= tc::kStreamRowMax && ntiles_long == 0;
    const bool short_rows = M > 0 && nnz_csr <= (int64_t)tc::kRowsMeanMax * M && (d.per_tile == 4 || rows_any);
    d.rows = 0;
    if ((d.per_tile == 4 || any_tiles) && !(params.flags & TC_FLAG_NO_ROWS))
        d.rows = (params.flags & TC_FLAG_ROWS) || (short_rows && tc::kRowsByDefault);
    d.rows_w = params.rows_w ? params.rows_w : rows_w;
    d.pos = hybrid && all_pos ? 1 : 0;
    // CTAs resident at once (the stream kernel's many-tile build, the rows
    // kernel): the CTA that starts when this one ends is about this far on
    d.prefetch = (params.flags & TC_FLAG_NO_PREFETCH) ? 0 : 1;
    d.ahead = (params.flags & TC_FLAG_NO_PREFETCH) ? (1 << 30)
            : (d.rows ? tc::kRowsMinBlocks : tc::kStreamManyMinBlocks) * tc::num_sms();
    d.wtiles = d_wtiles;
    d.nwtiles = nwtiles;
    d.wlo = wlo;
    d.whi = whi;
    d.w_rp = w_rp;
    d.w_cw = w_cw;
    d.w_xw = w_xw;
    d.w_stages = w_stages;
    d.w_grid = w_grid;
    return d;
}

void tc_plan::set_diags()
{
    diags = tc::PlanDiags{};
    if (dia_shapes != 1 || num_negs > tc::kMaxDiags || (int)h_offsets.size() < num_negs) return;
    // the rows where diag_row adds each offset's term (TaiChi.cu:1014-1023)
    const int xs = h_xStart[0], xe = h_xStop[0], ys = h_yStart[0];
    diags.n = num_negs;
    diags.rows = make_int2(std::max(xs, row_start), std::min(xe, row_stop));
    diags.cols = make_int2(ys, ys + xe - xs);
    diags.in = diags.rows;
    for (int i = 0; i < num_negs; ++i) {
        const int c = diags.col[i] = ys - xs + h_offsets[i];
        diags.in = make_int2(std::max(diags.in.x, diags.cols.x - c), std::min(diags.in.y, diags.cols.y - c));
    }
}

int64_t tc_plan::spmv_bytes() const
{
    // 4(M+1) row pointers + 4 per CSR entry + x read once + y written once +
    // 20 bytes per shape descriptor + 4 per dense-diagonal offset.
    return 4LL * (M + 1) + 4LL * nnz_csr + 4LL * N + 4LL * M + 20LL * dia_shapes +
           4LL * num_negs;
}
