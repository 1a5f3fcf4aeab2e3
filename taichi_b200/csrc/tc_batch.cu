// tc_batch.cu -- many resident plans multiplied in one launch.
//
// The batch flattens the tile lists of all its plans into one work list, an
// item per tile, and runs it with one CTA per item in one launch (captured
// once in a CUDA graph and replayed by tc_batch_graph_launch).  An item holds
// all that its CTA needs to start -- tile, plan arrays, x and y -- so its
// words and row pointers are one load away; an item that named a plan and a
// tile, with the plan descriptor copied to shared memory first, put four
// loads and a barrier before them.  Small plans bring the tiles planned for
// batches (tc_plan::d_btiles): a plan alone spreads its entries over the GPU,
// a batch has the other plans for that and does better with whole tiles.
// When every plan holds only stream, direct and long tiles the lean kernel
// (no lane-tile code, more CTAs per SM) runs.  Every tile runs the same
// device code as the single-plan kernel, so each matrix's y is bit-identical
// alone and inside a batch.  Measured on 256 matrices of 1e3 to 2e5 rows
// (92 M entries, 471 MB): 280 us with the longer chain, a launch per word
// kind and the plans' own tiles, 148 us now.

#include <cuda_runtime.h>

#include <algorithm>
#include <new>

#include "tc_internal.h"
#include "tc_tile.cuh"

namespace tc {
namespace {

// One CTA's work: 64 bytes, read as four int4s by every thread of the CTA.
struct alignas(64) BatchItem {
    const int *rowptr, *cols;
    const float *x;
    float *y;
    Tile tile;
    int N;
    int plan;          // index of its descriptor
    int part;          // part of a wide direct tile, else 0
    int hybrid_skew;   // bit 0: hybrid plan, bit 1: skewed slots
};
static_assert(sizeof(BatchItem) == 64, "read as four int4s");

// LEAN: no lane-tile code; B: resident CTAs per SM it is compiled for.
template <bool LEAN, int B>
__global__ void __launch_bounds__(kBlock, B)
    batch_kernel(const DevPlan *__restrict__ plans, const BatchItem *__restrict__ items)
{
    const BatchItem it = load64(items + blockIdx.x);
    run_item<LEAN>(it.rowptr, it.cols, it.N, it.hybrid_skew, plans + it.plan, it.tile, it.part, it.x, it.y, true);
}

}  // namespace
}  // namespace tc

struct tc_batch {
    int n = 0;
    int nitems = 0;
    bool lean = false;
    void *dev = nullptr;
    tc::DevPlan *d_plans = nullptr;
    tc::BatchItem *d_items = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
};

using tc::fail;

extern "C" {

tc_status tc_batch_create(int n, tc_plan *const *plans, const float *const *d_x, float *const *d_y,
                          tc_batch **out)
{
    if (n < 1 || !plans || !d_x || !d_y || !out) return fail(TC_ERR_INVALID, "tc_batch_create: bad arguments");
    *out = nullptr;
    std::vector<tc::DevPlan> dps(n);
    std::vector<tc::BatchItem> items;
    std::vector<tc::Tile> tiles;
    bool lean = true;
    for (int i = 0; i < n; ++i) {
        const tc_plan *p = plans[i];
        if (!p) return fail(TC_ERR_INVALID, "plan %d is null", i);
        const tc::DevPlan &dp = dps[i] = p->dev_plan();
        lean = lean && dp.per_tile >= 2;
        tiles.resize(p->nbtiles);
        if (p->nbtiles)
            TC_CUDA(cudaMemcpy(tiles.data(), p->d_btiles, sizeof(tc::Tile) * tiles.size(), cudaMemcpyDeviceToHost));
        for (const tc::Tile &t : tiles)
            for (int k = 0; k < tc::tile_parts(dp.per_tile, tc::tile_nrows(t)); ++k)
                items.push_back(tc::BatchItem{dp.rowptr, dp.cols, d_x[i], d_y[i], t, dp.N, i, k,
                                              (dp.hybrid ? 1 : 0) | (dp.skew ? 2 : 0)});
    }
    tc_batch *b = new (std::nothrow) tc_batch();
    if (!b) return fail(TC_ERR_ALLOC, "host allocation");
    b->lean = lean;
    b->n = n;
    b->nitems = (int)items.size();
    const size_t o_it = (sizeof(tc::DevPlan) * n + 255) & ~(size_t)255;
    char *base = nullptr;
    if (cudaMalloc(&base, o_it + sizeof(tc::BatchItem) * items.size() + 256) != cudaSuccess) {
        delete b;
        return fail(TC_ERR_ALLOC, "batch tables");
    }
    b->dev = base;
    b->d_plans = reinterpret_cast<tc::DevPlan *>(base);
    b->d_items = reinterpret_cast<tc::BatchItem *>(base + o_it);
    tc_status st = tc::upload(b->d_plans, dps.data(), sizeof(tc::DevPlan) * n);    // run on any stream
    if (st == TC_OK && !items.empty())
        st = tc::upload(b->d_items, items.data(), sizeof(tc::BatchItem) * items.size());
    if (st != TC_OK) {
        cudaFree(base);
        delete b;
        return st;
    }
    *out = b;
    return TC_OK;
}

tc_status tc_batch_run(tc_batch *b, void *stream)
{
    if (!b) return fail(TC_ERR_INVALID, "null batch");
    if (b->nitems == 0) return TC_OK;
    cudaStream_t s = (cudaStream_t)stream;
    constexpr int few = tc::kItemFewBlocks, many = tc::kItemManyBlocks;
    if (!b->lean) tc::batch_kernel<false, 1><<<b->nitems, tc::kBlock, 0, s>>>(b->d_plans, b->d_items);
    else if (b->nitems <= 2 * few * tc::num_sms())
        tc::batch_kernel<true, few><<<b->nitems, tc::kBlock, 0, s>>>(b->d_plans, b->d_items);
    else tc::batch_kernel<true, many><<<b->nitems, tc::kBlock, 0, s>>>(b->d_plans, b->d_items);
    TC_CUDA(cudaGetLastError());
    return TC_OK;
}

tc_status tc_batch_graph_launch(tc_batch *b, void *stream)
{
    if (!b) return fail(TC_ERR_INVALID, "null batch");
    cudaStream_t s = (cudaStream_t)stream;
    if (!b->exec) {
        cudaStream_t cap;
        TC_CUDA(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
        TC_CUDA(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
        tc_status st = tc_batch_run(b, cap);
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamEndCapture(cap, &g);
        cudaStreamDestroy(cap);
        if (st != TC_OK) return st;
        if (e != cudaSuccess) return fail(TC_ERR_CUDA, "graph capture: %s", cudaGetErrorString(e));
        b->graph = g;
        TC_CUDA(cudaGraphInstantiate(&b->exec, g, 0));
    }
    TC_CUDA(cudaGraphLaunch(b->exec, s));
    return TC_OK;
}

tc_status tc_batch_destroy(tc_batch *b)
{
    if (!b) return TC_OK;
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    if (b->dev) cudaFree(b->dev);
    delete b;
    return TC_OK;
}

}  // extern "C"
