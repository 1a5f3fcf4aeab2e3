// tc_partition.cu -- the TaiChi partitioner on the GPU.
//
// Replaces getSdf (morohutils.cu:153-291) and partition_shapes /
// partition_dia_shape (TaiChi.cu:313-879).  Output is bit-identical to the
// reference for the same parameters:
//
//  1. raster       512 x W thumbnail of the pattern (getSdf_GPU1), one CTA per
//                  thumbnail row, bits in shared memory.
//  2. morphology   hole fill (imfill) by union-find over runs of zeros; 30x1
//                  and 1x30 openings, subtraction and the eye(5) opening on
//                  bit-packed rows, with OpenCV's conventions
//                  (non-reflected element, anchor at the centre, erosion sees
//                  1 and dilation 0 outside the image).
//  3. contours     findContours(RETR_CCOMP, CHAIN_APPROX_NONE): union-find
//                  labelling of 8-connected ones and 4-connected zeros gives
//                  every border's start pixel (Suzuki & Abe: the first pixel of
//                  a component starts its outer border; the pixel left of the
//                  first pixel of a hole starts that hole's border), a scan
//                  gives their discovery order, and one thread per border
//                  follows it.  OpenCV lists outer borders newest first, each
//                  followed by its holes newest first.
//  4. shapes       per kept contour, in order: cal_shape_size, the band
//                  histogram of unclaimed entries, the density test, hole rows
//                  and the claim of dense-diagonal entries.
//  5. assembly     per row: holes (shape, diagonal, row order) then unclaimed
//                  entries in CSR order, with the sign bit.

#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "tc_ctxcache.h"
#include "tc_internal.h"
#include "tc_scan.cuh"
#include "tc_words.h"

namespace tc {
namespace {

// ------------------------------------------------------------- bit images
// An H x W binary image is stored as H rows of WW = ceil(W/32) uint32 words;
// pixel x of a row is bit (x & 31) of word (x >> 5).  Bits at x >= W are 0.

struct Img {
    unsigned *w;
    int H, W, WW;
    __device__ __forceinline__ unsigned lastmask() const
    {
        const int r = W & 31;
        return r ? (1u << r) - 1u : 0xffffffffu;
    }
    // word k of row y, with `fill` outside the image (also for x >= W)
    __device__ __forceinline__ unsigned get(int y, int k, unsigned fill) const
    {
        if (y < 0 || y >= H || k < 0 || k >= WW) return fill;
        unsigned v = w[y * WW + k];
        if (k == WW - 1) v = (v & lastmask()) | (fill & ~lastmask());
        return v;
    }
    // bits x+d (x = 32k..32k+31) of row y
    __device__ __forceinline__ unsigned shifted(int y, int k, int d, unsigned fill) const
    {
        const int q = d >> 5, r = d & 31;
        const unsigned lo = get(y, k + q, fill);
        if (r == 0) return lo;
        return __funnelshift_r(lo, get(y, k + q + 1, fill), r);
    }
    __device__ __forceinline__ int pix(int y, int x) const
    {
        if (y < 0 || y >= H || x < 0 || x >= W) return 0;
        return (w[y * WW + (x >> 5)] >> (x & 31)) & 1;
    }
};

// Raster (morohutils.cu:153-180): bit (px, col/pN) for every entry of the
// rows of thumbnail row px = row / pM, for px < H and col/pN < W.
__global__ void raster_kernel(const int *__restrict__ rowptr, const int *__restrict__ col, int M,
                              int pM, int pN, Img img)
{
    extern __shared__ unsigned srow[];
    const int px = blockIdx.x;
    for (int k = threadIdx.x; k < img.WW; k += blockDim.x) srow[k] = 0;
    __syncthreads();
    const long r0 = (long)px * pM;
    const long r1 = r0 + pM < (long)M ? r0 + pM : (long)M;   // rows >= H*pM are never drawn
    if (r0 < M) {
        unsigned cur_w = 0xffffffffu, cur_bits = 0;
        for (Words a(__ldg(rowptr + r0), __ldg(rowptr + r1), threadIdx.x); a.left > 0; a.skip(blockDim.x)) {
            const int py = __ldg(col + a.at) / pN;
            if (py < img.W) {
                const unsigned wi = (unsigned)py >> 5, bit = 1u << (py & 31);
                if (wi != cur_w) {
                    if (cur_bits) atomicOr(&srow[cur_w], cur_bits);
                    cur_w = wi;
                    cur_bits = 0;
                }
                cur_bits |= bit;
            }
        }
        if (cur_bits) atomicOr(&srow[cur_w], cur_bits);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < img.WW; k += blockDim.x) img.w[px * img.WW + k] = srow[k];
}

// ------------------------------------------------------- connected regions
// Union-find over runs.  A node is a maximal run of equal pixels within one
// word of a row, named 1 + the index of its first pixel; node 0 is the zero
// frame around the image.  Links always point to a smaller name, so a
// region's root names its first pixel in raster order.  Joining runs instead
// of pixels is what makes it cheap: a word of equal pixels is one node, zero
// runs on the image border start out linked to the frame, and vertical
// neighbours join once per overlap.  Hole filling of the 9-point mesh's
// thumbnail (512 x 512, noisy): 2.5 ms as alternating row and column closures
// in one CTA, 0.14 ms this way; labelling the opened image: 190 us per pixel,
// 100 us per run.  Every look-up halves the path it walks (a node is pointed
// at its grandparent: an ancestor for good, so a racing store loses nothing),
// as rows joined at the same time link into long chains: hole filling 130 ->
// 97 us, labelling 87 -> 61.  (Joining rows in pairs, then pairs of pairs,
// to keep the chains short: 300 us each, too few CTAs.)
__device__ __forceinline__ int uf_find(int *L, int a)
{
    int b = __ldcg(L + a);
    while (b != a) {
        const int c = __ldcg(L + b);
        if (c != b) __stcg(L + a, c);
        a = b;
        b = c;
    }
    return a;
}

__device__ void uf_union(int *L, int a, int b, int *flag)
{
    for (int it = 0; it < (1 << 24); ++it) {
        a = uf_find(L, a);
        b = uf_find(L, b);
        if (a == b) return;
        if (a < b) {
            const int old = atomicMin(L + b, a);
            if (old == b) return;
            b = old;
        } else {
            const int old = atomicMin(L + a, b);
            if (old == a) return;
            a = old;
        }
    }
    *flag = 2;   // no progress (cannot happen): reported, never waited on
}

// First bit of the run of set bits of v that holds bit p.
__device__ __forceinline__ int run_start(unsigned v, int p)
{
    return 32 - __clz(~v & ((1u << p) - 1u));
}
__device__ __forceinline__ unsigned run_starts(unsigned v) { return v & ~(v << 1); }
// The run of set bits of v that starts at bit p, as a mask.
__device__ __forceinline__ unsigned run_mask(unsigned v, int p)
{
    const unsigned past = ~(v >> p);                 // first clear bit above p ends the run
    const int n = past ? __ffs(past) - 1 : 32;
    return (n >= 32 ? 0xffffffffu : (1u << n) - 1u) << p;
}
// Bits of word k inside the image.
__device__ __forceinline__ unsigned word_mask(const Img &img, int k)
{
    return k == img.WW - 1 ? img.lastmask() : 0xffffffffu;
}

// Names every run of zeros, and with ONES every run of ones: itself, or the
// frame for a zero run that touches the image border.
template <bool ONES>
__global__ void regions_init(Img img, int *__restrict__ L)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) L[0] = 0;
    if (i >= img.H * img.WW) return;
    const int y = i / img.WW, k = i % img.WW;
    const unsigned in = word_mask(img, k), v = img.w[i] & in, z = ~v & in;
    const int name = 1 + y * img.W + 32 * k;
    const bool edge_row = y == 0 || y == img.H - 1;
    for (unsigned m = run_starts(z); m; m &= m - 1) {
        const int p = __ffs(m) - 1;
        const bool edge = edge_row || (k == 0 && p == 0) ||
                          (k == img.WW - 1 && (run_mask(z, p) & ~(in >> 1)));   // holds the last column
        L[name + p] = edge ? 0 : name + p;
    }
    if (ONES)
        for (unsigned m = run_starts(v); m; m &= m - 1) {
            const int p = __ffs(m) - 1;
            L[name + p] = name + p;
        }
}

// Joins neighbouring runs: zeros 4-connected, ones 8-connected.
template <bool ONES>
__global__ void regions_join(Img img, int *L, int *flag)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= img.H * img.WW) return;
    const int WW = img.WW, W = img.W, y = i / WW, k = i % WW;
    const unsigned in = word_mask(img, k), v = img.w[i] & in, z = ~v & in;
    const int name = 1 + y * W + 32 * k;
    const unsigned pv = k > 0 ? img.w[i - 1] : 0u;           // word to the left (whole)
    const unsigned uv = y > 0 ? img.w[i - WW] & in : 0u, uz = y > 0 ? ~uv & in : 0u;
    if (k > 0 && (z & 1u) && !(pv >> 31)) uf_union(L, name, name - 32 + run_start(~pv, 31), flag);
    for (unsigned m = run_starts(z & uz); m; m &= m - 1) {
        const int p = __ffs(m) - 1;
        uf_union(L, name + run_start(z, p), name - W + run_start(uz, p), flag);
    }
    if (!ONES) return;
    if (k > 0 && (v & 1u) && (pv >> 31)) uf_union(L, name, name - 32 + run_start(pv, 31), flag);
    if (y == 0) return;
    const unsigned ul = k > 0 ? img.w[i - WW - 1] : 0u, ur = k < WW - 1 ? img.w[i - WW + 1] & word_mask(img, k + 1) : 0u;
    for (unsigned m = run_starts(v); m; m &= m - 1) {
        const int p = __ffs(m) - 1;
        const unsigned run = run_mask(v, p), near = run | (run << 1) | (run >> 1);
        for (unsigned t = run_starts(uv & near); t; t &= t - 1)
            uf_union(L, name + p, name - W + run_start(uv, __ffs(t) - 1), flag);
        if (p == 0 && (ul >> 31)) uf_union(L, name, name - W - 32 + run_start(ul, 31), flag);
        if ((run >> 31) && (ur & 1u)) uf_union(L, name + p, name - W + 32, flag);
    }
}

// imfill (morohutils.cu:73-83): F = B | (zeros of B that are not 4-connected
// to the zero frame around the image).
__global__ void fill_holes(Img B, int *L, Img F)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B.H * B.WW) return;
    const int y = i / B.WW, k = i % B.WW;
    const unsigned in = word_mask(B, k), z = ~B.w[i] & in;
    unsigned f = B.w[i] & in;
    for (unsigned m = run_starts(z); m; m &= m - 1) {
        const int p = __ffs(m) - 1;
        if (uf_find(L, 1 + y * B.W + 32 * k + p) != 0) f |= run_mask(z, p);
    }
    F.w[i] = f;
}

// --------------------------------------------------------------- morphology
// The openings on bit-packed rows, a launch for each step that needs its
// neighbours' results: the 30x1 opening stays inside a row, the 1x30 one inside
// a column of words, so each is one launch with a barrier between its erosion
// and dilation; the eye crosses both and takes two.  Bound by launch latency
// on a 512 x 512 thumbnail: 17 us in four launches, 65 in one CTA.

// AND (erode) or OR over the L pixels x - a .. x - a + L - 1 of a row for the
// 32 pixels x of word k, a = L / 2; outside the image the neutral value.
// L <= 32: by doubling on three words in registers.
__device__ __forceinline__ unsigned line_h(const Img &src, int y, int k, int L, bool erode)
{
    const unsigned fill = erode ? 0xffffffffu : 0u;
    const int a = L / 2;
    if (L > 32) {
        unsigned v = fill;
        for (int d = -a; d < L - a; ++d) {
            const unsigned t = src.shifted(y, k, d, fill);
            v = erode ? v & t : v | t;
        }
        return v;
    }
    unsigned lo = src.get(y, k - 1, fill), mid = src.get(y, k, fill), hi = src.get(y, k + 1, fill);
    if (!erode) { lo = ~lo; mid = ~mid; hi = ~hi; }          // OR of pixels = not AND of their complements
    for (int m = 1; m < L;) {                                // windows of m pixels from each pixel on
        const int s = min(m, L - m);
        lo &= __funnelshift_r(lo, mid, s);
        mid &= __funnelshift_r(mid, hi, s);
        hi &= __funnelshift_r(hi, 0xffffffffu, s);
        m += s;
    }
    const unsigned v = a ? __funnelshift_r(lo, mid, 32 - a) : mid;
    return erode ? v : ~v;
}

// Opening by L x 1: blockDim.x / WW whole rows a CTA (at least one).
__global__ void open_rows(Img src, Img tmp, Img dst, int L)
{
    const int WW = src.WW, per = max(1, (int)blockDim.x / WW), y0 = blockIdx.x * per;
    const int n = min(per, src.H - y0) * WW;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int y = y0 + i / WW, k = i % WW;
        tmp.w[y * WW + k] = line_h(src, y, k, L, true) & word_mask(src, k);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int y = y0 + i / WW, k = i % WW;
        dst.w[y * WW + k] = line_h(tmp, y, k, L, false) & word_mask(src, k);
    }
}

// O = opening of src by 1 x L, D = B - O (saturating): a CTA per column of
// words, in shared memory (2 H words).
__global__ void open_cols(Img src, Img B, Img O, Img D, int L)
{
    extern __shared__ unsigned col[];
    const int k = blockIdx.x, H = src.H, WW = src.WW, a = L / 2;
    unsigned *const er = col + H;
    for (int y = threadIdx.x; y < H; y += blockDim.x) col[y] = src.w[y * WW + k];
    __syncthreads();
    for (int y = threadIdx.x; y < H; y += blockDim.x) {
        unsigned v = 0xffffffffu;
        for (int r = max(y - a, 0); r < min(y + L - a, H); ++r) v &= col[r];
        er[y] = v;
    }
    __syncthreads();
    for (int y = threadIdx.x; y < H; y += blockDim.x) {
        unsigned v = 0;
        for (int r = max(y - a, 0); r < min(y + L - a, H); ++r) v |= er[r];
        O.w[y * WW + k] = v;
        D.w[y * WW + k] = B.w[y * WW + k] & ~v;
    }
}

// Erosion or dilation by the K x K eye (diagonal line).
template <bool ERODE>
__global__ void eye_pass(Img src, Img dst, int K)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, WW = src.WW;
    if (i >= src.H * WW) return;
    const int y = i / WW, k = i % WW, a = K / 2;
    unsigned v = ERODE ? 0xffffffffu : 0u;
    for (int t = 0; t < K; ++t) {
        const unsigned u = src.shifted(y + t - a, k, t - a, ERODE ? 0xffffffffu : 0u);
        v = ERODE ? v & u : v | u;
    }
    dst.w[i] = v & word_mask(src, k);
}

struct MorphArgs {
    Img B, F;                 // raster ("rev" image: set where the matrix has entries), filled
    Img O2, D, E;             // open-open, subtracted, eye-opened
    Img T1, T2;               // scratch
    int open_len, eye;
};

// Raster of the CSR to the five stage images in `a` (a.B .. a.E), with L
// (H * W + 1 ints) and *flag as scratch of the hole filling; *flag stays 0
// unless a union gave up.
tc_status thumbnail_stages(const int *d_rowptr, const int *d_col, int M, int pM, int pN, MorphArgs &a, int *L,
                           int *flag, cudaStream_t s)
{
    const int H = a.B.H, WW = a.B.WW, n = H * WW, T = 128;
    raster_kernel<<<H, 512, sizeof(unsigned) * WW, s>>>(d_rowptr, d_col, M, pM, pN, a.B);
    regions_init<false><<<(n + T - 1) / T, T, 0, s>>>(a.B, L);
    regions_join<false><<<(n + T - 1) / T, T, 0, s>>>(a.B, L, flag);
    fill_holes<<<(n + T - 1) / T, T, 0, s>>>(a.B, L, a.F);
    const int per = std::max(1, 256 / WW);
    open_rows<<<(H + per - 1) / per, 256, 0, s>>>(a.F, a.T2, a.T1, a.open_len);
    open_cols<<<WW, std::min(1024, (H + 31) & ~31), 2 * sizeof(unsigned) * (size_t)H, s>>>(a.T1, a.B, a.O2, a.D,
                                                                                         a.open_len);
    eye_pass<true><<<(n + T - 1) / T, T, 0, s>>>(a.D, a.T2, a.eye);
    eye_pass<false><<<(n + T - 1) / T, T, 0, s>>>(a.T2, a.E, a.eye);
    TC_CUDA(cudaGetLastError());
    return TC_OK;
}

// Bytes (nonzero = set) -> bits, and bits -> 0/255 bytes.
__global__ void pack_kernel(const unsigned char *__restrict__ in, Img img)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= img.H * img.WW) return;
    const int y = i / img.WW, k = i % img.WW;
    unsigned v = 0;
    for (int b = 0; b < 32; ++b) {
        const int x = k * 32 + b;
        if (x < img.W && in[(size_t)y * img.W + x]) v |= 1u << b;
    }
    img.w[i] = v;
}

__global__ void unpack_kernel(Img img, unsigned char *__restrict__ out)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long)img.H * img.W) return;
    const int y = (int)(i / img.W), x = (int)(i % img.W);
    out[i] = img.pix(y, x) ? 255 : 0;
}

// ----------------------------------------------------------------- contours
struct Border {
    int start;      // pixel index y*W+x
    int hole;       // 0 outer, 1 hole
    int parent;     // hole: start pixel of the enclosing outer border
    int len;        // points of the traced contour
    int mid;        // pixel index of point len/2
    long long area2;   // twice the signed area of the contour polygon (shoelace sum)
};

// Border starts of a word: the roots of ones (an outer border starts at a
// region's first pixel) and of zeros that are not the frame's (a hole's
// border starts at the pixel left of its first one).  Returns the word's
// outer starts; *holes: the first pixels of its holes.
__device__ __forceinline__ unsigned border_bits(const Img &img, int *L, int i, unsigned *holes)
{
    const int y = i / img.WW, k = i % img.WW;
    const unsigned in = word_mask(img, k), v = img.w[i] & in, z = ~v & in;
    const int name = 1 + y * img.W + 32 * k;
    unsigned o = 0, h = 0;
    for (unsigned m = run_starts(v); m; m &= m - 1) {
        const int p = __ffs(m) - 1;
        if (__ldcg(L + name + p) == name + p) o |= 1u << p;
    }
    for (unsigned m = run_starts(z); m; m &= m - 1) {
        const int p = __ffs(m) - 1;
        if (__ldcg(L + name + p) == name + p) h |= 1u << p;
    }
    *holes = h;
    return o;
}

__global__ void border_count(Img img, int *L, int *__restrict__ cnt)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, n = img.H * img.WW;
    if (i == n) cnt[n] = 0;
    if (i >= n) return;
    unsigned h;
    const unsigned o = border_bits(img, L, i, &h);
    cnt[i] = __popc(o) + __popc(h);
}

// The borders in discovery order, which is the raster order of their starts.
// (A hole's border starts one pixel before its first zero, but no other start
// lies between the two: the pixel is a one that is not its region's first.)
__global__ void border_write(Img img, int *L, const int *__restrict__ at, Border *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= img.H * img.WW) return;
    unsigned h;
    const unsigned o = border_bits(img, L, i, &h);
    const int y = i / img.WW, k = i % img.WW, first = y * img.W + 32 * k;
    int slot = at[i];
    for (unsigned m = o | h; m; m &= m - 1) {
        const int p = __ffs(m) - 1;
        Border b;
        b.hole = h >> p & 1u;
        b.start = first + p - b.hole;
        b.parent = -1;
        if (b.hole) {                                // the region of the one to its left
            const int lk = p ? k : k - 1, lp = (p + 31) & 31;
            b.parent = uf_find(L, 1 + y * img.W + 32 * lk + run_start(img.w[y * img.WW + lk], lp)) - 1;
        }
        b.len = 0;
        b.mid = b.start;
        b.area2 = 0;
        out[slot++] = b;
    }
}

// Directions: 0 = +x, counter-clockwise on screen (y grows downward).

// Three pixels (y, x - 1 .. x + 1): bits 0 .. 2.  From the image in global
// memory, or from a copy in shared memory with a zero row above and below and
// a zero word left and right.
struct GlobalPixels {
    Img img;
    __device__ __forceinline__ unsigned three(int y, int x) const
    {
        const int k = (x - 1) >> 5;
        return __funnelshift_r(img.get(y, k, 0u), img.get(y, k + 1, 0u), (x - 1) & 31) & 7u;
    }
};
struct SharedPixels {
    const unsigned *w;
    int stride;
    __device__ __forceinline__ unsigned three(int y, int x) const
    {
        const unsigned *r = w + (y + 1) * stride + ((x + 31) >> 5);
        return __funnelshift_r(r[0], r[1], (x + 31) & 31) & 7u;
    }
};

// A position on a border and the direction it was entered from (Suzuki & Abe
// steps 3.1-3.5).
struct Walk {
    int y, x, s;
    // bit d: the neighbour in direction d is set
    template <class P>
    static __device__ __forceinline__ unsigned around(const P &px, int y, int x)
    {
        const unsigned u = px.three(y - 1, x), m = px.three(y, x), d = px.three(y + 1, x);
        return (m >> 2) | (u & 4u) >> 1 | (u & 2u) << 1 | (u & 1u) << 3 | (m & 1u) << 4 | d << 5;
    }
    // To the first set neighbour counter-clockwise after direction s (there
    // is one: the pixel the walk came from).
    template <class P>
    __device__ __forceinline__ void step(const P &px)
    {
        const unsigned a = around(px, y, x);
        const int from = (s + 1) & 7;
        const unsigned turned = ((a | a << 8) >> from) & 0xffu;
        const int k = turned ? (from + __ffs(turned) - 1) & 7 : s;
        // dx = 1, 1, 0, -1, -1, -1, 0, 1 and dy = 0, -1, -1, -1, 0, 1, 1, 1, two bits each (value + 1)
        x += (int)(0x901au >> (2 * k) & 3u) - 1;
        y += (int)(0xa901u >> (2 * k) & 3u) - 1;
        s = (k + 4) & 7;
    }
    // The position that step() came from: one pixel back, and the first set
    // neighbour clockwise before the direction it left by.
    template <class P>
    __device__ __forceinline__ void back(const P &px)
    {
        x += (int)(0x901au >> (2 * s) & 3u) - 1;
        y += (int)(0xa901u >> (2 * s) & 3u) - 1;
        const unsigned a = around(px, y, x);
        const int d = (s + 4) & 7;
        const unsigned turned = ((a | a << 8) >> d) & 0xffu;
        s = (d + 31 - __clz(turned | 1u)) & 7;
    }
    __device__ __forceinline__ bool operator==(const Walk &o) const { return x == o.x && y == o.y && s == o.s; }
};

// Follows one border: its length, middle point and polygon area.  Two walks
// leave the start, one forwards and one backwards (a step can be undone: see
// Walk::back), and meet half-way round, where point len / 2 is.
template <class P>
__device__ void follow(const P &px, int W, long cap, Border &b, int *flag)
{
    const int sy = b.start / W, sx = b.start % W;
    const int s0 = b.hole ? 0 : 4;
    const unsigned a = Walk::around(px, sy, sx);
    int s = s0;
    bool found = false;
    for (int t = 0; t < 8 && !found; ++t) {          // clockwise from the outside pixel
        s = (s - 1) & 7;
        found = a >> s & 1u;
    }
    b.len = 1;
    b.mid = b.start;
    if (!found) return;                              // a single pixel
    Walk f{sy, sx, s}, g = f;
    long long area = 0;
    for (long n = 1; n <= cap; n += 2) {
        const Walk f0 = f, g0 = g;
        f.step(px);
        g.back(px);
        area += (long long)f0.x * f.y - (long long)f.x * f0.y;
        if (f == g0) {                               // n steps round
            b.len = (int)n;
            b.mid = f0.y * W + f0.x;
            b.area2 = area;
            return;
        }
        area += (long long)g.x * g0.y - (long long)g0.x * g.y;
        if (f == g) {                                // n + 1
            b.len = (int)n + 1;
            b.mid = f.y * W + f.x;
            b.area2 = area;
            return;
        }
    }
    *flag = 3;   // longer than any border can be: reported
}

// One thread per border: bound by the longest border, each of whose steps
// waits on the one before.  A step waits on the image alone (two or three words
// of three rows), so the image is copied to shared memory when it fits
// (`shared`): a 512 x 512 thumbnail takes 35 KB, the eight neighbours come
// from three reads, and two walks share the way.  On the 9-point mesh's
// thumbnail: 787 us with one pixel test at a time and a second round for the
// middle, 209 with a second walk at half the pace, 100 from both ends.
constexpr int kTraceBlock = 256;

__global__ void __launch_bounds__(kTraceBlock) trace_kernel(Img img, Border *__restrict__ bs,
                                                            const int *__restrict__ count, int shared, int *flag)
{
    extern __shared__ unsigned sp[];
    const int nb = *count;
    if ((int)(blockIdx.x * blockDim.x) >= nb) return;
    const int stride = img.WW + 3;                   // a word each side, and one more for the last pair
    if (shared) {
        const int n = stride * (img.H + 2);
        for (int i = threadIdx.x; i < n; i += blockDim.x) sp[i] = img.get(i / stride - 1, i % stride - 1, 0u);
        __syncthreads();
    }
    const long cap = 8L * img.H * img.W + 16;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += gridDim.x * blockDim.x) {
        Border b = bs[i];
        if (shared) follow(SharedPixels{sp, stride}, img.W, cap, b, flag);
        else follow(GlobalPixels{img}, img.W, cap, b, flag);
        bs[i] = b;
    }
}

// ------------------------------------------------------------------ shapes
__device__ __forceinline__ bool is_unclaimed(float v)
{
    const float d = v - FLT_MAX;          // TaiChi.cu:730
    return fabs((double)d) > 1e-8;
}

__global__ void claim_init(const float *__restrict__ val, unsigned char *__restrict__ claimed, long nnz)
{
    const long j = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < nnz) claimed[j] = is_unclaimed(val[j]) ? 0 : 1;
}

struct ShapeBox {
    int x, y, a, b;   // row / column corner, column extent (a) and row extent (b)
    int w;            // band half-width
    int nd;           // 2w - 1 candidate diagonals
};

// The boxes of a launch of band_hist: row blockIdx.y of the grid counts b[y]
// into cnt[at[y]] on.
constexpr int kHistBoxes = 32;
struct HistBoxes {
    ShapeBox b[kHistBoxes];
    int at[kHistBoxes];
};

// Per-diagonal counts of unclaimed entries inside each box and its band
// (TaiChi.cu:723-734); one thread per row of the box, four of its entries in
// flight (9-point mesh 2048^2: 78 -> 57 us), all boxes in one launch (15 of
// R-MAT scale 20 with self loops: 86 us in a launch each, 38 in one).
constexpr int kHistLocal = 8192;     // most diagonals counted in shared memory
__global__ void band_hist(const int *__restrict__ rowptr, const int *__restrict__ col,
                          const unsigned char *__restrict__ claimed, const __grid_constant__ HistBoxes boxes,
                          unsigned *__restrict__ cnt_all)
{
    extern __shared__ unsigned sh[];
    const ShapeBox sb = boxes.b[blockIdx.y];
    unsigned *const cnt = cnt_all + boxes.at[blockIdx.y];
    if ((long)blockIdx.x * blockDim.x >= sb.b) return;
    const bool local = sb.nd <= kHistLocal;
    if (local) {
        for (int i = threadIdx.x; i < sb.nd; i += blockDim.x) sh[i] = 0;
        __syncthreads();
    }
    const int dof = sb.y - sb.x;
    for (long r = (long)blockIdx.x * blockDim.x + threadIdx.x + sb.x; r < (long)sb.x + sb.b;
         r += (long)gridDim.x * blockDim.x) {
        const int b = __ldg(rowptr + r), e = __ldg(rowptr + r + 1);
        const long lo = r + dof - sb.w + 1, hi = r + dof + sb.w - 1;
        for (Words a(b, e); a.left > 0; a.skip(4)) {
            int c[4];
            unsigned char k[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                c[u] = u < a.left ? __ldg(col + a.at + u) : -1;
                k[u] = u < a.left ? claimed[a.at + u] : 1;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (c[u] < sb.y || c[u] >= sb.y + sb.a || c[u] < lo || c[u] > hi || k[u]) continue;
                const int n = (int)(c[u] - r - dof + sb.w - 1);
                if (local) atomicAdd(sh + n, 1u);
                else atomicAdd(cnt + n, 1u);
            }
        }
    }
    if (local) {
        __syncthreads();
        for (int i = threadIdx.x; i < sb.nd; i += blockDim.x)
            if (sh[i]) atomicAdd(cnt + i, sh[i]);
    }
}

// Claims the entries of the dense diagonals (TaiChi.cu:848-874) with the
// shape's mark, one thread per row of the box, and notes the diagonals each
// row has an entry on: bit d & 31 of found[(d >> 5) * b + local row].  The
// row's words belong to its thread alone.  *dup: a row met a diagonal twice.
__global__ void band_claim(const int *__restrict__ rowptr, const int *__restrict__ col,
                           unsigned char *__restrict__ claimed, ShapeBox sb,
                           const int *__restrict__ dense_idx, unsigned char mark,
                           unsigned *__restrict__ found, int *__restrict__ dup)
{
    const int dof = sb.y - sb.x;
    for (long r = (long)blockIdx.x * blockDim.x + threadIdx.x + sb.x; r < (long)sb.x + sb.b;
         r += (long)gridDim.x * blockDim.x) {
        const int b = __ldg(rowptr + r), e = __ldg(rowptr + r + 1);
        const long lo = r + dof - sb.w + 1, hi = r + dof + sb.w - 1;
        unsigned bits = 0;
        int at = 0;                                  // the word that `bits` goes to
        auto flush = [&] {
            if (!bits) return;
            unsigned *const f = found + (long)at * sb.b + (r - sb.x);
            const unsigned old = *f;
            if (old & bits) *dup = 1;
            *f = old | bits;
            bits = 0;
        };
        for (Words a(b, e); a.left > 0; a.skip(4)) {
            int dd[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = u < a.left ? __ldg(col + a.at + u) : -1;
                const bool in = c >= sb.y && c < sb.y + sb.a && c >= lo && c <= hi && !claimed[a.at + u];
                dd[u] = in ? __ldg(dense_idx + (c - r - dof + sb.w - 1)) : -1;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int d = dd[u];
                if (d < 0) continue;
                claimed[a.at + u] = mark;
                if (d >> 5 != at) {
                    flush();
                    at = d >> 5;
                }
                if (bits >> (d & 31) & 1u) *dup = 1;
                bits |= 1u << (d & 31);
            }
        }
        flush();
    }
}

// Found bits to hole bits, in place: diagonal d has a hole in every local
// row of [start[d], end[d]) without an entry on it.
__global__ void hole_bits(unsigned *__restrict__ bits, int b, int neg, const int2 *__restrict__ range)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const int words = (neg + 31) >> 5;
    if (i >= (long)words * b) return;
    const int w = (int)(i / b), r = (int)(i % b);
    unsigned in = 0;
    for (int d = 32 * w; d < min(neg, 32 * w + 32); ++d) {
        const int2 se = __ldg(range + d);
        if (r >= se.x && r < se.y) in |= 1u << (d & 31);
    }
    bits[i] = in & ~bits[i];
}

// Duplicate entries: the reference's row walk (TaiChi.cu:809-827) consumes one
// listed entry per row once the row reaches it; a row is a hole when no entry
// is pending, and at most keep[d] holes are kept.  The entries per diagonal
// and row, then a sequential walk per diagonal (only run when duplicates
// exist).
__global__ void dup_counts(const int *__restrict__ rowptr, const int *__restrict__ col,
                           const unsigned char *__restrict__ claimed, ShapeBox sb,
                           const int *__restrict__ dense_idx, unsigned char mark, int *__restrict__ rowcnt)
{
    const int dof = sb.y - sb.x;
    for (long r = (long)blockIdx.x * blockDim.x + threadIdx.x + sb.x; r < (long)sb.x + sb.b;
         r += (long)gridDim.x * blockDim.x)
        for (int j = __ldg(rowptr + r); j < __ldg(rowptr + r + 1); ++j)
            if (claimed[j] == mark)                  // an entry of this shape
                rowcnt[(long)dense_idx[__ldg(col + j) - r - dof + sb.w - 1] * sb.b + (r - sb.x)] += 1;
}

__global__ void dup_holes(const int *__restrict__ rowcnt, int b, int neg, const int2 *__restrict__ range,
                          const int *__restrict__ keep, unsigned *__restrict__ bits)
{
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= neg) return;
    unsigned *const w = bits + (long)(d >> 5) * b;
    const unsigned bit = 1u << (d & 31);
    long pending = 0;
    int made = 0;
    for (int r = 0; r < b; ++r) {
        bool hole = false;
        if (r >= range[d].x && r < range[d].y) {
            pending += rowcnt[(long)d * b + r];
            if (pending > 0) --pending;
            else hole = made++ < keep[d];
        }
        if (hole) atomicOr(w + r, bit);              // a word holds 32 diagonals
        else atomicAnd(w + r, ~bit);
    }
}

// Any mark to 1, so that the marks can be given out again.
__global__ void settle_marks(unsigned char *__restrict__ claimed, long nnz)
{
    const long j = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < nnz && claimed[j]) claimed[j] = 1;
}

// --------------------------------------------------------------- assembly
// A shape with dense diagonals, for the assembly: rows [x, x + b), columns
// from y, `neg` diagonals from offset index `off0` on, hole bits as in
// hole_bits().
struct HoleShape {
    int x, y, b, neg, off0;
    const unsigned *bits;
};

// Row lengths of the remainder: the row's holes and its unclaimed entries.
__global__ void remainder_counts(const int *__restrict__ rowptr, const unsigned char *__restrict__ claimed,
                                 const HoleShape *__restrict__ shapes, int nshapes, int M, int *__restrict__ cnt)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < M; r += gridDim.x * blockDim.x) {
        int n = 0;
        for (int s = 0; s < nshapes; ++s) {
            const HoleShape h = shapes[s];
            if (r < h.x || r >= h.x + h.b) continue;
            for (int w = 0; w < (h.neg + 31) >> 5; ++w) n += __popc(__ldg(h.bits + (long)w * h.b + (r - h.x)));
        }
        const int e = __ldg(rowptr + r + 1);
        for (int j = __ldg(rowptr + r); j < e; ++j) n += !__ldg(claimed + j);
        cnt[r] = n;
    }
}

// The remainder's words: per row its holes (shape order, offset order), then
// its unclaimed entries (CSR order).
__global__ void remainder_words(const int *__restrict__ rowptr, const int *__restrict__ col,
                                const unsigned char *__restrict__ claimed, const HoleShape *__restrict__ shapes,
                                int nshapes, const int *__restrict__ offs, int M,
                                const int *__restrict__ rp_out, int *__restrict__ cols)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < M; r += gridDim.x * blockDim.x) {
        int at = __ldg(rp_out + r);
        for (int s = 0; s < nshapes; ++s) {
            const HoleShape h = shapes[s];
            if (r < h.x || r >= h.x + h.b) continue;
            const int rs = r - h.x;
            for (int w = 0; w < (h.neg + 31) >> 5; ++w)
                for (unsigned m = __ldg(h.bits + (long)w * h.b + rs); m; m &= m - 1)
                    cols[at++] = (h.y + rs + __ldg(offs + h.off0 + 32 * w + __ffs(m) - 1)) << 1;
        }
        const int e = __ldg(rowptr + r + 1);
        for (int j = __ldg(rowptr + r); j < e; ++j)
            if (!__ldg(claimed + j)) cols[at++] = (__ldg(col + j) << 1) + 1;
    }
}

inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }

// Input check: rowptr[0] == 0, non-decreasing, rowptr[M] == nnz, 0 <= col < N.
__global__ void validate_csr(const int *__restrict__ rowptr, const int *__restrict__ col, int M,
                             int N, long nnz, int *__restrict__ bad)
{
    const long stride = (long)gridDim.x * blockDim.x;
    for (long r = (long)blockIdx.x * blockDim.x + threadIdx.x; r < M; r += stride)
        if (rowptr[r + 1] < rowptr[r]) atomicOr(bad, 1);
    for (long j = (long)blockIdx.x * blockDim.x + threadIdx.x; j < nnz; j += stride) {
        const int c = col[j];
        if (c < 0 || c >= N) atomicOr(bad, 2);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && (rowptr[0] != 0 || rowptr[M] != nnz)) atomicOr(bad, 4);
}

int band_width(int s)     // TaiChi.cu:689-699
{
    double w;
    if (s >= 10000000) w = s * 0.000001;
    else if (s >= 1000000) w = s * 0.00001;
    else if (s >= 100000) w = s * 0.001;
    else if (s >= 10000) w = s * 0.01;
    else w = s * 0.1;
    return (int)w;
}

void start_end(int M_sub, int N_sub, int width, int off, int n, int &start, int &end)   // TaiChi.cu:881-916
{
    const int ao = off < 0 ? -off : off;
    if (M_sub >= N_sub) {
        if (n >= width - 1) { start = 0; end = N_sub - off; }
        else if (ao > M_sub - N_sub) { start = ao; end = M_sub; }
        else { start = ao; end = N_sub + ao; }
    } else {
        if (n <= width - 1) { start = ao; end = M_sub; }
        else if (ao > N_sub - M_sub) { start = 0; end = N_sub - ao; }
        else { start = 0; end = M_sub; }
    }
}

void shape_size(int M, int N, int mF, int x1, int y1, int a1, int b1, int &x, int &y, int &a, int &b)
{   // TaiChi.cu:280-311
    if (M > mF) {
        const float g = (float)M / (float)mF;
        x = (int)((float)x1 * g); y = (int)((float)y1 * g);
        a = (int)((float)a1 * g); b = (int)((float)b1 * g);
    } else if (M < mF) {
        const float g = (float)mF / (float)M;
        x = (int)((float)x1 / g); y = (int)((float)y1 / g);
        a = (int)((float)a1 / g); b = (int)((float)b1 / g);
    } else {
        x = x1; y = y1; a = a1; b = b1;
    }
    if (x < 0) x = 0;
    if (x > M - 1) x = M - 1;
    if (y < 0) y = 0;
    if (y > N - 1) y = N - 1;
    if (y + a > N) a = N - y;
    if (x + b > M) b = M - x;
    if (a > b) a = b; else b = a;
}

}  // namespace

// ======================================================================
// Contours of a bit image already on the device: ordered (len, start, mid).
// ======================================================================
struct ContourList {
    std::vector<int> lens, first, mid;   // pixel indices y*W+x
    std::vector<long long> area2;        // twice the polygon area (signed)
};

static tc_status contours_on_device(const Img &img, cudaStream_t s, ContourList &out)
{
    const int n = img.H * img.WW, T = 128;
    const long px = (long)img.H * img.W;
    // no two border starts are neighbours in a row (an outer one and a hole's
    // first pixel would share a corner with a one above)
    const long most = (long)img.H * ((img.W + 1) / 2);
    Scratch lab, cnt, tmp, bord, flag;
    TC_CHECK(lab.alloc(sizeof(int) * ((size_t)px + 1), s));
    TC_CHECK(cnt.alloc(sizeof(int) * 2 * ((size_t)n + 1), s));
    TC_CHECK(tmp.alloc(sizeof(int) * scan_tmp_ints(n), s));
    TC_CHECK(bord.alloc(sizeof(Border) * (size_t)most, s));
    TC_CHECK(flag.alloc(sizeof(int), s));
    int *const L = lab.as<int>(), *const at = cnt.as<int>() + n + 1;
    TC_CUDA(cudaMemsetAsync(flag.p, 0, sizeof(int), s));
    regions_init<true><<<cdiv(n, T), T, 0, s>>>(img, L);
    regions_join<true><<<cdiv(n, T), T, 0, s>>>(img, L, flag.as<int>());
    border_count<<<cdiv(n + 1, T), T, 0, s>>>(img, L, cnt.as<int>());
    TC_CUDA(cudaGetLastError());
    TC_CHECK(exclusive_scan(cnt.as<int>(), at, n, tmp.as<int>(), s));
    border_write<<<cdiv(n, T), T, 0, s>>>(img, L, at, bord.as<Border>());
    const size_t smem = sizeof(unsigned) * (size_t)(img.WW + 3) * (img.H + 2);
    const int shared = smem <= 200 * 1024;
    if (shared) TC_CHECK(ensure_smem((const void *)trace_kernel, smem));
    const int grid = (int)std::min<long>((most + kTraceBlock - 1) / kTraceBlock, num_sms());
    trace_kernel<<<grid, kTraceBlock, shared ? smem : 0, s>>>(img, bord.as<Border>(), at + n, shared, flag.as<int>());
    TC_CUDA(cudaGetLastError());
    int nb = 0, hflag = 0;
    std::vector<Border> hb((size_t)std::min(most, 2048L));   // usually all of them, in one round trip
    TC_CUDA(cudaMemcpyAsync(&nb, at + n, sizeof(int), cudaMemcpyDeviceToHost, s));
    TC_CUDA(cudaMemcpyAsync(&hflag, flag.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    TC_CUDA(cudaMemcpyAsync(hb.data(), bord.p, sizeof(Border) * hb.size(), cudaMemcpyDeviceToHost, s));
    TC_CUDA(cudaStreamSynchronize(s));
    const size_t have = hb.size();
    hb.resize(nb);
    if ((size_t)nb > have) {
        TC_CUDA(cudaMemcpyAsync(hb.data() + have, bord.as<Border>() + have, sizeof(Border) * (nb - have),
                                cudaMemcpyDeviceToHost, s));
        TC_CUDA(cudaStreamSynchronize(s));
    }
    if (hflag) return fail(TC_ERR_UNSUPPORTED, "contour labelling gave up (code %d)", hflag);
    // OpenCV order: outer borders newest first, each followed by its holes
    // newest first.  hb is in discovery order.
    std::vector<int> head(nb, -1), next(nb, -1);
    {
        // outer start pixels are unique and sorted (discovery order)
        std::vector<std::pair<int, int>> os;
        for (int i = 0; i < nb; ++i)
            if (!hb[i].hole) os.push_back({hb[i].start, i});
        for (int i = 0; i < nb; ++i) {
            if (!hb[i].hole) continue;
            auto it = std::lower_bound(os.begin(), os.end(), std::make_pair(hb[i].parent, -1));
            if (it == os.end() || it->first != hb[i].parent)
                return fail(TC_ERR_FORMAT, "hole border without an outer border");
            const int p = it->second;
            next[i] = head[p];
            head[p] = i;
        }
    }
    out.lens.clear(); out.first.clear(); out.mid.clear(); out.area2.clear();
    auto put = [&](const Border &b) {
        out.lens.push_back(b.len); out.first.push_back(b.start); out.mid.push_back(b.mid);
        out.area2.push_back(b.area2);
    };
    for (int i = nb - 1; i >= 0; --i) {
        if (hb[i].hole) continue;
        put(hb[i]);
        for (int j = head[i]; j >= 0; j = next[j]) put(hb[j]);
    }
    return TC_OK;
}


// ======================================================================
// getSdf on the device
// ======================================================================
struct SdfOut {
    int mF = 0, W = 0;
    std::vector<int> corners;               // 4 per kept contour
    std::vector<double> widths;             // per kept contour: area / corner distance
    std::vector<unsigned char> stages;      // 5*H*W when requested
    int ncontours = 0;                      // all contours before the length filter
};

static tc_status getsdf_device(int M, int N, const int *d_rowptr, const int *d_col, const tc_params &p,
                               bool keep_stages, cudaStream_t s, SdfOut &out)
{
    const int H = p.thumb_height;
    out = SdfOut();
    if (M <= H) return TC_OK;                 // morohutils.cu:192-196: no thumbnail
    const int pM = M / H;
    const double scale = (double)H / (double)M;
    const int W = (int)(scale * N);
    if (W <= 0) return fail(TC_ERR_UNSUPPORTED, "thumbnail width is 0 (N < M/%d)", H);
    if ((long)H * W > (1L << 26)) return fail(TC_ERR_UNSUPPORTED, "thumbnail %d x %d too large", H, W);
    const int pN = N / W;
    const int WW = (W + 31) / 32;
    const size_t nw = (size_t)H * WW;
    Scratch imgs, lab, flag;
    TC_CHECK(imgs.alloc(sizeof(unsigned) * nw * 7, s));
    TC_CHECK(lab.alloc(sizeof(int) * ((size_t)H * W + 1), s));
    TC_CHECK(flag.alloc(sizeof(int), s));
    TC_CUDA(cudaMemsetAsync(flag.p, 0, sizeof(int), s));
    auto img = [&](int k) { return Img{imgs.as<unsigned>() + k * nw, H, W, WW}; };
    MorphArgs a;
    a.B = img(0); a.F = img(1); a.O2 = img(2); a.D = img(3); a.E = img(4);
    a.T1 = img(5); a.T2 = img(6);
    a.open_len = p.open_len;
    a.eye = p.eye_size;
    TC_CHECK(thumbnail_stages(d_rowptr, d_col, M, pM, pN, a, lab.as<int>(), flag.as<int>(), s));
    ContourList cl;
    TC_CHECK(contours_on_device(a.E, s, cl));
    int hflag = 0;
    TC_CUDA(cudaMemcpyAsync(&hflag, flag.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    TC_CUDA(cudaStreamSynchronize(s));
    if (hflag) return fail(TC_ERR_UNSUPPORTED, "hole fill gave up (code %d)", hflag);
    out.mF = H;
    out.W = W;
    out.ncontours = (int)cl.lens.size();
    for (size_t i = 0; i < cl.lens.size(); ++i) {
        if (cl.lens[i] < p.min_contour) continue;           // morohutils.cu:138-151
        out.corners.push_back(cl.first[i] % W);             // contour[0].x (column)
        out.corners.push_back(cl.first[i] / W);             // contour[0].y (row)
        out.corners.push_back(cl.mid[i] % W);               // contour[size/2]
        out.corners.push_back(cl.mid[i] / W);
        // morohutils.cu:268-272: contourArea(contour) / |contour[0] - contour[size/2]|
        const double dx = cl.first[i] % W - cl.mid[i] % W, dy = cl.first[i] / W - cl.mid[i] / W;
        const double area = 0.5 * std::fabs((double)cl.area2[i]);
        out.widths.push_back(area / std::sqrt(dx * dx + dy * dy));
    }
    if (keep_stages) {
        Scratch bytes;
        const size_t px = (size_t)H * W;
        TC_CHECK(bytes.alloc(px * 5, s));
        for (int k = 0; k < 5; ++k)
            unpack_kernel<<<cdiv((long)px, 256), 256, 0, s>>>(img(k), bytes.as<unsigned char>() + k * px);
        out.stages.resize(px * 5);
        TC_CUDA(cudaMemcpyAsync(out.stages.data(), bytes.p, px * 5, cudaMemcpyDeviceToHost, s));
        TC_CUDA(cudaStreamSynchronize(s));
    }
    return TC_OK;
}

// ======================================================================
// Shapes: dense diagonals, claims, holes (TaiChi.cu:677-879)
// ======================================================================
struct ShapeResult {
    ShapeBox box{};
    int neg = 0;                     // dense diagonals
    long nnz = 0;
    int cnt0 = 0;                    // its counts' place in the shared histogram
    std::vector<int> offs, start, end, nzero;
    std::vector<int> dense_idx;      // of each candidate diagonal, -1: not dense
    unsigned char mark = 0;          // of its entries among the claims
    Scratch tab;                     // device: dense_idx, ranges {start, end}, nzero, dup flag
    Scratch bits;                    // hole bits (see hole_bits)
};

static int box_grid(const ShapeBox &sb) { return std::max(1, std::min(cdiv(sb.b, 256), num_sms() * 8)); }

// The box of a shape; nd <= 0 or b <= 0: no diagonal can be dense.
static ShapeBox shape_box(int x, int y, int a, int b)
{
    const int w = band_width(b < a ? b : a);
    return ShapeBox{x, y, a, b, w, 2 * w - 1};
}

// Which diagonals are dense (TaiChi.cu:740-760), from the box's counts.
static void dense_diagonals(const unsigned *cnt, double density, ShapeResult &R)
{
    const ShapeBox &sb = R.box;
    R.dense_idx.assign(sb.nd, -1);
    for (int n = 0; n < sb.nd; ++n) {
        const int off = n - sb.w + 1;
        int st, en;
        start_end(sb.b, sb.a, sb.w, off, n, st, en);
        const float dens = (float)cnt[n] / (float)(en - st);
        if ((double)dens >= density) {           // TaiChi.cu:756-757
            R.dense_idx[n] = R.neg++;
            R.offs.push_back(off);
            R.start.push_back(st);
            R.end.push_back(en);
            R.nzero.push_back(en - st - (int)cnt[n]);
            R.nnz += cnt[n];
        }
    }
}

// Where the parts of ShapeResult::tab start (ints).
static size_t tab_range(const ShapeResult &R) { return ((size_t)R.box.nd + 1) & ~(size_t)1; }
static size_t tab_keep(const ShapeResult &R) { return tab_range(R) + 2 * (size_t)R.neg; }
static size_t tab_dup(const ShapeResult &R) { return tab_keep(R) + (size_t)R.neg; }

// Claims the shape's dense entries and finds its holes, taking the entries
// for free of duplicates (R.tab's dup flag says whether they were).
static tc_status claim_shape(const int *d_rowptr, const int *d_col, unsigned char *d_claim, cudaStream_t s,
                             ShapeResult &R)
{
    const ShapeBox &sb = R.box;
    std::vector<int> tab(tab_dup(R) + 1, 0);
    std::copy(R.dense_idx.begin(), R.dense_idx.end(), tab.begin());
    for (int d = 0; d < R.neg; ++d) {
        tab[tab_range(R) + 2 * d] = R.start[d];
        tab[tab_range(R) + 2 * d + 1] = R.end[d];
        tab[tab_keep(R) + d] = R.nzero[d];
    }
    const size_t words = (size_t)((R.neg + 31) / 32) * sb.b;
    TC_CHECK(R.tab.alloc(sizeof(int) * tab.size(), s));
    TC_CHECK(R.bits.alloc(sizeof(unsigned) * words, s));
    TC_CUDA(cudaMemcpyAsync(R.tab.p, tab.data(), sizeof(int) * tab.size(), cudaMemcpyHostToDevice, s));
    TC_CUDA(cudaMemsetAsync(R.bits.p, 0, sizeof(unsigned) * words, s));
    int *const t = R.tab.as<int>();
    band_claim<<<box_grid(sb), 256, 0, s>>>(d_rowptr, d_col, d_claim, sb, t, R.mark, R.bits.as<unsigned>(),
                                            t + tab_dup(R));
    hole_bits<<<cdiv((long)words, 256), 256, 0, s>>>(R.bits.as<unsigned>(), sb.b, R.neg,
                                                     reinterpret_cast<const int2 *>(t + tab_range(R)));
    TC_CUDA(cudaGetLastError());
    return TC_OK;
}

// Redoes the holes of a shape whose rows hold duplicate entries, if it does.
static tc_status settle_duplicates(const int *d_rowptr, const int *d_col, const unsigned char *d_claim,
                                   cudaStream_t s, ShapeResult &R)
{
    int *const t = R.tab.as<int>();
    int dup = 0;
    TC_CUDA(cudaMemcpyAsync(&dup, t + tab_dup(R), sizeof(int), cudaMemcpyDeviceToHost, s));
    TC_CUDA(cudaStreamSynchronize(s));
    if (!dup) return TC_OK;
    Scratch rowcnt;
    const size_t bytes = sizeof(int) * (size_t)R.neg * R.box.b;
    TC_CHECK(rowcnt.alloc(bytes, s));
    TC_CUDA(cudaMemsetAsync(rowcnt.p, 0, bytes, s));
    dup_counts<<<box_grid(R.box), 256, 0, s>>>(d_rowptr, d_col, d_claim, R.box, t, R.mark, rowcnt.as<int>());
    dup_holes<<<cdiv(R.neg, 32), 32, 0, s>>>(rowcnt.as<int>(), R.box.b, R.neg,
                                            reinterpret_cast<const int2 *>(t + tab_range(R)), t + tab_keep(R),
                                            R.bits.as<unsigned>());
    TC_CUDA(cudaGetLastError());
    return TC_OK;
}

// The counts of shapes [i, stop), at most kHistBoxes of them.
static tc_status launch_hist(const int *d_rowptr, const int *d_col, const unsigned char *d_claim,
                             const std::vector<ShapeResult> &shapes, size_t i, size_t stop, unsigned *cnt,
                             cudaStream_t s)
{
    HistBoxes h{};
    int grid = 1, most = 0;
    for (size_t k = i; k < stop; ++k) {
        h.b[k - i] = shapes[k].box;
        h.at[k - i] = shapes[k].cnt0;
        grid = std::max(grid, box_grid(shapes[k].box));
        if (shapes[k].box.nd <= kHistLocal) most = std::max(most, shapes[k].box.nd);
    }
    band_hist<<<dim3((unsigned)grid, (unsigned)(stop - i)), 256, sizeof(unsigned) * (size_t)most, s>>>(
        d_rowptr, d_col, d_claim, h, cnt);
    TC_CUDA(cudaGetLastError());
    return TC_OK;
}

// The shapes in order (TaiChi.cu:361-421).  A shape's counts see the claims
// of the shapes before it, so they are taken for up to kHistBoxes shapes at
// once and taken again for the rest after a shape that claims.
constexpr int kMarks = 250;          // marks 2 .. 251; 1: claimed earlier

static tc_status process_shapes(const int *d_rowptr, const int *d_col, unsigned char *d_claim, int64_t nnz,
                                double density, cudaStream_t s, std::vector<ShapeResult> &shapes)
{
    const size_t n = shapes.size();
    Scratch cnt;
    std::vector<unsigned> hc;
    std::vector<ShapeResult *> open;             // claimed since the marks were last settled
    auto settle = [&](bool marks) -> tc_status {
        for (ShapeResult *R : open) TC_CHECK(settle_duplicates(d_rowptr, d_col, d_claim, s, *R));
        open.clear();
        if (marks && nnz) settle_marks<<<cdiv(nnz, 256), 256, 0, s>>>(d_claim, nnz);
        return TC_OK;
    };
    for (size_t i = 0; i < n;) {
        const size_t stop = std::min(n, i + kHistBoxes);
        int total = 0;
        for (size_t k = i; k < stop; ++k) {
            shapes[k].cnt0 = total;
            total += shapes[k].box.nd;
        }
        TC_CHECK(cnt.alloc(sizeof(unsigned) * (size_t)total, s));
        TC_CUDA(cudaMemsetAsync(cnt.p, 0, sizeof(unsigned) * (size_t)total, s));
        TC_CHECK(launch_hist(d_rowptr, d_col, d_claim, shapes, i, stop, cnt.as<unsigned>(), s));
        hc.resize(total);
        TC_CUDA(cudaMemcpyAsync(hc.data(), cnt.p, sizeof(unsigned) * (size_t)total, cudaMemcpyDeviceToHost, s));
        TC_CUDA(cudaStreamSynchronize(s));
        for (bool claimed = false; i < stop && !claimed; ++i) {
            ShapeResult &R = shapes[i];
            dense_diagonals(hc.data() + R.cnt0, density, R);
            if (R.neg == 0) continue;
            if (open.size() == kMarks) TC_CHECK(settle(true));
            R.mark = (unsigned char)(2 + open.size());
            TC_CHECK(claim_shape(d_rowptr, d_col, d_claim, s, R));
            open.push_back(&R);
            claimed = true;
        }
    }
    return settle(false);
}

// ======================================================================
// The whole partition
// ======================================================================
tc_status gpu_partition(int M, int N, int64_t nnz, const int *d_rowptr, const int *d_col,
                        const float *d_val, const tc_params &prm, bool keep_stages,
                        bool want_claimed, cudaStream_t s, PartitionOut &out)
{
    auto t0 = std::chrono::steady_clock::now();
    if (M < 0 || N < 0 || nnz < 0) return fail(TC_ERR_INVALID, "negative sizes");
    Scratch claim, bad;
    TC_CHECK(claim.alloc((size_t)std::max<int64_t>(nnz, 1), s));
    TC_CHECK(bad.alloc(sizeof(int), s));
    const int T = 256;
    TC_CUDA(cudaMemsetAsync(bad.p, 0, sizeof(int), s));
    validate_csr<<<std::max(1, std::min(cdiv(std::max<long>(nnz, M), T), num_sms() * 16)), T, 0, s>>>(
        d_rowptr, d_col, M, N, nnz, bad.as<int>());
    int hbad = 0;
    TC_CUDA(cudaMemcpyAsync(&hbad, bad.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    TC_CUDA(cudaStreamSynchronize(s));
    if (hbad) return fail(TC_ERR_FORMAT, "invalid CSR input (code %d: 1 rowptr decreases, 2 column "
                                         "outside [0, N), 4 rowptr[0]/rowptr[M] wrong)", hbad);
    if (nnz && d_val) claim_init<<<cdiv(nnz, T), T, 0, s>>>(d_val, claim.as<unsigned char>(), nnz);
    else TC_CUDA(cudaMemsetAsync(claim.p, 0, (size_t)std::max<int64_t>(nnz, 1), s));
    TC_CUDA(cudaGetLastError());

    SdfOut sdf;
    TC_CHECK(getsdf_device(M, N, d_rowptr, d_col, prm, keep_stages, s, sdf));
    out.thumb_W = sdf.W;
    out.thumb_H = sdf.mF ? prm.thumb_height : 0;
    out.corners = sdf.corners;
    out.stages.swap(sdf.stages);
    out.ncontours = sdf.ncontours;

    std::vector<ShapeBox> boxes;
    for (size_t i = 0; i + 3 < sdf.corners.size(); i += 4) {     // TaiChi.cu:361-421, in shape order
        const int x1 = sdf.corners[i], y1 = sdf.corners[i + 1];
        int x, y, a, b;
        shape_size(M, N, sdf.mF, x1, y1, sdf.corners[i + 2] - x1, sdf.corners[i + 3] - y1, x, y, a, b);
        if (a < prm.min_shape_side || b < prm.min_shape_side) continue;
        const ShapeBox sb = shape_box(x, y, a, b);
        if (sb.nd > 0 && sb.b > 0) boxes.push_back(sb);
    }
    std::vector<ShapeResult> shapes(boxes.size());
    for (size_t i = 0; i < boxes.size(); ++i) shapes[i].box = boxes[i];
    TC_CHECK(process_shapes(d_rowptr, d_col, claim.as<unsigned char>(), nnz, prm.density, s, shapes));
    long dense = 0;
    for (const ShapeResult &S : shapes)
        if (S.nnz > 0) {
            out.dia_shapes++;
            out.num_negs += S.neg;
            dense += S.nnz;
        }
    out.dense_nnz = (int)dense;
    out.sparse_nnz = (int)(nnz - dense);
    long zeros = 0, holes = 0;
    for (const ShapeResult &S : shapes)
        if (S.nnz > 0)
            for (int z : S.nzero) holes += std::max(z, 0);
    // a low density threshold can make more holes than a row pointer counts
    if (holes + out.sparse_nnz > 0x7fffffffL)
        return fail(TC_ERR_UNSUPPORTED, "%ld holes and %d entries left: more than 2^31 - 1 CSR words", holes, out.sparse_nnz);
    out.nDiasPtr.push_back(0);
    std::vector<HoleShape> hs;
    for (const ShapeResult &S : shapes) {
        if (S.nnz <= 0) continue;
        hs.push_back(HoleShape{S.box.x, S.box.y, S.box.b, S.neg, out.nDiasPtr.back(), S.bits.as<unsigned>()});
        out.xStart.push_back(S.box.x);
        out.yStart.push_back(S.box.y);
        out.xStop.push_back(S.box.x + S.box.b);
        out.nDiasPtr.push_back(out.nDiasPtr.back() + S.neg);
        for (int d = 0; d < S.neg; ++d) { out.offsets.push_back(S.offs[d]); zeros += S.nzero[d]; }
    }
    if (out.dia_shapes == 0) out.nDiasPtr.clear();
    out.zero_elements = (int)zeros;
    if (out.dia_shapes > 0) {
        out.row_start = *std::min_element(out.xStart.begin(), out.xStart.end());
        out.row_stop = *std::max_element(out.xStop.begin(), out.xStop.end());
    }

    if (dense == 0) {
        out.aliases_input = true;     // TaiChi.cu:575-578
        out.nnz_csr = nnz;
    } else {
        // TaiChi.cu:495-612: per row, holes then unclaimed entries
        Scratch tab, cnt, tmp;
        const size_t o_off = sizeof(HoleShape) * hs.size();
        TC_CHECK(tab.alloc(o_off + sizeof(int) * out.offsets.size(), s));
        TC_CHECK(cnt.alloc(sizeof(int) * ((size_t)M + 1), s));
        TC_CHECK(tmp.alloc(sizeof(int) * scan_tmp_ints(M), s));
        TC_CHECK(out.d_rowptr.alloc(sizeof(int) * ((size_t)M + 1), s));
        const HoleShape *const d_hs = tab.as<HoleShape>();
        const int *const d_offs = reinterpret_cast<const int *>(tab.as<char>() + o_off);
        TC_CUDA(cudaMemcpyAsync(tab.p, hs.data(), o_off, cudaMemcpyHostToDevice, s));
        TC_CUDA(cudaMemcpyAsync(tab.as<char>() + o_off, out.offsets.data(), sizeof(int) * out.offsets.size(),
                                cudaMemcpyHostToDevice, s));
        int *const rp_out = out.d_rowptr.as<int>();
        const int grid = std::max(1, std::min(cdiv(M, T), num_sms() * 8));
        TC_CUDA(cudaMemsetAsync(cnt.as<int>() + M, 0, sizeof(int), s));          // the scan's trailing 0
        remainder_counts<<<grid, T, 0, s>>>(d_rowptr, claim.as<unsigned char>(), d_hs, (int)hs.size(), M,
                                            cnt.as<int>());
        TC_CUDA(cudaGetLastError());
        TC_CHECK(exclusive_scan(cnt.as<int>(), rp_out, M, tmp.as<int>(), s));
        int total = 0;
        TC_CUDA(cudaMemcpyAsync(&total, rp_out + M, sizeof(int), cudaMemcpyDeviceToHost, s));
        TC_CUDA(cudaStreamSynchronize(s));
        out.nnz_csr = total;
        TC_CHECK(out.d_cols.alloc(sizeof(int) * (size_t)total, s));
        remainder_words<<<grid, T, 0, s>>>(d_rowptr, d_col, claim.as<unsigned char>(), d_hs, (int)hs.size(), d_offs,
                                           M, rp_out, out.d_cols.as<int>());
        TC_CUDA(cudaGetLastError());
        TC_CUDA(cudaStreamSynchronize(s));
    }
    if (want_claimed && nnz) {
        out.claimed.resize((size_t)nnz);
        TC_CUDA(cudaMemcpyAsync(out.claimed.data(), claim.p, (size_t)nnz, cudaMemcpyDeviceToHost, s));
    }
    TC_CUDA(cudaStreamSynchronize(s));
    out.ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return TC_OK;
}

// One shape on host arrays, for the reference's partition_dia_shape entry.
tc_status gpu_one_shape(int M, int64_t nnz, const int *h_rowptr, const int *h_col, float *h_val,
                        int x, int y, int a, int b, double density, OneShape &o)
{
    cudaStream_t s = 0;
    ScratchEnd end(s);
    Scratch rp, cl, va, claim;
    TC_CHECK(rp.alloc(sizeof(int) * ((size_t)M + 1), s));
    TC_CHECK(cl.alloc(sizeof(int) * (size_t)std::max<int64_t>(nnz, 1), s));
    TC_CHECK(va.alloc(sizeof(float) * (size_t)std::max<int64_t>(nnz, 1), s));
    TC_CHECK(claim.alloc((size_t)std::max<int64_t>(nnz, 1), s));
    TC_CUDA(cudaMemcpy(rp.p, h_rowptr, sizeof(int) * ((size_t)M + 1), cudaMemcpyHostToDevice));
    if (nnz) {
        TC_CUDA(cudaMemcpy(cl.p, h_col, sizeof(int) * (size_t)nnz, cudaMemcpyHostToDevice));
        TC_CUDA(cudaMemcpy(va.p, h_val, sizeof(float) * (size_t)nnz, cudaMemcpyHostToDevice));
        claim_init<<<cdiv(nnz, 256), 256, 0, s>>>(va.as<float>(), claim.as<unsigned char>(), nnz);
    }
    std::vector<ShapeResult> one(1);
    ShapeResult &R = one[0];
    R.box = shape_box(x, y, a, b);
    if (R.box.nd > 0 && b > 0)
        TC_CHECK(process_shapes(rp.as<int>(), cl.as<int>(), claim.as<unsigned char>(), nnz, density, s, one));
    o.width = R.box.w; o.neg = R.neg; o.nnz = R.nnz;
    o.offs = R.offs; o.start = R.start; o.end = R.end; o.nzero = R.nzero;
    o.holes.assign(R.neg, std::vector<int>());
    if (R.neg > 0) {
        std::vector<unsigned> bits((size_t)((R.neg + 31) / 32) * b);
        TC_CUDA(cudaMemcpy(bits.data(), R.bits.p, sizeof(unsigned) * bits.size(), cudaMemcpyDeviceToHost));
        for (int d = 0; d < R.neg; ++d)
            for (int r = 0; r < b; ++r)
                if (bits[(size_t)(d / 32) * b + r] >> (d & 31) & 1u) o.holes[d].push_back(r);
    }
    if (nnz && R.neg > 0) {
        std::vector<unsigned char> c((size_t)nnz);
        TC_CUDA(cudaMemcpy(c.data(), claim.p, (size_t)nnz, cudaMemcpyDeviceToHost));
        for (int64_t j = 0; j < nnz; ++j)
            if (c[j]) h_val[j] = FLT_MAX;
    }
    return TC_OK;
}

}  // namespace tc

using tc::fail;

extern "C" tc_status tc_getsdf(int M, int N, const int *d_rowptr, const int *d_col, const tc_params *p,
                               int *mF, int *W, int *corners, int max_corners, int *ncorners,
                               unsigned char *stages, void *stream)
{
    if (!mF || !W || !ncorners || M < 0 || N < 0) return fail(TC_ERR_INVALID, "tc_getsdf: bad arguments");
    tc_params prm;
    tc_params_default(&prm);
    if (p) prm = *p;
    TC_CHECK(tc::check_params(prm));
    tc::ScratchEnd end((cudaStream_t)stream, M > prm.thumb_height);
    tc::SdfOut o;
    TC_CHECK(tc::getsdf_device(M, N, d_rowptr, d_col, prm, stages != nullptr, (cudaStream_t)stream, o));
    *mF = o.mF;
    *W = o.W;
    const int n = (int)o.corners.size() / 4;
    *ncorners = n;
    if (corners) memcpy(corners, o.corners.data(), sizeof(int) * 4 * (size_t)std::min(n, max_corners));
    if (stages && !o.stages.empty()) memcpy(stages, o.stages.data(), o.stages.size());
    return n > max_corners && corners ? fail(TC_ERR_CAPACITY, "%d corners, room for %d", n, max_corners) : TC_OK;
}

extern "C" tc_status tc_trace_contours(const unsigned char *img, int H, int W, int *lens, int *ends,
                                       int max_contours, int *ncontours)
{
    if (!img || H <= 0 || W <= 0 || !ncontours) return fail(TC_ERR_INVALID, "tc_trace_contours: bad arguments");
    if ((long)H * W > (1L << 26)) return fail(TC_ERR_UNSUPPORTED, "image too large");
    const int WW = (W + 31) / 32;
    cudaStream_t s = nullptr;
    tc::ScratchEnd end(s);
    tc::Scratch bytes, bits;
    TC_CHECK(bytes.alloc((size_t)H * W, s));
    TC_CHECK(bits.alloc(sizeof(unsigned) * (size_t)H * WW, s));
    TC_CUDA(cudaMemcpy(bytes.p, img, (size_t)H * W, cudaMemcpyHostToDevice));
    tc::Img im{bits.as<unsigned>(), H, W, WW};
    tc::pack_kernel<<<tc::cdiv((long)H * WW, 256), 256>>>(bytes.as<unsigned char>(), im);
    TC_CUDA(cudaGetLastError());
    tc::ContourList cl;
    TC_CHECK(tc::contours_on_device(im, 0, cl));
    const int n = (int)cl.lens.size();
    *ncontours = n;
    for (int i = 0; i < n && i < max_contours; ++i) {
        if (lens) lens[i] = cl.lens[i];
        if (ends) {
            ends[4 * i + 0] = cl.first[i] % W;
            ends[4 * i + 1] = cl.first[i] / W;
            ends[4 * i + 2] = cl.mid[i] % W;
            ends[4 * i + 3] = cl.mid[i] / W;
        }
    }
    return n > max_contours ? fail(TC_ERR_CAPACITY, "%d contours, room for %d", n, max_contours) : TC_OK;
}

// ======================================================================
// Thumbnail stages without any allocation
// ======================================================================
// Some callers cannot allocate device memory at the point where they need
// the partitioner's thumbnail: code running while another framework owns the
// device allocator, or a caller that must not add cudaMalloc/cudaFree (which
// synchronize the device) to a latency-critical path.  This variant of the
// raster + morphology stages takes its scratch -- the seven bit-packed
// working images and a status word -- from the fixed array below instead of
// cudaMalloc.  The array holds at most a 512 x 1024 thumbnail (512 KB); it
// lives on every GPU that loads the library until the process exits.
namespace tc {
namespace {

constexpr int kNoAllocMaxH = 512, kNoAllocMaxW = 1024;
constexpr int kNoAllocWords = 8 * kNoAllocMaxH * (kNoAllocMaxW / 32);
static __device__ __align__(256) unsigned g_thumb_scratch[kNoAllocWords + 64];

ContextAddressCache<> g_noalloc_cache;

// Device address of g_thumb_scratch in the current context: looked up once
// per device and context (the host-side name is not a device address, and a
// context created after cudaDeviceReset gets a new lookup).
tc_status noalloc_scratch(unsigned **out)
{
    int dev = 0;
    TC_CUDA(cudaGetDevice(&dev));
    TC_CUDA(cudaSetDevice(dev));                 // initialises and makes current its primary context
    void *p = nullptr;
    cudaError_t err = cudaSuccess;
    const int rc = g_noalloc_cache.get(dev, current_context_id(), [&](void **a) {
        err = cudaGetSymbolAddress(a, g_thumb_scratch);
        return err == cudaSuccess ? 0 : 1;
    }, &p);
    if (rc < 0) return fail(TC_ERR_UNSUPPORTED, "device index %d", dev);
    if (rc != 0) {
        (void)cudaGetLastError();
        return fail(TC_ERR_CUDA, "cudaGetSymbolAddress(thumbnail scratch): %s", cudaGetErrorString(err));
    }
    *out = static_cast<unsigned *>(p);
    return TC_OK;
}

}  // namespace
}  // namespace tc

// Same images as tc_getsdf's `stages`, written to caller-owned device memory;
// allocates nothing.  The first call on a device looks up the scratch array's
// address (make it before any stream capture).  All calls share that array,
// so calls that overlap on the GPU (other streams, other threads) race; each
// call rewrites every word it reads before reading it and clears the status
// word itself.  Synchronizes `stream` to read the status word.
extern "C" tc_status tc_thumbnail_noalloc(int M, int N, const int *d_rowptr, const int *d_col,
                                          const tc_params *params, unsigned char *d_stages, int *W_out,
                                          void *stream)
{
    if (!W_out || M < 0 || N < 0 || (M > 0 && !d_rowptr)) return tc::fail(TC_ERR_INVALID, "tc_thumbnail_noalloc: bad arguments");
    *W_out = 0;
    tc_params p;
    tc_params_default(&p);
    if (params) p = *params;
    TC_CHECK(tc::check_params(p));
    const int H = p.thumb_height;
    if (M <= H) return TC_OK;                      // no thumbnail (morohutils.cu:192-196)
    const int W = (int)((double)H / (double)M * N);
    if (W <= 0) return tc::fail(TC_ERR_UNSUPPORTED, "thumbnail width is 0 (N < M/%d)", H);
    if (H > tc::kNoAllocMaxH || W > tc::kNoAllocMaxW)
        return tc::fail(TC_ERR_CAPACITY, "thumbnail %d x %d exceeds the fixed scratch (%d x %d)", H, W,
                        tc::kNoAllocMaxH, tc::kNoAllocMaxW);
    if (!d_stages || !d_col) return tc::fail(TC_ERR_INVALID, "tc_thumbnail_noalloc: null buffer");
    unsigned *scratch = nullptr;
    TC_CHECK(tc::noalloc_scratch(&scratch));
    cudaStream_t s = (cudaStream_t)stream;
    const int pM = M / H, pN = N / W, WW = (W + 31) / 32;
    const size_t nw = (size_t)H * WW;
    auto img = [&](int k) { return tc::Img{scratch + k * nw, H, W, WW}; };
    int *flag = reinterpret_cast<int *>(scratch + tc::kNoAllocWords);
    TC_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), s));
    tc::MorphArgs a;
    a.B = img(0); a.F = img(1); a.O2 = img(2); a.D = img(3); a.E = img(4);
    a.T1 = img(5); a.T2 = img(6);
    a.open_len = p.open_len;
    a.eye = p.eye_size;
    // the hole filling's H x W + 1 region names live in the output (5 H x W
    // bytes, written last), from its first 4-byte boundary on; those of a tiny
    // thumbnail, which would not fit there, behind the images
    const size_t px = (size_t)H * W;
    int *const names = px < 16 ? reinterpret_cast<int *>(scratch + 7 * nw)
                               : reinterpret_cast<int *>((reinterpret_cast<uintptr_t>(d_stages) + 3) & ~(uintptr_t)3);
    TC_CHECK(tc::thumbnail_stages(d_rowptr, d_col, M, pM, pN, a, names, flag, s));
    for (int k = 0; k < 5; ++k)
        tc::unpack_kernel<<<tc::cdiv((long)px, 256), 256, 0, s>>>(img(k), d_stages + k * px);
    TC_CUDA(cudaGetLastError());
    int hflag = 0;
    TC_CUDA(cudaMemcpyAsync(&hflag, flag, sizeof(int), cudaMemcpyDeviceToHost, s));
    TC_CUDA(cudaStreamSynchronize(s));
    if (hflag) return tc::fail(TC_ERR_UNSUPPORTED, "hole fill gave up (code %d)", hflag);
    *W_out = W;
    return TC_OK;
}

// ======================================================================
// getSdf with the reference's C++ signature (morphutils.h:40-41)
// ======================================================================
#include "morphutils.h"

void getSdf(std::string path, int M, int N, int nnz, int *&csrRowIndexHostPtr, int *&csrColIndexHostPtr,
            float *&csrValHostPtr, std::string &category, Point_t &size, int &shapeNum,
            std::vector<Point_t> &shapePoints, std::vector<double> &widths)
{
    (void)path;
    (void)csrValHostPtr;
    category = "diagonal";                        // morohutils.cu:186
    tc_params prm;
    tc_params_default(&prm);
    if (M <= prm.thumb_height) {                  // morohutils.cu:192-196
        printf("the matrix is too small! exit\n");
        return;
    }
    shapeNum = 0;
    auto report = [](tc_status st) {
        if (st != TC_OK) printf("getSdf: %s\n", tc_last_error());
    };
    if (M < 0 || N < 0 || nnz < 0 || !csrRowIndexHostPtr || (nnz > 0 && !csrColIndexHostPtr)) {
        report(tc::fail(TC_ERR_INVALID, "bad arguments"));
        return;
    }
    tc::ScratchEnd end(nullptr);
    tc::Scratch drp, dcol;
    tc_status st = drp.alloc(sizeof(int) * ((size_t)M + 1), nullptr);
    if (st == TC_OK) st = dcol.alloc(sizeof(int) * (size_t)std::max(nnz, 1), nullptr);
    if (st == TC_OK && cudaMemcpy(drp.p, csrRowIndexHostPtr, sizeof(int) * ((size_t)M + 1),
                                  cudaMemcpyHostToDevice) != cudaSuccess)
        st = tc::fail(TC_ERR_CUDA, "row pointer upload");
    if (st == TC_OK && nnz > 0 &&
        cudaMemcpy(dcol.p, csrColIndexHostPtr, sizeof(int) * (size_t)nnz, cudaMemcpyHostToDevice) != cudaSuccess)
        st = tc::fail(TC_ERR_CUDA, "column upload");
    tc::SdfOut o;
    if (st == TC_OK) st = tc::getsdf_device(M, N, drp.as<int>(), dcol.as<int>(), prm, false, nullptr, o);
    if (st != TC_OK) {
        report(st);
        return;
    }
    size.x = o.mF;                                // morohutils.cu:262-263
    size.y = o.W;
    shapeNum = (int)o.corners.size() / 4;
    for (int i = 0; i < shapeNum; ++i) {
        shapePoints.push_back(Point_t{o.corners[4 * i], o.corners[4 * i + 1]});
        shapePoints.push_back(Point_t{o.corners[4 * i + 2], o.corners[4 * i + 3]});
        widths.push_back(o.widths[i]);
    }
}
