// tdc_prep.cu -- per-acquisition preparation kernels of the GB300 TDC engine:
// the range window (tdc-lib/src/tdckernels.cu:32-64), its application to the
// raw chirps once per start() instead of once per pixel, focus-grid layout
// conversion and per-chirp position offsets (autofocus).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "tdc_device.cuh"
#include "tdc_internal.h"

namespace tdc {

namespace {

// w[n] = a - (1 - a) cos(2 pi n / N) (periodic), a = 25/46, or all ones.
__global__ void range_window_kernel(float *__restrict__ w, int n, int apply)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    w[i] = apply ? kRangeA - (1.0f - kRangeA) * cospif(2.0f * (float)i / (float)n) : 1.0f;
}

// In place on rows of s_pad complex samples (first S valid): x *= w[s]; padding -> 0.
__global__ void prewindow_kernel(float2 *__restrict__ xw, const float *__restrict__ w, int C, int S, int s_pad)
{
    const long long total = (long long)C * s_pad;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int s = (int)(idx % s_pad);
        float2 v = make_float2(0.f, 0.f);
        if (s < S) {
            const float ws = w[s];
            const float2 x = xw[idx];
            v = make_float2(x.x * ws, x.y * ws);
        }
        xw[idx] = v;
    }
}

// Range-windowed, zero-padded rows from a source the device can read directly
// (device memory, or pageable host memory on a system with coherent host access).
__global__ void prewindow_from_kernel(const float2 *__restrict__ src, const float *__restrict__ w, int C, int S,
                                      int s_pad, float2 *__restrict__ xw)
{
    const long long total = (long long)C * s_pad;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const long long c = idx / s_pad;
        const int s = (int)(idx - c * s_pad);
        float2 v = make_float2(0.f, 0.f);
        if (s < S) {
            const float2 x = src[c * S + s];
            const float ws = w[s];
            v = make_float2(x.x * ws, x.y * ws);
        }
        xw[idx] = v;
    }
}

// flag |= 1 when any sample of a chirp differs (bitwise) from the chirp's first sample;
// a is [C][S][k] floats.
__global__ void rows_differ_kernel(const unsigned int *__restrict__ a, int C, int S, int k, int *__restrict__ flag)
{
    const long long per = (long long)S * k;
    const long long total = (long long)C * per;
    bool differ = false;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const long long c = idx / per;
        const long long r = idx - c * per;
        differ |= a[idx] != a[c * per + (r % k)];
    }
    if (__syncthreads_or(differ) && threadIdx.x == 0) atomicOr(flag, 1);
}

// The same test of up to three arrays (blockIdx.y) reading 16 bytes per load (16-byte aligned, C x S x k
// < 2^31 elements, S >= 2, k of 3 or 4): all samples of a chirp equal its first exactly when
// each equals the one before, k elements back, which lies in this lane's vector or the previous
// lane's. A warp's first lane repeats the last vector of the warp before it instead of
// fetching it separately. The arrays usually sit in the caller's host memory: what counts
// is loads in flight, kScanLoads a thread.
constexpr int kScanLoads = 4;
struct RowScans {
    const uint4 *a[3];
    unsigned int total[3], per[3], k[3];
    int flag[3];
};

__global__ void __launch_bounds__(256) rows_differ_vec_kernel(const __grid_constant__ RowScans scans, int *__restrict__ flags)
{
    const int y = blockIdx.y, lane = threadIdx.x & 31;
    const uint4 *__restrict__ a4 = scans.a[y];
    const unsigned int total = scans.total[y], per = scans.per[y], k = scans.k[y];
    const unsigned int n4 = total / 4;
    const unsigned int warp = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, warps = gridDim.x * (blockDim.x / 32);
    bool differ = false;
    // 31 new vectors a warp and load
    for (unsigned int w0 = warp; w0 * 31u < n4; w0 += warps * kScanLoads) {
        uint4 v[kScanLoads];
#pragma unroll
        for (int u = 0; u < kScanLoads; ++u) {
            const unsigned int i = (w0 + u * warps) * 31u + lane;
            v[u] = i < n4 ? __ldg(&a4[i]) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int u = 0; u < kScanLoads; ++u) {
            const unsigned int i = (w0 + u * warps) * 31u + lane;
            const uint4 b = make_uint4(__shfl_up_sync(0xffffffffu, v[u].x, 1), __shfl_up_sync(0xffffffffu, v[u].y, 1),
                                       __shfl_up_sync(0xffffffffu, v[u].z, 1), __shfl_up_sync(0xffffffffu, v[u].w, 1));
            if (i >= n4) continue;
            const unsigned int cur[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
            // element k back of each; of a warp's first vector only what lies in it
            const unsigned int back[4] = {k == 3 ? b.y : b.x, k == 3 ? b.z : b.y, k == 3 ? b.w : b.z,
                                          k == 3 ? v[u].x : b.w};
            unsigned int r = 4u * i % per;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const bool known = lane > 0 || (k == 3 && q == 3);
                differ |= known && r >= k && cur[q] != back[q];
                if (++r == per) r = 0;
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x < total - 4 * n4) {
        const unsigned int *a = reinterpret_cast<const unsigned int *>(a4);
        const unsigned int el = 4 * n4 + threadIdx.x;
        differ |= el % per >= k && a[el] != a[el - k];
    }
    if (__syncthreads_or(differ) && threadIdx.x == 0) atomicOr(&flags[scans.flag[y]], 1);
}

// out[c][s] = s * rows[c][s]: rows pre-scaled by the sample index (the adjoint's B = sum_s s x_s z^s).
__global__ void scale_rows_kernel(const float2 *__restrict__ rows, long long total, int s_pad, float2 *__restrict__ out)
{
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const float s = (float)(idx % s_pad);
        const float2 x = rows[idx];
        out[idx] = make_float2(s * x.x, s * x.y);
    }
}

// Bounding box of the grid and the anchor span (GridBounds, which starts as grid_bounds_init sets it): the
// largest distance of a pixel from the anchor of its 32 consecutive pixels, the 17th or the last.
// Low parts count: half an ulp of a high float is 0.25 m at 4.5e6 m, many cells of a range profile.
__device__ __forceinline__ int float_key(float f)
{
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}

// (h, l) as one integer that orders as h + l does: the pair is normalised first.
__device__ __forceinline__ long long pair_key(float h, float l)
{
    float s = h, e = l;
    if (l != 0.f) two_sum(h, l, s, e);
    return (long long)float_key(s) << 32 | ((unsigned int)float_key(e) ^ 0x80000000u);
}

// Least (SIGN 1) or greatest (-1) key of the warp.
template <int SIGN>
__device__ __forceinline__ long long warp_extreme(long long key)
{
    const int h = (int)(key >> 32);
    const unsigned int l = (unsigned int)key;
    if (SIGN > 0) {
        const int m = __reduce_min_sync(0xffffffffu, h);
        return (long long)m << 32 | __reduce_min_sync(0xffffffffu, h == m ? l : 0xffffffffu);
    }
    const int m = __reduce_max_sync(0xffffffffu, h);
    return (long long)m << 32 | __reduce_max_sync(0xffffffffu, h == m ? l : 0u);
}

// Pixel p of a grid less a point (a, b) of it.
__device__ __forceinline__ float3 grid_offset(const float4 *hi, const float4 *lo, long long p, float4 a, float4 b)
{
    const float4 v = hi[p], l = lo ? lo[p] : make_float4(0.f, 0.f, 0.f, 0.f);
    return make_float3((v.x - a.x) + (l.x - b.x), (v.y - a.y) + (l.y - b.y), (v.z - a.z) + (l.z - b.z));
}

__device__ __forceinline__ float length2(float3 d) { return d.x * d.x + d.y * d.y + d.z * d.z; }

__global__ void __launch_bounds__(256) grid_bbox_kernel(const float4 *__restrict__ hi, const float4 *__restrict__ lo,
                                                        long long P, GridBounds *__restrict__ out)
{
    const long long top = 0x7fffffffffffffffLL;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    long long mn[3] = {top, top, top}, mx[3] = {-top - 1, -top - 1, -top - 1};
    float span2 = 0.f;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
        const float4 v = hi[p], l = lo ? lo[p] : zero;
        const long long k[3] = {pair_key(v.x, l.x), pair_key(v.y, l.y), pair_key(v.z, l.z)};
        for (int d = 0; d < 3; ++d) {
            mn[d] = min(mn[d], k[d]);
            mx[d] = max(mx[d], k[d]);
        }
        const long long a = min(P - 1, (p & ~31LL) + 16);
        const float d2 = length2(grid_offset(hi, lo, p, hi[a], lo ? lo[a] : zero));
        span2 = d2 > span2 || d2 != d2 ? d2 : span2;
    }
    const int span = __reduce_max_sync(0xffffffffu, __float_as_int(fabsf(sqrtf(span2))));
    __shared__ long long part[8][7];  // one row a warp: the block's atomics are 7, not 7 a warp
    for (int d = 0; d < 3; ++d) {
        mn[d] = warp_extreme<1>(mn[d]);
        mx[d] = warp_extreme<-1>(mx[d]);
    }
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        for (int d = 0; d < 3; ++d) {
            part[warp][d] = mn[d];
            part[warp][3 + d] = mx[d];
        }
        part[warp][6] = span;
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        const int d = threadIdx.x, n_warps = blockDim.x >> 5;
        long long v = part[0][d];
        for (int w = 1; w < n_warps; ++w) v = d < 3 ? min(v, part[w][d]) : max(v, part[w][d]);
        if (d < 3) atomicMin(&out->box[d], v);
        else if (d < 6) atomicMax(&out->box[d], v);
        else if (v > 0) atomicMax(&out->words[3], (int)v);
    }
}

// Largest distance from each work tile's centre pixel to its other pixels (see FocusJob::tile_cols);
// one warp a tile.
__global__ void tile_radius_kernel(const float4 *__restrict__ hi, const float4 *__restrict__ lo, long long P, int rows,
                                   int cols, int tile_cols, int n_tiles, float *__restrict__ radius)
{
    const int t = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (t >= n_tiles) return;
    long long centre;
    if (tile_cols) {
        const int n_tc = (cols + tile_cols - 1) / tile_cols, tile_rows = kFocusTile / tile_cols;
        const long long r = min((long long)rows - 1, (long long)(t / n_tc) * tile_rows + tile_rows / 2);
        const long long c = min((long long)cols - 1, (long long)(t % n_tc) * tile_cols + tile_cols / 2);
        centre = r * cols + c;
    } else {
        centre = min(P - 1, (long long)t * kFocusTile + kFocusTile / 2);
    }
    const float4 a = hi[centre], b = lo ? lo[centre] : make_float4(0.f, 0.f, 0.f, 0.f);
    float r2 = 0.f;
    for (int s = lane; s < kFocusTile; s += 32) {
        const long long p = tile_pixel(tile_cols, cols, P, t, s);
        if (p < 0) continue;
        const float d2 = length2(grid_offset(hi, lo, p, a, b));
        r2 = d2 > r2 || d2 != d2 ? d2 : r2;
    }
    const int m = __reduce_max_sync(0xffffffffu, __float_as_int(fabsf(r2)));
    if (lane == 0) radius[t] = sqrtf(__int_as_float(m));
}

// Reach of the anchored pixel groups of the range-profile focus: the largest distance from a
// group's anchor (its middle pixel) to its other pixels, for groups of 8, 4 and 2 consecutive
// pixels of a run and of 16, and the largest offset along each axis in the groups of 16
// (GridBounds::words); one thread per 8 pixels of a run.
__global__ void group_reach_kernel(const float4 *__restrict__ hi, const float4 *__restrict__ lo, long long P, int run,
                                   int *__restrict__ words)
{
    float spread[4] = {0.f, 0.f, 0.f, 0.f};
    const int per = (run + 7) / 8;
    const long long n = (P / run) * per + (P % run + 7) / 8;
    float reach[3] = {0.f, 0.f, 0.f};
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const long long r = q / per;
        const int col = (int)(q - r * per) * 8;
        const long long p0 = r * run + col;
        const int valid = (int)min((long long)min(8, run - col), P - p0);
        for (int k = 0; k < 3; ++k) {
            const int g = 8 >> k;
            for (int s = 0; s < valid; s += g) {
                const int m = min(g, valid - s);
                const float4 a = hi[p0 + s + m / 2], b = lo ? lo[p0 + s + m / 2] : zero;
                for (int i = 0; i < m; ++i) {
                    const float d = sqrtf(length2(grid_offset(hi, lo, p0 + s + i, a, b)));
                    reach[k] = d > reach[k] || d != d ? d : reach[k];
                }
            }
        }
        if (col & 15) continue;
        const int valid16 = (int)min((long long)min(16, run - col), P - p0);
        const float4 a = hi[p0 + valid16 / 2], b = lo ? lo[p0 + valid16 / 2] : zero;
        for (int i = 0; i < valid16; ++i) {
            const float3 v = grid_offset(hi, lo, p0 + i, a, b);
            const float o[4] = {fabsf(v.x), fabsf(v.y), fabsf(v.z), sqrtf(length2(v))};
            for (int d = 0; d < 4; ++d) spread[d] = o[d] > spread[d] || o[d] != o[d] ? o[d] : spread[d];
        }
    }
    for (int d = 0; d < 4; ++d) {
        const int v = __reduce_max_sync(0xffffffffu, __float_as_int(fabsf(spread[d])));
        if ((threadIdx.x & 31) == 0 && v > 0) atomicMax(&words[4 + d], v);
    }
    for (int k = 0; k < 3; ++k) {
        const int v = __reduce_max_sync(0xffffffffu, __float_as_int(fabsf(reach[k])));
        if ((threadIdx.x & 31) == 0 && v > 0) atomicMax(&words[k], v);
    }
}

__global__ void grid_f32_kernel(const float *__restrict__ g, long long P, float4 *__restrict__ hi)
{
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P) return;
    hi[p] = make_float4(g[3 * p], g[3 * p + 1], g[3 * p + 2], 0.f);
}

__device__ __forceinline__ void split_dd(double v, float &h, float &l)
{
    h = (float)v;
    l = (float)(v - (double)h);
}

__global__ void grid_f64_kernel(const double *__restrict__ g, long long P, float4 *__restrict__ hi,
                                float4 *__restrict__ lo)
{
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P) return;
    float h[3], l[3];
    for (int k = 0; k < 3; ++k) split_dd(g[3 * p + k], h[k], l[k]);
    hi[p] = make_float4(h[0], h[1], h[2], 0.f);
    lo[p] = make_float4(l[0], l[1], l[2], 0.f);
}

// recs[c].p = base[c] + off[c] as double-float pairs (off may be null).
__global__ void chirp_positions_kernel(ChirpRec *__restrict__ recs, const double *__restrict__ base,
                                       const double *__restrict__ off, int C)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    float h[3], l[3];
    for (int k = 0; k < 3; ++k) {
        const double v = base[3 * c + k] + (off ? off[3 * c + k] : 0.0);
        split_dd(v, h[k], l[k]);
    }
    ChirpRec r = recs[c];
    r.p_hi = make_float4(h[0], h[1], h[2], r.p_hi.w);
    r.p_lo = make_float4(l[0], l[1], l[2], 0.f);
    recs[c] = r;
}

}  // namespace

cudaError_t launch_range_window(float *w, int n, int apply, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    range_window_kernel<<<(n + 127) / 128, 128, 0, st>>>(w, n, apply);
    return cudaGetLastError();
}

cudaError_t launch_prewindow(float2 *xw, const float *w, int C, int S, int s_pad, cudaStream_t st)
{
    const long long total = (long long)C * s_pad;
    if (total <= 0) return cudaSuccess;
    long long blocks = (total + 255) / 256;
    if (blocks > 152 * 32) blocks = 152 * 32;
    prewindow_kernel<<<(unsigned)blocks, 256, 0, st>>>(xw, w, C, S, s_pad);
    return cudaGetLastError();
}

cudaError_t launch_prewindow_from(const float2 *src, const float *w, int C, int S, int s_pad, float2 *xw,
                                  cudaStream_t st)
{
    const long long total = (long long)C * s_pad;
    if (total <= 0) return cudaSuccess;
    long long blocks = (total + 255) / 256;
    if (blocks > 152 * 32) blocks = 152 * 32;
    prewindow_from_kernel<<<(unsigned)blocks, 256, 0, st>>>(src, w, C, S, s_pad, xw);
    return cudaGetLastError();
}

cudaError_t launch_rows_differ(const RowScan *scans, int n, int C, int S, int *flags, cudaStream_t st)
{
    RowScans vec{};
    int n_vec = 0;
    long long blocks = 1;
    for (int i = 0; i < n; ++i) {
        const RowScan &r = scans[i];
        const long long total = (long long)C * S * r.k;
        if (total <= 0 || S < 2) continue;
        if ((reinterpret_cast<uintptr_t>(r.a) & 15u) == 0 && total < (1LL << 31) && (r.k == 3 || r.k == 4) && n_vec < 3) {
            vec.a[n_vec] = reinterpret_cast<const uint4 *>(r.a);
            vec.total[n_vec] = (unsigned)total;
            vec.per[n_vec] = (unsigned)((long long)S * r.k);
            vec.k[n_vec] = (unsigned)r.k;
            vec.flag[n_vec] = r.flag;
            blocks = std::max(blocks, (total / 4 + 256 * kScanLoads - 1) / (256 * kScanLoads));
            ++n_vec;
            continue;
        }
        const long long b = std::min<long long>((total + 255) / 256, 152 * 16);
        rows_differ_kernel<<<(unsigned)b, 256, 0, st>>>(reinterpret_cast<const unsigned int *>(r.a), C, S, r.k,
                                                         flags + r.flag);
        if (const cudaError_t e = cudaGetLastError()) return e;
    }
    if (n_vec == 0) return cudaSuccess;
    rows_differ_vec_kernel<<<dim3((unsigned)std::min<long long>(blocks, 152 * 4), n_vec), 256, 0, st>>>(vec, flags);
    return cudaGetLastError();
}

cudaError_t launch_scale_rows(const float2 *rows, int C, int s_pad, float2 *rows_out, cudaStream_t st)
{
    const long long total = (long long)C * s_pad;
    if (total <= 0) return cudaSuccess;
    long long blocks = (total + 255) / 256;
    if (blocks > 152 * 32) blocks = 152 * 32;
    scale_rows_kernel<<<(unsigned)blocks, 256, 0, st>>>(rows, total, s_pad, rows_out);
    return cudaGetLastError();
}

cudaError_t launch_grid_bbox(const float4 *hi, const float4 *lo, long long P, GridBounds *out, cudaStream_t st)
{
    if (P <= 0) return cudaSuccess;
    long long blocks = (P + 255) / 256;
    if (blocks > 152 * 8) blocks = 152 * 8;
    grid_bbox_kernel<<<(unsigned)blocks, 256, 0, st>>>(hi, lo, P, out);
    return cudaGetLastError();
}

cudaError_t launch_tile_radius(const float4 *hi, const float4 *lo, long long P, int rows, int cols, int tile_cols,
                               int n_tiles, float *radius, cudaStream_t st)
{
    if (n_tiles <= 0) return cudaSuccess;
    tile_radius_kernel<<<(unsigned)((n_tiles * 32LL + 255) / 256), 256, 0, st>>>(hi, lo, P, rows, cols, tile_cols,
                                                                                n_tiles, radius);
    return cudaGetLastError();
}

cudaError_t launch_group_reach(const float4 *hi, const float4 *lo, long long P, int run, int *words, cudaStream_t st)
{
    if (P <= 0 || run <= 0) return cudaSuccess;
    long long blocks = (P / 8 + 255) / 256;
    if (blocks > 152 * 8) blocks = 152 * 8;
    if (blocks < 1) blocks = 1;
    group_reach_kernel<<<(unsigned)blocks, 256, 0, st>>>(hi, lo, P, run, words);
    return cudaGetLastError();
}

cudaError_t launch_grid_from_f32(const float *grid, long long P, float4 *hi, cudaStream_t st)
{
    if (P <= 0) return cudaSuccess;
    grid_f32_kernel<<<(unsigned)((P + 255) / 256), 256, 0, st>>>(grid, P, hi);
    return cudaGetLastError();
}

cudaError_t launch_grid_from_f64(const double *grid, long long P, float4 *hi, float4 *lo, cudaStream_t st)
{
    if (P <= 0) return cudaSuccess;
    grid_f64_kernel<<<(unsigned)((P + 255) / 256), 256, 0, st>>>(grid, P, hi, lo);
    return cudaGetLastError();
}

cudaError_t launch_chirp_positions(ChirpRec *recs, const double *base, const double *off, int C, cudaStream_t st)
{
    if (C <= 0) return cudaSuccess;
    chirp_positions_kernel<<<(C + 127) / 128, 128, 0, st>>>(recs, base, off, C);
    return cudaGetLastError();
}

}  // namespace tdc
