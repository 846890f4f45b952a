// tdc_profile.cu -- focus through range profiles: the FP32-bulk focus for grids of many pixels.
//
// With one range R per (pixel, chirp) and uniformly spaced samples, a pixel's sum over a
// chirp's samples is the chirp's centred spectrum at beta = g1 R [cycles / sample],
//
//   sum_s x[s] exp(j 2 pi (g0 + g1 s) R) = exp(j 2 pi gc R) A(beta),
//   A(beta) = sum_s x[s] exp(j 2 pi beta (s - sc)),  sc = S / 2,  gc = g0 + g1 sc,
//
// the same smooth function for every pixel. The direct kernels evaluate it from scratch, 4 S
// FMAs a pixel; here profile_build_kernel tabulates it once per chirp over the ranges the grid
// can take, and profile_focus_kernel reads one polynomial value per (pixel, chirp).
//
// The table ("cells"): A on cells of 1 / (4 S) cycles / sample (a quarter of the range
// resolution), each a polynomial of degree 7 in t = 4 S beta - cell, good for |t| <= 1.5, so
// that a group of neighbouring pixels reads one cell although their ranges differ. Built from
// A at nodes 1 / (2 S) apart (a product of the chirps' rows with a fixed matrix of phasors)
// by Kaiser-Bessel interpolation (9 nodes wide, the samples divided by the kernel's transform
// beforehand) at 8 Chebyshev points of the cell. Error of the interpolation and of the
// polynomial together: <= 2e-7 rms of a row's norm at |t| = 1.5, 1e-8 within the cell.
//
// Whole focus, direct kernels -> profiles (GB300, resident acquisition): 1024^2 pixels x 4096
// chirps x 1024 samples 532 -> 5.32 ms; 1.05 M voxels x 16,384 x 256 587 -> 20.1 ms; 256^2 x 1024 x
// 512 4.5 -> 0.164 ms; 256^2 x 64 x 12,345 6.5 -> 0.100 ms.
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>

#include <cooperative_groups.h>

#include "tdc_device.cuh"
#include "tdc_internal.h"

namespace cg = cooperative_groups;

namespace tdc {

namespace {

// ---- table construction -----------------------------------------------------

constexpr int kNodes = kProfileNodes;            // nodes one CTA forms
constexpr int kTaps = 11;                        // nodes a cell reads: -5 .. +5 about its own
constexpr int kOwn = kProfileNodes - kTaps + 1;  // nodes whose two cells the CTA writes
constexpr int kBuildChirps = 16;
constexpr int kBuildThreads = 256;
constexpr int kBuildStep = 64;                   // samples per shared-memory tile
constexpr double kKbWidth = 9.0;
constexpr double kKbBeta = 2.3 * kKbWidth;

// Real weights of a cell's polynomial coefficients: a_m = sum_j c[parity][m][j] V[node + j - 5].
struct ProfileStencil {
    float c[2][kProfileCoefs][kTaps];
};

double bessel_i0(double x)
{
    // sum_k (x^2 / 4)^k / (k!)^2
    double term = 1.0, sum = 1.0;
    for (int k = 1; k < 200 && term > 1e-18 * sum; ++k) {
        term *= (x * x / 4.0) / ((double)k * k);
        sum += term;
    }
    return sum;
}

ProfileStencil make_stencil()
{
    // f(x) = sum_j phi(x - j) V_j at the Chebyshev points t_i of the cell (x = t / 2 from the
    // cell's centre, which lies on a node or half way to the next), then the polynomial through
    // the 8 values: a = V^-1 f, V the Vandermonde matrix of the points (Gauss-Jordan in FP64).
    constexpr int n = kProfileCoefs;
    ProfileStencil st{};
    double t[n], a[n][2 * n];
    for (int i = 0; i < n; ++i) {
        t[i] = kProfileReach * std::cos(M_PI * (i + 0.5) / n);
        for (int m = 0; m < n; ++m) {
            a[i][m] = std::pow(t[i], m);
            a[i][n + m] = i == m ? 1.0 : 0.0;
        }
    }
    for (int k = 0; k < n; ++k) {
        int piv = k;
        for (int i = k + 1; i < n; ++i)
            if (std::fabs(a[i][k]) > std::fabs(a[piv][k])) piv = i;
        for (int m = 0; m < 2 * n; ++m) std::swap(a[k][m], a[piv][m]);
        const double d = a[k][k];
        for (int m = 0; m < 2 * n; ++m) a[k][m] /= d;
        for (int i = 0; i < n; ++i) {
            if (i == k) continue;
            const double f = a[i][k];
            for (int m = 0; m < 2 * n; ++m) a[i][m] -= f * a[k][m];
        }
    }
    // normalised so that the samples' factors (profile_twiddle_kernel) are about 1
    const double norm = kKbBeta / std::sinh(kKbBeta) / kKbWidth;
    for (int par = 0; par < 2; ++par)
        for (int m = 0; m < n; ++m)
            for (int j = 0; j < kTaps; ++j) {
                double s = 0.0;
                for (int i = 0; i < n; ++i) {
                    const double z = (0.5 * par + 0.5 * t[i] - (j - 5)) * 2.0 / kKbWidth;
                    if (std::fabs(z) < 1.0) s += a[m][n + i] * bessel_i0(kKbBeta * std::sqrt(1.0 - z * z)) * norm;
                }
                st.c[par][m][j] = (float)s;
            }
    return st;
}

// Per-length constants: phasors e^{j 2 pi n (s - sc) / (2 S)} for the nodes of one CTA
// ([S][kNodes]) and the samples' factors 1 / phi^ (the Kaiser-Bessel kernel's transform at the
// sample's frequency in node units).
__global__ void profile_twiddle_kernel(float2 *__restrict__ tw, float *__restrict__ factor, int S,
                                       const int *__restrict__ enabled)
{
    if (enabled && *enabled == 0) return;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)S * kNodes) return;
    const int s = (int)(i / kNodes), n = (int)(i - (long long)s * kNodes);
    const long long nn = 2LL * S, d = s - S / 2;
    int r = n * (int)d % (int)nn;  // (rows of up to 2^24 samples)
    if (r < 0) r += (int)nn;
    if (r > S) r -= (int)nn;
    // r / nn as a double-float pair, so that the sincos's rounding is all that is left (FP64: 142 us
    // for 12345 samples)
    const float fn = (float)nn, ratio = (float)r / fn, rest = fmaf(-ratio, fn, (float)r) / fn;
    float sn, cs;
    sincospif(2.0f * ratio, &sn, &cs);
    tw[i] = make_float2(fmaf(-kTwoPiF * rest, sn, cs), fmaf(kTwoPiF * rest, cs, sn));
    if (n == 0) {
        const double q2 = 0.5 * kKbWidth * 2.0 * 3.14159265358979323846 * (double)d / (double)nn;
        const double q = sqrt(kKbBeta * kKbBeta - q2 * q2);
        factor[s] = (float)(q / sinh(q) * (sinh(kKbBeta) / kKbBeta));
    }
}

// One CTA: 16 chirps x one block of kOwn nodes (2 kOwn cells). Blocks lie at multiples of kOwn
// of the absolute node index, so a cell's value does not depend on where the table starts
// (the row blocks of a sharded grid build the same cells bit for bit). The rows are shifted by
// the block's first node while they are staged, then multiplied by the fixed phasor matrix
// (2 nodes x 4 chirps per thread: 32 FFMA per 4 shared loads; the two halves of the warps take
// the two halves of a tile's samples), summed 64 samples at a time so that FP32 rounding does
// not grow with the row, and the cells' coefficients are formed from the nodes in shared memory.
// Bound: FP32 FMA; C x S x (nodes the grid spans + up to one block) complex MACs, a few per cent
// of the focus it serves.
// A cluster of `split` CTAs shares a row's samples (launch_build).
// INDIRECT: the inputs come from device memory (`dev`, written by an earlier kernel of the stream)
// and the CTAs return at once where *enabled is 0.
template <bool INDIRECT>
__global__ void __launch_bounds__(kBuildThreads)
    profile_build_kernel(const __grid_constant__ ProfileBuild direct, const __grid_constant__ ProfileStencil stencil,
                         const ProfileBuild *__restrict__ dev, const int *__restrict__ enabled, int split)
{
    __shared__ ProfileBuild sb;
    if (INDIRECT) {
        if (*enabled == 0) return;
        for (int i = threadIdx.x; i < (int)(sizeof(ProfileBuild) / sizeof(int)); i += kBuildThreads)
            reinterpret_cast<int *>(&sb)[i] = reinterpret_cast<const int *>(dev)[i];
        __syncthreads();
    }
    const ProfileBuild &b = INDIRECT ? sb : direct;
    __shared__ __align__(16) float2 sx[kBuildStep][kBuildChirps];
    __shared__ __align__(16) float2 sv[kBuildStep * kNodes];  // phasors of a tile; then the nodes' values
    __shared__ int s_base[kBuildChirps];            // the chirp's first cell (absolute, even)
    __shared__ int s_cell[kBuildChirps];            // the block's first cell within the chirp's table
    __shared__ unsigned int s_shift[kBuildChirps];  // first node of the block modulo 2 S
    static_assert(kBuildStep >= 2 * kBuildChirps, "node values reuse the phasor tile");
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)blockIdx.x % split;  // in the cluster: this CTA's part of the samples
    const int c0 = (int)blockIdx.x / split * kBuildChirps;
    const unsigned int nn = 2u * (unsigned)b.S;

    if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && tid == 0) *b.job_out = b.job;
    if (tid < kBuildChirps) {
        // first cell: the smallest cell coordinate of any point in the grid's bounding box
        const int c = min(c0 + tid, b.C - 1);
        const float4 ph = b.chirps[(size_t)c * b.chirp_words], pl = b.chirps[(size_t)c * b.chirp_words + 1];
        const double p[3] = {(double)ph.x + pl.x, (double)ph.y + pl.y, (double)ph.z + pl.z};
        double near2 = 0.0, far2 = 0.0;
        for (int k = 0; k < 3; ++k) {
            const double lo = b.box_min[k] - p[k], hi = p[k] - b.box_max[k];
            const double n = fmax(0.0, fmax(lo, hi)), f = fmax(fabs(lo), fabs(hi));
            near2 += n * n;
            far2 += f * f;
        }
        const double u = fmin(b.cells_per_m * sqrt(near2), b.cells_per_m * sqrt(far2));
        // (positions far outside what the table can index: any base will do, reads are clamped)
        const int base = fabs(u) < 1e9 ? 2 * (int)floor(0.5 * u) - 2 - b.margin : 0;
        if (rank == 0 && blockIdx.y == 0 && blockIdx.z == 0 && c0 + tid < b.C) b.cell_base[c0 + tid] = base;
        const int node = base >> 1;
        const int block = (node >= 0 ? node / kOwn : -((kOwn - 1 - node) / kOwn)) + (int)blockIdx.y;
        s_cell[tid] = 2 * (block * kOwn - node);
        // (cell indices stay below 2^22)
        const int n0 = (block * kOwn - kTaps / 2) % (int)nn;
        s_shift[tid] = (unsigned)(n0 < 0 ? n0 + (int)nn : n0);
    }
    __syncthreads();
    if (!__syncthreads_or(tid < kBuildChirps && s_cell[tid & (kBuildChirps - 1)] < b.n_cells)) return;

    const int cq = 4 * (warp & 3), half = warp >> 2;
    float2 acc[4][2], run[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < 2; ++k) acc[i][k] = run[i][k] = make_float2(0.f, 0.f);

    // A tile's samples and phasors are loaded into registers while the tile before it is worked on.
    constexpr int kRowsEach = kBuildStep * kBuildChirps / kBuildThreads;
    constexpr int kPhasorsEach = kBuildStep * kNodes / 2 / kBuildThreads;
    float2 ahead_x[kRowsEach];
    float4 ahead_z[kPhasorsEach];
    float ahead_f = 0.f;
    const int si_mine = (warp & 1) * 32 + lane;  // this thread's sample of a tile, for kRowsEach chirps
    auto load_ahead = [&](int s0) {
        const int s = s0 + si_mine;
        ahead_f = s < b.S ? b.factor[s] : 0.f;
#pragma unroll
        for (int i = 0; i < kRowsEach; ++i) {
            const int q = (warp >> 1) + 4 * i;
            ahead_x[i] = s < b.S && c0 + q < b.C ? b.rows[(size_t)(c0 + q) * b.s_pad + s] : make_float2(0.f, 0.f);
        }
        // phasors: kBuildStep x kNodes, contiguous in memory (rows past the end meet zero samples)
        const int ns = min(kBuildStep, b.S - s0);
        const float4 *src = reinterpret_cast<const float4 *>(b.twiddle + (size_t)s0 * kNodes);
#pragma unroll
        for (int i = 0; i < kPhasorsEach; ++i) {
            const int e = tid + i * kBuildThreads;
            ahead_z[i] = e < ns * kNodes / 2 ? __ldg(&src[e]) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    // this CTA's tiles, in whole pairs (the sums are carried over two)
    const int tiles = (b.S + kBuildStep - 1) / kBuildStep, each = ((tiles + split - 1) / split + 1) & ~1;
    const int s_begin = rank * each * kBuildStep, s_end = min(b.S, s_begin + each * kBuildStep);
    // shift's turns at this thread's sample, modulo 2 S: (first node) x (s - sc), advanced a tile at a time
    unsigned int turn[kRowsEach], turn_step[kRowsEach];
    {
        const int d = s_begin + si_mine - b.S / 2;
        const unsigned int dm = d < 0 ? (unsigned)(d + (int)nn) : (unsigned)d;
        // (64-bit remainders cost about 100 instructions each)
        auto mul_mod = [nn](unsigned int a, unsigned int m) {
            return nn <= 65536 ? a * m % nn : (unsigned)((unsigned long long)a * m % nn);
        };
#pragma unroll
        for (int i = 0; i < kRowsEach; ++i) {
            const unsigned int sh = s_shift[(warp >> 1) + 4 * i];
            turn[i] = mul_mod(sh, dm % nn);
            turn_step[i] = mul_mod(sh, (unsigned)kBuildStep % nn);
        }
    }
    const float fnn = (float)nn, inv_nn = 1.0f / fnn;
    // Vibration: table blockIdx.z is of the samples times 1, phi_x, phi_y, phi_z, chi^2, chi^3 (phi the
    // deviation from the smooth motion in radians of carrier phase, chi its principal component).
    const int family = blockIdx.z;
    auto family_weight = [&](int q, int s) {
        const int c = c0 + q;
        if (s >= b.S || c >= b.C) return 0.f;
        const float4 *rec = b.chirps + (size_t)c * b.chirp_words;
        const float4 w1 = rec[2], f0 = rec[4], n = rec[5];
        const float4 d = sample_table(b.traj + (size_t)c * b.s_pad, s);
        const float t = (float)(s - b.S / 2);
        const float g = fmaf(b.phase_g1, t, b.phase_g);
        const float x = g * fmaf(-w1.x, t, d.x - f0.x), y = g * fmaf(-w1.y, t, d.y - f0.y),
                    z = g * fmaf(-w1.z, t, d.z - f0.z);
        const float chi = fmaf(n.x, x, fmaf(n.y, y, n.z * z));
        return family == 1 ? x : family == 2 ? y : family == 3 ? z : family == 4 ? chi * chi : chi * chi * chi;
    };
    load_ahead(s_begin);

    for (int s0 = s_begin, tile = 0; s0 < s_end; s0 += kBuildStep, ++tile) {
        // rows: shifted by the block's first node, scaled, zero past the row's end
#pragma unroll
        for (int i = 0; i < kRowsEach; ++i) {
            const int rc = turn[i] > nn / 2 ? (int)turn[i] - (int)nn : (int)turn[i];
            turn[i] += turn_step[i];
            if (turn[i] >= nn) turn[i] -= nn;
            // rc / nn to FP32 rounding
            const float fr = (float)rc;
            float ratio = fr * inv_nn;
            ratio = fmaf(fmaf(-ratio, fnn, fr), inv_nn, ratio);
            float sn, cs;
            sincospif(2.0f * ratio, &sn, &cs);
            float2 x = ahead_x[i];
            if (family) {
                const float w = family_weight((warp >> 1) + 4 * i, s0 + si_mine);
                x = make_float2(w * x.x, w * x.y);
            }
            sx[si_mine][(warp >> 1) + 4 * i] =
                make_float2(ahead_f * fmaf(x.x, cs, -x.y * sn), ahead_f * fmaf(x.x, sn, x.y * cs));
        }
#pragma unroll
        for (int i = 0; i < kPhasorsEach; ++i) reinterpret_cast<float4 *>(sv)[tid + i * kBuildThreads] = ahead_z[i];
        __syncthreads();
        if (s0 + kBuildStep < s_end) load_ahead(s0 + kBuildStep);
#pragma unroll 8
        for (int si = 0; si < kBuildStep / 2; ++si) {
            const int s = half * (kBuildStep / 2) + si;
            const float4 xa = *reinterpret_cast<const float4 *>(&sx[s][cq]);
            const float4 xb = *reinterpret_cast<const float4 *>(&sx[s][cq + 2]);
            const float2 x[4] = {make_float2(xa.x, xa.y), make_float2(xa.z, xa.w), make_float2(xb.x, xb.y),
                                 make_float2(xb.z, xb.w)};
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const float2 z = sv[s * kNodes + lane + 32 * k];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    run[i][k].x = fmaf(x[i].x, z.x, run[i][k].x);
                    run[i][k].x = fmaf(-x[i].y, z.y, run[i][k].x);
                    run[i][k].y = fmaf(x[i].x, z.y, run[i][k].y);
                    run[i][k].y = fmaf(x[i].y, z.x, run[i][k].y);
                }
            }
        }
        if ((tile & 1) || s0 + kBuildStep >= s_end) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    acc[i][k].x += run[i][k].x;
                    acc[i][k].y += run[i][k].y;
                    run[i][k] = make_float2(0.f, 0.f);
                }
        }
        __syncthreads();
    }

#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < 2; ++k) sv[(half * kBuildChirps + cq + i) * kNodes + lane + 32 * k] = acc[i][k];
    __syncthreads();
    for (int i = tid; i < kBuildChirps * kNodes; i += kBuildThreads) {
        const float2 a = sv[i], z = sv[kBuildChirps * kNodes + i];
        sv[i] = make_float2(a.x + z.x, a.y + z.y);
    }
    // the cluster's sums, each CTA for its share of the chirps, in order of the samples
    const int share = kBuildChirps / split;
    float2 *nodes = sv;
    if (split > 1) {
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        nodes = &sx[0][0];
        for (int i = tid; i < share * kNodes; i += kBuildThreads) {
            float2 v = make_float2(0.f, 0.f);
            for (int r = 0; r < split; ++r) {
                const float2 x = cluster.map_shared_rank(sv, r)[rank * share * kNodes + i];
                v.x += x.x;
                v.y += x.y;
            }
            nodes[i] = v;
        }
        cluster.sync();
    } else {
        __syncthreads();
    }

    for (int i = tid; i < share * kOwn; i += kBuildThreads) {
        const int q = rank * share + i / kOwn, j = i % kOwn;
        const int c = c0 + q;
        if (c >= b.C) break;
        const int l = s_cell[q] + 2 * j;  // cell within the chirp's table
        if (l < 0 || l >= b.n_cells) continue;
        float2 v[kTaps];
#pragma unroll
        for (int k = 0; k < kTaps; ++k) v[k] = nodes[(q - rank * share) * kNodes + j + k];
        float4 *__restrict__ out =
            b.cells + (((size_t)family * b.C + c) * b.n_cells + l) * (kProfileCoefs / 2);
#pragma unroll
        for (int par = 0; par < 2; ++par)
#pragma unroll
            for (int m = 0; m < kProfileCoefs; m += 2) {
                float2 a0 = make_float2(0.f, 0.f), a1 = a0;
#pragma unroll
                for (int k = 0; k < kTaps; ++k) {
                    a0.x = fmaf(stencil.c[par][m][k], v[k].x, a0.x);
                    a0.y = fmaf(stencil.c[par][m][k], v[k].y, a0.y);
                    a1.x = fmaf(stencil.c[par][m + 1][k], v[k].x, a1.x);
                    a1.y = fmaf(stencil.c[par][m + 1][k], v[k].y, a1.y);
                }
                out[par * (kProfileCoefs / 2) + m / 2] = make_float4(a0.x, a0.y, a1.x, a1.y);
            }
    }
}

// One warp a chirp: least squares of D_s by a line in s (FP64), re-centred on the middle sample; then
// the covariance of the deviations, its principal direction by power iteration, and the largest
// deviation off it. (A quadratic would take part of the vibration's bow into the smooth
// motion, whose bend a group of pixels then shares.)
__global__ void __launch_bounds__(128)
    vib_fit_kernel(const float4 *__restrict__ traj, const ChirpRec *__restrict__ chirps, int C, int S, int s_pad,
                   float phase_per_m, VibRec *__restrict__ recs, int *__restrict__ maxima)
{
    const int c = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (c >= C) return;
    const float4 *row = traj + (size_t)c * s_pad;
    const double hs = 0.5 * (S - 1);
    double a[6] = {0, 0, 0, 0, 0, 0}, sxx = 0.0;
    for (int s = lane; s < S; s += 32) {
        const float4 d = sample_table(row, s);
        const double x = s - hs, v[3] = {d.x, d.y, d.z};
        sxx += x * x;
        for (int k = 0; k < 3; ++k) {
            a[k] += v[k];
            a[3 + k] += v[k] * x;
        }
    }
    for (int off = 16; off > 0; off >>= 1) {
        sxx += __shfl_xor_sync(0xffffffffu, sxx, off);
        for (int k = 0; k < 6; ++k) a[k] += __shfl_xor_sync(0xffffffffu, a[k], off);
    }
    const double xc = (double)(S / 2) - hs;
    double f0[3], w1[3], n1 = 0.0;
    for (int k = 0; k < 3; ++k) {
        w1[k] = sxx > 0.0 ? a[3 + k] / sxx : 0.0;
        f0[k] = a[k] / S + w1[k] * xc;
        n1 += w1[k] * w1[k];
    }
    const float ff[3] = {(float)f0[0], (float)f0[1], (float)f0[2]}, fw[3] = {(float)w1[0], (float)w1[1], (float)w1[2]};
    auto deviation = [&](int s, float &x, float &y, float &z) {
        const float4 d = sample_table(row, s);
        const float t = (float)(s - S / 2);
        x = fmaf(-fw[0], t, d.x - ff[0]);
        y = fmaf(-fw[1], t, d.y - ff[1]);
        z = fmaf(-fw[2], t, d.z - ff[2]);
    };
    float cov[6] = {0, 0, 0, 0, 0, 0}, most = 0.f;
    for (int s = lane; s < S; s += 32) {
        float x, y, z;
        deviation(s, x, y, z);
        cov[0] += x * x;
        cov[1] += y * y;
        cov[2] += z * z;
        cov[3] += x * y;
        cov[4] += x * z;
        cov[5] += y * z;
        const float m = sqrtf(x * x + y * y + z * z);
        most = m > most || m != m ? m : most;
    }
    for (int off = 16; off > 0; off >>= 1)
        for (int k = 0; k < 6; ++k) cov[k] += __shfl_xor_sync(0xffffffffu, cov[k], off);
    // power iteration from the axis of largest variance (scaled to its trace)
    float n[3] = {0.f, 0.f, 0.f};
    const int axis = cov[0] >= cov[1] && cov[0] >= cov[2] ? 0 : cov[1] >= cov[2] ? 1 : 2;
    n[axis] = 1.f;
    const float tr = cov[0] + cov[1] + cov[2];
    if (tr > 0.f)
        for (int it = 0; it < 24; ++it) {
            const float x = (cov[0] * n[0] + cov[3] * n[1] + cov[4] * n[2]) / tr,
                        y = (cov[3] * n[0] + cov[1] * n[1] + cov[5] * n[2]) / tr,
                        z = (cov[4] * n[0] + cov[5] * n[1] + cov[2] * n[2]) / tr;
            const float r = rsqrtf(x * x + y * y + z * z);
            n[0] = x * r;
            n[1] = y * r;
            n[2] = z * r;
        }
    float side = 0.f;
    for (int s = lane; s < S; s += 32) {
        float x, y, z;
        deviation(s, x, y, z);
        const float r = n[0] * x + n[1] * y + n[2] * z;
        const float px = x - r * n[0], py = y - r * n[1], pz = z - r * n[2];
        const float m = sqrtf(px * px + py * py + pz * pz);
        side = m > side || m != m ? m : side;
    }
    const int im = __reduce_max_sync(0xffffffffu, __float_as_int(fabsf(most)));
    const int is = __reduce_max_sync(0xffffffffu, __float_as_int(fabsf(side)));
    if (lane) return;
    VibRec r;
    const ChirpRec base = chirps[c];
    // (what is kept of f0 and W1 in FP32 is what the deviations were taken from)
    const double p[3] = {(double)base.p_hi.x + base.p_lo.x + ff[0], (double)base.p_hi.y + base.p_lo.y + ff[1],
                         (double)base.p_hi.z + base.p_lo.z + ff[2]};
    r.m.p_hi = make_float4((float)p[0], (float)p[1], (float)p[2], 0.f);
    r.m.p_lo = make_float4((float)(p[0] - r.m.p_hi.x), (float)(p[1] - r.m.p_hi.y), (float)(p[2] - r.m.p_hi.z), 0.f);
    r.m.w1 = make_float4(fw[0], fw[1], fw[2], (float)n1);
    r.m.v2 = make_float4(0.f, 0.f, 0.f, 0.f);
    r.f0 = make_float4(ff[0], ff[1], ff[2], 0.f);
    const float amp = phase_per_m * __int_as_float(im);
    r.n = make_float4(n[0], n[1], n[2], amp * amp);
    recs[c] = r;
    atomicMax(&maxima[0], im);
    atomicMax(&maxima[1], is);
    atomicMax(&maxima[2], __float_as_int((float)sqrt(n1)) & 0x7fffffff);
}

// ---- focus ------------------------------------------------------------------

constexpr int kThreads = kProfileThreads;
static_assert(kThreads == 64, "records are staged by 64 threads");
constexpr int kPT = kFocusTile / kProfileThreads;  // pixels per thread: consecutive pixels of a run
#ifndef TDC_PROFILE_MINB
#define TDC_PROFILE_MINB 8
#endif
constexpr int kFlush = kProfileBlock;                         // chirps summed in plain FP32 between Kahan steps

// (sqrt(1 + y) - 1) / (y / 2) = 1 - y / 4 + kRoot2 y^2 + kRoot3 y^3 on |y| <= Y = 0.061: the Taylor
// terms 1/8 and -5/64, with 7/128 y^4 replaced by its best multiple of y^2 there, 0.828 Y^2 y^2
// (error below 1.3e-7 at the end of the range, 4e-8 at 0.045, vanishing with y).
constexpr float kRootRange = 0.061f;
// The same to y^4 for groups of 16, |y| <= 0.1 (reach / R <= 1 / 21; 6e-8 left), the y^5 term
// economised: y^5 = 5/4 Y^2 y^3 - 5/16 Y^4 y within Y^5 / 16.
constexpr float kWide1 = -0.25f + 21.0f / 512.0f * 0.3125f * 1e-4f, kWide2 = 0.125f,
                kWide3 = -5.0f / 64.0f - 21.0f / 512.0f * 1.25f * 1e-2f, kWide4 = 7.0f / 128.0f;
constexpr float kRoot2 = 0.125f + 7.0f / 128.0f * 0.828f * kRootRange * kRootRange, kRoot3 = -5.0f / 64.0f;

template <int PT>
struct SharedSums {
    float4 s[PT][kThreads];       // (sum.re, sum.im, comp.re, comp.im)
    float2 dz[PT / 2][kThreads];  // z offsets and |d|^2 of the thread's pixel pairs
    float2 dd[PT / 2][kThreads];
};

// Chirp records of kFlush chirps at a time (position high and low; the velocity with a finite
// band; W1 and V2 with smooth motion) and their first cells.
template <int WORDS>
struct SharedChirps {
    float4 p[kFlush][WORDS];
    int base[kFlush];
};

// Kahan step of pixel i's sums: + sum over chirps of (cos + j sin) h, given as sum h cos, sum h sin.
template <int PT>
__device__ __forceinline__ void stash(SharedSums<PT> &sums, int i, int tid, float2 hc, float2 hs)
{
    float4 s = sums.s[i][tid];
    const float yr = (hc.x - hs.y) - s.z, yi = (hc.y + hs.x) - s.w;
    const float tr = s.x + yr, ti = s.y + yi;
    s.z = (tr - s.x) - yr;
    s.w = (ti - s.y) - yi;
    s.x = tr;
    s.y = ti;
    sums.s[i][tid] = s;
}

// First pixel of thread `tid` of tile t, and how many it has (consecutive ones, up to kPT; 0
// past the grid's end). Threads take kPT consecutive pixels of a run (a grid row: consecutive
// pixels without a jump), so no thread's pixels straddle the end of one. Groups are numbered
// down the runs of a band of 8 runs, then along it: a warp covers a block of 8 runs x 32
// pixels, whose ranges, and so the cells it reads, lie closer together than 256 pixels of one
// run's do.
template <int PT>
__device__ __forceinline__ long long run_pixels(long long P, int run, int t, int tid, int &count)
{
    const int per_run = (run + PT - 1) / PT;
    const long long runs = (P + run - 1) / run;
    const long long q = (long long)t * kThreads + tid;
    const long long band = q / ((long long)kProfileBand * per_run);
    const int rem = (int)(q - band * kProfileBand * per_run);
    const int height = (int)min((long long)kProfileBand, runs - band * kProfileBand);
    count = 0;
    if (height <= 0) return 0;
    const int col = rem / height * PT;
    const long long p = (band * kProfileBand + rem % height) * run + col;
    if (col < run && p < P) count = (int)min((long long)min(PT, run - col), P - p);
    return p;
}

// Pairs of FP32 values in one instruction (FFMA2 and its kin): the same FMA-pipe time as two
// scalar ones, half the issue slots, which is what bounds the scalar form of this kernel.
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }

// Asynchronous copy of 4 or 16 bytes into shared memory.
template <int BYTES>
__device__ __forceinline__ void copy_async(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES) : "memory");
}

__device__ __forceinline__ void copy_async_wait()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// Shared memory loaded where it is used: these values would otherwise sit in registers through the
// whole loop.
__device__ __forceinline__ float4 fresh(const float *p)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(smem_u32(p)));
    return v;
}

__device__ __forceinline__ float2 fresh2(const float2 *p)
{
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(smem_u32(p)));
    return v;
}

// dd_sub with its high part rounded from the whole difference. The high parts of antenna and pixel
// alone are an ulp of their coordinates off, and h stands for the direction of the group's range
// differences here: at coordinates of 1 km and ranges of 0.3 m, 5e-4 of the image without the
// low parts and 3e-7 with them.
__device__ __forceinline__ void difference(float ah, float al, float bh, float bl, float &h, float &l)
{
    float s, e;
    dd_sub(ah, al, bh, bl, s, e);
    h = s + e;
    l = e - (h - s);
}

// One (chirp, anchor pixel): e = antenna - anchor, R0, gc / (2 R0), the carrier phase 2 pi frac(gc R0),
// and the anchor's cell and place in it.
struct Anchor {
    float ex, ey, ez, rh, h, turn, t0;
    const float4 *cell;  // its first table's cell (MOVE == 2)
    float w;  // Doppler window (BAND with every pixel its own anchor); cell shift of its motion (MOVE)
    float2 a[kProfileCoefs];
};

// turn + 2 pi psi [rad], psi modulo one cycle unless SMALL (the sincos's argument is then rounded at up
// to 2 pi kLineMaxCycles + pi: 1e-6 rad rms at a group's edge, 5e-7 over it).
template <bool SMALL>
__device__ __forceinline__ float2 phase_of(float2 psi, float turn)
{
    if (SMALL) return __ffma2_rn(psi, both(kTwoPiF), both(turn));
    const float2 n = __fadd2_rn(__fadd2_rn(psi, both(12582912.0f)), both(-12582912.0f));  // nearest integer
    return __ffma2_rn(__fadd2_rn(psi, make_float2(-n.x, -n.y)), both(kTwoPiF), both(turn));
}

// One chirp's contributions to two pixels with phase differences psi (cycles) from their
// anchor: e^{j (turn + 2 pi psi)} A(t0 + psi cells_per_cycle), A the cell's polynomial with
// coefficients a, times its window (WEIGHTED). Real and imaginary part of the value h advance together; the product with
// the phasor is kept as h cos and h sin (c_i, s_i) and combined when the sums are flushed.
template <bool WEIGHTED, bool LINE>
__device__ __forceinline__ void add_pair(float2 psi, float turn, float t0, float cells_per_cycle,
                                         const float2 (&a)[kProfileCoefs], float w0, float w1, float2 &c0, float2 &s0, float2 &c1,
                                         float2 &s1)
{
    const float2 x = phase_of<LINE>(psi, turn);
    const float2 t = __ffma2_rn(psi, both(cells_per_cycle), both(t0));
    float sn0, cs0, sn1, cs1;
    __sincosf(x.x, &sn0, &cs0);
    __sincosf(x.y, &sn1, &cs1);
    if (WEIGHTED) {
        cs0 *= w0;
        sn0 *= w0;
        cs1 *= w1;
        sn1 *= w1;
    }
    const float2 ta = both(t.x), tb = both(t.y);
    float2 h0 = a[kProfileCoefs - 1], h1 = h0;
#pragma unroll
    for (int m = kProfileCoefs - 2; m >= 0; --m) {
        h0 = __ffma2_rn(h0, ta, a[m]);
        h1 = __ffma2_rn(h1, tb, a[m]);
    }
    c0 = __ffma2_rn(h0, both(cs0), c0);
    s0 = __ffma2_rn(h0, both(sn0), s0);
    c1 = __ffma2_rn(h1, both(cs1), c1);
    s1 = __ffma2_rn(h1, both(sn1), s1);
}

// Smooth motion: the anchor's bend eps0 [rad at the row's ends]; a := coefficients of
// e^{j (eps0 s^2 + cubic s^3)} A, bend := of the pixel's first-order term, s^2 (1 + j eps0 s^2) A
// (s = s~ / (S / 2) = -j (4 / pi) d/dt).
__device__ __forceinline__ float move_coefs(const Anchor &n, float4 w1, float4 v2, const ProfileJob &job,
                                            float2 (&a)[kProfileCoefs], float2 (&bend)[kProfileCoefs - 2])
{
    const float ri = n.rh > 0.0f ? 2.0f * n.h * job.inv_gc : 0.0f;
    const float rate = fmaf(n.ex, w1.x, fmaf(n.ey, w1.y, n.ez * w1.z)) * ri;
    const float ev = fmaf(n.ex, v2.x, fmaf(n.ey, v2.y, n.ez * v2.z));
    const float curve = ri * fmaf(0.5f, fmaf(-rate, rate, w1.w), ev);  // b
    const float eps = fmaf(job.bend1, rate, 2.0f * job.bend2 * curve);
    const float cubic = job.bend3 * curve;
    constexpr float q = -16.0f / (kPiF * kPiF);
    float2 b[kProfileCoefs - 2], c[kProfileCoefs - 4], e[kProfileCoefs - 6];
#pragma unroll
    for (int m = 0; m < kProfileCoefs - 2; ++m) b[m] = __fmul2_rn(a[m + 2], both(q * (float)((m + 2) * (m + 1))));
#pragma unroll
    for (int m = 0; m < kProfileCoefs - 4; ++m) c[m] = __fmul2_rn(b[m + 2], both(q * (float)((m + 2) * (m + 1))));
#pragma unroll
    for (int m = 0; m < kProfileCoefs - 6; ++m) e[m] = __fmul2_rn(c[m + 2], both(q * (float)((m + 2) * (m + 1))));
    const float e2 = -0.5f * eps * eps, e3 = -eps * eps * eps * (1.0f / 6.0f);
#pragma unroll
    for (int m = 0; m < kProfileCoefs - 2; ++m) {
        // + j eps b; + j cubic s b = cubic (4 / pi) b'
        a[m] = make_float2(fmaf(-eps, b[m].y, a[m].x), fmaf(eps, b[m].x, a[m].y));
        if (m + 1 < kProfileCoefs - 2)
            a[m] = __ffma2_rn(b[m + 1], both(cubic * (4.0f / kPiF) * (float)(m + 1)), a[m]);
        bend[m] = b[m];
        if (m < kProfileCoefs - 4) {
            a[m] = __ffma2_rn(c[m], both(e2), a[m]);
            bend[m] = make_float2(fmaf(-eps, c[m].y, b[m].x), fmaf(eps, c[m].x, b[m].y));
        }
        if (m < kProfileCoefs - 6) a[m] = make_float2(fmaf(-e3, e[m].y, a[m].x), fmaf(e3, e[m].x, a[m].y));
    }
    return eps;
}

__device__ __forceinline__ float2 neg(float2 v) { return make_float2(-v.x, -v.y); }
// a + j s b
__device__ __forceinline__ float2 plus_j(float2 a, float s, float2 b)
{
    return make_float2(fmaf(-s, b.y, a.x), fmaf(s, b.x, a.y));
}

// Vibration: a (the first table's cell) := the combined cell polynomial for the anchor's direction;
// turn_k := its gradient in the direction, coefficients of degree < kVibCoefs (it is multiplied
// by changes of direction of a few per cent; the terms left out are below 1e-3 of it).
constexpr int kVibCoefs = 6;
template <bool TURN>
__device__ __forceinline__ void vib_coefs(const Anchor &n, float4 w1, float4 axis, size_t table, int samples,
                                          const ProfileJob &job, float2 (&a)[kProfileCoefs],
                                          float2 (&tx)[kVibCoefs], float2 (&ty)[kVibCoefs], float2 (&tz)[kVibCoefs])
{
    const float ri = n.rh > 0.0f ? 2.0f * n.h * job.inv_gc : 0.0f;
    const float u[3] = {n.ex * ri, n.ey * ri, n.ez * ri};
    const float rate = fmaf(u[0], w1.x, fmaf(u[1], w1.y, u[2] * w1.z));
    const float un = fmaf(u[0], axis.x, fmaf(u[1], axis.y, u[2] * axis.z));
    // direction's turn along the chirp, times s~ = -j (2 S / pi) d/dt of j phi_k: (2 S / pi) w_k a_k'
    const float scale = (float)samples * (2.0f / kPiF) * ri;
    const float w[3] = {scale * fmaf(-rate, u[0], w1.x), scale * fmaf(-rate, u[1], w1.y),
                        scale * fmaf(-rate, u[2], w1.z)};
    // cosine to fourth order, economised over |(u.n) chi| <= A: 1 - x^2 / 2 + x^4 / 24 = 1 - A^4 / 192
    // - x^2 (1 / 2 - A^2 / 24) within A^4 / 192; and the range's second order, chi^2 (1 - (u.n)^2) / (2 2 pi gc R)
    const float u2 = un * un, ua = u2 * axis.w;
    const float c4 = u2 * fmaf(ua, 1.0f / 24.0f, -0.5f), d4 = un * fmaf(ua, 1.0f / 6.0f, -1.0f);
    const float c5 = -u2 * un * (1.0f / 6.0f), d5 = -0.5f * u2;
    const float bow = (1.0f - u2) * n.h * (job.inv_gc * job.inv_gc) * (0.5f / kPiF);
    const float one = fmaf(ua * ua, -1.0f / 192.0f, 1.0f);
#pragma unroll
    for (int m = 0; m < kProfileCoefs; ++m) a[m] = __fmul2_rn(a[m], both(one));
    const float4 *p = n.cell;
    if (!TURN) {  // (one table at a time: all five at once do not fit the registers)
#pragma unroll 1
        for (int f = 1; f < kVibTables; ++f) {
            p += table;
            const float im = f == 1 ? u[0] : f == 2 ? u[1] : f == 3 ? u[2] : f == 4 ? bow : c5;
            const float re = f == 4 ? c4 : 0.f;
            const float wf = f == 1 ? w[0] : f == 2 ? w[1] : f == 3 ? w[2] : 0.f;
#pragma unroll
            for (int m = 0; m < kProfileCoefs / 2; ++m) {
                const float4 q = __ldg(p + m);
                const float2 v0 = make_float2(q.x, q.y), v1 = make_float2(q.z, q.w);
                if (m) a[2 * m - 1] = __ffma2_rn(v0, both(wf * (float)(2 * m)), a[2 * m - 1]);
                a[2 * m] = __ffma2_rn(v1, both(wf * (float)(2 * m + 1)), __ffma2_rn(v0, both(re), plus_j(a[2 * m], im, v0)));
                a[2 * m + 1] = __ffma2_rn(v1, both(re), plus_j(a[2 * m + 1], im, v1));
            }
        }
        return;
    }
#pragma unroll
    for (int f = 1; f < kVibTables; ++f) {
        p += table;
        float2 v[kProfileCoefs];
#pragma unroll
        for (int m = 0; m < kProfileCoefs / 2; ++m) {
            const float4 q = __ldg(p + m);
            v[2 * m] = make_float2(q.x, q.y);
            v[2 * m + 1] = make_float2(q.z, q.w);
        }
        if (f < 4) {
            float2(&t)[kVibCoefs] = f == 1 ? tx : f == 2 ? ty : tz;
#pragma unroll
            for (int m = 0; m < kProfileCoefs; ++m) {
                a[m] = plus_j(a[m], u[f - 1], v[m]);
                if (m + 1 < kProfileCoefs) a[m] = __ffma2_rn(v[m + 1], both(w[f - 1] * (float)(m + 1)), a[m]);
                if (m < kVibCoefs) t[m] = make_float2(-v[m].y, v[m].x);
            }
        } else {
            // - (u.n)^2 / 2 v4, - j (u.n)^3 / 6 v5, and their gradients along n
            const float c = f == 4 ? c4 : c5, d = f == 4 ? d4 : d5;
#pragma unroll
            for (int m = 0; m < kProfileCoefs; ++m) {
                const float2 x = f == 4 ? v[m] : make_float2(-v[m].y, v[m].x);
                a[m] = __ffma2_rn(x, both(c), a[m]);
                if (f == 4) a[m] = plus_j(a[m], bow, v[m]);
                if (m < kVibCoefs) {
                    tx[m] = __ffma2_rn(x, both(d * axis.x), tx[m]);
                    ty[m] = __ffma2_rn(x, both(d * axis.y), ty[m]);
                    tz[m] = __ffma2_rn(x, both(d * axis.z), tz[m]);
                }
            }
        }
    }
}

// The gradient's change for a change (x, y, z) of direction, at place t of the cell.
__device__ __forceinline__ float2 turn_value(const float2 (&tx)[kVibCoefs], const float2 (&ty)[kVibCoefs],
                                             const float2 (&tz)[kVibCoefs], float x, float y, float z, float t)
{
    float2 h = both(0.f);
#pragma unroll
    for (int m = kVibCoefs - 1; m >= 0; --m) {
        const float2 c = __ffma2_rn(tx[m], both(x), __ffma2_rn(ty[m], both(y), __fmul2_rn(tz[m], both(z))));
        h = m == kVibCoefs - 1 ? c : __ffma2_rn(h, both(t), c);
    }
    return h;
}

// add_pair with the pixels' places t in the cell and bends eps beside the anchor's.
__device__ __forceinline__ void add_moving_pair(float2 psi, float turn, float2 t, float2 eps,
                                                const float2 (&a)[kProfileCoefs],
                                                const float2 (&bend)[kProfileCoefs - 2], float2 more0, float2 more1,
                                                float2 &c0, float2 &s0,
                                                float2 &c1, float2 &s1)
{
    const float2 n = __fadd2_rn(__fadd2_rn(psi, both(12582912.0f)), both(-12582912.0f));  // nearest integer
    const float2 x = __ffma2_rn(__fadd2_rn(psi, make_float2(-n.x, -n.y)), both(kTwoPiF), both(turn));
    float sn0, cs0, sn1, cs1;
    __sincosf(x.x, &sn0, &cs0);
    __sincosf(x.y, &sn1, &cs1);
    const float2 ta = both(t.x), tb = both(t.y);
    float2 h0 = a[kProfileCoefs - 1], h1 = h0, b0 = bend[kProfileCoefs - 3], b1 = b0;
#pragma unroll
    for (int m = kProfileCoefs - 2; m >= 0; --m) {
        h0 = __ffma2_rn(h0, ta, a[m]);
        h1 = __ffma2_rn(h1, tb, a[m]);
    }
#pragma unroll
    for (int m = kProfileCoefs - 4; m >= 0; --m) {
        b0 = __ffma2_rn(b0, ta, bend[m]);
        b1 = __ffma2_rn(b1, tb, bend[m]);
    }
    h0 = __fadd2_rn(h0, more0);
    h1 = __fadd2_rn(h1, more1);
    h0 = make_float2(fmaf(-eps.x, b0.y, h0.x), fmaf(eps.x, b0.x, h0.y));  // + j eps b
    h1 = make_float2(fmaf(-eps.y, b1.y, h1.x), fmaf(eps.y, b1.x, h1.y));
    c0 = __ffma2_rn(h0, both(cs0), c0);
    s0 = __ffma2_rn(h0, both(sn0), s0);
    c1 = __ffma2_rn(h1, both(cs1), c1);
    s1 = __ffma2_rn(h1, both(sn1), s1);
}

// Coefficients of D = A - j kappa A', kappa = cells per cycle / 2 pi (the adjoint).
__device__ __forceinline__ void adjoint_coefs(const float2 (&a)[kProfileCoefs], float cells_per_cycle,
                                              float2 (&d)[kProfileCoefs - 1])
{
    const float kappa = cells_per_cycle * (0.5f / kPiF);
#pragma unroll
    for (int m = 0; m < kProfileCoefs - 1; ++m) {
        const float c = kappa * (float)(m + 1);
        d[m] = make_float2(fmaf(c, a[m + 1].y, a[m].x), fmaf(-c, a[m + 1].x, a[m].y));
    }
}

// One chirp's terms of the adjoint for two pixels: with D = (dF/dR) / (j 2 pi gc e^{j phase}) given
// by the coefficients d, gi the image gradient (re, im) and range = R, adds
// dl = Im(conj(gi) e^{j phase} D) / R and dl x offset to the sums.
template <bool LINE>
__device__ __forceinline__ void adjoint_pair(float2 psi, float turn, float t0, float cells_per_cycle,
                                             const float2 (&d)[kProfileCoefs - 1], float w0, float w1, float2 g0,
                                             float2 g1, float2 range, float2 dx, float2 dy, float2 dz, float2 &s,
                                             float2 &sx, float2 &sy, float2 &sz)
{
    const float2 x = phase_of<LINE>(psi, turn);
    const float2 t = __ffma2_rn(psi, both(cells_per_cycle), both(t0));
    float sn0, cs0, sn1, cs1;
    __sincosf(x.x, &sn0, &cs0);
    __sincosf(x.y, &sn1, &cs1);
    const float2 ta = both(t.x), tb = both(t.y);
    float2 h0 = d[kProfileCoefs - 2], h1 = h0;
#pragma unroll
    for (int m = kProfileCoefs - 3; m >= 0; --m) {
        h0 = __ffma2_rn(h0, ta, d[m]);
        h1 = __ffma2_rn(h1, tb, d[m]);
    }
    // Im(conj(g) e^{j x} h) = (g.im cos - g.re sin)... written out: g = gi, t = e^{j x} h,
    // g.im t.re - g.re t.im
    const float p0 = g0.y * cs0 - g0.x * sn0, q0 = g0.y * sn0 + g0.x * cs0;
    const float p1 = g1.y * cs1 - g1.x * sn1, q1 = g1.y * sn1 + g1.x * cs1;
    const float2 dl = make_float2(w0 * __fdividef(p0 * h0.x - q0 * h0.y, range.x),
                                  w1 * __fdividef(p1 * h1.x - q1 * h1.y, range.y));
    s = __fadd2_rn(s, dl);
    sx = __ffma2_rn(dl, dx, sx);
    if (LINE) return;  // (offsets along one axis only)
    sy = __ffma2_rn(dl, dy, sy);
    sz = __ffma2_rn(dl, dz, sz);
}

// CTAs per SM the registers of an instance are limited to.
constexpr int focus_ctas(int group, bool band, bool adjoint, int motion)
{
    if (group == 16) return adjoint ? 4 : 6;
    if (motion == 2) return 4;
    if (group == 1) return band || adjoint ? 4 : 6;
    return band || motion || (adjoint && group == 2) ? 6 : TDC_PROFILE_MINB;
}

// Persistent CTAs of 64 threads over units (tile x chirp group) from an atomic counter, 8
// pixels a thread. Per chirp, each G consecutive pixels share an anchor pixel: its range R0,
// the carrier phase frac(gc R0) and the cell it reads (64 bytes, from L1 / L2: neighbouring
// threads read the same few cells) are formed once in double-float. A pixel then takes its
// phase difference from the anchor, psi = gc (R - R0) cycles, from
//   Q = gc (R^2 - R0^2) / (2 R0) = d.e' + |d|^2 h     (d = pixel - anchor, 4 operations),
//   psi = Q (1 + b1 Q + b2 Q^2 + b3 Q^3)              (sqrt(1 + y) - 1, y = Q k2 small),
// where y is small (|y| <= 0.061, reach / R0 <= 0.03), or from the exact
// quotient otherwise, and the cell's polynomial at t0 + psi x cells per cycle. About 28
// operations a pixel and chirp on runs along an axis, 33 off it, plus 110 per anchor, whatever the
// row's length.
//
// Bound: the FMA pipe (72% busy, 61% of the issue slots, on 512^2 x 2048 x 1024). What brought it
// there, 1024^2 x 4096 x 1024 each: scalar FMAs 9.6 ms; pairs of pixels in FFMA2 (half the issue
// slots) 7.7; the next anchor formed beside this one's pixels 7.5; blocks of 8 runs x 32 pixels a
// warp instead of 256 pixels of a run, and chirp records staged in shared memory 32 at a time,
// 7.2-7.4 (the cells' wait for memory: 1.5 -> 0.4 cycles an instruction). 64-thread CTAs at 128
// registers: 16 warps an SM; 12 or 18 warps are 2-6% slower. With the cells in L1, forming the next
// anchor ahead costs more registers than it hides (7.05 -> 6.72 ms without).
//
// G = 16: 16 pixels a thread and one anchor for them (LINE only: the offsets of 16 vectors do not fit the
// registers), 162 registers, 12 warps an SM: 6.06 -> 5.27 ms (5 CTAs an SM 5.42). FMA pipe 66%, issue
// 53%; half the cells' sectors come from L2.
//
// BAND: a finite Doppler band. Chirps out of band for all of a warp's pixels are found first, 32
// at a time, from the anchors' Doppler and a bound on its change over a group (about 20
// operations an anchor and chirp); the others weight each pixel with its own window.
//
// ADJ: the adjoint with respect to the chirps' positions. F(R) = e^{j 2 pi gc R} A(t), so
// dF/dR = j 2 pi gc e^{j ...} D, D = A - j (cells per cycle / 2 pi) A'(t): the same evaluation with
// the coefficients of D, formed once an anchor. Each chirp's sum over the tile's pixels (two
// shuffle steps, then shared memory, 32 chirps at a time) goes to gpart[tile][chirp].
//
// MOVE: positions moving within each chirp, R_s = R + a s~ + b s~^2 about the middle sample (s~ = s -
// sc, a = e.W1 / R, b = (|W1|^2 - a^2) / (2 R) + e.V2 / R), so the phase of sample s is
//   gc R + s~ (g1 R + gc a) + s~^2 (g1 a + gc b) + s~^3 g1 b  cycles.
// The linear part is a shift of the cell coordinate by 4 S gc a. The rest is small (the host
// bounds it to 0.1 rad at the row's ends, eps there): s~ is -j (2 S / pi) d/dt on A(t), so with
// B = s~^2 A (in units of the half row) and so on, e^{j eps s~^2} A = A + j eps B - eps^2 / 2 C
// - j eps^3 / 6 E, all polynomials of the cell formed once an anchor; the pixel's difference in
// eps from its anchor, at most a few per cent of it, enters to first order. 64 x 512 pixels x 512
// chirps x 1024 samples: 2.64 ms in the per-segment kernel of tdc_motion.cu, 0.092 ms here.
//
// MOVE = 2: vibration about a constant velocity, rho_s = P[c, s] minus the chirp's line. Its phase is
// psi_s = u.phi_s (u = e / R the direction of the antenna, phi = 2 pi g_s rho, at most 0.1 rad), so
//   e^{j psi} = 1 + j u.phi - (u.n)^2 chi^2 / 2 - j (u.n)^3 chi^3 / 6,
// six tables of the same samples times 1, phi_x, phi_y, phi_z, chi^2 and chi^3 (chi = n.phi, n the
// principal direction of the chirp's deviations: what lies off it, the rounding of the FP32
// positions, is kept to first order). An anchor combines them for its own u into one cell
// polynomial; the direction turning along the chirp (W1 / R) enters through the derivative of
// the phi tables, a pixel's own direction as the polynomial's gradient in u, to first order.
// 151 x 97 pixels x 333 chirps x 500 samples: 1930 us in the general kernel of tdc_general.cu, which
// corrects every sample, 94 us here (40 the six tables, 52 this kernel).
//
// LINE: every group's pixels lie on a line parallel to one axis (sP.axis; checked when the grid is
// measured: the offsets along the others are exactly zero) and span at most kLineMaxCycles carrier
// cycles. The offsets are one number a pixel, in registers: Q = d (e' + d h) in 2 operations, and
// the phase needs no reduction: 5 operations of 45 a pixel and chirp less (1024^2 x 4096 x 1024: 6.52 ->
// 6.06 ms; adjoint and finite band likewise 7-10%).
template <int G, bool BAND, bool ADJ, int MOVE, bool LINE>
__global__ void __launch_bounds__(kThreads, focus_ctas(G, BAND, ADJ, MOVE))
    profile_focus_kernel(const FocusJob *__restrict__ jobs, const FocusUnit *__restrict__ units, int n_units,
                         int *__restrict__ counter, const float2 *__restrict__ gimg, float4 *__restrict__ gpart)
{
    constexpr int PT = G == 16 ? 16 : kPT;  // pixels per thread
    constexpr int kSub = PT / G;            // anchors per thread
    __shared__ SharedSums<PT> sums;
    static_assert(!MOVE || (!BAND && !ADJ), "smooth motion: unbounded band, forward only");
    static_assert(!LINE || (G > 1 && !MOVE), "runs along an axis: still antennas, shared anchors");
    static_assert(G < 16 || (LINE && !BAND), "groups of 16: runs along an axis, unbounded band");
    constexpr int kWords = MOVE == 2 ? 6 : MOVE ? 4 : BAND ? 3 : 2;  // float4 staged per record
    constexpr int kStride = MOVE ? kWords : 3;                      // float4 per record in memory
    __shared__ __align__(16) SharedChirps<kWords> recs[2];
    __shared__ float red[ADJ ? kFlush : 1][3][kThreads / 4];  // (ADJ) 8 partial sums a warp
    __shared__ int s_unit;
    __shared__ FocusUnit un;
    __shared__ FocusJob sJ;
    __shared__ ProfileJob sP;
    const int tid = threadIdx.x;

    for (;;) {
        __syncthreads();
        if (tid == 0) {
            s_unit = atomicAdd(counter, 1);
            if (s_unit < n_units) un = units[s_unit];
        }
        __syncthreads();
        if (s_unit >= n_units) break;
        for (int i = tid; i < (int)(sizeof(FocusJob) / sizeof(int)); i += kThreads)
            reinterpret_cast<int *>(&sJ)[i] = reinterpret_cast<const int *>(&jobs[un.job])[i];
        if (tid < (int)(sizeof(ProfileJob) / 16))
            reinterpret_cast<float4 *>(&sP)[tid] = reinterpret_cast<const float4 *>(jobs[un.job].profile)[tid];
        __syncthreads();

        const int c0 = un.group * sJ.chirps_per_group;
        const int c1 = min(sJ.C, c0 + sJ.chirps_per_group);
        const int axis = LINE ? sP.axis : 0;
        auto along = [&](float x, float y, float z) { return axis == 0 ? x : axis == 1 ? y : z; };

        // anchors (the middle pixel of each group) and the pixels' offsets from them, in pairs
        float ax[kSub][6];
        float2 dx[PT / 2], dy[PT / 2];
        int count;
        long long p0 = run_pixels<PT>(sJ.P, sJ.grid_cols, un.tile, tid, count);
#pragma unroll
        for (int g = 0; g < kSub; ++g) {
            const int valid = min(max(count - g * G, 0), G);
            float4 hi = make_float4(0.f, 0.f, 0.f, 0.f), lo = hi;
            if (valid) {
                const long long a = p0 + g * G + valid / 2;
                hi = __ldg(&sJ.grid_hi[a]);
                if (sJ.grid_lo) lo = __ldg(&sJ.grid_lo[a]);
            }
            ax[g][0] = hi.x;
            ax[g][1] = hi.y;
            ax[g][2] = hi.z;
            ax[g][3] = lo.x;
            ax[g][4] = lo.y;
            ax[g][5] = lo.z;
            if (G > 1) {
                float ox[G], oy[G], oz[G];
#pragma unroll
                for (int i = 0; i < G; ++i) {
                    const int s = g * G + i;
                    ox[i] = oy[i] = oz[i] = 0.f;
                    if (s < count) {
                        const float4 h = __ldg(&sJ.grid_hi[p0 + s]);
                        const float4 l = sJ.grid_lo ? __ldg(&sJ.grid_lo[p0 + s]) : make_float4(0.f, 0.f, 0.f, 0.f);
                        float rest;  // (rounded as e is: they are equal where the antenna is on the pixel)
                        difference(h.x, l.x, hi.x, lo.x, ox[i], rest);
                        difference(h.y, l.y, hi.y, lo.y, oy[i], rest);
                        difference(h.z, l.z, hi.z, lo.z, oz[i], rest);
                    }
                }
#pragma unroll
                for (int i = 0; i + 1 < G; i += 2) {
                    const int q = (g * G + i) / 2;
                    if (LINE) {
                        dx[q] = make_float2(along(ox[i], oy[i], oz[i]), along(ox[i + 1], oy[i + 1], oz[i + 1]));
                        continue;
                    }
                    dx[q] = make_float2(ox[i], ox[i + 1]);
                    dy[q] = make_float2(oy[i], oy[i + 1]);
                    const float2 dz = make_float2(oz[i], oz[i + 1]);
                    sums.dz[q][tid] = dz;
                    sums.dd[q][tid] = __ffma2_rn(dx[q], dx[q], __ffma2_rn(dy[q], dy[q], __fmul2_rn(dz, dz)));
                }
            }
        }
        float2 hc[PT], hs[PT];  // (hs stays zero where a pixel is its own anchor)
#pragma unroll
        for (int i = 0; i < PT; ++i) {
            hc[i] = hs[i] = make_float2(0.f, 0.f);
            sums.s[i][tid] = make_float4(0.f, 0.f, 0.f, 0.f);
        }

        float2 gi[PT];  // (ADJ) image gradient of the pixels
        auto load_gradient = [&](unsigned int without) {
#pragma unroll
            for (int i = 0; i < PT; ++i)
                gi[i] = i < count && !(without >> i & 1u) ? __ldg(&gimg[p0 + i]) : make_float2(0.f, 0.f);
        };
        if (ADJ) load_gradient(0);

        const float4 *__restrict__ chirps = reinterpret_cast<const float4 *>(sJ.chirps);
        const int *__restrict__ cell_base = sP.cell_base;
        const float4 *__restrict__ cells = sP.cells;
        const bool skip_test = (sJ.flags & kFlagSkipTest) != 0;
        unsigned int dropped = 0;  // pixels whose current chunk the skip test drops
        int chunk_end = c0;

        int b0 = c0, buf = 0;  // first chirp of the staged records, and their buffer
        auto anchor_of = [&](int k, const float (&p)[6]) {
            Anchor n;
            const float4 ph = recs[buf].p[k][0], pl = recs[buf].p[k][1];
            const int base = recs[buf].base[k];
            const float4 g = fresh(&sP.gc_hi);  // gc and cells per metre, high and low parts
            const int n_cells = __float_as_int(fresh(&sP.inv_gc2x4).w);
            float exl, eyl, ezl, rl, rs, dh;
            difference(ph.x, pl.x, p[0], p[3], n.ex, exl);
            difference(ph.y, pl.y, p[1], p[4], n.ey, eyl);
            difference(ph.z, pl.z, p[2], p[5], n.ez, ezl);
            dd_range(n.ex, exl, n.ey, eyl, n.ez, ezl, n.rh, rl, rs, dh);
            // gc / (2 R0), 1 / R0 to FP32 rounding (rsqrt is not)
            const float rinv = fmaf(rs, fmaf(-rl, rs, fmaf(-n.rh, rs, 1.0f)), rs);
            n.h = 0.5f * g.x * rinv;
            // its cell, and its place in it
            float shift = 0.f;
            if (MOVE) {
                const float4 w1 = recs[buf].p[k][MOVE ? 2 : 0];
                shift = sP.rate_cells * (fmaf(n.ex, w1.x, fmaf(n.ey, w1.y, n.ez * w1.z)) * rinv);
                if (!(n.rh > 0.0f)) shift = 0.f;
            }
            const float kf = rintf(fmaf(g.z, n.rh, shift));
            n.t0 = fmaf(g.z, n.rh, -kf);
            n.t0 = fmaf(g.z, rl, n.t0);
            n.t0 = fmaf(g.w, n.rh, n.t0);
            if (MOVE) n.t0 += shift;
            const int cell = min(max((int)kf - base, 0), n_cells - 1);
            const float4 *__restrict__ pc = cells + ((size_t)(b0 + k) * n_cells + cell) * (kProfileCoefs / 2);
            if (MOVE == 2) n.cell = pc;
#pragma unroll
            for (int m = 0; m < kProfileCoefs / 2; ++m) {
                const float4 v = __ldg(pc + m);
                n.a[2 * m] = make_float2(v.x, v.y);
                n.a[2 * m + 1] = make_float2(v.z, v.w);
            }
            n.turn = kTwoPiF * dd_frac_mul(g.x, g.y, n.rh, rl);
            if (MOVE) n.w = shift;
            if (BAND && G == 1) {
                const float4 v = recs[buf].p[k][2];
                // (from the high parts, as the direct kernels, unless the low parts move the direction)
                float dx = ph.x - p[0], dy = ph.y - p[1], dz = ph.z - p[2];
                if (fabsf(n.ex - dx) + fabsf(n.ey - dy) + fabsf(n.ez - dz) > 2e-6f * n.rh) {
                    dx = n.ex;
                    dy = n.ey;
                    dz = n.ez;
                }
                const float fd = doppler_freq(sJ.two_over_lambda, v.x, v.y, v.z, dx, dy, dz, rs);
                n.w = doppler_window(fd, ph.w, sJ.half_bw, sJ.inv_bw, (sJ.flags & kFlagTaper) != 0, sJ.az_a);
            }
            return n;
        };
        // the next block's records are copied while this one is worked on: thread tid copies half of
        // record tid / 2
        auto copy_ahead = [&](int first, int to) {
            if (first + (tid >> 1) < c1)
                copy_async<16>(&recs[to].p[tid >> 1][tid & 1], chirps + (size_t)(first + (tid >> 1)) * kStride + (tid & 1));
            if (kWords > 2 && tid < kFlush && first + tid < c1)
#pragma unroll
                for (int v = 2; v < kWords; ++v)
                    copy_async<16>(&recs[to].p[tid][v], chirps + (size_t)(first + tid) * kStride + v);
            if (tid < kFlush && first + tid < c1) copy_async<4>(&recs[to].base[tid], &cell_base[first + tid]);
        };
        copy_ahead(c0, 0);

        while (b0 < c1) {
            copy_async_wait();
            __syncthreads();  // this block's records are in, every thread is done with the last one's
            if (skip_test && b0 >= chunk_end) {
                // (unbounded band: a chunk is dropped only where the test's first point is NaN)
                const int k = b0 / sJ.chunk;
                chunk_end = (k + 1) * sJ.chunk;
                dropped = 0;
                p0 = run_pixels<PT>(sJ.P, sJ.grid_cols, un.tile, tid, count);  // (cheaper than two registers)
                const float4 pf = __ldg(&sJ.skip[(size_t)k * 9].pos_fdc);
                const float4 v = __ldg(&sJ.skip[(size_t)k * 9].vel);
#pragma unroll 1
                for (int i = 0; i < count; ++i) {
                    const float4 h = __ldg(&sJ.grid_hi[p0 + i]);
                    if (BAND) {
                        if (!chunk_is_nonzero(sJ.skip + (size_t)k * 9, h.x, h.y, h.z, sJ.two_over_lambda, sJ.half_bw))
                            dropped |= 1u << i;
                        continue;
                    }
                    const float ex = pf.x - h.x, ey = pf.y - h.y, ez = pf.z - h.z;
                    const float rs = rsqrtf(ex * ex + ey * ey + ez * ez);
                    const float val =
                        fabsf(doppler_freq(sJ.two_over_lambda, v.x, v.y, v.z, ex, ey, ez, rs) - pf.w);
                    if (!(val <= sJ.half_bw)) dropped |= 1u << i;
                }
                if (ADJ) load_gradient(dropped);
            }
            int n = min(kFlush, c1 - b0);
            if (skip_test) n = min(n, chunk_end - b0);
            copy_ahead(b0 + n, buf ^ 1);
            if (ADJ && BAND) {  // (chirps out of band keep zero sums)
                if ((tid & 31) < 8)
                    for (int i = 0; i < kFlush * 3; ++i) red[i / 3][i % 3][(tid >> 5) * 8 + (tid & 31)] = 0.f;
                __syncwarp();
            }
            unsigned int todo = 0xffffffffu >> (kFlush - n);  // chirps of the block still to add
            if constexpr (BAND) {
                unsigned int live = 0;
                if (dropped != (1u << count) - 1u)  // (some pixel's chunk is seen)
                    for (int k = 0; k < n; ++k) {
                        const float4 p = recs[buf].p[k][0], pl = recs[buf].p[k][1], v = recs[buf].p[k][2];
                        bool any = false;
#pragma unroll
                        for (int g = 0; g < kSub; ++g) {
                            // (the low parts are a direction of their own: 1e-3 at 1 km and ranges of 6 cm)
                            const float ex = (p.x - ax[g][0]) + (pl.x - ax[g][3]),
                                        ey = (p.y - ax[g][1]) + (pl.y - ax[g][4]),
                                        ez = (p.z - ax[g][2]) + (pl.z - ax[g][5]);
                            const float rs = rsqrtf(fmaf(ex, ex, fmaf(ey, ey, ez * ez)));
                            const float tol = sJ.two_over_lambda;
                            const float fd = doppler_freq(tol, v.x, v.y, v.z, ex, ey, ez, rs);
                            // directions within the group differ by at most 2 sin(asin(reach / R) / 2)
                            const float rel = sP.reach * rs;
                            const float bound = 1.05f * tol * (fabsf(v.x) + fabsf(v.y) + fabsf(v.z)) * rel +
                                                1e-4f * (fabsf(fd) + fabsf(p.w) + sJ.half_bw) + 1e-6f;
                            any |= !(fabsf(fd - p.w) > sJ.half_bw + bound) || !(rel < 0.4f);
                        }
                        if (any) live |= 1u << k;
                    }
                todo &= __reduce_or_sync(0xffffffffu, live);
            }
            int k = __ffs(todo) - 1;
            while (todo) {
                todo &= todo - 1;
                const int k_next = __ffs(todo) - 1;
                float grad[3] = {0.f, 0.f, 0.f};
#pragma unroll
                for (int g = 0; g < kSub; ++g) {
                    const Anchor cur = anchor_of(k, ax[g]);
                    if constexpr (G == 1) {
                        // (the antenna on the pixel: NaN Doppler, zero window)
                        float sn, cs;
                        __sincosf(cur.turn, &sn, &cs);
                        if (!(cur.rh > 0.0f)) sn = cs = 0.0f;
                        if (BAND) {
                            sn *= cur.w;
                            cs *= cur.w;
                        }
                        if constexpr (ADJ) {
                            float2 d[kProfileCoefs - 1];
                            adjoint_coefs(cur.a, fresh(&sP.inv_gc2x4).y, d);
                            float2 h = d[kProfileCoefs - 2];
#pragma unroll
                            for (int m = kProfileCoefs - 3; m >= 0; --m) h = __ffma2_rn(h, both(cur.t0), d[m]);
                            const float p = gi[g].y * cs - gi[g].x * sn, q = gi[g].y * sn + gi[g].x * cs;
                            const float dl = cur.rh > 0.0f ? __fdividef(p * h.x - q * h.y, cur.rh) : 0.0f;
                            grad[0] = fmaf(dl, cur.ex, grad[0]);
                            grad[1] = fmaf(dl, cur.ey, grad[1]);
                            grad[2] = fmaf(dl, cur.ez, grad[2]);
                            continue;
                        }
                        float2 a[kProfileCoefs];
#pragma unroll
                        for (int m = 0; m < kProfileCoefs; ++m) a[m] = cur.a[m];
                        if constexpr (MOVE) {
                            float2 bend[kProfileCoefs - 2];
                            if constexpr (MOVE == 2) {
                                float2 turn_x[kVibCoefs], turn_y[kVibCoefs], turn_z[kVibCoefs];
                                vib_coefs<false>(cur, recs[buf].p[k][2], recs[buf].p[k][kWords - 1],
                                          (size_t)sJ.C * sP.n_cells * (kProfileCoefs / 2), sJ.S, sP, a, turn_x, turn_y,
                                          turn_z);
                            }
                            move_coefs(cur, recs[buf].p[k][2], recs[buf].p[k][3 % kWords], sP, a, bend);
                        }
                        float2 h = a[kProfileCoefs - 1];
#pragma unroll
                        for (int m = kProfileCoefs - 2; m >= 0; --m) h = __ffma2_rn(h, both(cur.t0), a[m]);
                        hc[g].x = fmaf(cs, h.x, fmaf(-sn, h.y, hc[g].x));
                        hc[g].y = fmaf(cs, h.y, fmaf(sn, h.x, hc[g].y));
                    } else if constexpr (G == 16 && !ADJ) {
                        // (as below, each pair's phase difference formed where it is used: 16 at once do not
                        // fit the registers)
                        const float4 jc = fresh(&sP.inv_gc2x4);
                        const float ea = along(cur.ex, cur.ey, cur.ez);
                        if (cur.rh >= jc.z) {
                            const float h = cur.h, e2 = -2.0f * h * ea, k2 = h * jc.x;
                            const float b1 = kWide1 * k2, b2 = kWide2 * k2 * k2, b3 = kWide3 * k2 * k2 * k2,
                                        b4 = kWide4 * (k2 * k2) * (k2 * k2);
#pragma unroll
                            for (int i = 0; i < G; i += 2) {
                                const float2 q = __fmul2_rn(dx[i / 2], __ffma2_rn(dx[i / 2], both(h), both(e2)));
                                float2 f = __ffma2_rn(q, both(b4), both(b3));
                                f = __ffma2_rn(q, f, both(b2));
                                f = __ffma2_rn(q, f, both(b1));
                                add_pair<false, true>(__ffma2_rn(__fmul2_rn(q, q), f, q), cur.turn, cur.t0, jc.y, cur.a,
                                                      1.f, 1.f, hc[i], hs[i], hc[i + 1], hs[i + 1]);
                            }
                        } else if (cur.rh >= jc.z * (10.0f / 21.0f)) {
                            // |y| <= 0.2: the Taylor series to y^7, 6e-8 left
                            const float h = cur.h, e2 = -2.0f * h * ea, k2 = h * jc.x;
#pragma unroll
                            for (int i = 0; i < G; i += 2) {
                                const float2 q = __fmul2_rn(dx[i / 2], __ffma2_rn(dx[i / 2], both(h), both(e2)));
                                const float2 y = __fmul2_rn(q, both(k2));
                                float2 f = __ffma2_rn(y, both(-429.0f / 16384.0f), both(33.0f / 1024.0f));
                                f = __ffma2_rn(y, f, both(-21.0f / 512.0f));
                                f = __ffma2_rn(y, f, both(7.0f / 128.0f));
                                f = __ffma2_rn(y, f, both(-5.0f / 64.0f));
                                f = __ffma2_rn(y, f, both(0.125f));
                                f = __ffma2_rn(y, f, both(-0.25f));
                                add_pair<false, true>(__ffma2_rn(__fmul2_rn(q, y), f, q), cur.turn, cur.t0, jc.y, cur.a, 1.f,
                                                      1.f, hc[i], hs[i], hc[i + 1], hs[i + 1]);
                            }
                        } else {
                            // e's part off the axis, squared
                            const float sx = axis == 0 ? 0.f : cur.ex, sy = axis == 1 ? 0.f : cur.ey,
                                        sz = axis == 2 ? 0.f : cur.ez;
                            const float off2 = fmaf(sx, sx, fmaf(sy, sy, sz * sz));
#pragma unroll
                            for (int i = 0; i < G; i += 2) {
                                float2 psi;
                                bool on[2];
#pragma unroll
                                for (int j = 0; j < 2; ++j) {
                                    const float x = j ? dx[i / 2].y : dx[i / 2].x, v = ea - x;
                                    const float r2 = fmaf(v, v, off2), den = cur.rh + sqrtf(r2);
                                    const float d = den > 0.0f ? sP.gc_hi * (x * fmaf(-2.0f, ea, x) / den) : 0.0f;
                                    if (j) psi.y = d;
                                    else psi.x = d;
                                    on[j] = !(r2 > 0.0f);  // (the antenna on the pixel: NaN Doppler, zero window)
                                    if (on[j] && !(dropped >> (i + j) & 1u)) stash(sums, i + j, tid, hc[i + j], hs[i + j]);
                                }
                                add_pair<false, true>(psi, cur.turn, cur.t0, jc.y, cur.a, 1.f, 1.f, hc[i], hs[i], hc[i + 1],
                                                      hs[i + 1]);
#pragma unroll
                                for (int j = 0; j < 2; ++j)
                                    if (on[j]) hc[i + j] = hs[i + j] = make_float2(0.f, 0.f);
                            }
                        }
                    } else {
                        float2 psi[G / 2];
                        unsigned int zero = 0;  // pixels the antenna stands on
                        const float4 jc = fresh(&sP.inv_gc2x4);  // 4 / gc^2, cells per cycle, r_safe
                        if (cur.rh >= jc.z) {
                            const float h = cur.h, h2 = -2.0f * h;
                            const float e2x = h2 * cur.ex, e2y = h2 * cur.ey, e2z = h2 * cur.ez;
                            const float k2 = h * jc.x;
                            constexpr bool kWide = G == 16;
                            const float b1 = (kWide ? kWide1 : -0.25f) * k2, b2 = (kWide ? kWide2 : kRoot2) * k2 * k2;
                            const float b3 = (kWide ? kWide3 : kRoot3) * k2 * k2 * k2;
                            const float b4 = kWide4 * (k2 * k2) * (k2 * k2);
#pragma unroll
                            for (int i = 0; i < G / 2; ++i) {
                                const int s = g * (G / 2) + i;
                                const float2 q =
                                    LINE ? __fmul2_rn(dx[s], __ffma2_rn(dx[s], both(h), both(along(e2x, e2y, e2z))))
                                         : __ffma2_rn(dx[s], both(e2x),
                                                      __ffma2_rn(dy[s], both(e2y),
                                                                 __ffma2_rn(fresh2(&sums.dz[s][tid]), both(e2z),
                                                                            __fmul2_rn(fresh2(&sums.dd[s][tid]), both(h)))));
                                float2 f = kWide ? __ffma2_rn(q, both(b4), both(b3)) : both(b3);
                                f = __ffma2_rn(q, f, both(b2));
                                f = __ffma2_rn(q, f, both(b1));
                                psi[i] = __ffma2_rn(__fmul2_rn(q, q), f, q);
                            }
                        } else {
                            // R - R0 = d.(d - 2 e) / (R0 + R): no cancellation, any R0
#pragma unroll
                            for (int i = 0; i < G; ++i) {
                                const int s = (g * G + i) / 2;
                                float x = i & 1 ? dx[s].y : dx[s].x, y, z;
                                if (LINE) {
                                    y = axis == 1 ? x : 0.f;
                                    z = axis == 2 ? x : 0.f;
                                    x = axis == 0 ? x : 0.f;
                                } else {
                                    y = i & 1 ? dy[s].y : dy[s].x;
                                    z = i & 1 ? sums.dz[s][tid].y : sums.dz[s][tid].x;
                                }
                                const float vx = cur.ex - x, vy = cur.ey - y, vz = cur.ez - z;
                                const float num = fmaf(x, fmaf(-2.0f, cur.ex, x),
                                                       fmaf(y, fmaf(-2.0f, cur.ey, y), z * fmaf(-2.0f, cur.ez, z)));
                                const float r2 = fmaf(vx, vx, fmaf(vy, vy, vz * vz));
                                const float den = cur.rh + sqrtf(r2);
                                const float v = den > 0.0f ? sP.gc_hi * (num / den) : 0.0f;
                                if (i & 1) psi[i / 2].y = v;
                                else psi[i / 2].x = v;
                                // (the antenna on the pixel: NaN Doppler, zero window)
                                if (!(r2 > 0.0f)) zero |= 1u << i;
                            }
                        }
                        if (!BAND && !ADJ && zero) {
#pragma unroll
                            for (int i = 0; i < G; ++i)
                                if ((zero & ~(dropped >> (g * G))) >> i & 1u)
                                    stash(sums, g * G + i, tid, hc[g * G + i], hs[g * G + i]);
                        }
                        // Doppler windows of the pixels, fd = -(2 / lambda) v.(e - d) / R
                        float w[G];
                        if constexpr (BAND) {
                            const float4 v = recs[buf].p[k][2];
                            const float fdc = recs[buf].p[k][0].w, tol = sJ.two_over_lambda;
                            const float half = sJ.half_bw, inv_bw = sJ.inv_bw, az = sJ.az_a;
                            const bool taper = (sJ.flags & kFlagTaper) != 0;
                            const float tx = tol * v.x, ty = tol * v.y, tz = tol * v.z;
                            const float te = -fmaf(tx, cur.ex, fmaf(ty, cur.ey, tz * cur.ez));
                            const float slack = 2e-6f * (fabsf(tx) + fabsf(ty) + fabsf(tz)) +
                                                1e-6f * (fabsf(fdc) + half);
                            unsigned int edge = 0;  // pixels at the band's edge to FP32 rounding
#pragma unroll
                            for (int i = 0; i < G; i += 2) {
                                const int s = (g * G + i) / 2;
                                const float2 dot =
                                    LINE ? __ffma2_rn(dx[s], both(along(tx, ty, tz)), both(te))
                                         : __ffma2_rn(dx[s], both(tx),
                                                      __ffma2_rn(dy[s], both(ty),
                                                                 __ffma2_rn(fresh2(&sums.dz[s][tid]), both(tz), both(te))));
                                const float2 r = __ffma2_rn(psi[i / 2], both(sP.inv_gc), both(cur.rh));
#pragma unroll
                                for (int q = 0; q < 2; ++q) {
                                    const float df = __fdividef(q ? dot.y : dot.x, q ? r.y : r.x) - fdc;
                                    w[i + q] = 0.0f;
                                    if (fabsf(df) <= half)
                                        w[i + q] = taper ? fmaf(1.0f - az, __cosf(kTwoPiF * df * inv_bw), az) : 1.0f;
                                    if (fabsf(fabsf(df) - half) <= slack) edge |= 1u << (i + q);
                                }
                            }
                            while (edge) {
                                // the side of the edge is decided as the direct kernels decide it, from the high
                                // parts of the direction; low parts that move it further than the doubt count
                                const int i = __ffs(edge) - 1;
                                edge &= edge - 1;
                                int m;
                                const long long p = run_pixels<PT>(sJ.P, sJ.grid_cols, un.tile, tid, m) + g * G + i;
                                const float4 ph = recs[buf].p[k][0], pl = recs[buf].p[k][1];
                                const float4 hi = g * G + i < m ? __ldg(&sJ.grid_hi[p]) : ph;
                                const float4 lo = g * G + i < m && sJ.grid_lo ? __ldg(&sJ.grid_lo[p])
                                                                              : make_float4(0.f, 0.f, 0.f, 0.f);
                                float ex, ey, ez, exl, eyl, ezl, rh, rl, rs, dh;
                                dd_sub(ph.x, pl.x, hi.x, lo.x, ex, exl);
                                dd_sub(ph.y, pl.y, hi.y, lo.y, ey, eyl);
                                dd_sub(ph.z, pl.z, hi.z, lo.z, ez, ezl);
                                if (fabsf(exl) + fabsf(eyl) + fabsf(ezl) > 2e-6f * cur.rh) {
                                    difference(ph.x, pl.x, hi.x, lo.x, ex, exl);
                                    difference(ph.y, pl.y, hi.y, lo.y, ey, eyl);
                                    difference(ph.z, pl.z, hi.z, lo.z, ez, ezl);
                                }
                                dd_range(ex, exl, ey, eyl, ez, ezl, rh, rl, rs, dh);
                                const float fd = doppler_freq(tol, v.x, v.y, v.z, ex, ey, ez, rs);
                                const float we = doppler_window(fd, fdc, half, inv_bw, taper, az);
#pragma unroll
                                for (int q = 0; q < G; ++q)
                                    if (q == i) w[q] = we;
                            }
#pragma unroll
                            for (int i = 0; i < G; ++i)
                                if (zero >> i & 1u) w[i] = 0.0f;
                        } else {
#pragma unroll
                            for (int i = 0; i < G; ++i) w[i] = ADJ && (zero >> i & 1u) ? 0.0f : 1.0f;
                        }
                        if constexpr (ADJ) {
                            float2 d[kProfileCoefs - 1];
                            adjoint_coefs(cur.a, jc.y, d);
                            float2 sum = both(0.f), sx = sum, sy = sum, sz = sum;
#pragma unroll
                            for (int i = 0; i < G; i += 2) {
                                const int s = (g * G + i) / 2;
                                float2 r = __ffma2_rn(psi[i / 2], both(sP.inv_gc), both(cur.rh));
                                if (zero >> i & 1u) r.x = 1.0f;
                                if (zero >> (i + 1) & 1u) r.y = 1.0f;
                                float2 oy = both(0.f), oz = oy;
                                if (!LINE) {
                                    oy = dy[s];
                                    oz = fresh2(&sums.dz[s][tid]);
                                }
                                adjoint_pair<LINE>(psi[i / 2], cur.turn, cur.t0, jc.y, d, w[i], w[i + 1], gi[g * G + i],
                                                   gi[g * G + i + 1], r, dx[s], oy, oz, sum, sx, sy, sz);
                            }
                            // sum over the pixels of dl (e - d)
                            const float all = sum.x + sum.y;
                            float bx = sx.x + sx.y, by = sy.x + sy.y, bz = sz.x + sz.y;
                            if (LINE) {
                                by = axis == 1 ? bx : 0.f;
                                bz = axis == 2 ? bx : 0.f;
                                bx = axis == 0 ? bx : 0.f;
                            }
                            grad[0] += fmaf(all, cur.ex, -bx);
                            grad[1] += fmaf(all, cur.ey, -by);
                            grad[2] += fmaf(all, cur.ez, -bz);
                            continue;
                        }
                        if constexpr (MOVE) {
                            const float4 w1 = recs[buf].p[k][2], v2 = recs[buf].p[k][3 % kWords];
                            float2 a[kProfileCoefs], bend[kProfileCoefs - 2];
#pragma unroll
                            for (int m = 0; m < kProfileCoefs; ++m) a[m] = cur.a[m];
                            constexpr int kTurn = MOVE == 2 ? kVibCoefs : 1;
                            float2 turn_x[kTurn], turn_y[kTurn], turn_z[kTurn];
                            if constexpr (MOVE == 2)
                                vib_coefs<true>(cur, w1, recs[buf].p[k][kWords - 1],
                                          (size_t)sJ.C * sP.n_cells * (kProfileCoefs / 2), sJ.S, sP, a, turn_x, turn_y,
                                          turn_z);
                            const float ri0 = 2.0f * cur.h * sP.inv_gc;
                            const float eps0 = move_coefs(cur, w1, v2, sP, a, bend);
                            const float ew = fmaf(cur.ex, w1.x, fmaf(cur.ey, w1.y, cur.ez * w1.z));
                            const float bend_v = 2.0f * sP.bend2 * fmaf(cur.ex, v2.x, fmaf(cur.ey, v2.y, cur.ez * v2.z));
#pragma unroll
                            for (int i = 0; i < G; i += 2) {
                                const int s = g * G + i, q = s / 2;
                                const float2 dot = __ffma2_rn(dx[q], both(-w1.x),
                                                              __ffma2_rn(dy[q], both(-w1.y),
                                                                         __ffma2_rn(fresh2(&sums.dz[q][tid]),
                                                                                    both(-w1.z), both(ew))));
                                const float2 r = __ffma2_rn(psi[i / 2], both(sP.inv_gc), both(cur.rh));
                                float2 ri = make_float2(rcp(r.x), rcp(r.y));
                                if (zero) {
                                    if (zero >> i & 1u) ri.x = 0.f;
                                    if (zero >> (i + 1) & 1u) ri.y = 0.f;
                                }
                                const float2 rate = __fmul2_rn(dot, ri);
                                // place in the cell: the anchor's, less its shift, plus the pixel's
                                const float2 t = __ffma2_rn(rate, both(sP.rate_cells),
                                                            __ffma2_rn(psi[i / 2], both(jc.y), both(cur.t0 - cur.w)));
                                const float2 bow = __fmul2_rn(
                                    __ffma2_rn(both(sP.bend2), __ffma2_rn(rate, make_float2(-rate.x, -rate.y), both(w1.w)),
                                               both(bend_v)),
                                    ri);
                                const float2 eps = __ffma2_rn(both(sP.bend1), rate, bow);
                                float2 h0 = both(0.f), h1 = h0;
                                if constexpr (MOVE == 2) {
                                    // the pixels' directions less the anchor's
                                    const float2 ux = __ffma2_rn(__fadd2_rn(both(cur.ex), neg(dx[q])), ri, both(-cur.ex * ri0)),
                                                 uy = __ffma2_rn(__fadd2_rn(both(cur.ey), neg(dy[q])), ri, both(-cur.ey * ri0)),
                                                 uz = __ffma2_rn(__fadd2_rn(both(cur.ez), neg(fresh2(&sums.dz[q][tid]))), ri,
                                                                 both(-cur.ez * ri0));
                                    h0 = turn_value(turn_x, turn_y, turn_z, ux.x, uy.x, uz.x, t.x);
                                    h1 = turn_value(turn_x, turn_y, turn_z, ux.y, uy.y, uz.y, t.y);
                                }
                                add_moving_pair(psi[i / 2], cur.turn, t, __fadd2_rn(eps, both(-eps0)), a, bend, h0, h1,
                                                hc[s], hs[s], hc[s + 1], hs[s + 1]);
                            }
                            if (zero) {
#pragma unroll
                                for (int i = 0; i < G; ++i)
                                    if (zero >> i & 1u) hc[g * G + i] = hs[g * G + i] = make_float2(0.f, 0.f);
                            }
                            continue;
                        }
#pragma unroll
                        for (int i = 0; i < G; i += 2) {
                            const int s = g * G + i;
                            add_pair<BAND, LINE>(psi[i / 2], cur.turn, cur.t0, jc.y, cur.a, w[i], w[i + 1], hc[s], hs[s], hc[s + 1],
                                           hs[s + 1]);
                        }
                        if (!BAND && !ADJ && zero) {
#pragma unroll
                            for (int i = 0; i < G; ++i)
                                if (zero >> i & 1u) hc[g * G + i] = hs[g * G + i] = make_float2(0.f, 0.f);
                        }
                    }
                }
                if constexpr (ADJ) {
#pragma unroll
                    for (int v = 0; v < 3; ++v) {
                        grad[v] += __shfl_xor_sync(0xffffffffu, grad[v], 16);
                        grad[v] += __shfl_xor_sync(0xffffffffu, grad[v], 8);
                    }
                    if ((tid & 31) < 8)
#pragma unroll
                        for (int v = 0; v < 3; ++v) red[k][v][(tid >> 5) * 8 + (tid & 31)] = grad[v];
                }
                k = k_next;
            }
            if constexpr (ADJ) {
                __syncthreads();
                float *__restrict__ out = reinterpret_cast<float *>(gpart + (size_t)un.tile * sJ.C + b0);
                for (int i = tid; i < 3 * n; i += kThreads) {
                    float s = 0.f;
#pragma unroll
                    for (int j = 0; j < kThreads / 4; ++j) s += red[i / 3][i % 3][j];
                    out[4 * (i / 3) + i % 3] = kTwoPiF * sP.gc_hi * s;
                }
            }
            // the plain sums of these chirps (of one skip-test chunk) into the Kahan sums
#pragma unroll
            for (int i = 0; i < (ADJ ? 0 : PT); ++i) {
                if (!(dropped >> i & 1u)) stash(sums, i, tid, hc[i], hs[i]);
                hc[i] = hs[i] = make_float2(0.f, 0.f);
            }
            b0 += n;
            buf ^= 1;
        }

        if (ADJ) continue;
        p0 = run_pixels<PT>(sJ.P, sJ.grid_cols, un.tile, tid, count);
        float4 *__restrict__ part = sJ.partial + (size_t)un.group * sJ.P;
#pragma unroll
        for (int i = 0; i < PT; ++i)
            if (i < count) part[p0 + i] = sums.s[i][tid];
    }
}

}  // namespace

cudaError_t launch_profile_twiddle(float2 *twiddle, float *factor, int S, cudaStream_t st, const int *enabled)
{
    const long long n = (long long)S * kNodes;
    profile_twiddle_kernel<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(twiddle, factor, S, enabled);
    return cudaGetLastError();
}

// A row's samples are split over the CTAs of a cluster (their sums meet in its shared memory) while
// the chirps alone leave SMs idle: up to 8 ways, at least two tiles a CTA, at most 5/3 CTAs an SM. By
// chirps and samples only: the sums must not depend on where a row block of a grid lies. Whole
// focus, split or not: 256^2 pixels x 64 chirps x 12345 samples 103 / 511 us, 64 x 512 x 512 x 1024
// (moving) 117 / 148, 128^2 x 256 x 256 50 / 54, vibration (151 x 97 x 333 x 500) 107 / 126; up to 2
// CTAs an SM, 256^2 x 1024 x 512 179 / 175.
constexpr int kBuildMaxSplit = 8, kBuildMaxCtas = 152 * 5 / 3;

template <bool INDIRECT>
static cudaError_t launch_build(const ProfileBuild &b, const ProfileStencil &stencil, const ProfileBuild *dev,
                                const int *enabled, int C, int S, int blocks, int tables, cudaStream_t st)
{
    const int chirp_blocks = (C + kBuildChirps - 1) / kBuildChirps, tiles = (S + kBuildStep - 1) / kBuildStep;
    int split = 1;
    while (split < kBuildMaxSplit && 2LL * split * chirp_blocks * tables <= kBuildMaxCtas && tiles >= 4 * split) split *= 2;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(chirp_blocks * split, blocks, tables);
    cfg.blockDim = dim3(kBuildThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = split;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = split > 1;
    return cudaLaunchKernelEx(&cfg, profile_build_kernel<INDIRECT>, b, stencil, dev, enabled, split);
}

cudaError_t launch_profile_build(const ProfileBuild &b, cudaStream_t st)
{
    static const ProfileStencil stencil = make_stencil();
    // nodes of n_cells / 2 from an even cell on, wherever the first block starts
    const int blocks = (b.n_cells / 2 + kOwn - 2) / kOwn + 1;
    return launch_build<false>(b, stencil, nullptr, nullptr, b.C, b.S, blocks, b.traj ? kVibTables : 1, st);
}

cudaError_t launch_profile_build_indirect(const ProfileBuild *dev, const int *enabled, int C, int S, int max_cells,
                                          cudaStream_t st)
{
    static const ProfileStencil stencil = make_stencil();
    return launch_build<true>(ProfileBuild{}, stencil, dev, enabled, C, S, (max_cells / 2 + kOwn - 2) / kOwn + 1, 1, st);
}

using ProfileFn = void (*)(const FocusJob *, const FocusUnit *, int, int *, const float2 *, float4 *);

template <bool BAND, bool ADJ, int MOVE>
static ProfileFn profile_fn(int group)
{
    switch (group) {
    case 8: return profile_focus_kernel<8, BAND, ADJ, MOVE, false>;
    case 4: return profile_focus_kernel<4, BAND, ADJ, MOVE, false>;
    case 2: return profile_focus_kernel<2, BAND, ADJ, MOVE, false>;
    default: return profile_focus_kernel<1, BAND, ADJ, MOVE, false>;
    }
}

static ProfileFn profile_fn(int group, bool band, bool adjoint, int motion, bool line)
{
    if (line && group == 16) {
        if (adjoint) return profile_focus_kernel<16, false, true, 0, true>;
        return profile_focus_kernel<16, false, false, 0, true>;
    }
    if (line && adjoint)
        return band ? profile_focus_kernel<8, true, true, 0, true> : profile_focus_kernel<8, false, true, 0, true>;
    if (line)
        return band ? profile_focus_kernel<8, true, false, 0, true> : profile_focus_kernel<8, false, false, 0, true>;
    if (motion == 2) return profile_fn<false, false, 2>(group);
    if (motion) return profile_fn<false, false, 1>(group);
    if (adjoint) return band ? profile_fn<true, true, 0>(group) : profile_fn<false, true, 0>(group);
    return band ? profile_fn<true, false, 0>(group) : profile_fn<false, false, 0>(group);
}

cudaError_t launch_vib_fit(const float4 *traj, const ChirpRec *chirps, int C, int S, int s_pad, float phase_per_m,
                           VibRec *recs, int *maxima, cudaStream_t st)
{
    vib_fit_kernel<<<(C + 3) / 4, 128, 0, st>>>(traj, chirps, C, S, s_pad, phase_per_m, recs, maxima);
    return cudaGetLastError();
}

cudaError_t launch_focus_profile(int group, bool band, int motion, bool line, const FocusJob *jobs_dev,
                                 const FocusUnit *units_dev, int n_units, int *counter_dev, int grid_ctas,
                                 cudaStream_t st)
{
    if (band && motion) return cudaErrorInvalidValue;
    profile_fn(group, band, false, motion, line)<<<grid_ctas, kThreads, 0, st>>>(jobs_dev, units_dev, n_units, counter_dev,
                                                                           nullptr, nullptr);
    return cudaGetLastError();
}

cudaError_t launch_adjoint_profile(int group, bool band, bool line, const FocusJob *jobs_dev, const FocusUnit *units_dev,
                                   int n_units, int *counter_dev, int grid_ctas, const float2 *gimg, float4 *gpart,
                                   cudaStream_t st)
{
    profile_fn(group, band, true, 0, line)<<<grid_ctas, kThreads, 0, st>>>(jobs_dev, units_dev, n_units, counter_dev,
                                                                         gimg, gpart);
    return cudaGetLastError();
}

int focus_profile_blocks_per_sm(int group, bool band, bool adjoint, int motion, bool line)
{
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, profile_fn(group, band, adjoint, motion, line), kThreads, 0) !=
        cudaSuccess)
        return 0;
    return blocks;
}

}  // namespace tdc
