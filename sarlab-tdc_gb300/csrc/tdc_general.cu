// tdc_general.cu -- FP32 general focus kernel of the GB300 TDC engine: the
// inputs the FP32-bulk kernel does not take, at FP32-bulk-like accuracy.
//
//   * per-sample antenna positions (position[c][s] varies within a chirp, as the
//     reference's tdckernels.cu:204-208 reads it per element);
//   * per-sample Doppler windows (velocity / attitude varying within a chirp,
//     tdckernels.cu:106-130 evaluates the window per element);
//   * non-uniform sample times (2 f_s / c0 not affine in s).
//
// Phase of sample s of chirp c at pixel T, in cycles:
//   g_s R_s,  R_s = |P[c,s] - T|,  g_s = 2 f_s / c0.
// Split about sample 0 (R0 = |P[c,0] - T| in double-float, as in the bulk kernel)
// and the affine fit g_s = g0 + g1 s + r_s:
//   g_s R_s = (g0 + g1 s) R0  +  r_s R0  +  g_s d_s,   d_s = R_s - R0.
// The first term is alpha + beta s; the rest, psi_s, is a phase of every (pixel, sample). Where
// there is one (all variants but per-sample windows alone) each sample takes one sincos of
// 2 pi (beta s + psi_s): beta s is the block of 8's turn, a 32-bit fraction of a cycle stepped by
// 8 beta, plus a table of k beta. (Correcting the sample by psi_s first and feeding it to the
// bulk kernel's Horner recurrence took 4 more operations and as much state.) With per-sample
// windows alone the recurrence runs on the weighted samples.
// d_s comes without cancellation from the per-sample offset D_s = P[c,s] - P[c,0]
// (host table: D_s and |D_s|^2 per (chirp, sample)):
//   m = n0.D + |D|^2 / 2R0 = (R_s^2 - R0^2) / 2R0,   d_s = m f(e),   e = 2 m / R0,
//   f(e) = 2 / (1 + sqrt(1 + e)) = 1 - e/4 + e^2/8 - 5e^3/64 + 7e^4/128 - ...,
// the series taken to e^2 when the host bounds |e| <= 0.02 and |psi| <= 4 cycles (then
// the sincos takes the phase unreduced: its argument scaling adds < 2e-6 rad), else to e^4 with
// the phase reduced modulo one cycle ("wide" variants, which also carry the non-uniform
// sampling residual; the host routes |e| > 0.1 to the FP64 kernel; at 0.1 the
// truncation is 4e-7 of d_s).
//
// Bound: the FMA pipe (63% busy, 63% of the issue slots). Two samples stand side by side in the
// two halves of FFMA2, which halves the issue slots (the tables are laid out for it; what is a
// pixel's own sits in both halves). 128^2 pixels x 512 chirps x 512 samples, 256 threads x 2 CTAs an SM
// throughout: positions and windows per sample 5.19 ms as scalar code with a Horner recurrence,
// 4.54 with pairs and dead chirps left out (23% of them there), 3.70 with one sincos for the whole
// phase and the reciprocal by the special-function unit, 3.50 in units half as long. 128^2 x
// 256 x 512: positions alone 1.62 -> 1.37 ms, windows alone 1.49 -> 1.16, non-uniform times 1.26
// -> 1.17, windows and times 3.03 -> 1.72, all three 3.53 -> 2.52.
//
// Same unit decomposition, staging (cp.async.bulk + mbarrier pipeline), skip test,
// Kahan accumulation and group reduction as the bulk kernel. A chirp skips its samples where its
// chirp-level weight is zero, or every sample provably out of band, for every pixel of a warp (see
// window_bounds_kernel).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "tdc_device.cuh"
#include "tdc_internal.h"

namespace tdc {

namespace {

#ifndef TDC_GENERAL_MINB
#define TDC_GENERAL_MINB 2
#endif

constexpr int kL = 8;                   // in-block phasor table length
constexpr int kPT = kGeneralPT;         // pixels per thread
constexpr int kT = kFocusTile / kPT;    // threads per CTA (a CTA covers one 512-pixel tile)
constexpr int kTile = kT * kPT;
// Double buffering: a chirp row takes tens of microseconds of arithmetic per CTA, far
// longer than its copy, and the smaller footprint keeps two CTAs resident per SM.
constexpr int kStages = 2;
static_assert(kTile == kFocusTile, "work units tile the grid like the FP32-bulk kernel");

__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 neg(float2 v) { return make_float2(-v.x, -v.y); }

struct GenShared {
    float t[kPT * 6][kT];  // (x_hi, y_hi, z_hi, x_lo, y_lo, z_lo) per pixel slot
};

__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}

// Nearest integer for |v| < 2^22 without a conversion instruction.
__device__ __forceinline__ float round_small(float v)
{
    constexpr float kMagic = 12582912.0f;  // 1.5 x 2^23
    return (v + kMagic) - kMagic;
}

// The window-and-residual variant without per-sample positions keeps more samples in
// flight than 128 registers hold: it runs one CTA per SM instead of spilling.
//
// Stages: rows of job.seg_len samples. When a whole row fits (seg_len = s_pad) a stage
// holds stage_chirps chirps; otherwise each chirp's row is staged in segments, last
// segment first, and the chirp's Horner state carries from segment to segment. Stage
// layout: [x rows][trajectory rows][window rows][window-offset rows][residual r_s][g_s]
// [records], the per-sample tables only where the variant reads them.
template <bool TRAJ, bool WIN, bool WIDE>
__global__ void __launch_bounds__(kT, (!TRAJ && WIN && WIDE) ? 1 : TDC_GENERAL_MINB)
    focus_general_kernel(const FocusJob *__restrict__ jobs, const FocusUnit *__restrict__ units, int n_units,
                         int *__restrict__ counter, int *__restrict__ status, int stage_bytes)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t full_bar[kStages];
    __shared__ int s_unit;
    __shared__ FocusJob sJ;

    GenShared &sp = *reinterpret_cast<GenShared *>(smem + kStages * stage_bytes);

    constexpr bool TW = TRAJ && WIN;  // per-sample positions and windows: window-offset rows staged
    constexpr bool PHASE = TRAJ || WIDE;  // a phase of its own for every sample
    const int tid = threadIdx.x;
    if (tid == 0) {
        for (int i = 0; i < kStages; ++i) mbar_init(&full_bar[i], 1);
        fence_barrier_init();
    }
    __syncthreads();

    uint32_t n_issued = 0;
    uint32_t n_consumed = 0;

    for (;;) {
        if (tid == 0) s_unit = atomicAdd(counter, 1);
        __syncthreads();
        const int u = s_unit;
        if (u >= n_units) break;
        const FocusUnit un = units[u];
        if (tid < (int)(sizeof(FocusJob) / sizeof(int)))
            reinterpret_cast<int *>(&sJ)[tid] = reinterpret_cast<const int *>(&jobs[un.job])[tid];
        __syncthreads();

        const int C = sJ.C;
        const int c0 = un.group * sJ.chirps_per_group;
        const int c1 = min(C, c0 + sJ.chirps_per_group);
        const int s_pad = sJ.s_pad;
        const int seg = sJ.seg_len;  // samples per staged row segment (multiple of 16)
        const int nseg = (s_pad + seg - 1) / seg;
        const int CB = nseg == 1 ? sJ.stage_chirps : 1;
        const int nblk = nseg == 1 ? (c1 - c0 + CB - 1) / CB : (c1 - c0) * nseg;
        const uint32_t xrow = static_cast<uint32_t>(seg) * 8u;
        const uint32_t arow = static_cast<uint32_t>(seg) * 16u;
        const uint32_t grow = static_cast<uint32_t>(seg) * 4u;
        const uint32_t off_a = CB * xrow;
        const uint32_t off_b = off_a + (TRAJ ? CB * arow : 0u);
        const uint32_t off_w = off_b + (WIN ? CB * arow : 0u);
        const uint32_t off_g = off_w + (TW ? CB * grow : 0u);
        const uint32_t off_r = off_g + (WIDE ? grow : 0u) + (TRAJ ? grow : 0u);
        const float4 *__restrict__ xw = sJ.xw;
        const float4 *__restrict__ traj = sJ.traj;
        const float4 *__restrict__ wins = sJ.wins;
        const float4 *__restrict__ bounds = wins + (size_t)C * s_pad;  // see window_bounds_kernel
        const float *__restrict__ wdot = sJ.wdot;
        const float *__restrict__ gres = sJ.gres;
        const float *__restrict__ gsam = sJ.gsam;
        const ChirpRec *__restrict__ chirps = sJ.chirps;

        // stage j -> first chirp, chirps, segment, sample offset, samples
        auto stage_of = [&](int j, int &cb0, int &cnt, int &sg, int &off, int &len) {
            if (nseg == 1) {
                cb0 = c0 + j * CB;
                cnt = min(CB, c1 - cb0);
                sg = 0;
            } else {
                cb0 = c0 + j / nseg;
                cnt = 1;
                sg = nseg - 1 - j % nseg;
            }
            off = sg * seg;
            len = min(seg, s_pad - off);
        };

        auto issue = [&](int j) {
            int cb0, cnt, sg, off, len;
            stage_of(j, cb0, cnt, sg, off, len);
            const int st = n_issued % kStages;
            unsigned char *base = smem + st * stage_bytes;
            const uint32_t lx = static_cast<uint32_t>(len) * 8u, la = static_cast<uint32_t>(len) * 16u,
                           lg = static_cast<uint32_t>(len) * 4u;
            uint32_t total =
                cnt * (lx + (TRAJ ? la : 0u) + (WIN ? la : 0u) + (TW ? lg : 0u) + (uint32_t)sizeof(ChirpRec));
            if (WIDE) total += lg;
            if (TRAJ) total += lg;
            mbar_arrive_expect_tx(&full_bar[st], total);
            for (int cc = 0; cc < cnt; ++cc) {
                const size_t row = (size_t)(cb0 + cc) * s_pad + off;
                bulk_g2s(base + cc * xrow, xw + row / 2, lx, &full_bar[st]);
                if (TRAJ) bulk_g2s(base + off_a + cc * arow, traj + row, la, &full_bar[st]);
                if (WIN) bulk_g2s(base + off_b + cc * arow, wins + row, la, &full_bar[st]);
                if (TW) bulk_g2s(base + off_w + cc * grow, wdot + row, lg, &full_bar[st]);
            }
            uint32_t og = off_g;
            if (WIDE) {
                bulk_g2s(base + og, gres + off, lg, &full_bar[st]);
                og += grow;
            }
            if (TRAJ) bulk_g2s(base + og, gsam + off, lg, &full_bar[st]);
            bulk_g2s(base + off_r, chirps + cb0, cnt * (uint32_t)sizeof(ChirpRec), &full_bar[st]);
            ++n_issued;
        };

        if (tid == 0) {
            fence_proxy_async_smem();
            const int npro = nblk < kStages ? nblk : kStages;
            for (int j = 0; j < npro; ++j) issue(j);
        }

        const long long P = sJ.P;
#pragma unroll
        for (int i = 0; i < kPT; ++i) {
            const long long p = tile_pixel(sJ.tile_cols, sJ.grid_cols, P, un.tile, i * kT + tid);
            float4 hi = make_float4(0.f, 0.f, 0.f, 0.f), lo = hi;
            if (p >= 0) {
                hi = __ldg(&sJ.grid_hi[p]);
                if (sJ.grid_lo) lo = __ldg(&sJ.grid_lo[p]);
            }
            sp.t[i * 6 + 0][tid] = hi.x;
            sp.t[i * 6 + 1][tid] = hi.y;
            sp.t[i * 6 + 2][tid] = hi.z;
            sp.t[i * 6 + 3][tid] = lo.x;
            sp.t[i * 6 + 4][tid] = lo.y;
            sp.t[i * 6 + 5][tid] = lo.z;
        }

        const float g0h = sJ.g0_hi, g0l = sJ.g0_lo, g1 = sJ.g1, g1l = sJ.g1_lo;
        const float tol = sJ.two_over_lambda, half_bw = sJ.half_bw, inv_bw = sJ.inv_bw, az_a = sJ.az_a;
        const bool taper = (sJ.flags & kFlagTaper) != 0;
        const bool skip_test = (sJ.flags & kFlagSkipTest) != 0;
        const float taper_a = taper ? az_a : 1.0f, taper_b = taper ? 1.0f - az_a : 0.0f;
        const int chunk = sJ.chunk;
        const SkipPoint *__restrict__ skip = sJ.skip;

        float2 sum[kPT], comp[kPT];
        float wskip[kPT];
#pragma unroll
        for (int i = 0; i < kPT; ++i) {
            sum[i] = make_float2(0.f, 0.f);
            comp[i] = make_float2(0.f, 0.f);
            wskip[i] = 1.0f;
        }
        // per-(pixel, chirp) state, carried across the segments of a chirp; what two samples side by
        // side share is kept in both halves
        constexpr int kTab = kL / 2, kRot = PHASE ? 1 : kTab, kTurns = PHASE ? kTab : 1;
        float2 px[kPT][kRot], py[kPT][kRot], ql[kPT], h[kPT];  // in-block phasors, block step, Horner state
        float2 turns[kPT][kTurns];                             // (PHASE) k beta of the block's samples
        unsigned int step[kPT];                                // (PHASE) 8 beta [2^-32 cycles]
        float2 accx[kPT], accy[kPT];                           // (PHASE) sums of the even and the odd samples
        float2 q0[kPT];
        float2 nx[kPT], ny[kPT], nz[kPT];   // (P0 - T) / R0
        float2 r0[kPT], rs1[kPT];           // R0, 1 / R0
        float2 a2[kPT], k2[kPT];            // 1 / 2R0, 1 / 2R0^2
        bool live = true;
        int cur_chunk = -1;
        bool timed_out = false;

        for (int j = 0; j < nblk; ++j) {
            const int st = n_consumed % kStages;
            const uint32_t parity = (n_consumed / kStages) & 1u;
            const bool ok = mbar_wait_bounded(&full_bar[st], parity, kWaitLimitNs);
            if (__syncthreads_or(!ok)) {
                timed_out = true;
                break;
            }
            const unsigned char *base = smem + st * stage_bytes;
            const ChirpRec *recs = reinterpret_cast<const ChirpRec *>(base + off_r);
            const float *sgr = reinterpret_cast<const float *>(base + off_g);           // r_s of the segment
            const float *sgg = sgr + (WIDE ? seg : 0);                                  // g_s of the segment
            int cb0, cnt, sg, off, len;
            stage_of(j, cb0, cnt, sg, off, len);

            for (int cc = 0; cc < cnt; ++cc) {
                const int c = cb0 + cc;
                const float4 *xs = reinterpret_cast<const float4 *>(base) + (size_t)cc * (seg / 2);
                const float4 *as = reinterpret_cast<const float4 *>(base + off_a) + (size_t)cc * seg;
                const float4 *bs = reinterpret_cast<const float4 *>(base + off_b) + (size_t)cc * seg;
                const float *us = reinterpret_cast<const float *>(base + off_w) + (size_t)cc * seg;

                if (sg == nseg - 1) {
                    // first staged segment of the chirp: skip weight, range, phase set-up
                    if (skip_test) {
                        const int k = c / chunk;
                        if (k != cur_chunk) {
                            cur_chunk = k;
#pragma unroll
                            for (int i = 0; i < kPT; ++i)
                                wskip[i] = chunk_is_nonzero(skip + (size_t)k * 9, sp.t[i * 6 + 0][tid],
                                                            sp.t[i * 6 + 1][tid], sp.t[i * 6 + 2][tid], tol,
                                                            half_bw)
                                               ? 1.0f
                                               : 0.0f;
                        }
                    }
                    const ChirpRec r = recs[cc];
                    bool any = false;
#pragma unroll
                    for (int i = 0; i < kPT; ++i) {
                        float dxh, dxl, dyh, dyl, dzh, dzl;
                        dd_sub(r.p_hi.x, r.p_lo.x, sp.t[i * 6 + 0][tid], sp.t[i * 6 + 3][tid], dxh, dxl);
                        dd_sub(r.p_hi.y, r.p_lo.y, sp.t[i * 6 + 1][tid], sp.t[i * 6 + 4][tid], dyh, dyl);
                        dd_sub(r.p_hi.z, r.p_lo.z, sp.t[i * 6 + 2][tid], sp.t[i * 6 + 5][tid], dzh, dzl);
                        float rh, rl, rs, dh;
                        dd_range(dxh, dxl, dyh, dyl, dzh, dzl, rh, rl, rs, dh);
                        // 1 / R0 to FP32 rounding (rsqrt is not)
                        const float rinv = fmaf(rs, fmaf(-rl, rs, fmaf(-rh, rs, 1.0f)), rs);
                        const float alpha = dd_frac_mul(g0h, g0l, rh, rl);
                        float bh = g1 * rh;
                        float bl = fmaf(g1, rh, -bh);
                        bl = fmaf(g1, rl, bl);
                        bl = fmaf(g1l, rh, bl);
                        bh -= rintf(bh);
                        const float lbh = (float)kL * bh;
                        if constexpr (PHASE) {
#pragma unroll
                            for (int k = 0; k < kL; k += 2) {
                                const float e = (float)k * bh, o = (float)(k + 1) * bh;
                                const float2 v = make_float2(fmaf((float)k, bh, -rintf(e)) + (float)k * bl,
                                                             fmaf((float)(k + 1), bh, -rintf(o)) + (float)(k + 1) * bl);
                                turns[i][k / 2] = WIDE ? v : __fmul2_rn(v, both(kTwoPiF));
                            }
                            step[i] = (unsigned)__float2int_rn((lbh - rintf(lbh)) * 4294967296.0f) +
                                      (unsigned)__float2int_rn(((float)kL * bl) * 4294967296.0f);
                            accx[i] = accy[i] = both(0.f);
                        } else {
                            float s1, c1s;
                            __sincosf(kTwoPiF * (bh + bl), &s1, &c1s);
                            const float2 p1 = make_float2(c1s, s1);
                            float2 pe = make_float2(1.f, 0.f);
#pragma unroll
                            for (int k = 0; k < kL; k += 2) {
                                const float2 po = cmul(pe, p1);
                                px[i][k / 2] = make_float2(pe.x, po.x);
                                py[i][k / 2] = make_float2(pe.y, po.y);
                                pe = cmul(po, p1);
                            }
                            const float lfr = (lbh - rintf(lbh)) + (float)kL * bl;
                            float sl, cl;
                            sincospif(2.0f * lfr, &sl, &cl);
                            ql[i] = make_float2(cl, sl);
                            h[i] = make_float2(0.f, 0.f);
                        }
                        float w = wskip[i];
                        if (!WIN) {
                            const float fd = doppler_freq(tol, r.vel.x, r.vel.y, r.vel.z, dxh, dyh, dzh, rs);
                            w *= doppler_window(fd, r.p_hi.w, half_bw, inv_bw, taper, az_a);
                        }
                        bool out = false;
                        if (WIN) {
                            // every sample's window angle lies within `span` of this one
                            const float4 wr = __ldg(&bounds[2 * c]), wb = __ldg(&bounds[2 * c + 1]);
                            const float q = fmaf(rs, fmaf(wr.x, dxh, fmaf(wr.y, dyh, wr.z * dzh)), -wr.w);
                            const float span = TRAJ ? fmaf(wb.y, __fdividef(wb.z, fmaxf(rh - wb.z, 0.0f)), wb.x) : wb.x;
                            out = fabsf(q) > kPiF + span;
                        }
                        any |= w != 0.0f && !out;
                        float sa, ca;
                        __sincosf(kTwoPiF * alpha, &sa, &ca);
                        q0[i] = make_float2(w * ca, w * sa);
                        nx[i] = both(rinv * dxh);
                        ny[i] = both(rinv * dyh);
                        nz[i] = both(rinv * dzh);
                        r0[i] = both(rh);
                        rs1[i] = both(rinv);
                        a2[i] = both(0.5f * rinv);
                        k2[i] = both(0.5f * rinv * rinv);
                    }
                    // a chirp whose chirp-level weight (skip test, and the window unless it is
                    // per sample) is zero for every pixel of the warp contributes nothing
                    live = __any_sync(0xffffffffu, any);
                }
                if (!live) continue;

                // This segment's blocks; each sample corrected per pixel.
                for (int b = len / kL - 1; b >= 0; --b) {
                    float2 base[kPT];  // (PHASE) turn of the block's first sample, beta s
                    float2 bx[kPT], by[kPT];
#pragma unroll
                    for (int i = 0; i < kPT; ++i) {
                        if constexpr (PHASE) {
                            const int turn = (int)((unsigned)(off / kL + b) * step[i]);
                            base[i] = both((float)turn * (WIDE ? 1.0f / 4294967296.0f : kTwoPiF / 4294967296.0f));
                        } else {
                            const float2 v = cmul(h[i], ql[i]);
                            bx[i] = make_float2(v.x, 0.f);
                            by[i] = make_float2(v.y, 0.f);
                        }
                    }
#pragma unroll
                    for (int k = 0; k < kL; k += 2) {
                        const int s = b * kL + k;  // samples s and s + 1 within the segment
                        const float4 xv = xs[s >> 1];
                        const float2 xr = make_float2(xv.x, xv.z), xi = make_float2(xv.y, xv.w);
                        float4 a01 = make_float4(0.f, 0.f, 0.f, 0.f), a23 = a01, b01 = a01, b23 = a01;
                        if (TRAJ) {
                            a01 = as[s];
                            a23 = as[s + 1];
                        }
                        if (WIN) {
                            b01 = bs[s];
                            b23 = bs[s + 1];
                        }
                        const float2 uD = TW ? *reinterpret_cast<const float2 *>(us + s) : both(0.f);
                        const float2 res = WIDE ? *reinterpret_cast<const float2 *>(sgr + s) : both(0.f);
                        const float2 gsv = TRAJ ? *reinterpret_cast<const float2 *>(sgg + s) : both(0.f);
#pragma unroll
                        for (int i = 0; i < kPT; ++i) {
                            float2 d = both(0.f);  // R_s - R0
                            if (TRAJ) {
                                // m = (R_s^2 - R0^2) / 2R0, d = m f(e), e = 2 m / R0
                                const float2 m = __ffma2_rn(
                                    nx[i], make_float2(a01.x, a01.y),
                                    __ffma2_rn(ny[i], make_float2(a01.z, a01.w),
                                               __ffma2_rn(nz[i], make_float2(a23.x, a23.y),
                                                          __fmul2_rn(a2[i], make_float2(a23.z, a23.w)))));
                                if (WIDE) {
                                    const float2 e = __fmul2_rn(m, __fadd2_rn(rs1[i], rs1[i]));
                                    float2 f = __ffma2_rn(e, both(7.0f / 128.0f), both(-5.0f / 64.0f));
                                    f = __ffma2_rn(f, e, both(0.125f));
                                    f = __ffma2_rn(f, e, both(-0.25f));
                                    f = __ffma2_rn(f, e, both(1.0f));
                                    d = __fmul2_rn(m, f);
                                } else {
                                    d = __ffma2_rn(__fmul2_rn(m, m), __ffma2_rn(m, k2[i], neg(a2[i])), m);
                                }
                            }
                            float2 cs = both(1.f), sn = both(0.f);
                            if constexpr (PHASE) {
                                float2 th = __fadd2_rn(base[i], turns[i][k / 2]);
                                if (TRAJ) th = __ffma2_rn(gsv, d, th);  // g_s d_s (radians when narrow)
                                if (WIDE) {
                                    th = __ffma2_rn(res, r0[i], th);
                                    th = make_float2(th.x - round_small(th.x), th.y - round_small(th.y));
                                    th = __fmul2_rn(th, both(kTwoPiF));
                                }
                                __sincosf(th.x, &sn.x, &cs.x);
                                __sincosf(th.y, &sn.y, &cs.y);
                            }
                            float2 w = both(1.f);
                            if (WIN) {
                                // per-sample window at P[c,s] (d = P0 - T + D_s), as an angle:
                                // q = 2 pi (fDop - centre) / B, the table's velocity scaled by
                                // -4 pi / (lambda B) and centre by 2 pi / B; in band for |q| <= pi, taper
                                // a - (1-a) cos(q - pi) = a + (1-a) cos(q) (with moving positions
                                // u.d / R_s = (u.n0 + u.D / R0) / (1 + d_s / R0), u.D from the table)
                                float2 q = __ffma2_rn(make_float2(b01.x, b01.y), nx[i],
                                                      __ffma2_rn(make_float2(b01.z, b01.w), ny[i],
                                                                 __fmul2_rn(make_float2(b23.x, b23.y), nz[i])));
                                if (TRAJ) {
                                    q = __ffma2_rn(uD, rs1[i], q);
                                    const float2 y = __ffma2_rn(d, rs1[i], both(1.0f));
                                    q = __ffma2_rn(q, make_float2(rcp(y.x), rcp(y.y)),
                                                   make_float2(-b23.z, -b23.w));
                                } else {
                                    q = __fadd2_rn(q, make_float2(-b23.z, -b23.w));
                                }
                                w = __ffma2_rn(make_float2(__cosf(q.x), __cosf(q.y)), both(taper_b), both(taper_a));
                                w.x = fabsf(q.x) <= kPiF ? w.x : 0.0f;
                                w.y = fabsf(q.y) <= kPiF ? w.y : 0.0f;
                            }
                            if constexpr (PHASE) {
                                if (WIN) {
                                    cs = __fmul2_rn(cs, w);
                                    sn = __fmul2_rn(sn, w);
                                }
                                accx[i] = __ffma2_rn(xr, cs, accx[i]);
                                accx[i] = __ffma2_rn(neg(xi), sn, accx[i]);
                                accy[i] = __ffma2_rn(xr, sn, accy[i]);
                                accy[i] = __ffma2_rn(xi, cs, accy[i]);
                            } else {
                                const float2 yr = __fmul2_rn(xr, w), yi = __fmul2_rn(xi, w);
                                bx[i] = __ffma2_rn(yr, px[i][k / 2], bx[i]);
                                bx[i] = __ffma2_rn(neg(yi), py[i][k / 2], bx[i]);
                                by[i] = __ffma2_rn(yr, py[i][k / 2], by[i]);
                                by[i] = __ffma2_rn(yi, px[i][k / 2], by[i]);
                            }
                        }
                    }
                    if constexpr (!PHASE) {
#pragma unroll
                        for (int i = 0; i < kPT; ++i) h[i] = make_float2(bx[i].x + bx[i].y, by[i].x + by[i].y);
                    }
                }

                if (sg == 0) {
#pragma unroll
                    for (int i = 0; i < kPT; ++i) {
                        if constexpr (PHASE) h[i] = make_float2(accx[i].x + accx[i].y, accy[i].x + accy[i].y);
                        const float2 v = cmul(q0[i], h[i]);
                        const float yr = v.x - comp[i].x, yi = v.y - comp[i].y;
                        const float tr = sum[i].x + yr, ti = sum[i].y + yi;
                        comp[i].x = (tr - sum[i].x) - yr;
                        comp[i].y = (ti - sum[i].y) - yi;
                        sum[i].x = tr;
                        sum[i].y = ti;
                    }
                }
            }

            __syncthreads();
            ++n_consumed;
            if (tid == 0 && j + kStages < nblk) {
                fence_proxy_async_smem();
                issue(j + kStages);
            }
        }

        if (timed_out) {
            if (tid == 0) {
                for (uint32_t k = n_consumed; k < n_issued; ++k)
                    mbar_wait_bounded(&full_bar[k % kStages], (k / kStages) & 1u, kWaitLimitNs);
                atomicOr(status, kStatusTimeout);
            }
            __syncthreads();
            return;
        }

        float4 *__restrict__ part = sJ.partial + (size_t)un.group * P;
#pragma unroll
        for (int i = 0; i < kPT; ++i) {
            const long long pidx = tile_pixel(sJ.tile_cols, sJ.grid_cols, P, un.tile, i * kT + tid);
            if (pidx >= 0) part[pidx] = make_float4(sum[i].x, sum[i].y, comp[i].x, comp[i].y);
        }
        __syncthreads();
    }
}

// Entries (x, y, z, w) of samples 2 i and 2 i + 1 to (x0, x1, y0, y1)(z0, z1, w0, w1), in place (the host's
// loops that fill the tables are faster with whole entries).
__global__ void __launch_bounds__(256) pair_samples_kernel(float4 *__restrict__ t, long long pairs)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < pairs;
         i += (long long)gridDim.x * blockDim.x) {
        const float4 a = t[2 * i], b = t[2 * i + 1];
        t[2 * i] = make_float4(a.x, b.x, a.y, b.y);
        t[2 * i + 1] = make_float4(a.z, b.z, a.w, b.w);
    }
}

// Per chirp, how far the per-sample windows stray from one: with u_s the scaled velocity, c_s the
// scaled window centre, and n_s the unit vector from the pixel, q_s = u_s.n_s - c_s. About the
// mean (u, c) and the direction n_0 from sample 0, |q_s - (u.n_0 - c)| <= max|u_s - u| + max|c_s - c|
// + max|u_s| |n_s - n_0|, and |n_s - n_0| <= max|D_s| / (R0 - max|D_s|). Writes (u, c) and (the first two
// terms plus FP32 rounding, max|u_s|, max|D_s|) behind the windows. A row with a sample, or a position
// of one, that is not finite is never skipped (its product with a zero window is NaN). One warp a
// chirp.
__global__ void __launch_bounds__(128)
    window_bounds_kernel(float4 *__restrict__ wins, const float4 *__restrict__ traj, const float2 *__restrict__ xw,
                         int C, int S, int s_pad)
{
    const int c = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (c >= C) return;
    const size_t row = (size_t)c * s_pad;
    auto window = [&](int s) { return sample_table(wins + row, s); };
    float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = lane; s < S; s += 32) {
        const float4 w = window(s);
        m = make_float4(m.x + w.x, m.y + w.y, m.z + w.z, m.w + w.w);
    }
    const float inv = 1.0f / (float)S;
    for (int off = 16; off > 0; off >>= 1)
        m = make_float4(m.x + __shfl_xor_sync(0xffffffffu, m.x, off), m.y + __shfl_xor_sync(0xffffffffu, m.y, off),
                        m.z + __shfl_xor_sync(0xffffffffu, m.z, off), m.w + __shfl_xor_sync(0xffffffffu, m.w, off));
    m = make_float4(m.x * inv, m.y * inv, m.z * inv, m.w * inv);
    float du = 0.f, dc = 0.f, dd = 0.f;
    bool bad = false;
    for (int s = lane; s < S; s += 32) {
        const float4 w = window(s);
        const float x = w.x - m.x, y = w.y - m.y, z = w.z - m.z;
        du = fmaxf(du, sqrtf(x * x + y * y + z * z));
        dc = fmaxf(dc, fabsf(w.w - m.w));
        const float d = traj ? sqrtf(sample_table(traj + row, s).w) : 0.f;
        dd = fmaxf(dd, d);  // (drops a NaN)
        const float2 v = xw[row + s];
        bad |= !isfinite(v.x) || !isfinite(v.y) || !isfinite(x + y + z + w.w + d);
    }
    for (int off = 16; off > 0; off >>= 1) {
        du = fmaxf(du, __shfl_xor_sync(0xffffffffu, du, off));
        dc = fmaxf(dc, __shfl_xor_sync(0xffffffffu, dc, off));
        dd = fmaxf(dd, __shfl_xor_sync(0xffffffffu, dd, off));
    }
    bad = __any_sync(0xffffffffu, bad);
    if (lane) return;
    const float u = sqrtf(m.x * m.x + m.y * m.y + m.z * m.z) + du;
    const float slack = 1.01f * (du + dc) + 1e-5f * (1.0f + u + fabsf(m.w));
    float4 *out = wins + (size_t)C * s_pad + 2 * (size_t)c;
    out[0] = m;
    out[1] = make_float4(bad ? INFINITY : slack, 1.01f * u, 1.001f * dd, 0.f);
}

template <bool TRAJ, bool WIN, bool WIDE>
struct GeneralKernel {
    static constexpr auto fn = focus_general_kernel<TRAJ, WIN, WIDE>;
};

using KernelFn = void (*)(const FocusJob *, const FocusUnit *, int, int *, int *, int);

KernelFn select_kernel(int variant)
{
    switch (variant & 7) {
        case 1: return GeneralKernel<true, false, false>::fn;
        case 2: return GeneralKernel<false, true, false>::fn;
        case 3: return GeneralKernel<true, true, false>::fn;
        case 4: return GeneralKernel<false, false, true>::fn;
        case 5: return GeneralKernel<true, false, true>::fn;
        case 6: return GeneralKernel<false, true, true>::fn;
        case 7: return GeneralKernel<true, true, true>::fn;
        default: return nullptr;
    }
}

}  // namespace

cudaError_t launch_pair_samples(float4 *table, long long n, cudaStream_t st)
{
    pair_samples_kernel<<<(unsigned)std::min<long long>((n / 2 + 255) / 256, 152 * 16), 256, 0, st>>>(table, n / 2);
    return cudaGetLastError();
}

cudaError_t launch_window_bounds(float4 *wins, const float4 *traj, const float2 *xw, int C, int S, int s_pad,
                                 cudaStream_t st)
{
    window_bounds_kernel<<<(C + 3) / 4, 128, 0, st>>>(wins, traj, xw, C, S, s_pad);
    return cudaGetLastError();
}

int focus_general_smem_bytes(int stage_bytes)
{
    return kStages * stage_bytes + (int)sizeof(GenShared);
}

int focus_general_blocks_per_sm(int variant, int stage_bytes)
{
    KernelFn fn = select_kernel(variant);
    if (!fn) return 0;
    const int smem = focus_general_smem_bytes(stage_bytes);
    if (allow_max_dynamic_smem(fn) != cudaSuccess) return 0;
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, fn, kT, smem) != cudaSuccess) return 0;
    return blocks;
}

cudaError_t launch_focus_general(int variant, const FocusJob *jobs_dev, const FocusUnit *units_dev, int n_units,
                                 int *counter_dev, int *status_dev, int stage_bytes, int grid_ctas, cudaStream_t st)
{
    KernelFn fn = select_kernel(variant);
    if (!fn) return cudaErrorInvalidValue;
    const int smem = focus_general_smem_bytes(stage_bytes);
    cudaError_t e = allow_max_dynamic_smem(fn);
    if (e != cudaSuccess) return e;
    fn<<<grid_ctas, kT, smem, st>>>(jobs_dev, units_dev, n_units, counter_dev, status_dev, stage_bytes);
    return cudaGetLastError();
}

}  // namespace tdc
