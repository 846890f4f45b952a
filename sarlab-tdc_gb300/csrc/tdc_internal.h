// tdc_internal.h -- structures shared by the host code and the kernels of the
// GB300 TDC engine. Not part of the public ABI (include/tdc_gb300.h is).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <string>

namespace tdc {

constexpr double kC0 = 299792458.0;  // SPEED_OF_LIGHT, tdcprocessor.cpp:37
constexpr int kChunk = 128;          // PRI_CHUNKSIZE, tuning.h:18
constexpr float kRangeA = 25.0f / 46.0f;    // RANGE_WINDOW_A_PARAMETER, tuning.h:31
constexpr float kAzimuthA = 25.0f / 46.0f;  // AZIMUTH_WINDOW_A_PARAMETER, tuning.h:38

// Focus tile geometry of the FP32-bulk kernel: 128 threads x TDC_FOCUS_PT pixels.
#ifndef TDC_FOCUS_PT
#define TDC_FOCUS_PT 4
#endif
constexpr int kFocusThreads = 128;
constexpr int kFocusPT = TDC_FOCUS_PT;
constexpr int kFocusTile = kFocusThreads * kFocusPT;
constexpr int kFocusStages = 3;
constexpr int kSampleAlign = 16;  // s_pad is a multiple of this (bulk-copy rows stay 128-byte sized)
#ifndef TDC_FOCUS_STAGE_TARGET
#define TDC_FOCUS_STAGE_TARGET 16640
#endif
constexpr int kFocusStageTarget = TDC_FOCUS_STAGE_TARGET;  // bytes of chirp rows + records per pipeline stage
// Anchored ranges of the FP32-bulk kernel (pixels of a warp share a double-float anchor
// range per chirp, each adds its FP32 range difference): at most this many chirps per stage,
// and no pixel farther than kAnchorMaxDistance from its anchor. At 5 cm the FP32 range
// difference keeps the phase within ~3e-5 rad of the double-float range's at 77 GHz (1e-5 at
// the 1.6 cm of a 1 mm grid; tests/test_anchor_error_cpu.py).
constexpr int kAnchorMaxStageChirps = 16;
constexpr double kAnchorMaxDistance = 0.05;  // metres
// Fewest work units per CTA slot the planner aims for where the grid and chirps allow
// it. CTAs that share an SM need not progress at the same rate, so with a few long
// units per slot the last units end far apart (measured on 256^2 pixels x 256 chirps
// x 1024 samples, general kernel: SMs busy 72-100% of the launch at 3 units per slot,
// +14% throughput at 4 or more; with dead chirps skipped, 128^2 x 512 x 512, 4.08 ms at 2 units a
// slot, 3.70 at 4, 3.50 at 8, 3.47 at 16).
#ifndef TDC_GENERAL_MIN_UNITS
#define TDC_GENERAL_MIN_UNITS 8
#endif
#ifndef TDC_FOCUS_MIN_UNITS
#define TDC_FOCUS_MIN_UNITS 8
#endif
constexpr int kGeneralMinUnitsPerSlot = TDC_GENERAL_MIN_UNITS;
constexpr int kFocusMinUnitsPerSlot = TDC_FOCUS_MIN_UNITS;
// Pixels per thread of the FP32 general kernel (per-sample trajectories / windows, non-uniform sampling).
#ifndef TDC_GENERAL_PT
#define TDC_GENERAL_PT 2
#endif
constexpr int kGeneralPT = TDC_GENERAL_PT;

// One chirp's trajectory record, 48 bytes (3 x float4):
//   p_hi.xyz  antenna position, high float of a double-float pair; p_hi.w = Doppler window centre [Hz]
//   p_lo.xyz  low float of the position pair; p_lo.w = 0
//   vel.xyz   velocity; vel.w = 0
struct __align__(16) ChirpRec {
    float4 p_hi;
    float4 p_lo;
    float4 vel;
};
static_assert(sizeof(ChirpRec) == 48, "ChirpRec must be 48 bytes");

// One chirp's record for the smooth-motion kernel, 80 bytes (5 x float4): positions of
// the chirp's samples as P[c, s] = P0 + V1 s + V2 s^2 (the host's fit of the per-sample
// positions).
//   p_hi.xyz, p_lo.xyz  P0 as double-float pairs; p_hi.w = Doppler window centre [Hz]; p_lo.w = 0
//   vel.xyz             velocity at sample 0 (Doppler window); vel.w = 2 V1.V2
//   v1.xyz              V1 [m / sample]; v1.w = |V1|^2
//   v2.xyz              V2 [m / sample^2]; v2.w = |V2|^2
struct __align__(16) MotionRec {
    float4 p_hi;
    float4 p_lo;
    float4 vel;
    float4 v1;
    float4 v2;
};
static_assert(sizeof(MotionRec) == 80, "MotionRec must be 80 bytes");

// One chirp's record for the smooth motion through range profiles, 64 bytes: the same positions
// about the middle sample sc = S / 2, P[c, s] = P(sc) + W1 (s - sc) + V2 (s - sc)^2.
//   p_hi.xyz, p_lo.xyz  P(sc) as double-float pairs
//   w1.xyz              W1 = V1 + 2 sc V2 [m / sample]; w1.w = |W1|^2
//   v2.xyz              V2 [m / sample^2]
struct __align__(16) MoveRec {
    float4 p_hi;
    float4 p_lo;
    float4 w1;
    float4 v2;
};
static_assert(sizeof(MoveRec) == 64, "MoveRec must be 64 bytes");

// One chirp's record for vibration about a constant velocity, 96 bytes: the smooth part as above (V2
// zero), and
//   f0.xyz  P(sc) - P[c, 0], so that the deviation of sample s is D_s - f0 - W1 (s - sc)
//   n.xyz   its principal direction (unit); n.w = its largest carrier phase squared [rad^2]
struct __align__(16) VibRec {
    MoveRec m;
    float4 f0;
    float4 n;
};
static_assert(sizeof(VibRec) == 96, "VibRec must be 96 bytes");
constexpr int kVibTables = 6;  // range-profile tables of a vibrating acquisition (tdc_profile.cu)

// One sample point of the reference's chunk skip test (tdcprocessor.cpp:355-378).
struct __align__(16) SkipPoint {
    float4 pos_fdc;  // position xyz, window centre
    float4 vel;      // velocity xyz, 0
};
static_assert(sizeof(SkipPoint) == 32, "SkipPoint must be 32 bytes");

enum FocusFlags : int {
    kFlagTaper = 1,     // dopplerWinTaper
    kFlagSkipTest = 2,  // apply the per-chunk skip test
    kFlagMotionExactQL = 4,  // smooth-motion kernel: block step per segment from an accurate sincos
};

// Everything a focus kernel needs about one job (acquisition x grid).
struct FocusJob {
    const float4 *xw;        // [C][s_pad/2]: pairs of windowed complex samples
    const ChirpRec *chirps;  // [C] (or [C][S] for per-sample trajectories)
    const float4 *grid_hi;   // [P]
    const float4 *grid_lo;   // [P] or nullptr
    const SkipPoint *skip;   // [n_chunks][9]
    const double *gs;        // [S] 2 f_s / c0 (FP64 kernels only)
    const float4 *traj;      // [C][s_pad] (P[c,s] - P[c,0], |P[c,s] - P[c,0]|^2) (FP32 general kernel, per-sample
                             // positions), two samples side by side: (x0, x1, y0, y1)(z0, z1, w0, w1)
    const float4 *wins;      // [C][s_pad] 2 pi / B (velocity x -2 / lambda, window centre) per sample, likewise (FP32
                             // general kernel, per-sample windows); then [C][2] bounds (launch_window_bounds)
    const float *wdot;       // [C][s_pad] 2 pi / B velocity x -2 / lambda . (P[c,s] - P[c,0]) (per-sample positions
                             // and windows)
    const float *gres;       // [s_pad] 2 f_s / c0 - (g0 + g1 s) (FP32 general kernel, non-uniform sampling)
    const float *gsam;       // [s_pad] 2 f_s / c0 [cycles / m] (wide variants) or 2 pi x that [rad / m]
                             // (narrow variants) (FP32 general kernel, per-sample positions)
    float4 *partial;         // [n_groups][P]: (sum.re, sum.im, comp.re, comp.im)
    float2 *chirp_sums;      // [C][P] per-(chirp, pixel) sums A = sum_s x_s z^s: written by the storing
                             // focus instance, read by the adjoint that uses them (else null)
    long long P;
    int C;
    int S;
    int s_pad;
    int n_groups;
    int chirps_per_group;
    int chunk;
    int stage_chirps;        // chirps per pipeline stage
    int flags;
    int n_tiles;
    int per_sample;          // ChirpRec per sample instead of per chirp
    float g0_hi, g0_lo;      // 2 f_0 / c0 as a double-float pair [cycles / m]
    float g1;                // 2 df / c0 per sample [cycles / m]
    float two_over_lambda;   // 2 / lambda_centre
    float half_bw;           // dopplerBandwidth / 2
    float inv_bw;            // 1 / dopplerBandwidth
    float az_a;              // azimuth window a
    float g1_lo;             // low part of g1 (double-float pair)
    int seg_len;             // samples per pipeline stage of a chirp staged in segments (FP32 bulk: 0 for
                             // whole rows; FP32 general: s_pad for whole rows)
    int tile_cols;           // 0: a tile is kFocusTile consecutive pixels; else kFocusTile / tile_cols grid
                             // rows x tile_cols columns of the grid_cols-wide row-major grid
    int grid_cols;           // columns of the focus grid (block tiles); length of its runs (range profiles)
    int pad_;
    const struct ProfileJob *profile;  // range profiles (tdc_profile.cu), else null
};

// What a focus through range profiles needs beside its FocusJob (16-byte groups: the kernel
// loads four words together).
struct __align__(16) ProfileJob {
    float gc_hi, gc_lo;        // g0 + g1 (S / 2) as a double-float pair: carrier phase [cycles / m]
    float cells_hi, cells_lo;  // cells per metre of range, 4 S g1, as a double-float pair
    float inv_gc2x4;           // 4 / gc^2
    float cells_per_cycle;     // cells per cycle of carrier phase
    float r_safe;              // ranges below take the exact range difference (reach of a group / 0.03)
    int n_cells;               // cells per chirp
    const float4 *cells;       // [C][n_cells][kProfileCoefs / 2]: pairs of complex polynomial coefficients
    const int *cell_base;      // [C] absolute index of each chirp's first cell
    float inv_gc;              // 1 / gc
    float reach;               // largest distance of a pixel from its anchor [m]
    int axis;                  // axis the runs are parallel to (kernels with LINE)
    float pad_;
    // smooth motion: cells per (m / sample) of range rate, 4 S gc; with h = S / 2, the bend of the
    // phase at the row's ends is bend1 a + bend2 (|W1|^2 - a^2) / R + 2 bend2 e.V2 / R radians
    // (a = e.W1 / R), and its cubic part bend3 d2R/ds2 / 2
    float rate_cells;
    float bend1;               // 2 pi h^2 g1
    float bend2;               // pi h^2 gc
    float bend3;               // 2 pi h^3 g1
};
static_assert(sizeof(ProfileJob) == 80, "ProfileJob layout");

// Kernels copy a FocusJob into shared memory one int per thread (128 threads); the
// no-allocation scratch reserves 256 bytes for it.
static_assert(sizeof(FocusJob) <= 256 && sizeof(FocusJob) % 8 == 0, "FocusJob layout");

// Tiles of a P-pixel grid (see FocusJob::tile_cols).
inline long long tile_count(long long P, int tile_cols, int grid_cols)
{
    if (tile_cols <= 0 || grid_cols <= 0) return (P + kFocusTile - 1) / kFocusTile;
    const long long rows = (P + grid_cols - 1) / grid_cols;
    const int tile_rows = kFocusTile / tile_cols;
    return ((rows + tile_rows - 1) / tile_rows) * ((grid_cols + tile_cols - 1) / tile_cols);
}

// ---- range profiles (tdc_profile.cu) ----
constexpr int kProfileThreads = 64;     // a tile's kFocusTile pixels, 8 consecutive pixels a thread
constexpr int kProfilePixels = kFocusTile / kProfileThreads;
constexpr int kProfileNodes = 64;       // nodes one CTA of the table's construction forms
constexpr int kProfileBlock = 32;       // chirp records the focus stages at a time
constexpr int kProfileCoefs = 8;        // complex coefficients per cell
constexpr double kProfileReach = 1.5;   // |t| a cell's polynomial is made for [cells]
// CTAs per SM the planner counts on (the focus kernel's launch bound), and units per CTA.
#ifndef TDC_PROFILE_CTAS
#define TDC_PROFILE_CTAS 8
#endif
constexpr int kProfileCtasPerSm = TDC_PROFILE_CTAS;
#ifndef TDC_PROFILE_MIN_UNITS
#define TDC_PROFILE_MIN_UNITS 1
#endif
constexpr int kProfileMinUnitsPerSlot = TDC_PROFILE_MIN_UNITS;
constexpr int kProfileBandMinUnitsPerSlot = 8;  // (units differ in their live chirps)

// Groups of at most this many carrier cycles take their phase unreduced (kernels with LINE).
constexpr double kLineMaxCycles = 4.5;

// Inputs and outputs of profile_build_kernel.
struct ProfileBuild {
    const float2 *rows;      // [C][s_pad] windowed samples
    const float4 *chirps;    // [C] records of chirp_words float4: position high, low, ...
    const float2 *twiddle;   // [S][kProfileNodes], launch_profile_twiddle
    const float *factor;     // [S]
    float4 *cells;           // [C][n_cells][kProfileCoefs / 2]
    int *cell_base;          // [C]
    ProfileJob *job_out;     // receives `job`
    ProfileJob job;
    double box_min[3], box_max[3];  // bounding box of the grid
    double cells_per_m;
    int C, S, s_pad, n_cells;
    int chirp_words;
    int margin;              // cells the table starts early (even; smooth motion)
    const float4 *traj;      // vibration: FocusJob::traj (else null)
    float phase_g, phase_g1; // 2 pi gc and 2 pi g1 [rad / m]
};

// Tiles of a P-pixel grid whose runs are `run` pixels long: groups of kProfilePixels
// consecutive pixels of a run, kProfileThreads groups a tile (in bands of kProfileBand runs).
constexpr int kProfileBand = 8;
inline long long profile_tiles(long long P, int run, int pixels = kProfilePixels)
{
    const long long per = (run + pixels - 1) / pixels;
    const long long groups = (P + run - 1) / run * per;
    return (groups + kProfileThreads - 1) / kProfileThreads;
}

struct FocusUnit {
    int job;
    int tile;
    int group;
    int span;  // 0: the group's chirps; else unit_span(lo, hi): the chirps group x cpg + [lo, hi)
               // (the FP32-bulk kernels; the host sets it only for chirps the tile cannot see in band)
};
// FocusUnit::span: a marker bit and two 15-bit chirp offsets within the group (groups of
// fewer than kUnitSpanMax chirps).
constexpr int kUnitSpanMax = 1 << 15;
__host__ __device__ constexpr int unit_span(int lo, int hi) { return (1 << 30) | (lo << 15) | hi; }
__host__ __device__ constexpr int unit_span_lo(int span) { return (span >> 15) & (kUnitSpanMax - 1); }
__host__ __device__ constexpr int unit_span_hi(int span) { return span & (kUnitSpanMax - 1); }

// Kernel-side status bits (written to the status word in scratch).
enum StatusBits : int {
    kStatusTimeout = 1,
    kStatusBadJob = 2,  // a kernel found a job record outside what it takes (no work done for it)
};

// ---- launchers (defined in the .cu files) ----
cudaError_t launch_range_window(float *w, int n, int apply, cudaStream_t st);
cudaError_t launch_prewindow(float2 *xw, const float *w, int C, int S, int s_pad, cudaStream_t st);
cudaError_t launch_chirp_positions(ChirpRec *recs, const double *base, const double *off, int C, cudaStream_t st);
// Direct-read ingest (source may be pageable host memory where the device reads it coherently).
cudaError_t launch_prewindow_from(const float2 *src, const float *w, int C, int S, int s_pad, float2 *xw,
                                  cudaStream_t st);
// flags[flag] |= 1 when a sample of any chirp differs (bitwise) from the chirp's first; a is [C][S][k].
struct RowScan {
    const float *a;
    int k, flag;
};
cudaError_t launch_rows_differ(const RowScan *scans, int n, int C, int S, int *flags, cudaStream_t st);
cudaError_t launch_tile_radius(const float4 *hi, const float4 *lo, long long P, int rows, int cols, int tile_cols,
                               int n_tiles, float *radius, cudaStream_t st);

// What is measured of a grid on the device. box: minima and maxima of x, y, z as order-preserving keys of
// the double-float values (pair_key; pair_value on the host and device). words (float bits, starting
// at 0; a NaN compares above any distance): 0..2 and 7 reach of the groups of 8, 4, 2 and 16 pixels, 3
// the anchor span, 4..6 largest offset along each axis in the groups of 16.
struct GridBounds {
    long long box[6];
    int words[8];
};

inline void grid_bounds_init(GridBounds &b)
{
    for (int k = 0; k < 3; ++k) {
        b.box[k] = 0x7fffffffffffffffLL;
        b.box[3 + k] = -0x7fffffffffffffffLL - 1;
    }
    for (int &w : b.words) w = 0;
}

// The value of a key: the upper word is the high float, the lower one the low float.
#ifdef __CUDACC__
__host__ __device__
#endif
inline double pair_value(long long key)
{
    const int k[2] = {(int)(key >> 32), (int)((unsigned int)key ^ 0x80000000u)};
    union {
        int i;
        float f;
    } v[2];
    for (int j = 0; j < 2; ++j) v[j].i = k[j] >= 0 ? k[j] : k[j] ^ 0x7fffffff;
    // (no low part beside an infinity or NaN)
    return v[0].f - v[0].f == 0.0f ? (double)v[0].f + (double)v[1].f : (double)v[0].f;
}

cudaError_t launch_grid_bbox(const float4 *hi, const float4 *lo, long long P, GridBounds *out, cudaStream_t st);
cudaError_t launch_grid_from_f32(const float *grid, long long P, float4 *hi, cudaStream_t st);
cudaError_t launch_grid_from_f64(const double *grid, long long P, float4 *hi, float4 *lo, cudaStream_t st);

// FP32-bulk focus over a unit list. `jobs` and `units` are device arrays.
// Long chirps (rows longer than the stages hold): the same focus with rows staged in
// segments of job.seg_len samples; stage_bytes >= seg_len x 8 + one record.
cudaError_t launch_focus_fp32_seg(const FocusJob *jobs_dev, const FocusUnit *units_dev, int n_units,
                                  int *counter_dev, int *status_dev, int stage_bytes, int grid_ctas, bool skip_zero,
                                  cudaStream_t st);
int focus_fp32_seg_blocks_per_sm(int stage_bytes);
// skip_zero: skip chirps whose window is zero for a whole warp (any job with a finite band).
// store_sums: also write job.chirp_sums (whole-row staging only).
// anchored: anchored ranges (neither skip_zero nor store_sums; flat tiles; at most
// kAnchorMaxStageChirps chirps a stage; every pixel within kAnchorMaxDistance of its anchor).
cudaError_t launch_focus_fp32(const FocusJob *jobs_dev, const FocusUnit *units_dev, int n_units,
                              int *counter_dev, int *status_dev, int stage_bytes, int grid_ctas,
                              bool skip_zero, bool store_sums, bool anchored, cudaStream_t st);
int focus_fp32_anchor_blocks_per_sm(int stage_bytes);
// Smooth-motion focus (tdc_motion.cu): per-sample positions given by job.chirps as
// MotionRec records, rows staged whole (stage_bytes >= chirps x (s_pad x 8 + 80)),
// psi linearised over segments of job.seg_len samples (a power of two >= 8).
cudaError_t launch_focus_motion(const FocusJob *jobs_dev, const FocusUnit *units_dev, int n_units, int *counter_dev,
                                int *status_dev, int stage_bytes, int grid_ctas, bool skip_zero, cudaStream_t st);
int focus_motion_blocks_per_sm(int stage_bytes);
int focus_motion_smem_bytes(int stage_bytes);
// Plain FP64-phase focus (comparator and general fallback), one CTA per unit.
cudaError_t launch_focus_fp64(const FocusJob *jobs_dev, const FocusUnit *units_dev, int n_units,
                              int *status_dev, int per_sample, cudaStream_t st);
// (plan_pixels: pixels of the grid that the groups were planned for; enabled, when given: the launch does
// nothing unless *enabled == want.)
cudaError_t launch_focus_reduce(const float4 *partial, int n_groups, long long P, long long plan_pixels, float2 *image,
                                cudaStream_t st, const int *enabled = nullptr, int want = 0);
// FP32 general focus (tdc_general.cu). variant bits: 1 per-sample positions, 2 per-sample
// windows, 4 wide (non-uniform sampling residual, large intra-chirp motion: reduced phase
// correction, longer range-change series); at least one set. Rows are staged job.seg_len
// samples at a time: whole rows (seg_len = s_pad, job.stage_chirps chirps a stage) or
// segments of one chirp; stage_bytes = chirps x (seg_len x row bytes per sample + one
// record) + seg_len x table bytes per sample (see general_stage_bytes_for).
// n (even) entries of a per-sample table to two samples side by side (FocusJob::traj).
cudaError_t launch_pair_samples(float4 *table, long long n, cudaStream_t st);
// Bounds on each chirp's windows over its samples, behind the table wins [C][s_pad].
cudaError_t launch_window_bounds(float4 *wins, const float4 *traj, const float2 *xw, int C, int S, int s_pad,
                                 cudaStream_t st);
cudaError_t launch_focus_general(int variant, const FocusJob *jobs_dev, const FocusUnit *units_dev, int n_units,
                                 int *counter_dev, int *status_dev, int stage_bytes, int grid_ctas, cudaStream_t st);
int focus_general_blocks_per_sm(int variant, int stage_bytes);
int focus_general_smem_bytes(int stage_bytes);

// Range profiles: the per-length constants (twiddle [S][kProfileNodes], factor [S]), the table
// of the resident acquisition over the grid's ranges, and the focus that reads it, with
// `group` (16, 8, 4, 2 or 1) consecutive pixels sharing an anchor (band: a finite Doppler band; line: runs
// parallel to an axis, the only form with 16).
// (enabled, when given: nothing where *enabled is 0)
cudaError_t launch_profile_twiddle(float2 *twiddle, float *factor, int S, cudaStream_t st, const int *enabled = nullptr);
cudaError_t launch_profile_build(const ProfileBuild &b, cudaStream_t st);
// The same with its inputs in device memory, of at most max_cells cells; nothing where *enabled is 0.
cudaError_t launch_profile_build_indirect(const ProfileBuild *dev, const int *enabled, int C, int S, int max_cells,
                                          cudaStream_t st);
// motion: 1, the records are MoveRec, every sample of a chirp at a range of its own; 2, they are
// VibRec and there are kVibTables tables.
cudaError_t launch_focus_profile(int group, bool band, int motion, bool line, const FocusJob *jobs_dev, const FocusUnit *units_dev, int n_units,
                                 int *counter_dev, int grid_ctas, cudaStream_t st);
// Its adjoint: gpart[tile][C] = (d/dx, d/dy, d/dz) of each chirp over the tile's pixels (sums of
// Re(conj(G) dI/dR) (P - T) / R; .w is not written).
cudaError_t launch_adjoint_profile(int group, bool band, bool line, const FocusJob *jobs_dev, const FocusUnit *units_dev,
                                   int n_units, int *counter_dev, int grid_ctas, const float2 *gimg, float4 *gpart,
                                   cudaStream_t st);
int focus_profile_blocks_per_sm(int group, bool band, bool adjoint, int motion, bool line);
// Straight-line fit of every chirp's offsets (FocusJob::traj, chirps with sample-0 positions) and the
// principal direction of what it leaves, as VibRec; maxima[0..2] = max(maxima, largest deviation,
// deviation off that direction, |W1|) as float bits (starting at 0; NaN above all).
cudaError_t launch_vib_fit(const float4 *traj, const ChirpRec *chirps, int C, int S, int s_pad, float phase_per_m,
                           VibRec *recs, int *maxima, cudaStream_t st);
// GridBounds::words but the anchor span, for groups of consecutive pixels of a run.
cudaError_t launch_group_reach(const float4 *hi, const float4 *lo, long long P, int run, int *words, cudaStream_t st);

// Adjoint of the FP32-bulk focus w.r.t. per-chirp position offsets: per-(tile, chirp)
// float4 partials, then an FP64 sum over tiles into grad[C][3]. stored: job.xw holds the
// rows pre-scaled by the sample index and job.chirp_sums the forward's per-(chirp, pixel)
// sums (flat tiles).
cudaError_t launch_adjoint_fp32(const FocusJob *jobs_dev, const FocusUnit *units_dev, int n_units, int *counter_dev,
                                int *status_dev, int stage_bytes, int stage_chirps, int grid_ctas,
                                const float2 *gimg, float4 *gpart, bool stored, cudaStream_t st);
cudaError_t launch_adjoint_reduce(const float4 *gpart, int n_tiles, int C, double *grad, cudaStream_t st);
int adjoint_fp32_blocks_per_sm(int stage_bytes, int stage_chirps, bool stored);
// rows_out[c][s] = s * rows[c][s] (complex, [C][s_pad]): the adjoint's pre-scaled rows.
cudaError_t launch_scale_rows(const float2 *rows, int C, int s_pad, float2 *rows_out, cudaStream_t st);
int adjoint_fp32_smem_bytes(int stage_bytes, int stage_chirps);

// Let `fn` launch with as much dynamic shared memory as the device allows. The attribute
// is process-wide per kernel: every caller sets this same value, so threads that plan
// and launch with different sizes at the same time cannot undercut one another.
template <class F>
inline cudaError_t allow_max_dynamic_smem(F *fn)
{
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes a{};
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, reinterpret_cast<const void *>(fn));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(reinterpret_cast<const void *>(fn), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 optin - (int)a.sharedSizeBytes);
    return e;
}

// Record `msg` as the calling thread's tdc_last_error() and return `code`.
int set_last_error(int code, const char *msg);
inline int set_last_error(int code, const std::string &msg) { return set_last_error(code, msg.c_str()); }

// Occupancy of the FP32-bulk kernel at a given dynamic shared memory size.
int focus_fp32_blocks_per_sm(int stage_bytes);
int focus_fp32_smem_bytes(int stage_bytes, bool anchored = false);

}  // namespace tdc
