// tdc_noalloc.cu -- the focus entry point that allocates nothing.
//
// Some callers cannot allocate device memory when they focus: radar processing
// chains that provision all device memory once at start-up and must not
// allocate afterwards (real-time and certified pipelines with a fixed memory
// budget), plug-ins running inside a host framework that owns the device
// allocator, and code that must not call cudaMalloc while a stream is being
// captured. For them, tdc_focus_noalloc runs the same FP32-bulk focus kernel
// (focus_fp32_kernel) and reduce kernel as tdc_processor_focus_device, on
// device inputs and an output the caller provides, with the kernel's scratch
// (work counter, status word, job record, unit table, per-group partial sums)
// taken from a file-scope __device__ array of TDC_NOALLOC_SCRATCH_BYTES instead
// of cudaMalloc. Every GPU that loads this library holds that array until the
// process exits.
//
// Large calls take range profiles (tdc_profile.cu, every range in double-float) when the table
// fits the array. The host knows neither the grid's extent nor the trajectory, so a kernel
// decides from the inputs on the device (noalloc_decide_kernel): both forms are enqueued, and
// the one not taken finds its work counter already past its last unit. 200 x 150 pixels x 300
// chirps x 256 samples: 395 -> 144 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <limits>
#include <mutex>
#include <string>

#include "tdc_gb300.h"
#include "tdc_internal.h"
#include "tdc_processor_impl.h"

using namespace tdc;

namespace {

static __device__ __align__(256) unsigned char g_noalloc_scratch[TDC_NOALLOC_SCRATCH_BYTES];

constexpr int kMaxDevices = 64;
std::mutex g_mu;
// Device address of g_noalloc_scratch per device, as last looked up with that device
// current. Calls outside stream capture look it up again (cheap), so a device reset or
// another context made current since is picked up; calls under capture use this copy.
unsigned char *g_scratch_addr[kMaxDevices] = {};

size_t round_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

constexpr size_t kOffStatus = 0;    // int counter, int status
constexpr size_t kOffJob = 256;     // FocusJob
constexpr size_t kOffUnits = 512;   // FocusUnit[n_units]
// Words at kOffStatus.
constexpr int kWordCounter = 0, kWordStatus = 1, kWordProfile = 2, kWordProfileCounter = 3;
constexpr size_t kOffBounds = 32;  // GridBounds
constexpr int kSpent = 1 << 30;  // a work counter past every unit

size_t layout_bytes(long long P, long long n_units, int n_groups, size_t &off_partial)
{
    off_partial = round_up(kOffUnits + (size_t)n_units * sizeof(FocusUnit), 256);
    return off_partial + (size_t)n_groups * (size_t)P * 16;
}

// Job record, unit table (tile-major, one unit per tile x chirp group) and zeroed
// counter / status written into the scratch array by the device itself.
__global__ void noalloc_setup_kernel(FocusJob job, GridBounds bounds, int n_tiles, int n_groups, unsigned char *base)
{
    const long long n_units = (long long)n_tiles * n_groups;
    const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i0 == 0) {
        int *words = reinterpret_cast<int *>(base + kOffStatus);
        words[kWordCounter] = 0;
        words[kWordStatus] = 0;
        words[kWordProfile] = 0;
        *reinterpret_cast<GridBounds *>(base + kOffBounds) = bounds;
        *reinterpret_cast<FocusJob *>(base + kOffJob) = job;
    }
    FocusUnit *units = reinterpret_cast<FocusUnit *>(base + kOffUnits);
    for (long long u = i0; u < n_units; u += (long long)gridDim.x * blockDim.x) {
        units[u] = FocusUnit{0, (int)(u / n_groups), (int)(u % n_groups), 0};
    }
}

// The profile form of a call: its job, its unit table and what its table is built from, in the
// scratch array.
struct ProfilePlan {
    FocusJob job;
    ProfileBuild build;  // box, n_cells and the job record are filled in on the device
    FocusJob *job_out;
    ProfileBuild *build_out;
    FocusUnit *units;
    int n_tiles, n_groups, max_cells;
    double g1, gc;
};

// Whether range profiles apply, from the grid's bounding box (bounds, from grid_bbox_kernel) and
// the chirp records, as the processor decides it from its host copies: finite inputs, a grid
// within the unambiguous range, ranges the cell index resolves, a table that fits. Fills in the
// build inputs and leaves one of the two work counters spent: the first block, with the farthest range in
// FP32 (FP64 runs at 1/64 of its rate); the others write the unit table.
__global__ void noalloc_decide_kernel(ProfilePlan plan, const GridBounds *__restrict__ bounds, int *__restrict__ words,
                                      bool band)
{
    __shared__ float far2[8];
    __shared__ double box[6];
    const int tid = threadIdx.x;
    if (blockIdx.x > 0) {
        const int n = plan.n_tiles * plan.n_groups;
        for (int u = (blockIdx.x - 1) * blockDim.x + tid; u < n; u += (gridDim.x - 1) * blockDim.x)
            plan.units[u] = FocusUnit{0, u % plan.n_tiles, u / plan.n_tiles, 0};
        return;
    }
    if (tid < 6) box[tid] = pair_value(bounds->box[tid]);
    __syncthreads();
    float most = 0.f;
    bool finite = true;
    const ChirpRec *recs = reinterpret_cast<const ChirpRec *>(plan.build.chirps);
    for (int c = tid; c < plan.build.C; c += blockDim.x) {
        const ChirpRec r = recs[c];
        float f = 0.f;
        const float p[3] = {r.p_hi.x, r.p_hi.y, r.p_hi.z};
        for (int k = 0; k < 3; ++k) {
            const float d = fmaxf(fabsf((float)box[k] - p[k]), fabsf(p[k] - (float)box[3 + k]));
            f += d * d;
        }
        finite = finite && f < 1e30f && isfinite(r.p_lo.x + r.p_lo.y + r.p_lo.z) &&
                 (band || (isfinite(r.vel.x) && isfinite(r.vel.y) && isfinite(r.vel.z) && isfinite(r.p_hi.w)));
        most = fmaxf(most, f);
    }
    most = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(most)));
    if ((tid & 31) == 0) far2[tid >> 5] = most;
    finite = __syncthreads_and(finite);
    if (tid) return;
    for (int w = 1; w < 8; ++w) far2[0] = fmaxf(far2[0], far2[w]);
    ProfileBuild &b = plan.build;
    double diag2 = 0.0;
    for (int k = 0; k < 3; ++k) {
        b.box_min[k] = box[k];
        b.box_max[k] = box[3 + k];
        diag2 += (b.box_max[k] - b.box_min[k]) * (b.box_max[k] - b.box_min[k]);
    }
    const double span = fabs(b.cells_per_m) * sqrt(diag2);
    const bool take = finite && diag2 < 1e30 && fabs(b.cells_per_m) * (1.0f + 1e-6f) * sqrtf(far2[0]) < 2097152.0 &&
                      span + 7.0 <= (double)plan.max_cells && span + 7.0 <= 4.0 * b.S;
    if (take) {
        b.n_cells = ((int)ceil(span) + 7) / 2 * 2;
        b.job.n_cells = b.n_cells;
        *plan.build_out = b;
        *plan.job_out = plan.job;
    }
    words[kWordProfile] = take;
    words[kWordCounter] = take ? kSpent : 0;
    words[kWordProfileCounter] = take ? 0 : kSpent;
}

int fail(int code, const std::string &msg) { return set_last_error(code, msg); }

void split_dd(double v, float &h, float &l)
{
    h = static_cast<float>(v);
    l = static_cast<float>(v - static_cast<double>(h));
}

// Chirp groups so that tiles x groups fill whole waves of `slots` (among the splits
// with at least kFocusMinUnitsPerSlot units per slot when there are any), limited to
// what fits in the scratch array.
bool plan(long long P, int C, int slots, int &n_groups, int &cpg, size_t &off_partial)
{
    const long long n_tiles = (P + kFocusTile - 1) / kFocusTile;
    const long long min_units = (long long)kFocusMinUnitsPerSlot * slots;
    const int gmax = std::max(1, std::min(C, 1024));
    for (int pass = 0; pass < 2; ++pass) {
        double best = std::numeric_limits<double>::infinity();
        for (int g = 1; g <= gmax; ++g) {
            const int c = (C + g - 1) / g;
            const int geff = (C + c - 1) / c;
            if (geff != g) continue;
            size_t off;
            if (layout_bytes(P, n_tiles * geff, geff, off) > TDC_NOALLOC_SCRATCH_BYTES) break;
            if (pass == 0 && n_tiles * geff < min_units) continue;
            const long long waves = (n_tiles * geff + slots - 1) / slots;
            const double cost = (double)waves * (c + 0.5);
            if (cost < best - 1e-9) {
                best = cost;
                n_groups = geff;
                cpg = c;
                off_partial = off;
            }
        }
        if (best < std::numeric_limits<double>::infinity()) return true;
    }
    return false;
}

// Checks, plans and enqueues the setup, focus and reduce kernels on `st`; nothing
// blocks. `status_word` receives the device address of the kernels' status word.
int enqueue(const tdc_noalloc_focus_args *a, float *image_dev, cudaStream_t st, int **status_word)
{
    // ---- argument and size checks first: nothing below runs for rejected sizes ----
    if (!a || !image_dev) return fail(TDC_ERR_INVALID_ARGUMENT, "null argument");
    if (a->n_pri <= 0) return fail(TDC_ERR_INVALID_ARGUMENT, "nPri must be greater than 0");
    if (a->n_samples <= 0) return fail(TDC_ERR_INVALID_ARGUMENT, "nSamples must be greater than 0");
    if (a->n_pix <= 0) return fail(TDC_ERR_INVALID_ARGUMENT, "n_pix must be greater than 0");
    if (!a->samples || !a->chirps || !a->grid_hi) return fail(TDC_ERR_INVALID_ARGUMENT, "null input array");
    if ((reinterpret_cast<uintptr_t>(a->samples) | reinterpret_cast<uintptr_t>(a->chirps) |
         reinterpret_cast<uintptr_t>(a->grid_hi) | reinterpret_cast<uintptr_t>(a->grid_lo) |
         reinterpret_cast<uintptr_t>(a->skip_points)) & 15u)
        return fail(TDC_ERR_INVALID_ARGUMENT, "input arrays must be 16-byte aligned");
    const long long P = a->n_pix;
    const int C = a->n_pri, S = a->n_samples;
    const int s_pad = (int)round_up((size_t)S, kSampleAlign);
    const long long n_tiles = (P + kFocusTile - 1) / kFocusTile;
    size_t min_off;
    const size_t min_bytes = layout_bytes(P, n_tiles, 1, min_off);
    if (min_bytes > TDC_NOALLOC_SCRATCH_BYTES || n_tiles > (1LL << 30)) {
        return fail(TDC_ERR_UNSUPPORTED, "tdc_focus_noalloc: " + std::to_string(P) + " pixels need " +
                                             std::to_string(min_bytes) + " bytes of scratch; the fixed array "
                                             "holds " + std::to_string((size_t)TDC_NOALLOC_SCRATCH_BYTES) +
                                             " (about 2M pixels)");
    }
    // Whole rows only (the processor stages longer rows in segments): the same limit as
    // the processor's choice between the two, TDC_NOALLOC_MAX_SAMPLES samples.
    if (impl::needs_segments(s_pad))
        return fail(TDC_ERR_UNSUPPORTED, "tdc_focus_noalloc: nSamples " + std::to_string(S) + " above " +
                                             std::to_string(TDC_NOALLOC_MAX_SAMPLES) +
                                             " (whole rows must fit the shared-memory stages)");
    int cb = 1;
    const int stage_bytes = impl::stage_bytes_for(s_pad, cb);

    // ---- per-device set-up: the device address of the scratch array ----
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(TDC_ERR_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxDevices) return fail(TDC_ERR_UNSUPPORTED, "device index out of range");
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    e = cudaStreamIsCapturing(st, &cap);
    if (e != cudaSuccess) return fail(TDC_ERR_CUDA, std::string("cudaStreamIsCapturing: ") + cudaGetErrorString(e));
    unsigned char *base = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        if (cap == cudaStreamCaptureStatusNone) {
            void *ptr = nullptr;
            e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
            if (e != cudaSuccess || !ptr)
                return fail(TDC_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
            g_scratch_addr[dev] = static_cast<unsigned char *>(ptr);
        } else if (!g_scratch_addr[dev]) {
            return fail(TDC_ERR_UNSUPPORTED, "tdc_focus_noalloc: the first call on a device must come before "
                                             "any stream capture (it looks up the scratch array's address)");
        }
        base = g_scratch_addr[dev];
    }

    int n_sm = 0;
    e = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return fail(TDC_ERR_CUDA, std::string("device query: ") + cudaGetErrorString(e));
    const int bps = focus_fp32_blocks_per_sm(stage_bytes);
    if (bps <= 0) return fail(TDC_ERR_CUDA, "focus kernel does not fit on the device");
    const int slots = n_sm * bps;
    int n_groups = 1, cpg = C;
    size_t off_partial = min_off;
    if (!plan(P, C, slots, n_groups, cpg, off_partial)) {
        n_groups = 1;
        cpg = C;
        off_partial = min_off;
    }

    FocusJob job{};
    job.xw = reinterpret_cast<const float4 *>(a->samples);
    job.chirps = reinterpret_cast<const ChirpRec *>(a->chirps);
    job.grid_hi = reinterpret_cast<const float4 *>(a->grid_hi);
    job.grid_lo = reinterpret_cast<const float4 *>(a->grid_lo);
    job.skip = reinterpret_cast<const SkipPoint *>(a->skip_points);
    job.gs = nullptr;
    job.partial = reinterpret_cast<float4 *>(base + off_partial);
    job.P = P;
    job.C = C;
    job.S = S;
    job.s_pad = s_pad;
    job.n_groups = n_groups;
    job.chirps_per_group = cpg;
    job.chunk = kChunk;
    job.stage_chirps = cb;
    job.flags = (a->doppler_win_taper ? kFlagTaper : 0) | (a->skip_points ? kFlagSkipTest : 0);
    job.n_tiles = (int)n_tiles;
    job.per_sample = 0;
    split_dd(a->g0, job.g0_hi, job.g0_lo);
    split_dd(a->g1, job.g1, job.g1_lo);
    job.two_over_lambda = 2.0f / a->lambda;
    job.half_bw = a->doppler_bandwidth / 2.0f;
    job.inv_bw = 1.0f / a->doppler_bandwidth;
    job.az_a = kAzimuthA;

    const long long n_units = n_tiles * n_groups;
    const int setup_blocks = (int)std::min<long long>((n_units + 255) / 256, 1024);
    GridBounds bounds;
    grid_bounds_init(bounds);
    noalloc_setup_kernel<<<setup_blocks, 256, 0, st>>>(job, bounds, (int)n_tiles, n_groups, base);
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail(TDC_ERR_CUDA, std::string("setup kernel: ") + cudaGetErrorString(e));
    int *words = reinterpret_cast<int *>(base + kOffStatus);

    // ---- range profiles, where the call is large enough and a table may fit ----
    const bool band = std::isfinite(job.half_bw);
    ProfilePlan pp{};
    bool profile = impl::profile_pays((double)P, C, S, band) && impl::profile_own_pays(S, band) &&
                   (band || job.half_bw > 0.0f);
    if (profile) {
        const double gc = a->g0 + a->g1 * (S / 2), cells_per_m = 4.0 * S * a->g1;
        const int tiles = (int)profile_tiles(P, (int)std::min<long long>(P, 1 << 30));
        // two units per CTA, partials in at most a third of the array
        const int pslots = n_sm * focus_profile_blocks_per_sm(1, band, false, 0, false);
        const long long fit = (long long)(TDC_NOALLOC_SCRATCH_BYTES / 3) / (P * 16);
        int pg = (int)std::max<long long>(1, std::min<long long>({(long long)C, fit, (2LL * pslots + tiles - 1) / tiles}));
        const int pcpg = (C + pg - 1) / pg;
        pg = (C + pcpg - 1) / pcpg;
        // (laid over the direct form's partials: one of the two runs)
        size_t off = round_up(kOffUnits + (size_t)n_units * sizeof(FocusUnit), 256);
        auto take = [&](size_t bytes) {
            const size_t at = off;
            off = round_up(off + bytes, 256);
            return at;
        };
        const size_t o_job = take(sizeof(FocusJob)), o_pjob = take(sizeof(ProfileJob)),
                     o_build = take(sizeof(ProfileBuild)), o_units = take((size_t)tiles * pg * sizeof(FocusUnit)),
                     o_base = take((size_t)C * 4), o_tw = take((size_t)S * (kProfileNodes * 8 + 4)),
                     o_part = take((size_t)pg * P * 16);
        const long long left = (long long)TDC_NOALLOC_SCRATCH_BYTES - (long long)off;
        pp.max_cells = (int)std::max<long long>(0, std::min<long long>(4LL * S, left / ((long long)C * kProfileCoefs * 8)));
        profile = pp.max_cells >= 16 && std::isfinite(gc) && std::fabs(gc) > 0.0 && std::isfinite(cells_per_m);
        pp.n_tiles = tiles;
        pp.n_groups = pg;
        pp.job_out = reinterpret_cast<FocusJob *>(base + o_job);
        pp.build_out = reinterpret_cast<ProfileBuild *>(base + o_build);
        pp.units = reinterpret_cast<FocusUnit *>(base + o_units);
        pp.job = job;
        pp.job.partial = reinterpret_cast<float4 *>(base + o_part);
        pp.job.n_groups = pg;
        pp.job.chirps_per_group = pcpg;
        pp.job.n_tiles = tiles;
        pp.job.grid_cols = (int)std::min<long long>(P, 1 << 30);
        ProfileBuild &b = pp.build;
        b.job_out = reinterpret_cast<ProfileJob *>(base + o_pjob);
        pp.job.profile = b.job_out;
        b.rows = reinterpret_cast<const float2 *>(a->samples);
        b.chirps = reinterpret_cast<const float4 *>(a->chirps);
        b.twiddle = reinterpret_cast<const float2 *>(base + o_tw);
        b.factor = reinterpret_cast<const float *>(b.twiddle + (size_t)S * kProfileNodes);
        b.cells = reinterpret_cast<float4 *>(base + off);
        b.cell_base = reinterpret_cast<int *>(base + o_base);
        b.cells_per_m = cells_per_m;
        b.C = C;
        b.S = S;
        b.s_pad = s_pad;
        b.chirp_words = (int)(sizeof(ChirpRec) / 16);
        split_dd(gc, b.job.gc_hi, b.job.gc_lo);
        split_dd(cells_per_m, b.job.cells_hi, b.job.cells_lo);
        b.job.inv_gc2x4 = (float)(4.0 / (gc * gc));
        b.job.cells_per_cycle = (float)(cells_per_m / gc);
        b.job.cells = b.cells;
        b.job.cell_base = b.cell_base;
        b.job.inv_gc = (float)(1.0 / gc);
    }
    if (profile) {
        GridBounds *bounds_dev = reinterpret_cast<GridBounds *>(base + kOffBounds);
        e = launch_grid_bbox(job.grid_hi, job.grid_lo, P, bounds_dev, st);
        if (e == cudaSuccess) {
            noalloc_decide_kernel<<<9, 256, 0, st>>>(pp, bounds_dev, words, band);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess)
            e = launch_profile_twiddle(const_cast<float2 *>(pp.build.twiddle), const_cast<float *>(pp.build.factor), S, st,
                                       words + kWordProfile);
        if (e == cudaSuccess)
            e = launch_profile_build_indirect(pp.build_out, words + kWordProfile, C, S, pp.max_cells, st);
        const int n = pp.n_tiles * pp.n_groups;
        const int ctas = std::min(n, n_sm * focus_profile_blocks_per_sm(1, band, false, 0, false));
        if (e == cudaSuccess)
            e = launch_focus_profile(1, band, 0, false, pp.job_out, pp.units, n, words + kWordProfileCounter, ctas, st);
        if (e == cudaSuccess)
            e = launch_focus_reduce(pp.job.partial, pp.n_groups, P, P, reinterpret_cast<float2 *>(image_dev), st,
                                    words + kWordProfile, 1);
        if (e != cudaSuccess)
            return fail(TDC_ERR_CUDA, std::string("range profile kernels: ") + cudaGetErrorString(e));
    }
    const int grid = (int)std::min<long long>(n_units, slots);
    e = launch_focus_fp32(reinterpret_cast<const FocusJob *>(base + kOffJob),
                          reinterpret_cast<const FocusUnit *>(base + kOffUnits), (int)n_units,
                          reinterpret_cast<int *>(base + kOffStatus), reinterpret_cast<int *>(base + kOffStatus) + 1,
                          stage_bytes, grid, std::isfinite(job.half_bw), false, false, st);
    if (e != cudaSuccess) return fail(TDC_ERR_CUDA, std::string("focus kernel: ") + cudaGetErrorString(e));
    e = launch_focus_reduce(job.partial, n_groups, P, P, reinterpret_cast<float2 *>(image_dev), st,
                            words + kWordProfile, 0);
    if (e != cudaSuccess) return fail(TDC_ERR_CUDA, std::string("reduce kernel: ") + cudaGetErrorString(e));
    *status_word = reinterpret_cast<int *>(base + kOffStatus) + 1;
    return TDC_OK;
}

}  // namespace

extern "C" int tdc_focus_noalloc(const tdc_noalloc_focus_args *a, float *image_dev, void *stream)
{
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int *status_word = nullptr;
    if (int rc = enqueue(a, image_dev, st, &status_word)) return rc;
    // Blocking: collect the kernels' status word before returning.
    int status = 0;
    cudaError_t e = cudaMemcpyAsync(&status, status_word, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(TDC_ERR_CUDA, std::string("focus: ") + cudaGetErrorString(e));
    if (status & kStatusTimeout) return fail(TDC_ERR_TIMEOUT, "focus kernel wait timed out");
    if (status & kStatusBadJob) return fail(TDC_ERR_CUDA, "focus kernel rejected its job record");
    return TDC_OK;
}

extern "C" int tdc_focus_noalloc_async(const tdc_noalloc_focus_args *a, float *image_dev, int *status_dev,
                                       void *stream)
{
    if (!status_dev) return fail(TDC_ERR_INVALID_ARGUMENT, "null status word");
    if (reinterpret_cast<uintptr_t>(status_dev) & 3u)
        return fail(TDC_ERR_INVALID_ARGUMENT, "status word must be 4-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int *status_word = nullptr;
    if (int rc = enqueue(a, image_dev, st, &status_word)) return rc;
    const cudaError_t e = cudaMemcpyAsync(status_dev, status_word, sizeof(int), cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return fail(TDC_ERR_CUDA, std::string("status copy: ") + cudaGetErrorString(e));
    return TDC_OK;
}
