// Focus and adjoint where device memory runs short, on a fake of the CUDA runtime: the engine's host code
// (tdc_capi.cpp) linked against allocations from a stated capacity and kernel launches that only count.
// What pays through range profiles takes them while their table fits, and the direct kernels otherwise.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <vector>

#include "tdc_gb300.h"
#include "tdc_internal.h"

using namespace tdc;

namespace {
size_t g_capacity = (size_t)1 << 40, g_used = 0, g_taken_after_query = 0, g_largest = 0;
std::map<void *, size_t> g_blocks;
cudaError_t g_last = cudaSuccess;
int g_profile = 0, g_direct = 0;  // focus and adjoint launches of either form

cudaError_t give(void **p, size_t n)
{
    g_largest = n > g_largest ? n : g_largest;
    if (g_used + n > g_capacity) return g_last = cudaErrorMemoryAllocation;
    *p = std::calloc(n, 1);
    g_blocks[*p] = n;
    g_used += n;
    return cudaSuccess;
}

cudaError_t take(void *p)
{
    auto it = g_blocks.find(p);
    if (it != g_blocks.end()) {
        g_used -= it->second;
        g_blocks.erase(it);
    }
    std::free(p);
    return cudaSuccess;
}

// A launch reports what is left of an earlier error, as a real one does.
cudaError_t launch() { return cudaGetLastError(); }
cudaError_t launch(int &count)
{
    ++count;
    return launch();
}
}  // namespace

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) { return give(p, n); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return give(p, n); }
cudaError_t cudaMallocHost(void **p, size_t n) { return (*p = std::calloc(n, 1)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void *p) { return take(p); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return take(p); }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *free_b, size_t *total)
{
    *free_b = g_capacity - g_used;
    *total = g_capacity;
    g_capacity -= g_taken_after_query;  // (another thread allocates)
    g_taken_after_query = 0;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void *, size_t, const void *, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) { *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t, cudaEvent_t) { *t = 0.f; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
}

namespace tdc {
cudaError_t launch_vib_fit(const float4 *, const ChirpRec *, int, int, int, float, VibRec *, int *, cudaStream_t) { return launch(); }
cudaError_t launch_grid_bbox(const float4 *, const float4 *, long long, GridBounds *b, cudaStream_t)
{
    // a square of 5.6 m: keys of (high, 0)
    for (int k = 0; k < 6; ++k) {
        const float v = k >= 3 && k < 5 ? 5.6f : 0.0f;
        int bits;
        std::memcpy(&bits, &v, 4);
        b->box[k] = (long long)bits << 32 | 0x80000000u;
    }
    return launch();
}
cudaError_t launch_group_reach(const float4 *, const float4 *, long long, int, int *w, cudaStream_t)
{
    const float reach = 4e-3f;
    for (int k : {0, 1, 2, 4, 7}) std::memcpy(&w[k], &reach, 4);
    return launch();
}
cudaError_t launch_prewindow(float2 *, const float *, int, int, int, cudaStream_t) { return launch(); }
cudaError_t launch_focus_fp32(const FocusJob *, const FocusUnit *, int, int *, int *, int, int, bool, bool, bool, cudaStream_t) { return launch(g_direct); }
cudaError_t launch_focus_fp64(const FocusJob *, const FocusUnit *, int, int *, int, cudaStream_t) { return launch(); }
cudaError_t launch_scale_rows(const float2 *, int, int, float2 *, cudaStream_t) { return launch(); }
cudaError_t launch_rows_differ(const RowScan *, int, int, int, int *, cudaStream_t) { return launch(); }
cudaError_t launch_tile_radius(const float4 *, const float4 *, long long, int, int, int, int, float *, cudaStream_t) { return launch(); }
cudaError_t launch_adjoint_fp32(const FocusJob *, const FocusUnit *, int, int *, int *, int, int, int, const float2 *, float4 *, bool, cudaStream_t) { return launch(g_direct); }
cudaError_t launch_focus_motion(const FocusJob *, const FocusUnit *, int, int *, int *, int, int, bool, cudaStream_t) { return launch(); }
cudaError_t launch_focus_reduce(const float4 *, int, long long, long long, float2 *, cudaStream_t, const int *, int) { return launch(); }
cudaError_t launch_pair_samples(float4 *, long long, cudaStream_t) { return launch(); }
cudaError_t launch_range_window(float *, int, int, cudaStream_t) { return launch(); }
cudaError_t launch_focus_general(int, const FocusJob *, const FocusUnit *, int, int *, int *, int, int, cudaStream_t) { return launch(g_direct); }
cudaError_t launch_focus_profile(int, bool, int, bool, const FocusJob *, const FocusUnit *, int, int *, int, cudaStream_t) { return launch(g_profile); }
cudaError_t launch_grid_from_f32(const float *, long long, float4 *, cudaStream_t) { return launch(); }
cudaError_t launch_grid_from_f64(const double *, long long, float4 *, float4 *, cudaStream_t) { return launch(); }
cudaError_t launch_profile_build(const ProfileBuild &, cudaStream_t) { return launch(); }
cudaError_t launch_window_bounds(float4 *, const float4 *, const float2 *, int, int, int, cudaStream_t) { return launch(); }
cudaError_t launch_adjoint_reduce(const float4 *, int, int, double *, cudaStream_t) { return launch(); }
cudaError_t launch_focus_fp32_seg(const FocusJob *, const FocusUnit *, int, int *, int *, int, int, bool, cudaStream_t) { return launch(g_direct); }
cudaError_t launch_prewindow_from(const float2 *, const float *, int, int, int, float2 *, cudaStream_t) { return launch(); }
cudaError_t launch_adjoint_profile(int, bool, bool, const FocusJob *, const FocusUnit *, int, int *, int, const float2 *, float4 *, cudaStream_t) { return launch(g_profile); }
cudaError_t launch_chirp_positions(ChirpRec *, const double *, const double *, int, cudaStream_t) { return launch(); }
cudaError_t launch_profile_twiddle(float2 *, float *, int, cudaStream_t, const int *) { return launch(); }
int focus_fp32_blocks_per_sm(int) { return 3; }
int adjoint_fp32_blocks_per_sm(int, int, bool) { return 3; }
int focus_motion_blocks_per_sm(int) { return 3; }
int focus_general_blocks_per_sm(int, int) { return 2; }
int focus_profile_blocks_per_sm(int, bool, bool, int, bool) { return 8; }
int focus_fp32_seg_blocks_per_sm(int) { return 3; }
int focus_fp32_anchor_blocks_per_sm(int) { return 3; }
int focus_fp32_smem_bytes(int, bool) { return 0; }
int focus_motion_smem_bytes(int) { return 0; }
int focus_general_smem_bytes(int) { return 0; }
}  // namespace tdc

namespace {
int g_failed = 0;
void expect(bool ok, const char *what)
{
    if (!ok) {
        std::printf("failed: %s (%s)\n", what, tdc_last_error());
        g_failed = 1;
    }
}

struct Scene {
    static constexpr int C = 1000, S = 256, N = 64;
    std::vector<float> raw = std::vector<float>(2 * C * S, 1.f), pri = std::vector<float>(C), times = std::vector<float>(S),
                       pos = std::vector<float>(3 * C * S), vel = std::vector<float>(3 * C * S),
                       att = std::vector<float>(4 * C * S, 0.f), grid = std::vector<float>(3 * N * N);
    std::vector<float> image = std::vector<float>(2 * N * N);
    std::vector<double> grad = std::vector<double>(3 * C);
    tdc_processor *p = nullptr;

    Scene()
    {
        for (int s = 0; s < S; ++s) times[s] = (float)(s * (40e-6 / S));
        for (int i = 0; i < C * S; ++i) pos[3 * i + 2] = 0.3f, att[4 * i] = 1.f;
        for (int i = 0; i < N * N; ++i) grid[3 * i] = (i % N) * 1e-3f, grid[3 * i + 1] = (i / N) * 1e-3f;
        const float bore[3] = {0.f, 1.f, 0.f};
        expect(tdc_processor_create(0, &p) == TDC_OK, "create");
        expect(tdc_processor_set_raw_data(p, raw.data(), pri.data(), times.data(), pos.data(), vel.data(), att.data(), C, S,
                                          1e14f, 77e9f, bore) == TDC_OK, "raw data");
        expect(tdc_processor_set_focus_grid(p, grid.data(), N, N) == TDC_OK, "grid");
        expect(tdc_processor_prepare(p, 0.f, __builtin_inff(), 0, 0, 1) == TDC_OK, "prepare");
        expect(tdc_processor_upload_grid(p) == TDC_OK, "upload");
        g_profile = g_direct = 0;
        g_largest = 0;
        g_last = cudaSuccess;
    }
    ~Scene()
    {
        tdc_processor_destroy(p);
        expect(g_used == 0, "every allocation is given back");
        g_capacity = (size_t)1 << 40;
    }
    int focus() { return tdc_processor_focus_device(p, image.data(), nullptr); }
    int adjoint() { return tdc_processor_adjoint_device(p, image.data(), grad.data(), nullptr); }
};
}  // namespace

int main()
{
    size_t table = 0, scratch = 0;
    {
        Scene s;
        expect(s.focus() == TDC_OK && g_profile == 1 && g_direct == 0, "memory for everything: profiles");
        table = g_largest;
        expect(s.adjoint() == TDC_OK && g_profile == 2 && g_direct == 0, "and their adjoint");
    }
    {
        Scene s;
        g_capacity = g_used + table;  // less than two tables: not planned
        expect(s.focus() == TDC_OK && g_profile == 0 && g_direct == 1, "half the free memory is no table");
        scratch = g_largest;
        expect(scratch < table, "the direct scratch is the smaller");
    }
    {
        Scene s;
        g_capacity = g_used + 2 * table + scratch;
        g_taken_after_query = 2 * table;  // free when planned, taken before the table was allocated
        expect(s.focus() == TDC_OK && g_profile == 0 && g_direct == 1, "memory taken in between: direct");
        expect(s.focus() == TDC_OK && g_direct == 2, "and again");
    }
    {
        Scene s;
        g_capacity = g_used + 2 * table;
        g_taken_after_query = table - ((size_t)1 << 20);  // the table fits, the scratch beside it does not
        expect(s.focus() == TDC_OK && g_profile == 0 && g_direct == 1, "no scratch beside the table: direct");
    }
    {
        Scene s;
        g_capacity = g_used + 2 * table + scratch;
        g_taken_after_query = 2 * table;
        expect(s.adjoint() == TDC_OK && g_profile == 0 && g_direct == 1, "adjoint, memory taken in between: direct");
    }
    {
        Scene s;
        expect(s.focus() == TDC_OK && g_profile == 1, "a focus with its table");
        g_capacity = g_used;  // nothing left for the adjoint's sums until the table is given back
        expect(s.adjoint() == TDC_OK && g_profile == 1 && g_direct == 1, "adjoint without the table: direct");
        g_capacity = (size_t)1 << 40;
        expect(s.adjoint() == TDC_OK && g_profile == 2, "and with memory again: profiles");
    }
    std::puts(g_failed ? "FAILED" : "ok");
    return g_failed;
}
