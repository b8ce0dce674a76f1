// The plans' choices of buffers and kernels, without a GPU: ykb_api.cpp and
// ykb_geometry.cpp linked with a fake CUDA runtime, whose device memory is a
// number of bytes, and fake launchers, which count their calls.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>

#include "ykb_internal.hpp"

namespace {

size_t g_capacity = ~size_t(0), g_used = 0;
std::map<void*, size_t> g_blocks;
int g_failures = 0, g_lines = 0, g_walks = 0;
bool g_capturing = false;

void expect(bool ok, const char* what)
{
    if (!ok) {
        ++g_failures;
        std::fprintf(stderr, "FAILED: %s\n", what);
    }
}

} // namespace

extern "C" {
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorName(cudaError_t) { return "error"; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaMalloc(void** p, size_t n)
{
    if (g_used + n > g_capacity) return cudaErrorMemoryAllocation;
    static char* next = reinterpret_cast<char*>(size_t(1) << 40);
    *p = next;
    next += (n + 511) / 512 * 512;
    g_blocks[*p] = n;
    g_used += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
    g_used -= g_blocks.at(p);
    g_blocks.erase(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* to, const void*, size_t n, cudaMemcpyKind kind, cudaStream_t)
{
    if (kind == cudaMemcpyDeviceToHost) std::memset(to, 0, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* status)
{
    *status = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
{
    *e = reinterpret_cast<cudaEvent_t>(1);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
}

namespace ykb {
cudaError_t launch_joseph_ray_table(const JosephView*, int, int, int, float4*, float*, cudaStream_t)
{
    return cudaSuccess;
}
cudaError_t launch_joseph_column_table(const float4*, int, int, int, float2*, int*, cudaStream_t)
{
    return cudaSuccess;
}
cudaError_t launch_joseph_ray_heights(const float4*, long, float2*, cudaStream_t) { return cudaSuccess; }
JosephFpLines joseph_fp_lines_shape(const std::vector<JosephView>&, int) { return {128, 144}; }
bool joseph_bp_runs(const std::vector<JosephView>&, int) { return true; }
int joseph_bp_splits(const ykb_volume&, int) { return 4; }
bool siddon_lines_apply(const ykb_cone_view*, int, int, const VolumeGrid&) { return true; }
cudaError_t launch_siddon_fp(const float*, const ykb_cone_view*, int, int, int, const VolumeGrid&, float*, int,
    cudaStream_t)
{
    ++g_walks;
    return cudaSuccess;
}
cudaError_t launch_siddon_bp(const float* in, const ykb_cone_view* v, int n, int nu, int nv, const VolumeGrid& g,
    float* out, int accumulate, cudaStream_t s)
{
    return launch_siddon_fp(in, v, n, nu, nv, g, out, accumulate, s);
}
cudaError_t launch_siddon_fp_lines(const float*, float* vt, const ykb_cone_view*, int, int, int,
    const VolumeGrid&, float*, int, cudaStream_t)
{
    expect(vt != nullptr, "the projector's copy");
    ++g_lines;
    return cudaSuccess;
}
cudaError_t launch_siddon_bp_lines(const float* in, float* vt, float* odd, const ykb_cone_view* v, int n,
    int nu, int nv, const VolumeGrid& g, float* out, int accumulate, cudaStream_t s)
{
    expect(odd != nullptr && odd != vt, "the backprojector's second copy");
    return launch_siddon_fp_lines(in, vt, v, n, nu, nv, g, out, accumulate, s);
}
} // namespace ykb

using namespace ykb;

namespace {

struct Scan {
    std::vector<ykb_cone_view> views;
    int nu, nv;
    ykb_volume volume{};
    Scan(int n_views, int nu_, int nv_, int nx, int ny, int nz) : views(n_views), nu(nu_), nv(nv_)
    {
        ykb_circular_flat spec{};
        spec.total_views = spec.views_per_turn = n_views;
        spec.rotation_direction = 1;
        spec.sid_mm = 500.f;
        spec.sdd_mm = 1000.f;
        spec.channels = nu;
        spec.rows = nv;
        spec.channel_size_mm = spec.row_size_mm = 0.1f;
        expect(ykb_build_circular_flat(&spec, views.data(), n_views) == YKB_OK, "views");
        volume.nx = nx; volume.ny = ny; volume.nz = nz;
        volume.vox_x = volume.vox_y = volume.vox_z = 100.f / std::max({nx, ny, nz});
    }
    ykb_joseph_plan* joseph(size_t capacity = ~size_t(0)) const
    {
        g_capacity = capacity;
        ykb_joseph_plan* p = nullptr;
        const ykb_status st = ykb_joseph_plan_create(views.data(), static_cast<int>(views.size()), nu, nv,
            &volume, 0, &p);
        expect((st == YKB_OK) == (p != nullptr), "a plan or an error");
        return p;
    }
};

// The line projector's copy where 32 unsigned bits of quads reach all of it, the
// slabs where they do not
void line_volume()
{
    for (int n : {64, 2048, 2500, 2700}) {
        const Scan scan(4, 32, 32, n, n, n);
        ykb_joseph_plan* p = scan.joseph();
        if (!p) continue;
        const bool fits = n <= 2500;
        expect((p->vt.ptr != nullptr) == fits && (p->fp_lines.rows > 0) == fits, "line copy or not");
        expect((p->slab_x.ptr != nullptr && p->slab_y.ptr != nullptr) == !fits, "slabs or not");
        if (fits) {
            // the first element of the copy's last row
            const long row = static_cast<long>(joseph_line_elems(scan.volume)) - joseph_line_pitch(n);
            expect(4 * static_cast<long>(joseph_line_quad(row)) == row, "quad of the last row");
        }
        ykb_joseph_plan_destroy(p);
    }
    const Scan tall(4, 32, 32, 8, 70000, 8);
    if (ykb_joseph_plan* p = tall.joseph()) {
        expect(p->fp_lines.rows == 0, "y past the launch's third dimension");
        ykb_joseph_plan_destroy(p);
    }
    expect(g_used == 0 && g_blocks.empty(), "everything given back");
}

// A plan is refused only when what it cannot do without has no room; the split
// views' sums and the table of ray heights give way first
void optional_buffers()
{
    const Scan scan(24, 40, 36, 64, 60, 48);
    ykb_joseph_plan* p = scan.joseph();
    if (!p) return;
    expect(p->heights.ptr && p->bp_splits > 1 && p->bp_parts && p->fp_lines.rows > 0, "all with room");
    const size_t full = g_used, heights = p->heights.bytes;
    const size_t sums = sizeof(double) * p->bp_splits * 64 * 60 * 48;
    ykb_joseph_plan_destroy(p);
    for (const size_t capacity : {full, full - 1, full - heights, full - heights - 1, full - heights - sums}) {
        p = scan.joseph(capacity);
        expect(p != nullptr, "a plan");
        if (!p) continue;
        expect(g_used <= capacity && p->weighted.ptr && p->vt.ptr, "what it needs");
        expect((p->heights.ptr != nullptr) == (capacity == full ||
                   (capacity < full - heights && heights <= sums && capacity >= full - sums)), "heights");
        expect((p->bp_splits > 1) == (capacity >= full - heights) &&
                   (p->bp_parts != nullptr) == (p->bp_splits > 1), "sums");
        expect(p->ray_heights().bytes == (p->heights.ptr ? 8 : 16), "heights read from");
        ykb_joseph_plan_destroy(p);
    }
    g_capacity = full - heights - sums - 1;
    p = nullptr;
    expect(ykb_joseph_plan_create(scan.views.data(), 24, scan.nu, scan.nv, &scan.volume, 0, &p) ==
               YKB_ERR_OUT_OF_MEMORY && !p, "refused below");
    expect(g_used == 0 && g_blocks.empty(), "everything given back");
}

// The projector holds one volume copy, the backprojector two; without room for
// them, and under capture, the rays are walked one by one
void siddon_copies()
{
    const Scan scan(24, 40, 36, 64, 60, 48);
    const size_t copy = sizeof(float) * joseph_line_elems(scan.volume);
    float in = 0.f, out = 0.f;
    // room for: nothing of it, the views, one copy, both
    for (int room = 0; room < 4; ++room) {
        ykb_joseph_plan* p = scan.joseph();
        if (!p) return;
        const size_t before = g_used, views = 24 * sizeof(ykb_cone_view);
        const size_t one = (views + 255) / 256 * 256 + copy;
        g_capacity = before + (room == 0 ? views - 1 : room == 1 ? one - 1 : room == 2 ? one + copy - 1 : one + copy);
        g_lines = g_walks = 0;
        ykb_status st = ykb_operator_apply(p, YKB_TASK_FP_SIDDON, &in, &out, 0, nullptr);
        expect((st == YKB_OK) == (room > 0), "views are needed");
        expect(g_lines == (room > 1) && g_walks == (room == 1), "the projector's kernel");
        expect(g_used - before == (room == 0 ? 0 : room == 1 ? views : one), "one copy for the projector");
        st = ykb_operator_apply(p, YKB_TASK_BP_SIDDON_RAY_DRIVEN, &in, &out, 0, nullptr);
        expect((st == YKB_OK) == (room > 0), "views are needed");
        expect(g_lines == (room > 1) + (room > 2) && g_walks == (room == 1 ? 2 : room == 2), "the backprojector's");
        expect(g_used - before == (room == 3 ? one + copy : room == 2 ? one : room == 1 ? views : 0), "both copies");
        if (room == 3) {
            g_capturing = true;
            ykb_operator_apply(p, YKB_TASK_FP_SIDDON, &in, &out, 0, nullptr);
            g_capturing = false;
            expect(g_walks == 1 && g_lines == 2, "captured calls walk");
        }
        ykb_joseph_plan_destroy(p);
        expect(g_used == 0, "everything given back");
    }
}

} // namespace

int main(int argc, char** argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "line_volume") line_volume();
    else if (what == "optional_buffers") optional_buffers();
    else if (what == "siddon_copies") siddon_copies();
    else return 2;
    return g_failures ? 1 : 0;
}
