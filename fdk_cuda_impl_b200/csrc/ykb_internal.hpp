// Internal declarations shared by the host and CUDA translation units of
// libykb.so.  Nothing here crosses the C-ABI.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <cstddef>
#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "ykb.h"

namespace ykb {

// --------------------------------------------------------------- errors ---
void set_error(const std::string& msg);
void clear_error();
const char* last_error();

// Returns YKB_ERR_CUDA (and records the message) when status is an error.
ykb_status cuda_status(cudaError_t status, const char* what);

#define YKB_TRY_CUDA(expr)                                                   \
    do {                                                                     \
        const cudaError_t ykb_e_ = (expr);                                   \
        if (ykb_e_ != cudaSuccess) return ::ykb::cuda_status(ykb_e_, #expr); \
    } while (0)

// Device buffer owned by a plan (RAII; no exceptions).
struct DeviceBuffer {
    void* ptr = nullptr;
    size_t bytes = 0;
    DeviceBuffer() = default;
    DeviceBuffer(const DeviceBuffer&) = delete;
    DeviceBuffer& operator=(const DeviceBuffer&) = delete;
    ~DeviceBuffer() { reset(); }
    cudaError_t alloc(size_t n)
    {
        reset();
        if (n == 0) return cudaSuccess;
        const cudaError_t e = cudaMalloc(&ptr, n);
        if (e == cudaSuccess) bytes = n; else ptr = nullptr;
        return e;
    }
    void reset()
    {
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        bytes = 0;
    }
    template <typename T> T* as() const { return static_cast<T*>(ptr); }
};

// Switches to a device for the lifetime of the object and restores the
// caller's device afterwards.
struct DeviceGuard {
    int previous = -1;
    explicit DeviceGuard(int device)
    {
        if (cudaGetDevice(&previous) != cudaSuccess) previous = -1;
        if (previous != device) cudaSetDevice(device);
    }
    ~DeviceGuard()
    {
        int now = -1;
        if (previous >= 0 && cudaGetDevice(&now) == cudaSuccess && now != previous)
            cudaSetDevice(previous);
    }
};

// ------------------------------------------------------------- geometry ---
struct dvec3 { double x, y, z; };

// Per-view FDK quantities derived in FP64 from the float geometry
// (definitions of src/Reconstruction/Analytic/Circular/Flat/FDK/
// YkFDKVecGeoDerived.hpp:58-304).
struct FdkDerived {
    double theta, dtheta, fscale;
    double sid;     // source_to_axis_mm
    double dsd;     // source_to_radial_detector_mm
    double plane;   // source_to_detector_plane_mm
    double off_u, off_v;
    double du, dv;
    dvec3 src, detS, detU, detV, normal, radial;
    double UU, VV, UV, inv_gram;
    int start_u;    // placement of the row inside the padded FFT row
};

bool derive_fdk_geometry(const ykb_cone_view* views, int n, int nu, int nv,
    float scan_range, std::vector<FdkDerived>& out, std::string& why);

int padded_fft_length(int nu);

// Device-side per-view FDK coefficients (FP64).  Affine rows over world
// coordinates (X, Y, Z, 1): u = cu.P/cd.P, v = cv.P/cd.P (pixel units,
// pixel (0,0) at detS), radial depth = cr.P; wbase = SID^2 dtheta 2pi/range.
struct alignas(16) FdkViewCoef {
    double cu[4];
    double cv[4];
    double cd[4];
    double cr[4];
    double wbase;
    double pad[3];
};

// Device-side per-view preweight + placement data.
struct alignas(16) FdkPreweightView {
    double src[4];
    double detS[4];
    double detU[4];
    double detV[4];
    double dsd;     // cosine-weight numerator
    double wgeom;   // DSD / DSO / 2
    int in_lo, in_hi;   // input samples [in_lo, in_hi) are placed in the padded row
    int out_lo, out_hi; // outputs [out_lo, out_hi) fall inside the padded row
};

bool build_parker_weights(const std::vector<FdkDerived>& g, const ykb_cone_view* views, int nu,
    int nv, double scan_range, double start_angle, int direction, std::vector<float>& w,
    std::string& why);
void build_fdk_coefficients(const std::vector<FdkDerived>& g, int nu,
    std::vector<FdkViewCoef>& coef, std::vector<FdkPreweightView>& pw,
    bool& axial);

void build_ramp_kernel(int nu, double du, const ykb_filter& f,
    std::vector<double>& h);

// Per-view data of the pseudo-matched backprojection (BP_FDK_PseudoMatched,
// src/FlatFpBp/BP/kernels/YkBpFdkKernel.cu:356-450).  A voxel P projecting to
// detector pixel coordinates (u, v) receives k L^3 / |P - S|^2 times the
// bilinear sample, where L^2 = |detS + u detU + v detV - S|^2 is expanded
// once per view as a quadratic in (u, v) and k = voxel volume /
// (du dv |SDD_plane|) (src/Reconstruction/Analytic/Circular/Flat/FDK/kernels/
// YkFDKBpPrecompute.cu:104-122).
// Since |P - S| = L den / SDD_plane for the detector point of P (den =
// (P - S).n, n the unit detector normal), the weight equals
// kq |P - S| / den^3 with kq = voxel volume SDD_plane^2 / (du dv); the TMA
// kernel uses that form, in which only |P - S| varies along an axial z-column.
struct alignas(16) PseudoViewCoef {
    double src[4];
    float l2[6];  // l2[0] + u l2[1] + v l2[2] + u^2 l2[3] + u v l2[4] + v^2 l2[5]
    float k;
    float kq;
};

void build_pseudo_coefficients(const std::vector<FdkDerived>& g, const ykb_volume& vol,
    std::vector<PseudoViewCoef>& out);

// Joseph per-view data (FP64), volume-centred voxel units.
struct alignas(16) JosephView {
    double src[4];
    double detS[4];
    double detU[4];
    double detV[4];
    int axis;        // 0: X main axis, 1: Y, 2: Z
    int n0, n1, n2;  // volume extents along (main, minor1, minor2)
    double v0, v1, v2;  // voxel sizes (mm) along the same axes
    double pad;
};

bool build_joseph_views(const ykb_cone_view* views, int n, int nu, int nv,
    const ykb_volume& vol, std::vector<JosephView>& out, std::string& why);

bool build_circular_flat(const ykb_circular_flat& spec, ykb_cone_view* out,
    std::string& why);

// -------------------------------------------------------------- kernels ---
struct VolumeGrid {
    int nx, ny, nz;
    double vx, vy, vz;
    double ox, oy, oz;  // centre of voxel (0,0,0), FP64
};

VolumeGrid make_grid(const ykb_volume& v);

// FDK
// Layouts of filtered rows: plain floats [view][nv][ld], or row pairs
// [view][nv + 1][ld] float2 where element (n + 1, u) = (f[n][u],
// f[n + 1][u] - f[n][u]) for n = -1 .. nv - 1, f zero outside the detector.
// The TMA backprojection reads a voxel's four taps with two adjacent 8-byte
// loads and lerps each column with one FMA.
enum FilteredLayout : int { kFilteredScalar = 0, kFilteredPairs = 1 };
// parker: per-(view, column) weights [n_views][nu] multiplied in after the
// cosine weight (short scans), or nullptr
cudaError_t launch_fdk_preweight(const void* proj, int proj_dtype,
    const FdkPreweightView* pw, const float* parker, int n_views, int nu, int nv, float* out,
    cudaStream_t s);
cudaError_t launch_fdk_ramp_fp32(const float* pw_rows, const float* h_dev,
    const FdkPreweightView* pwv, int n_views, int nu, int nv, float* out,
    int ldc, cudaStream_t s);
// BF16 split parts of the preweighted rows: parts[0], parts[1] and, when
// parts[2] is not null, a third part (FP32-equivalent split)
cudaError_t launch_fdk_preweight_split_bf16(const void* proj, int proj_dtype,
    const FdkPreweightView* pw, const float* parker, int n_views, int nu, int nv, int ld,
    __nv_bfloat16* const parts[3], cudaStream_t s);
// tcgen05 Toeplitz filter over split operands: two parts each (3 products,
// BF16 plans) or three (6 products, FP32 accuracy) when a_parts[2] and
// t_parts[2] are given.  With three parts the three products at the 2^-16
// level run only over the K chunks (64 columns each) within `near_chunks`
// chunks of each output tile; tc_filter_near_chunks(h, nu) picks the
// fewest chunks for which the filter taps left out carry at most 2^-8 of
// the taps' absolute sum.
cudaError_t launch_fdk_ramp_tcgen05(const __nv_bfloat16* const a_parts[3],
    const __nv_bfloat16* const t_parts[3], int rows, int nu, int ld,
    const FdkPreweightView* pwv, int nv, float* out, int layout, int ldc, int tn, int near_chunks,
    int* err_flag, cudaStream_t s);
int tc_filter_near_chunks(const std::vector<double>& h, int nu);
bool tcgen05_filter_supported(int nu);
// Tile width tn (columns) for calls of `rows` rows.  The 2^-16 products reach whole
// tiles, so a row's last bits depend on it: a plan keeps one width for all of its
// calls, however the views are batched
int tc_filter_tile(int nu, long rows);
// view sub-batches (1 to 4) in which the preweight of one runs under the filter
// of the one before
int tc_filter_sub_batches(int tn, int nu, long rows);
int tc_filter_lda(int nu);
cudaError_t launch_fdk_backproject(const void* filtered, int dtype,
    const FdkViewCoef* coef, int n_views, int nu, int nv, int ld,
    const VolumeGrid& grid, bool axial, float* vol, int accumulate,
    cudaStream_t s);
// TMA-staged backprojection (fdk_bp_tma.cu)
bool fdk_tma_available();
// staged projection box as row pairs and as plain rows (width 0: not staged)
struct FdkTmaBox { int pair_w = 0, pair_h = 0, row_w = 0, row_h = 0; };
// z slices per tile of the TMA backprojection (slab work starts on a tile)
int fdk_tma_z_tile();
cudaError_t fdk_tma_box(const FdkViewCoef* coef, int n_views, const VolumeGrid& g,
    int* scratch3, FdkTmaBox* box, cudaStream_t s);
// floats of workspace for the sums of split views (0: the volume has tiles
// enough to fill the GPU)
size_t fdk_tma_part_floats(const VolumeGrid& g, int n_views);
// Limit of the TMA backprojection's pipeline waits (a wait that runs out
// sets the error word and stops the CTA) and, for tests of that path, a view
// whose copy is withheld (-1: none).  Waits that drain copies in
// flight keep the default limit.
struct PipelineWait {
    unsigned long long limit_ns = 2000000000ull;
    int withheld_view = -1;
};
// parts: workspace of part_floats floats for the sums of split views, or
// nullptr.  pseudo != nullptr: the pseudo-matched weight of PseudoViewCoef
// replaces the FDK depth weight (row pairs only)
cudaError_t launch_fdk_backproject_tma(const float* filtered, int layout, int ld,
    const FdkViewCoef* coef, int n_views, int nu, int nv, const VolumeGrid& g, bool axial,
    const FdkTmaBox& box, float* vol, int accumulate, int* err, float* parts, size_t part_floats,
    cudaStream_t s, const PseudoViewCoef* pseudo = nullptr, PipelineWait pw = PipelineWait{});
// Pseudo-matched backprojection straight from projections [n][nv][nu] with
// bounds-checked loads (used when the TMA box does not fit)
cudaError_t launch_pseudo_backproject(const float* proj, const FdkViewCoef* coef,
    const PseudoViewCoef* pseudo, int n_views, int nu, int nv, const VolumeGrid& grid,
    float* vol, int accumulate, cudaStream_t s);
// plain rows [views][nv][ld_in] -> row pairs [views][nv + 1][ldp]
cudaError_t launch_fdk_pairify(const float* in, int ld_in, long views, int nu, int nv, float* out,
    int ldp, cudaStream_t s);

// Joseph
// zero voxels bordering each slice of the transposed slabs on both minor axes
constexpr int kSlabPad = 2;
// slab of main axis x ([x][z][y]) or y ([y][z][x]) with its zero border
inline size_t joseph_slab_elems(const ykb_volume& v, int axis)
{
    const size_t n0 = static_cast<size_t>(axis == 0 ? v.nx : v.ny);
    const size_t n1 = static_cast<size_t>(axis == 0 ? v.ny : v.nx) + 2 * kSlabPad;
    return n0 * (static_cast<size_t>(v.nz) + 2 * kSlabPad) * n1;
}
cudaError_t launch_joseph_transpose(const float* vol, int nx, int ny, int nz,
    float* vol_yzx, float* vol_xzy, cudaStream_t s);
cudaError_t launch_joseph_fp(const float* slabs[3], const JosephView* views,
    const int* view_axis_host, int n_views, int nu, int nv, float* proj,
    int accumulate, cudaStream_t s);
// Axial-column scans: how far the rays of a view reach over the volume's slices
// and `margin` voxels around them.  ratio: a voxel's distance from the source
// over the detector's, along the detector normal.
struct JosephColumnReach {
    double near = 0.0, far = 0.0;  // extremes of the ratio
    double slope = 0.0;            // its change per voxel
    double pitch = 0.0;            // largest distance along z (voxels) of adjacent rows' rays
    double tall = 0.0;             // largest height of a detector row over the source (voxels)
};
JosephColumnReach joseph_column_reach(const JosephView& j, int nv, double margin);
// Whether adjacent rows' rays are less than a voxel apart along z everywhere in
// the volume (and far enough for FP32 to keep them in order)
bool joseph_bp_runs(const std::vector<JosephView>& views, int nv);
// (a2, e2) of the rays, `bytes` from one ray to the next: a table of their own,
// or without room for it the last two floats of the ray records
struct JosephHeights {
    const char* first;
    int bytes;
};
cudaError_t launch_joseph_ray_heights(const float4* rays, long n, float2* out, cudaStream_t s);
// Forward projection of axial-column scans by detector-column lines
// (joseph_fp_lines.cu): detector rows of a CTA (0: the lines do not fit, the
// slab kernel projects) and window of its lines
struct JosephFpLines { int rows = 0, window = 0; };
JosephFpLines joseph_fp_lines_shape(const std::vector<JosephView>& views, int nv);
// z pitch (floats) of the volume copy [x][y][z] that the lines are formed from,
// zero rows around x and y, and its size
constexpr int kLinePad = 2;
inline int joseph_line_pitch(int nz) { return (nz + 3) / 4 * 4; }
inline size_t joseph_line_elems(const ykb_volume& v)
{
    return static_cast<size_t>(v.nx + 2 * kLinePad) * (v.ny + 2 * kLinePad) * joseph_line_pitch(v.nz);
}
// The lines' tables name a row of the copy by its first quad, in 32 unsigned bits
constexpr uint32_t joseph_line_quad(long row) { return static_cast<uint32_t>(row / 4); }
// Volumes whose copy they reach, and whose y fits the third dimension of the copy's
// launch; the slab kernel projects the others
inline bool joseph_line_volume_fits(const ykb_volume& v)
{
    return v.ny <= 65535 && joseph_line_elems(v) <= (size_t(1) << 34);
}
cudaError_t launch_joseph_line_volume(const float* vol, int nx, int ny, int nz, float* vt, cudaStream_t s);
// vt: joseph_line_elems floats, zeroed once; every call rewrites its interior
cudaError_t launch_joseph_fp_lines(const float* vol, int nx, int ny, int nz, float* vt,
    const JosephView* views, const float2* cols, JosephHeights heights, const float* lens, int n_views,
    int nu, int nv, JosephFpLines shape, float* proj, int accumulate, cudaStream_t s);
cudaError_t launch_joseph_ray_table(const JosephView* views, int n_views,
    int nu, int nv, float4* rays, float* lens, cudaStream_t s);
// Iterative-solver vectors (iter_kernels.cu)
int dot_partial_count();
cudaError_t launch_dot_f64(const float* a, const float* b, size_t n, double* partials,
    double* result, cudaStream_t s);
cudaError_t launch_cgls_xr(const double* gamma, const double* ww, float* x, const float* p,
    size_t nx, float* r, const float* w, size_t nr, cudaStream_t s);
cudaError_t launch_cgls_p(const double* gamma_new, const double* gamma_old, float* p,
    const float* z, size_t n, cudaStream_t s);

// Siddon (siddon_kernels.cu); views in world coordinates
cudaError_t launch_siddon_fp(const float* vol, const ykb_cone_view* views, int n_views, int nu,
    int nv, const VolumeGrid& g, float* proj, int accumulate, cudaStream_t s);
cudaError_t launch_siddon_bp(const float* proj, const ykb_cone_view* views, int n_views, int nu,
    int nv, const VolumeGrid& g, float* vol, int accumulate, cudaStream_t s);
// The same pair for axial-column scans by detector columns, over the volume copy
// of joseph_line_elems floats (see launch_joseph_line_volume); the backprojector
// sums even and odd views in a copy each (vt, odd): half the additions to a voxel,
// to sums half as large, so half their rounding
bool siddon_lines_apply(const ykb_cone_view* views, int n_views, int nv, const VolumeGrid& g);
cudaError_t launch_siddon_fp_lines(const float* vol, float* vt, const ykb_cone_view* views, int n_views,
    int nu, int nv, const VolumeGrid& g, float* proj, int accumulate, cudaStream_t s);
cudaError_t launch_siddon_bp_lines(const float* proj, float* vt, float* odd, const ykb_cone_view* views,
    int n_views, int nu, int nv, const VolumeGrid& g, float* vol, int accumulate, cudaStream_t s);
// (a1, e1) of every detector column from its first row into cols[n][nu];
// flag[0] = 1 when any ray of a column differs (the line backprojector
// then does not apply)
cudaError_t launch_joseph_column_table(const float4* rays, int n_views, int nu, int nv,
    float2* cols, int* flag, cudaStream_t s);
// splits of the views of the line backprojector; with more than one its CTAs
// write FP64 sums to parts[splits][voxels]
int joseph_bp_splits(const ykb_volume& v, int n_views);
// matched backprojection for axial-column scans (see launch_joseph_column_table):
// weighted receives input x chord length per ray; runs: adjacent rows' rays are
// less than a voxel apart along z (joseph_bp_runs)
cudaError_t launch_joseph_bp_lines(const float* proj, const float4* rays, JosephHeights heights,
    const float* lens, const float2* cols, const float* view_proj, const JosephView* views, int n_views,
    int nu, int nv, const ykb_volume& vol, bool runs, float* weighted, int splits, double* parts,
    float* out, int accumulate, cudaStream_t s);
cudaError_t launch_joseph_bp(const float* proj, const float4* rays, const float* lens,
    const float* view_proj, const JosephView* views, int n_views, int nu, int nv,
    const ykb_volume& vol, float* weighted, float* out, int accumulate, cudaStream_t s);

} // namespace ykb

// Plan objects (opaque at the C-ABI).
struct ykb_fdk_plan {
    int device = 0;
    int n_views = 0, nu = 0, nv = 0;
    float scan_range = 0.f;
    ykb_volume volume{};
    ykb_filter filter{};
    int precision = YKB_PRECISION_FP32;
    bool axial = false;
    bool tc_filter = false;
    int tc_parts = 0;            // BF16 parts per operand of the tensor-core filter (2 or 3)
    int tc_tile = 0;             // its tile width
    int tc_near = 0;             // K chunks each side of a tile that its 2^-16 products cover
    int batch_capacity = 0;      // views the workspace holds
    int ld = 0;                  // row pitch (elements) of the filtered workspace
    int layout = 0;              // FilteredLayout of the filtered workspace
    int lda = 0;                 // row pitch of the bf16 GEMM operands (tensor-core filter)
    bool use_tma = false;        // TMA-staged backprojection
    ykb::FdkTmaBox tma_box;      // its projection box
    ykb::PipelineWait bp_wait;   // its pipeline-wait limit (tests shorten it)
    std::vector<ykb::FdkDerived> derived;
    ykb::DeviceBuffer coef;      // FdkViewCoef[n_views]
    ykb::DeviceBuffer pwv;       // FdkPreweightView[n_views]
    ykb::DeviceBuffer ramp;      // float[2*nu-1]
    ykb::DeviceBuffer parker;    // float[n_views][nu] short-scan weights, or empty
    ykb::DeviceBuffer toeplitz_hi, toeplitz_lo, toeplitz_lo2;  // bf16 [nu][lda] split parts
    ykb::DeviceBuffer work_a;    // preweighted rows: float, or the bf16 split parts in turn
    // filtered projections (layout, pitch ld), filtered_floats of them, then
    // part_floats for the sums of split views
    ykb::DeviceBuffer work_filtered;
    size_t filtered_floats = 0, part_floats = 0;
    ykb::DeviceBuffer err_flag;  // int[8]: device error word, box pre-pass scratch
    // stage timing (ykb_fdk_stage_timing): a start and a stop event around
    // each filter (stage 0) and backprojection (stage 1) launch group, on the
    // stream that launches it; events are pooled and reused
    struct StageEvents { cudaEvent_t start = nullptr, stop = nullptr; int stage = 0; };
    bool timing = false;
    std::vector<StageEvents> stage_events;
    size_t stage_events_used = 0;
    // tensor-core filter: the preweight of the next sub-batch of views runs on
    // this stream while the ramp filter of the current one runs on the
    // caller's (created on first use)
    static constexpr int kFilterSubBatches = 4;
    cudaStream_t aux_stream = nullptr;
    cudaEvent_t aux_in = nullptr;                       // the caller's stream reached the filter
    cudaEvent_t aux_done[kFilterSubBatches] = {};       // sub-batch preweighted
    // host-input streaming (ykb_fdk_execute_host), created on first use
    ykb::DeviceBuffer stage_in;  // two batches of input views
    int stage_views = 0;         // views per batch slot
    cudaStream_t copy_stream = nullptr;
    cudaEvent_t copied[2] = {nullptr, nullptr};    // batch slot filled
    cudaEvent_t consumed[2] = {nullptr, nullptr};  // batch slot read by the filter
    ~ykb_fdk_plan()
    {
        for (auto& e : stage_events) {
            if (e.start) cudaEventDestroy(e.start);
            if (e.stop) cudaEventDestroy(e.stop);
        }
        for (cudaEvent_t e : aux_done) if (e) cudaEventDestroy(e);
        if (aux_in) cudaEventDestroy(aux_in);
        if (aux_stream) cudaStreamDestroy(aux_stream);
        for (cudaEvent_t e : copied) if (e) cudaEventDestroy(e);
        for (cudaEvent_t e : consumed) if (e) cudaEventDestroy(e);
        if (copy_stream) cudaStreamDestroy(copy_stream);
    }
};

struct ykb_joseph_plan {
    int device = 0;
    int n_views = 0, nu = 0, nv = 0;
    ykb_volume volume{};
    std::vector<ykb::JosephView> host_views;
    std::vector<ykb_cone_view> cone_views;
    std::vector<int> axes;
    ykb::DeviceBuffer views;     // JosephView[n]
    ykb::DeviceBuffer view_proj; // float[n][12]: voxel-space 3x4 projection
    ykb::DeviceBuffer rays;      // float4[n*nv*nu]: (a1, e1, a2, e2)
    ykb::DeviceBuffer lens;      // float[n*nv*nu]: chord length per step
    // backprojector input x chord length: float[n*nv*nu]
    ykb::DeviceBuffer weighted;
    int bp_splits = 1;           // of the line backprojector's views
    double* bp_parts = nullptr;  // their sums (behind the weighted rays)
    bool bp_runs = false;        // the line backprojector's lines form in runs
    bool column_bp = false;      // every view's detector columns are axial (line backprojector)
    ykb::DeviceBuffer cols;      // float2[n*nu]: (a1, e1) per detector column
    ykb::DeviceBuffer heights;   // float2[n*nv*nu]: (a2, e2), or empty (read from rays)
    ykb::JosephHeights ray_heights() const
    {
        return heights.ptr ? ykb::JosephHeights{heights.as<char>(), 8}
                           : ykb::JosephHeights{rays.as<char>() + 8, 16};
    }
    ykb::DeviceBuffer slab_y, slab_x;  // transposed volume copies (scans without fp_lines)
    ykb::JosephFpLines fp_lines;       // forward projection by lines (column_bp scans)
    ykb::DeviceBuffer vt;              // its volume copy [x][y][z]
    // Siddon, set up on first use: the views, and for untilted scans a volume copy
    // behind them; the first backprojection adds the copy that sums the odd views.
    // Calls on different streams take turns on the copies
    ykb::DeviceBuffer world_views;     // ykb_cone_view[n], then the copy
    float* siddon_vt = nullptr;        // (null: the rays are walked one by one)
    ykb::DeviceBuffer siddon_odd;      // (empty: the backprojector walks them so)
    cudaEvent_t siddon_done = nullptr; // the last call's work on the copy
    std::mutex siddon_mutex;
    ~ykb_joseph_plan() { if (siddon_done) cudaEventDestroy(siddon_done); }
    // pseudo-matched backprojection, set up on first use
    bool pseudo_ready = false;
    bool pseudo_axial = false;         // untilted detector: the axial column walk
    ykb::FdkTmaBox pseudo_box;         // TMA projection box (width 0: bounds-checked loads)
    int pseudo_ld = 0;                 // row pitch of the row pairs
    ykb::DeviceBuffer fdk_coef;        // FdkViewCoef[n]
    ykb::DeviceBuffer pseudo_coef;     // PseudoViewCoef[n]
    ykb::DeviceBuffer pairs;           // projections as row pairs [n][nv + 1][pseudo_ld], then
    float* pseudo_parts = nullptr;     // the sums of split views
    size_t pseudo_part_floats = 0;
    ykb::DeviceBuffer err_flag;        // int[8]: device error word, box pre-pass scratch
};

struct ykb_iter {
    int device = 0;
    ykb::DeviceBuffer partials;  // double[dot_partial_count()]
};
