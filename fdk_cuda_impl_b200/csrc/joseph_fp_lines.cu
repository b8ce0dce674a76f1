// Joseph forward projector of axial-column scans by detector-column lines
// (sm_100a).
//
// All rays of a detector column share their minor-1 samples (a1, e1), so on a
// slice the column's rays sample one line along z, the lerp of two volume rows:
//   L(s, z) = (1 - w1) x[s][i1][z] + w1 x[s][i1 + 1][z],
//   sample  = lerp of L(s, .) at f2.
// A CTA owns kCols detector columns and 32 to 384 rows of one view, a thread a
// row with its kCols rays.  Per batch of kSlices slices the CTA forms the lines
// over the z window of its rays in shared memory (16-byte loads of volume rows
// that lie z-contiguous, each line entry formed once for the 1.5 rays that
// sample it), then every thread takes its kCols x kSlices samples: one shared
// address and two 4-byte loads each, where joseph_fp_padded_kernel gathers four
// taps from global memory and lerps them anew for every ray.  The window
// comes from the CTA's corner rays (positions are monotonic along a column and
// linear over slices), so a sample needs no bounds check: line entries outside
// the volume are zero.  Two buffers, one barrier a batch.
// Samples, weights and their order are those of joseph_fp_padded_kernel, summed
// in FP64.
// Bound: the L1 data path (73 % of its wavefronts: line loads and stores, 8 bytes
// of taps a sample) and instruction issue (62 %, 16 a sample).  256^3 x 360 x
// 384^2: 9.7 ms (128 rows, windows of 144 floats, 20 warps an SM), before 14.3
// (27 instructions a sample and four gathers of 4.65 sectors); whole (slice, quad)
// tasks, whose second round is nearly empty: 11.3; 192 rows and windows of 320,
// which leave 12 warps an SM: 20.7.
#include "ykb_internal.hpp"

#include <algorithm>
#include <cmath>
#include <iterator>

namespace ykb {
namespace {

constexpr int kCols = 8;     // detector columns of a CTA
constexpr int kSlices = 4;   // slices of a batch
constexpr int kMaxRows = 384;
constexpr int kTables = 3;   // (row, weight) tables: one read, one ahead, one being written
static_assert(kCols * kSlices == 32, "a warp's lanes form a batch's table");

constexpr float kFloorMagic = 12582912.0f;  // 1.5 * 2^23: v + it rounded down holds floor(v)
constexpr uint32_t kFloorMagicBits = 0x4B400000u;

// Packed FP32 pairs (sm_100 f32x2 arithmetic): two columns' rays.
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2pack(float lo, float hi)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2unpack(f2 v, float& lo, float& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 f2fma(f2 a, f2 b, f2 c)
{
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2 f2add_rm(f2 a, f2 b)
{
    f2 d;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 f2sub(f2 a, f2 b)
{
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

template <int OFF>
__device__ __forceinline__ float lds(uint32_t addr)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(addr), "n"(OFF));
    return v;
}

// the samples of columns C .. kCols - 1 of slice J (two columns at a time)
template <int W, int J, int C>
__device__ __forceinline__ void sample_columns(const f2 (&a2)[kCols / 2], const f2 (&e2)[kCols / 2],
    f2 c0, uint32_t base, double (&acc)[kCols])
{
    if constexpr (C < kCols) {
        const f2 M = f2pack(kFloorMagic, kFloorMagic);
        const f2 f = f2fma(a2[C / 2], c0, e2[C / 2]);
        const f2 t = f2add_rm(f, M);
        const f2 w = f2sub(f, f2sub(t, M));
        float ta, tb;
        f2unpack(t, ta, tb);
        const uint32_t at = __float_as_uint(ta) * 4u + base, bt = __float_as_uint(tb) * 4u + base;
        constexpr int off = (J * kCols + C) * W * 4;
        const f2 p0 = f2pack(lds<off>(at), lds<off + W * 4>(bt));
        const f2 p1 = f2pack(lds<off + 4>(at), lds<off + W * 4 + 4>(bt));
        float ra, rb;
        f2unpack(f2fma(w, f2sub(p1, p0), p0), ra, rb);
        acc[C] += static_cast<double>(ra);
        acc[C + 1] += static_cast<double>(rb);
        sample_columns<W, J, C + 2>(a2, e2, c0, base, acc);
    }
}
template <int W, int J>
__device__ __forceinline__ void sample_slices(const f2 (&a2)[kCols / 2], const f2 (&e2)[kCols / 2],
    float c0, uint32_t base, double (&acc)[kCols])
{
    if constexpr (J < kSlices) {
        const float c = c0 + static_cast<float>(J);
        sample_columns<W, J, 0>(a2, e2, f2pack(c, c), base, acc);
        sample_slices<W, J + 1>(a2, e2, c0, base, acc);
    }
}

// the same samples taken from the volume
__device__ __noinline__ float line_entry(const float* __restrict__ vt, long st_1, int nz, int2 t, int z)
{
    if (z < 0 || z >= nz) return 0.f;
    const float* p = vt + 4 * static_cast<long>(static_cast<uint32_t>(t.x)) + z;
    return fmaf(__int_as_float(t.y), p[st_1] - p[0], p[0]);
}
__device__ __forceinline__ void sample_volume(const float* __restrict__ vt, long st_1, int nz,
    const int2* table, const f2 (&a2)[kCols / 2], const f2 (&e2)[kCols / 2], float c0,
    double (&acc)[kCols])
{
#pragma unroll 1
    for (int js = 0; js < kSlices; ++js) {
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
            float a[2], e[2];
            f2unpack(a2[c / 2], a[0], a[1]);
            f2unpack(e2[c / 2], e[0], e[1]);
            const float f = fminf(fmaxf(fmaf(a[c & 1], c0 + js, e[c & 1]), -4.f), nz + 4.f), fl = floorf(f);
            const int2 t = table[js * kCols + c];
            const float p0 = line_entry(vt, st_1, nz, t, static_cast<int>(fl));
            const float p1 = line_entry(vt, st_1, nz, t, static_cast<int>(fl) + 1);
            acc[c] += static_cast<double>(fmaf(f - fl, p1 - p0, p0));
        }
    }
}

// slices with f1 = a1 (s - (n0 - 1) / 2) + e1 in [-3/2, n1 + 1/2]: every
// slice with a non-zero weight (FP64 from the floats the kernel evaluates)
__device__ __forceinline__ void slice_span(float a, float e, int n1, int n0, int& lo, int& hi)
{
    const double L = -1.5, U = n1 + 0.5, h = 0.5 * (n0 - 1), ad = a, ed = e;
    lo = 0; hi = n0 - 1;
    if (fabs(ad) < 1e-300) {
        if (!(ed >= L && ed <= U)) { lo = 1; hi = 0; }
        return;
    }
    double t0 = (L - ed) / ad + h, t1 = (U - ed) / ad + h;
    if (t0 > t1) { const double t = t0; t0 = t1; t1 = t; }
    lo = max(lo, static_cast<int>(ceil(fmin(fmax(t0, -1e9), 1e9))));
    hi = min(hi, static_cast<int>(floor(fmin(fmax(t1, -1e9), 1e9))));
}

// W: floats of a line's window (a multiple of 4)
template <int W>
__global__ void __launch_bounds__(kMaxRows, 2) joseph_fp_lines_kernel(const float* __restrict__ vt,
    const JosephView* __restrict__ views, const float2* __restrict__ cols,
    const char* __restrict__ heights, int ray_bytes, const float* __restrict__ lens, int view0, int nu, int nv,
    int nz, int nzp, float* __restrict__ proj, int accumulate)
{
    extern __shared__ __align__(16) float smem[];
    float* const lines = smem;                                             // [2][slice][column][W]
    int2* const tables = reinterpret_cast<int2*>(smem + 2 * 32 * W);       // [kTables][slice][column]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int k = view0 + blockIdx.z;
    const int iu0 = blockIdx.x * kCols, row0 = blockIdx.y * blockDim.x;
    const int iv = row0 + tid;
    const JosephView& j = views[k];
    const int n0 = j.n0, n1 = j.n1;
    // the volume is [x][y][z], z rows of nzp floats, kLinePad zero rows around x
    // and y
    const long row_x = static_cast<long>((j.axis == 0 ? n1 : n0) + 2 * kLinePad) * nzp;
    const long st_s = j.axis == 0 ? row_x : nzp, st_1 = j.axis == 0 ? nzp : row_x;
    const float half = 0.5f * (n0 - 1);
    const long ray_row = static_cast<long>(k) * nv;

    // rows and columns past the detector repeat the last one (never stored)
    f2 a2[kCols / 2], e2[kCols / 2];
    {
        const char* r = heights + (ray_row + min(iv, nv - 1)) * nu * ray_bytes;
#pragma unroll
        for (int c = 0; c < kCols; c += 2) {
            const float2 q = __ldg(reinterpret_cast<const float2*>(r + min(iu0 + c, nu - 1) * ray_bytes));
            const float2 p = __ldg(reinterpret_cast<const float2*>(r + min(iu0 + c + 1, nu - 1) * ray_bytes));
            a2[c / 2] = f2pack(q.x, p.x);
            e2[c / 2] = f2pack(q.y, p.y);
        }
    }
    // each lane: one column of the table, and a corner ray of the window
    const int lc = lane & (kCols - 1);
    const float2 col = __ldg(cols + static_cast<long>(k) * nu + min(iu0 + lc, nu - 1));
    float ca, ce;
    {
        const int edge = (lane & 8) ? min(row0 + static_cast<int>(blockDim.x) - 1, nv - 1) : row0;
        const float2 q = __ldg(reinterpret_cast<const float2*>(heights +
            ((ray_row + edge) * nu + min(iu0 + lc, nu - 1)) * ray_bytes));
        ca = q.x;
        ce = q.y;
    }
    const float corner_slice = (lane & 16) ? static_cast<float>(kSlices - 1) : 0.f;
    int slo, shi;
    slice_span(col.x, col.y, n1, n0, slo, shi);
    const int first = __reduce_min_sync(0xffffffffu, slo <= shi ? slo : 0x7fffffff);
    const int last = __reduce_max_sync(0xffffffffu, slo <= shi ? shi : -1);

    // table of batch b: per (slice, column) the place of volume row i1 (in
    // quads) and its weight w1; rows outside the volume, and slices past the
    // columns', are the zero rows around it
    auto form_table = [&](int b) {
        const int s = first + b * kSlices + (lane >> 3);
        const float f1 = fmaf(col.x, static_cast<float>(s) - half, col.y);
        const float fl = floorf(fminf(fmaxf(f1, static_cast<float>(-kLinePad)), static_cast<float>(n1)));
        const bool in = s <= last && f1 > -1.f && f1 < static_cast<float>(n1);
        const long row = (s + kLinePad) * st_s + (static_cast<int>(fl) + kLinePad) * st_1;
        tables[(b % kTables) * 32 + lane] =
            in ? make_int2(static_cast<int>(joseph_line_quad(row)), __float_as_int(f1 - fl)) : make_int2(0, 0);
    };
    if (warp == 0) {
        form_table(0);
        form_table(1);
    }
    double acc[kCols];
#pragma unroll
    for (int c = 0; c < kCols; ++c) acc[c] = 0.0;
    __syncthreads();

    const uint32_t lines_addr = static_cast<uint32_t>(__cvta_generic_to_shared(lines));
    for (int b = 0, s0 = first; s0 <= last; ++b, s0 += kSlices) {
        const float c0 = static_cast<float>(s0) - half;
        // the window: taps floor(f2) and + 1 of every ray of the CTA
        const float fc = fminf(fmaxf(fmaf(ca, c0 + corner_slice, ce), -1e6f), 1e6f);
        const int fz = static_cast<int>(floorf(fc));
        const int zlo = __reduce_min_sync(0xffffffffu, fz) - 1;
        const int zhi = __reduce_max_sync(0xffffffffu, fz) + 2;
        const int zb = zlo & ~3;  // 16-byte loads of the volume rows
        bool some = zhi >= 0 && zlo < nz;
        if (some && zhi - zb >= W) {
            // wider than the host's bound (no scan is known; a test narrows the
            // window): straight from the volume, so that no shared access leaves
            // its line
            some = false;
            sample_volume(vt, st_1, nz, tables + (b % kTables) * 32, a2, e2, c0, acc);
        }
        float* const buffer = lines + (b & 1) * 32 * W;
        if (some) {
            // a thread takes a quad of two columns' lines at a time: the lines are
            // about as long as the CTA has rows, so whole (slice, quad) tasks would
            // leave a second, nearly empty round
            const uint32_t quads = static_cast<uint32_t>(min((zhi - zb) / 4 + 1, W / 4));
            const uint32_t per_quads = ((1u << 20) + quads - 1) / quads;  // exact for q < 2^20 / quads
            const int2* const table = tables + (b % kTables) * 32;
#pragma unroll 2
            for (uint32_t q = tid; q < kSlices * kCols / 2 * quads; q += blockDim.x) {
                const uint32_t line = q * per_quads >> 20;  // slice x column pair
                const int zq = 4 * static_cast<int>(q - line * quads), z = zb + zq;
                float* const out = buffer + 2 * line * W + zq;
                const int4 t = *reinterpret_cast<const int4*>(table + 2 * line);
                float4 p0 = make_float4(0.f, 0.f, 0.f, 0.f), r0 = p0, p1 = p0, r1 = p0;
                if (z >= 0 && z < nz) {  // else above or below the volume (its rows are padded to quads)
                    const float4* const src = reinterpret_cast<const float4*>(vt + z);
                    const float4* const src1 = reinterpret_cast<const float4*>(vt + z + st_1);
                    p0 = __ldg(src + static_cast<uint32_t>(t.x));
                    r0 = __ldg(src1 + static_cast<uint32_t>(t.x));
                    p1 = __ldg(src + static_cast<uint32_t>(t.z));
                    r1 = __ldg(src1 + static_cast<uint32_t>(t.z));
                }
                const float w0 = __int_as_float(t.y), w1 = __int_as_float(t.w);
                *reinterpret_cast<float4*>(out) = make_float4(fmaf(w0, r0.x - p0.x, p0.x),
                    fmaf(w0, r0.y - p0.y, p0.y), fmaf(w0, r0.z - p0.z, p0.z), fmaf(w0, r0.w - p0.w, p0.w));
                *reinterpret_cast<float4*>(out + W) = make_float4(fmaf(w1, r1.x - p1.x, p1.x),
                    fmaf(w1, r1.y - p1.y, p1.y), fmaf(w1, r1.z - p1.z, p1.z), fmaf(w1, r1.w - p1.w, p1.w));
            }
        }
        __syncthreads();
        // (the table being written was last read two batches ago, before the
        // barrier of the previous one)
        if (warp == (b + 1) % (blockDim.x >> 5)) form_table(b + 2);
        if (some) {
            const uint32_t base = lines_addr + static_cast<uint32_t>((b & 1) * 32 * W * 4) -
                4u * (kFloorMagicBits + static_cast<uint32_t>(zb));
            sample_slices<W, 0>(a2, e2, c0, base, acc);
        }
    }
    if (iv >= nv) return;
    const long at = (ray_row + iv) * nu + iu0;
#pragma unroll
    for (int c = 0; c < kCols; ++c) {
        if (iu0 + c >= nu) break;
        const double v = acc[c] * __ldg(lens + at + c);
        proj[at + c] = static_cast<float>(accumulate ? proj[at + c] + v : v);
    }
}

// vol[z][y][x] -> vt[x][y][z], z rows padded with zeros to nzp (the zero rows
// around x and y are written once, when the plan is built)
__global__ void __launch_bounds__(256) transpose_xyz_kernel(const float* __restrict__ in, int nx,
    int ny, int nz, int nzp, float* __restrict__ out)
{
    __shared__ float tile[32][33];
    const int y = blockIdx.z, x0 = blockIdx.x * 32, z0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int z = z0 + r, x = x0 + threadIdx.x;
        tile[r][threadIdx.x] = (x < nx && z < nz) ? in[(static_cast<long>(z) * ny + y) * nx + x] : 0.f;
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int x = x0 + r, z = z0 + threadIdx.x;
        if (x < nx && z < nzp)
            out[(static_cast<long>(x + kLinePad) * (ny + 2 * kLinePad) + y + kLinePad) * nzp + z] =
                tile[threadIdx.x][r];
    }
}

constexpr int kWindows[] = {64, 96, 112, 128, 144, 160, 176, 208, 256, 304, 400};

template <int W> constexpr int lines_smem() { return 2 * 32 * W * 4 + kTables * 32 * 8; }

template <int W>
cudaError_t launch_window(dim3 grid, int threads, const float* vt, const JosephView* views,
    const float2* cols, JosephHeights heights, const float* lens, int view0, int nu, int nv, int nz,
    int nzp, float* proj, int accumulate, cudaStream_t s)
{
    constexpr int smem = lines_smem<W>();
    auto k = joseph_fp_lines_kernel<W>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    // the CTAs of an SM share 200 KB of it
    e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 88);
    if (e != cudaSuccess) return e;
    k<<<grid, threads, smem, s>>>(vt, views, cols, heights.first, heights.bytes, lens, view0, nu, nv, nz, nzp, proj, accumulate);
    return cudaGetLastError();
}

} // namespace

JosephColumnReach joseph_column_reach(const JosephView& j, int nv, double margin)
{
    // a detector point S + t (P - S) lies at t = 1 / ratio from the source, ratio
    // = (P - S).n / (D - S).n, which has no z part here (the detector's v axis is
    // along z): its extremes over the volume are at the corners of a slice
    const double n[2] = {j.detU[1] * j.detV[2] - j.detU[2] * j.detV[1],
                         j.detU[2] * j.detV[0] - j.detU[0] * j.detV[2]};
    const double plane = (j.detS[0] - j.src[0]) * n[0] + (j.detS[1] - j.src[1]) * n[1];
    const double hx = 0.5 * (j.axis == 0 ? j.n0 : j.n1) + margin;
    const double hy = 0.5 * (j.axis == 0 ? j.n1 : j.n0) + margin;
    JosephColumnReach r;
    r.near = 1e300;
    for (int q = 0; q < 4; ++q) {
        const double p = (((q & 1) ? hx : -hx) - j.src[0]) * n[0] + (((q & 2) ? hy : -hy) - j.src[1]) * n[1];
        r.near = std::min(r.near, p / plane);
        r.far = std::max(r.far, p / plane);
    }
    r.slope = std::sqrt(n[0] * n[0] + n[1] * n[1]) / std::fabs(plane);
    r.pitch = std::fabs(j.detV[2]) * r.far;
    r.tall = std::max(std::fabs(j.detS[2] - j.src[2]),
        std::fabs(j.detS[2] + (nv - 1) * j.detV[2] - j.src[2]));
    return r;
}

// A ray of a line reaches at most a voxel past the volume on the minor axis and
// the slice of a pair past the last one; 4 voxels cover both.  0.999 and 0.001:
// two roundings of a coordinate below 2^13 voxels.
bool joseph_bp_runs(const std::vector<JosephView>& views, int nv)
{
    for (const JosephView& j : views) {
        const JosephColumnReach r = joseph_column_reach(j, nv, 4.0);
        if (!(r.near > 0.0) || !(r.pitch <= 0.999) || !(std::fabs(j.detV[2]) * r.near >= 1e-3) ||
            j.n2 > 8192)
            return false;
    }
    return true;
}

// Rows of a CTA and window of its lines, from the largest spread of the rays of
// kCols columns and `rows` rows over kSlices slices of any view (FP64, plus
// floor, taps, alignment and a voxel of margin each side).
JosephFpLines joseph_fp_lines_shape(const std::vector<JosephView>& views, int nv)
{
    double pitch = 0.0, fixed = 0.0;  // voxels along z per row; of the columns and slices
    for (const JosephView& j : views) {
        const double column = std::sqrt(j.detU[0] * j.detU[0] + j.detU[1] * j.detU[1]);
        const JosephColumnReach r = joseph_column_reach(j, nv, kCols * column + kSlices + 2);
        if (j.axis == 2 || !(r.near > 0.0) || !(r.far < 1e6)) return {};
        pitch = std::max(pitch, r.pitch);
        fixed = std::max(fixed, r.tall * r.slope * (kCols * column * r.far + 2 * kSlices));
    }
    fixed += 9.0;
    const auto window = [&](int rows) { return pitch * (std::min(rows, nv) - 1) + fixed; };
    // the most warps on an SM (24 fit its registers) for the work of a row: 8
    // instructions a sample and 4.5 an entry of the lines
    JosephFpLines best;
    double best_score = 0.0;
    for (int chunks = (nv + kMaxRows - 1) / kMaxRows; ; ++chunks) {
        const int rows = ((nv + chunks - 1) / chunks + 31) / 32 * 32;
        const double need = window(rows);
        const int* w = std::find_if(std::begin(kWindows), std::end(kWindows), [&](int x) { return need <= x; });
        if (w != std::end(kWindows)) {
            const int ctas = std::min(200 * 1024 / (256 * *w + 2 * 1024), 24 * 32 / rows);
            const double score = ctas * rows / 32 / (8.0 + 4.5 * need / std::min(rows, nv));
            if (score > best_score) {
                best_score = score;
                best = {rows, *w};
            }
        }
        if (rows <= 32) break;
    }
    return best;
}

cudaError_t launch_joseph_line_volume(const float* vol, int nx, int ny, int nz, float* vt, cudaStream_t s)
{
    const int nzp = joseph_line_pitch(nz);
    transpose_xyz_kernel<<<dim3((nx + 31) / 32, (nzp + 31) / 32, ny), dim3(32, 8), 0, s>>>(vol, nx, ny,
        nz, nzp, vt);
    return cudaGetLastError();
}

cudaError_t launch_joseph_fp_lines(const float* vol, int nx, int ny, int nz, float* vt,
    const JosephView* views, const float2* cols, JosephHeights heights, const float* lens, int n_views,
    int nu, int nv, JosephFpLines shape, float* proj, int accumulate, cudaStream_t s)
{
    const int nzp = joseph_line_pitch(nz);
    cudaError_t e = launch_joseph_line_volume(vol, nx, ny, nz, vt, s);
    for (int done = 0; e == cudaSuccess && done < n_views; done += 65535) {
        const dim3 grid((nu + kCols - 1) / kCols, (nv + shape.rows - 1) / shape.rows,
            std::min(n_views - done, 65535));
        decltype(&launch_window<64>) launch = nullptr;
        switch (shape.window) {
        case 64: launch = launch_window<64>; break;
        case 96: launch = launch_window<96>; break;
        case 112: launch = launch_window<112>; break;
        case 128: launch = launch_window<128>; break;
        case 144: launch = launch_window<144>; break;
        case 160: launch = launch_window<160>; break;
        case 176: launch = launch_window<176>; break;
        case 208: launch = launch_window<208>; break;
        case 256: launch = launch_window<256>; break;
        case 304: launch = launch_window<304>; break;
        default: launch = launch_window<400>; break;
        }
        e = launch(grid, shape.rows, vt, views, cols, heights, lens, done, nu, nv, nz, nzp, proj,
            accumulate, s);
    }
    return e;
}

} // namespace ykb
