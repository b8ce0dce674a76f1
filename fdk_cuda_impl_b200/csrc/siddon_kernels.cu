// Siddon projector pair (FP_Siddon, BP_Siddon_RayDriven): exact
// intersection lengths of the ray from the source to each detector pixel
// centre with the voxels it crosses.
//
// Same model as src/FlatFpBp/FP/kernels/YkFPSiddonKernel.cu:19-129 and
// src/FlatFpBp/BP/kernels/YkBPSiddonKernel.cu:31-127: the ray
// S + t (D - S), t in [0, 1], clipped to the volume's outer faces, entered at
// the voxel nearest its entry point, then walked voxel by voxel
// (Amanatides-Woo) with segment length (t_next - t) |D - S|.  Both kernels
// run the one walk below, so the backprojector is the exact transpose of the
// projector.
//
// Organised for the GPU: one thread per ray, 32 channels of a detector row
// per warp (neighbouring rays walk neighbouring voxels, so the gathers and
// the reductions hit the same L1/L2 lines).  The ray is set up in FP64 and
// walked in FP32 in mm from its entry point, each face crossing evaluated
// from its index (a + j d) instead of accumulated along the ray as the
// reference does over the whole source-detector parameter, so the split of
// the length between voxels does not drift over long rays.  The choice of
// axis is branch-free and the walk runs in batches of kBatch segments whose
// gathers are issued together.  The walk is bounded by nx + ny + nz + 3
// steps.  The backprojector adds each segment to
// its voxel with a global reduction (red.global.add.f32): the sum is exact
// up to FP32 rounding, in an order that varies from run to run, as the
// reference's atomicAdd.
#include "ykb_internal.hpp"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace ykb {
namespace {

struct SiddonRay {
    float smax;              // length of the ray inside the volume (mm)
    float len;               // |D - S| (mm)
    float aX, aY, aZ;        // distance from the entry to the next face on each axis
    float dX, dY, dZ;        // distance between consecutive faces on each axis
    float mX, mY, mZ;        // interior faces ahead on each axis (crossings allowed)
    int ix, iy, iz;          // entry voxel
    int sx, sy, sz;          // step directions
};

// slab clip of one axis; false when the ray misses
__device__ __forceinline__ bool clip_axis(double s, double r, double lo, double hi, double& tmin,
    double& tmax)
{
    if (fabs(r) > 1e-8) {
        double ta = (lo - s) / r, tb = (hi - s) / r;
        if (ta > tb) { const double t = ta; ta = tb; tb = t; }
        tmin = fmax(tmin, ta);
        tmax = fmin(tmax, tb);
        return true;
    }
    return s >= lo && s <= hi;
}

// entry voxel (nearest centre to the entry point), step direction, and the
// walk's distances along this axis, measured in mm from the entry point:
// the first face crossed at a, the following ones every d
// (or from a point `origin` mm past it)
__device__ __forceinline__ void axis_setup(double s, double r, double tmin, double len, double o,
    double v, int n, int& i, int& step, float& a, float& d, float& m, double origin = 0.0)
{
    const double e = s + tmin * r;
    i = max(0, min(n - 1, static_cast<int>(floor((e - o) / v + 0.5))));
    step = r >= 0.0 ? 1 : -1;
    // faces between the entry voxel and the volume's far side: crossing
    // more would leave the volume, so the walk's indices stay in range
    m = static_cast<float>(step > 0 ? n - 1 - i : i);
    if (fabs(r) > 1e-8) {
        // face k lies at o + (k - 1/2) v
        const double k = step > 0 ? i + 1.0 : static_cast<double>(i);
        a = static_cast<float>(fmax(((o + (k - 0.5) * v - s) / r - tmin) * len, 0.0) - origin);
        d = static_cast<float>(v / fabs(r) * len);
    } else {
        a = 3e38f;  // never crossed
        d = 0.f;
        m = 0.f;
    }
    if (m == 0.f) a = 3e38f;
}

__device__ __forceinline__ bool siddon_setup(const ykb_cone_view& v, int iu, int iv,
    const VolumeGrid& g, SiddonRay& R)
{
    const double Sx = v.src.x, Sy = v.src.y, Sz = v.src.z;
    const double Dx = v.detS.x + iu * static_cast<double>(v.detU.x) + iv * static_cast<double>(v.detV.x);
    const double Dy = v.detS.y + iu * static_cast<double>(v.detU.y) + iv * static_cast<double>(v.detV.y);
    const double Dz = v.detS.z + iu * static_cast<double>(v.detU.z) + iv * static_cast<double>(v.detV.z);
    const double rx = Dx - Sx, ry = Dy - Sy, rz = Dz - Sz;
    const double len = sqrt(rx * rx + ry * ry + rz * rz);
    double tmin = 0.0, tmax = 1.0;
    if (!clip_axis(Sx, rx, g.ox - 0.5 * g.vx, g.ox + (g.nx - 0.5) * g.vx, tmin, tmax) ||
        !clip_axis(Sy, ry, g.oy - 0.5 * g.vy, g.oy + (g.ny - 0.5) * g.vy, tmin, tmax) ||
        !clip_axis(Sz, rz, g.oz - 0.5 * g.vz, g.oz + (g.nz - 0.5) * g.vz, tmin, tmax))
        return false;
    if (!(tmin < tmax)) return false;
    R.len = static_cast<float>(len);
    R.smax = static_cast<float>((tmax - tmin) * len);
    axis_setup(Sx, rx, tmin, len, g.ox, g.vx, g.nx, R.ix, R.sx, R.aX, R.dX, R.mX);
    axis_setup(Sy, ry, tmin, len, g.oy, g.vy, g.ny, R.iy, R.sy, R.aY, R.dY, R.mY);
    axis_setup(Sz, rz, tmin, len, g.oz, g.vz, g.nz, R.iz, R.sz, R.aZ, R.dZ, R.mZ);
    return true;
}

// Walks the ray in batches of kBatch segments: the walk of a batch is pure
// arithmetic, then f(index[], length[]) consumes it, so a thread has several
// independent gathers (or reductions) in flight.  Each axis crosses at most
// its interior faces ahead (mX, mY, mZ), after which its next face is at
// infinity: the voxel index never leaves the volume, and the walk ends when
// the distance reaches smax.  Segments past the exit have length 0 and the
// entry voxel's index.  I is the voxel index type (int below 2^31 voxels).
constexpr int kBatch = 4;

template <typename I, typename F>
__device__ __forceinline__ void siddon_walk(const SiddonRay& R, const VolumeGrid& g, F&& f)
{
    const I entry = (static_cast<I>(R.iz) * g.ny + R.iy) * g.nx + R.ix;
    const I stepX = R.sx, stepY = static_cast<I>(R.sy) * g.nx,
            stepZ = static_cast<I>(R.sz) * g.nx * g.ny;
    I idx = entry;
    float s = 0.f, sX = R.aX, sY = R.aY, sZ = R.aZ;
    float jx = 0.f, jy = 0.f, jz = 0.f;  // faces crossed so far (exact small integers)
    const int max_steps = g.nx + g.ny + g.nz + 3;
    for (int it = 0; it < max_steps && s < R.smax; it += kBatch) {
        I id[kBatch];
        float ds[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const bool inside = s < R.smax;
            // never behind s: an entry point on a face can round to the
            // voxel before it, whose far face then lies at s
            const float sn = fmaxf(s, fminf(fminf(sX, sY), fminf(sZ, R.smax)));
            ds[u] = inside ? sn - s : 0.f;
            id[u] = inside ? idx : entry;
            s = inside ? sn : R.smax;
            const bool xm = sX <= sY && sX <= sZ;
            const bool ym = !xm && sY <= sZ;
            idx += xm ? stepX : (ym ? stepY : stepZ);
            if (xm) {
                jx += 1.f;
                sX = jx < R.mX ? fmaf(jx, R.dX, R.aX) : 3e38f;
            } else if (ym) {
                jy += 1.f;
                sY = jy < R.mY ? fmaf(jy, R.dY, R.aY) : 3e38f;
            } else {
                jz += 1.f;
                sZ = jz < R.mZ ? fmaf(jz, R.dZ, R.aZ) : 3e38f;
            }
        }
        f(id, ds);
    }
}

template <typename I>
__global__ void __launch_bounds__(128) siddon_fp_kernel(const float* __restrict__ vol,
    const ykb_cone_view* __restrict__ views, int view0, int nu, int nv, VolumeGrid g,
    float* __restrict__ proj, int accumulate)
{
    const int iu = blockIdx.x * 32 + threadIdx.x;
    const int iv = blockIdx.y * 4 + threadIdx.y;
    const int k = view0 + blockIdx.z;
    if (iu >= nu || iv >= nv) return;
    SiddonRay R;
    float acc = 0.f;
    if (siddon_setup(views[k], iu, iv, g, R)) {
        siddon_walk<I>(R, g, [&](const I* id, const float* ds) {
            float x[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; ++u) x[u] = __ldg(vol + id[u]);
#pragma unroll
            for (int u = 0; u < kBatch; ++u) acc = fmaf(x[u], ds[u], acc);
        });
    }
    float* dst = proj + (static_cast<long>(k) * nv + iv) * nu + iu;
    *dst = accumulate ? *dst + acc : acc;
}

template <typename I>
__global__ void __launch_bounds__(128) siddon_bp_kernel(const float* __restrict__ proj,
    const ykb_cone_view* __restrict__ views, int view0, int nu, int nv, VolumeGrid g,
    float* __restrict__ vol)
{
    const int iu = blockIdx.x * 32 + threadIdx.x;
    const int iv = blockIdx.y * 4 + threadIdx.y;
    const int k = view0 + blockIdx.z;
    if (iu >= nu || iv >= nv) return;
    SiddonRay R;
    if (!siddon_setup(views[k], iu, iv, g, R)) return;
    const float p = proj[(static_cast<long>(k) * nv + iv) * nu + iu];
    if (p == 0.f) return;
    siddon_walk<I>(R, g, [&](const I* id, const float* ds) {
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
            if (ds[u] != 0.f) atomicAdd(vol + id[u], p * ds[u]);
    });
}

bool small_volume(const VolumeGrid& g)
{
    return static_cast<long>(g.nx) * g.ny * g.nz < (1L << 31);
}

// ---------------------------------------------------------------------------
// Axial-column scans: the rays of a detector column cross the same x and y
// faces at the same in-plane distances, so that walk is done once a column, and
// each ray follows its segments with its own height: within a segment it stays
// in one voxel or crosses one z face (checked by the host: it climbs less than a
// voxel over the longest segment).  A CTA owns kLineCols detector columns and up
// to 128 rows; an extra warp walks the columns a batch of segments ahead, a lane
// a column.  Against the walk above: 22 instructions per in-plane segment in the
// projector and 29 in the backprojector for 35 per voxel crossed, all lanes alive
// to the end, and the volume copy [x][y][z] makes a warp's accesses a run of
// neighbouring z.
// Distances are measured from the middle of the ray's way through the volume and
// heights from the voxel it is in there, so that both stay small and face
// crossings of flat rays keep their place.
// Bound: issue and the latency of its gathers in the projector (66 % issue), issue
// in the backprojector (76 %), whose reductions keep L2 half busy.  256^3 x 120 x 384^2:
// 5.2 and 6.0 ms, before 7.3 and 11.9; error against FP64 7.5e-7, before 7.7e-7
// (8.1e-7 while the face distances were rounded once per axis).
// ---------------------------------------------------------------------------
constexpr int kLineCols = 4;
constexpr int kLineRows = 128;
constexpr int kLineSegments = 32;  // of a column per batch
constexpr float kFloorMagic = 12582912.0f;  // 1.5 * 2^23: v + it rounded down holds floor(v)
constexpr int kFloorMagicBits = 0x4B400000;

// the in-plane walk of one column
struct ColumnWalk {
    float smax;             // half the length of the column's rays inside the volume, in the plane (mm)
    float aX, aY, dX, dY, mX, mY;
    float loX, loY;         // what dX and dY round off
    float sX, sY, jx, jy, s;
    int row, stepX, stepY;  // row: (x, y) row of the volume copy, its first element
};

// entry and exit of the column's rays (fractions of source to detector), in-plane length
__device__ __forceinline__ bool column_clip(const ykb_cone_view& v, int iu, const VolumeGrid& g,
    double& rx, double& ry, double& tmin, double& tmax)
{
    rx = v.detS.x + iu * static_cast<double>(v.detU.x) - v.src.x;
    ry = v.detS.y + iu * static_cast<double>(v.detU.y) - v.src.y;
    tmin = 0.0;
    tmax = 1.0;
    return clip_axis(v.src.x, rx, g.ox - 0.5 * g.vx, g.ox + (g.nx - 0.5) * g.vx, tmin, tmax) &&
        clip_axis(v.src.y, ry, g.oy - 0.5 * g.vy, g.oy + (g.ny - 0.5) * g.vy, tmin, tmax) && tmin < tmax;
}

__device__ __forceinline__ void column_start(const ykb_cone_view& v, int iu, const VolumeGrid& g, int nzp,
    ColumnWalk& w)
{
    const int row_x = (g.ny + 2 * kLinePad) * nzp;
    double rx, ry, tmin, tmax;
    w = ColumnWalk{};
    w.row = kLinePad * row_x + kLinePad * nzp;
    if (!column_clip(v, iu, g, rx, ry, tmin, tmax)) return;
    const double len = sqrt(rx * rx + ry * ry);
    const double half = 0.5 * (tmax - tmin) * len;
    w.smax = static_cast<float>(half);
    w.s = -w.smax;
    int ix, iy, sx, sy;
    axis_setup(v.src.x, rx, tmin, len, g.ox, g.vx, g.nx, ix, sx, w.aX, w.dX, w.mX, half);
    axis_setup(v.src.y, ry, tmin, len, g.oy, g.vy, g.ny, iy, sy, w.aY, w.dY, w.mY, half);
    w.loX = fabs(rx) > 1e-8 ? static_cast<float>(g.vx / fabs(rx) * len - w.dX) : 0.f;
    w.loY = fabs(ry) > 1e-8 ? static_cast<float>(g.vy / fabs(ry) * len - w.dY) : 0.f;
    w.sX = w.aX;
    w.sY = w.aY;
    w.row += ix * row_x + iy * nzp;
    w.stepX = sx * row_x;
    w.stepY = sy * nzp;
}

// the next segment: its end and its row; past the exit, empty ones in the zero row
// at the copy's start
__device__ __forceinline__ float2 column_segment(ColumnWalk& w)
{
    const float2 out = make_float2(fmaxf(w.s, fminf(fminf(w.sX, w.sY), w.smax)), __int_as_float(w.row));
    if (out.x < w.smax) {
        if (w.sX <= w.sY) {
            w.row += w.stepX;
            w.jx += 1.f;
            w.sX = w.jx < w.mX ? fmaf(w.jx, w.dX, fmaf(w.jx, w.loX, w.aX)) : 3e38f;
        } else {
            w.row += w.stepY;
            w.jy += 1.f;
            w.sY = w.jy < w.mY ? fmaf(w.jy, w.dY, fmaf(w.jy, w.loY, w.aY)) : 3e38f;
        }
    } else {
        w.row = 0;
    }
    w.s = out.x;
    return out;
}

// a ray over its column's segments
struct LineRay {
    float mz, ze, inv;  // voxels per mm; height in the middle over zref's floor; mm per voxel
    int zref;           // voxel in the middle
    float scale;        // length over in-plane length
    float s, t;         // where it is: distance and floor word of the height
};

__device__ __forceinline__ void line_ray(const ykb_cone_view& v, int iu, int iv, const VolumeGrid& g,
    LineRay& r, bool& inside)
{
    double rx, ry, tmin, tmax;
    r.mz = r.ze = r.inv = 0.f;
    r.zref = -(1 << 20);  // a ray that misses the volume is never inside
    r.scale = 0.f;
    r.s = 0.f;
    const bool hits = column_clip(v, iu, g, rx, ry, tmin, tmax);
    if (!hits) inside = false;
    if (hits) {
        const double rz = v.detS.z + iv * static_cast<double>(v.detV.z) - v.src.z;
        const double len = sqrt(rx * rx + ry * ry);
        const double z0 = (v.src.z + tmin * rz - g.oz) / g.vz + 0.5;
        const double z1 = (v.src.z + tmax * rz - g.oz) / g.vz + 0.5;
        const double zm = 0.5 * (z0 + z1), f = floor(fmin(fmax(zm, -1e8), 1e8));
        r.zref = static_cast<int>(f);
        r.ze = static_cast<float>(zm - f);
        r.s = static_cast<float>(-0.5 * (tmax - tmin) * len);
        r.mz = static_cast<float>(rz / (len * g.vz));
        r.inv = rz != 0.0 ? static_cast<float>(len * g.vz / rz) : 0.f;
        r.scale = static_cast<float>(sqrt(1.0 + (rz / len) * (rz / len)));
        if (!(fmin(z0, z1) >= 1e-3 && fmax(z0, z1) <= g.nz - 1e-3)) inside = false;
    }
    r.t = __fadd_rd(fmaf(r.s, r.mz, r.ze), kFloorMagic);
}

// One segment of a ray: the voxel it enters in (i0, weight w0) and the one it
// leaves in (i1, w1), indices in z.  Where they are the same, the projector has
// the whole length in w0 (in1 false: one gather); the backprojector has it in
// either, from the same expression held between zero and the segment's length: no
// weight is negative where the face rounds to a place outside the segment, and
// one that is zero marks a voxel that is not crossed.
struct LineStep { int i0, i1; float w0, w1; bool in1; };
template <bool FORWARD>
__device__ __forceinline__ LineStep line_step(LineRay& r, float s1)
{
    LineStep st;
    const float t1 = __fadd_rd(fmaf(s1, r.mz, r.ze), kFloorMagic);
    st.i0 = __float_as_int(r.t) - kFloorMagicBits + r.zref;
    st.i1 = __float_as_int(t1) - kFloorMagicBits + r.zref;
    const float face = fmaxf(t1, r.t) - kFloorMagic, length = s1 - r.s;
    st.w1 = s1 - (face - r.ze) * r.inv;
    if constexpr (FORWARD) {
        st.in1 = t1 != r.t;
        if (!st.in1) st.w1 = 0.f;
    } else {
        st.w1 = fminf(fmaxf(st.w1, 0.f), length);
        st.in1 = st.w1 != 0.f;
    }
    st.w0 = length - st.w1;
    r.s = s1;
    r.t = t1;
    return st;
}

template <bool FORWARD>
__global__ void __launch_bounds__(kLineRows + 32, 6) siddon_lines_kernel(const float* __restrict__ in,
    const ykb_cone_view* __restrict__ views, int view0, int nu, int nv, const __grid_constant__ VolumeGrid g,
    int nzp, float* __restrict__ out, float* __restrict__ odd, int accumulate)
{
    if constexpr (!FORWARD)
        if ((view0 + blockIdx.z) & 1) out = odd;
    __shared__ float2 segments[2][kLineSegments][kLineCols];
    __shared__ int more[2];
    const int tid = threadIdx.x, rows = blockDim.x - 32;
    const int iu0 = blockIdx.x * kLineCols, k = view0 + blockIdx.z;
    const ykb_cone_view& v = views[k];
    if (tid >= rows) {
        // the walking warp
        const int lane = tid - rows;
        ColumnWalk w{};
        if (lane < kLineCols) column_start(v, min(iu0 + lane, nu - 1), g, nzp, w);
        for (int b = 0;; ++b) {
            if (lane < kLineCols)
                for (int q = 0; q < kLineSegments; ++q) segments[b & 1][q][lane] = column_segment(w);
            const bool on = __any_sync(0xffffffffu, lane < kLineCols && w.s < w.smax);
            if (lane == 0) more[b & 1] = on;
            __syncthreads();
            if (!on) return;
        }
    }
    const int iv = blockIdx.y * rows + tid;
    const bool pixel = iv < nv;
    LineRay r[kLineCols];
    bool inside = true;
#pragma unroll
    for (int c = 0; c < kLineCols; ++c)
        line_ray(v, min(iu0 + c, nu - 1), min(iv, nv - 1), g, r[c], inside);
    inside = __all_sync(0xffffffffu, inside);
    const long at = (static_cast<long>(k) * nv + min(iv, nv - 1)) * nu + iu0;
    float acc[kLineCols], p[kLineCols];
#pragma unroll
    for (int c = 0; c < kLineCols; ++c) {
        acc[c] = 0.f;
        p[c] = !FORWARD && pixel && iu0 + c < nu ? in[at + c] * r[c].scale : 0.f;
    }
    for (int b = 0;; ++b) {
        __syncthreads();
        const float2 (*seg)[kLineCols] = segments[b & 1];
        const bool on = more[b & 1];
        const auto walk = [&](auto checked) {
#pragma unroll 2
            for (int q = 0; q < kLineSegments; ++q) {
#pragma unroll
                for (int c = 0; c < kLineCols; ++c) {
                    const float2 e = seg[q][c];
                    const LineStep st = line_step<FORWARD>(r[c], e.x);
                    const int row = __float_as_int(e.y);
                    const bool in0 = !decltype(checked)::value ||
                        static_cast<unsigned>(st.i0) < static_cast<unsigned>(g.nz);
                    const bool in1 = st.in1 && (!decltype(checked)::value ||
                        static_cast<unsigned>(st.i1) < static_cast<unsigned>(g.nz));
                    if constexpr (FORWARD) {
                        if (in0) acc[c] = fmaf(__ldg(in + (row + st.i0)), st.w0, acc[c]);
                        if (in1) acc[c] = fmaf(__ldg(in + (row + st.i1)), st.w1, acc[c]);
                    } else {
                        if (in0 && st.w0 != 0.f && p[c] != 0.f) atomicAdd(out + (row + st.i0), p[c] * st.w0);
                        if (in1 && p[c] != 0.f) atomicAdd(out + (row + st.i1), p[c] * st.w1);
                    }
                }
            }
        };
        if (inside) walk(std::false_type{});
        else walk(std::true_type{});
        if (!on) break;
    }
    if constexpr (FORWARD) {
        if (!pixel) return;
#pragma unroll
        for (int c = 0; c < kLineCols; ++c) {
            if (iu0 + c >= nu) break;
            const float a = acc[c] * r[c].scale;
            out[at + c] = accumulate ? out[at + c] + a : a;
        }
    }
}

// vol[z][y][x] (+)= vt[x][y][z] + odd[x][y][z] (rows of nzp, kLinePad rows around
// x and y)
__global__ void __launch_bounds__(256) untranspose_xyz_kernel(const float* __restrict__ vt,
    const float* __restrict__ odd, int nx, int ny, int nz, int nzp, float* __restrict__ vol, int accumulate)
{
    __shared__ float tile[32][33];
    const int y = blockIdx.z, x0 = blockIdx.x * 32, z0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int x = x0 + r, z = z0 + threadIdx.x;
        if (x < nx && z < nz)
        {
            const long at = (static_cast<long>(x + kLinePad) * (ny + 2 * kLinePad) + y + kLinePad) * nzp + z;
            tile[r][threadIdx.x] = vt[at] + odd[at];
        }
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int z = z0 + r, x = x0 + threadIdx.x;
        if (x >= nx || z >= nz) continue;
        float* dst = vol + (static_cast<long>(z) * ny + y) * nx + x;
        *dst = accumulate ? *dst + tile[threadIdx.x][r] : tile[threadIdx.x][r];
    }
}

dim3 line_grid(int nu, int nv, int count, int& threads)
{
    const int chunks = (nv + kLineRows - 1) / kLineRows;
    const int rows = ((nv + chunks - 1) / chunks + 31) / 32 * 32;
    threads = rows + 32;
    return dim3((nu + kLineCols - 1) / kLineCols, (nv + rows - 1) / rows, count);
}

} // namespace

bool siddon_lines_apply(const ykb_cone_view* views, int n_views, int nv, const VolumeGrid& g)
{
    // 32-bit indices into the volume copy, one dimension of the launch over y
    const double elems = (g.nx + 2.0 * kLinePad) * (g.ny + 2.0 * kLinePad) * joseph_line_pitch(g.nz);
    if (elems >= 2147483648.0 || g.ny > 65535 || g.nz > (1 << 20)) return false;
    const double longest = std::sqrt(g.vx * g.vx + g.vy * g.vy) / g.vz;
    for (int k = 0; k < n_views; ++k) {
        const ykb_cone_view& v = views[k];
        if (v.detU.z != 0.f || v.detV.x != 0.f || v.detV.y != 0.f) return false;
        const double u = std::hypot(static_cast<double>(v.detU.x), static_cast<double>(v.detU.y));
        const double plane = std::fabs((static_cast<double>(v.detS.x) - v.src.x) * v.detU.y -
            (static_cast<double>(v.detS.y) - v.src.y) * v.detU.x) / u;
        const double z0 = std::fabs(static_cast<double>(v.detS.z) - v.src.z);
        const double z1 = std::fabs(v.detS.z + (nv - 1) * static_cast<double>(v.detV.z) - v.src.z);
        if (!(std::max(z0, z1) / plane * longest <= 0.99)) return false;
    }
    return true;
}

cudaError_t launch_siddon_fp_lines(const float* vol, float* vt, const ykb_cone_view* views, int n_views,
    int nu, int nv, const VolumeGrid& g, float* proj, int accumulate, cudaStream_t s)
{
    cudaError_t e = launch_joseph_line_volume(vol, g.nx, g.ny, g.nz, vt, s);
    for (int done = 0; e == cudaSuccess && done < n_views; done += 65535) {
        int threads = 0;
        const dim3 grid = line_grid(nu, nv, min(n_views - done, 65535), threads);
        siddon_lines_kernel<true><<<grid, threads, 0, s>>>(vt, views, done, nu, nv, g,
            joseph_line_pitch(g.nz), proj, nullptr, accumulate);
        e = cudaGetLastError();
    }
    return e;
}

cudaError_t launch_siddon_bp_lines(const float* proj, float* vt, float* odd, const ykb_cone_view* views,
    int n_views, int nu, int nv, const VolumeGrid& g, float* vol, int accumulate, cudaStream_t s)
{
    const int nzp = joseph_line_pitch(g.nz);
    const size_t elems = static_cast<size_t>(g.nx + 2 * kLinePad) * (g.ny + 2 * kLinePad) * nzp;
    cudaError_t e = cudaMemsetAsync(vt, 0, sizeof(float) * elems, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(odd, 0, sizeof(float) * elems, s);
    for (int done = 0; e == cudaSuccess && done < n_views; done += 65535) {
        int threads = 0;
        const dim3 grid = line_grid(nu, nv, min(n_views - done, 65535), threads);
        siddon_lines_kernel<false><<<grid, threads, 0, s>>>(proj, views, done, nu, nv, g, nzp, vt, odd, 0);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return e;
    untranspose_xyz_kernel<<<dim3((g.nx + 31) / 32, (g.nz + 31) / 32, g.ny), dim3(32, 8), 0, s>>>(vt, odd,
        g.nx, g.ny, g.nz, nzp, vol, accumulate);
    return cudaGetLastError();
}

cudaError_t launch_siddon_fp(const float* vol, const ykb_cone_view* views, int n_views, int nu,
    int nv, const VolumeGrid& g, float* proj, int accumulate, cudaStream_t s)
{
    for (int done = 0; done < n_views; done += 65535) {
        const int count = min(n_views - done, 65535);
        const dim3 grid((nu + 31) / 32, (nv + 3) / 4, count);
        if (small_volume(g))
            siddon_fp_kernel<int><<<grid, dim3(32, 4), 0, s>>>(vol, views, done, nu, nv, g, proj, accumulate);
        else
            siddon_fp_kernel<long><<<grid, dim3(32, 4), 0, s>>>(vol, views, done, nu, nv, g, proj, accumulate);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_siddon_bp(const float* proj, const ykb_cone_view* views, int n_views, int nu,
    int nv, const VolumeGrid& g, float* vol, int accumulate, cudaStream_t s)
{
    if (!accumulate) {
        const cudaError_t e = cudaMemsetAsync(vol,
            0, static_cast<size_t>(g.nx) * g.ny * g.nz * sizeof(float), s);
        if (e != cudaSuccess) return e;
    }
    for (int done = 0; done < n_views; done += 65535) {
        const int count = min(n_views - done, 65535);
        const dim3 grid((nu + 31) / 32, (nv + 3) / 4, count);
        if (small_volume(g))
            siddon_bp_kernel<int><<<grid, dim3(32, 4), 0, s>>>(proj, views, done, nu, nv, g, vol);
        else
            siddon_bp_kernel<long><<<grid, dim3(32, 4), 0, s>>>(proj, views, done, nu, nv, g, vol);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

} // namespace ykb
