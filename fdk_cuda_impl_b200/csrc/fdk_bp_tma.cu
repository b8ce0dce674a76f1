// FDK weighted backprojection with TMA-staged projection tiles (sm_100a).
//
// Same arithmetic as fdk_bp_kernel in fdk_kernels.cu (the math of
// .../FDK/kernels/YkFDKBpKernels.cu:112-209 with exact software bilinear
// weights), organised for Blackwell:
//   * a persistent CTA per SM walks voxel tiles of 16 x 32 x 64; each of its
//     512 threads keeps the 64 sums of a z column in registers over all views
//     (the longer the column, the more voxels share the per-view column
//     terms); a remainder of at most 32 slices runs as 32-voxel columns, the
//     launch's last z layer.  A volume of few tiles also splits its views
//     into jobs of their own (see split_count);
//   * per view the detector box covering the tile's footprint is loaded with
//     cp.async.bulk.tensor (3D tile mode, this GPU's memory only, no
//     multicast) into a ring of shared-memory stages.  Out-of-detector
//     elements are zero-filled by TMA, which is the reference's Border
//     addressing;
//   * there is no producer warp: the sixteen warps take turns at computing a
//     view's box and FP64-derived terms a ring's length ahead, and the last
//     warp to finish with a stage issues the copy that refills it.  A
//     seventeenth warp would cost each thread a quarter of its registers
//     (65536 are granted to whole groups of four warps: 96 a thread with 17
//     warps, 128 with 16), which the 64 sums, the addresses and a few voxels'
//     taps in flight need;
//   * filtered rows arrive either as plain floats or as row pairs: element
//     (n + 1, u) = (f[n][u], f[n + 1][u] - f[n][u]) for n = -1 .. nv - 1, rows
//     outside the detector zero (written so by the filter epilogue).  The two
//     8-byte shared loads at columns u and u + 1 then hold a voxel's four taps
//     with the vertical differences already formed, at one row address;
//   * the taps are read without bounds checks: the box is sized by a pre-pass
//     over all (tile, view) pairs with the same footprint function, and each
//     (column, view) checks its end points.
// Bound: the shared-memory data path, 16 bytes of taps per voxel and view (84 %
// of its wavefront peak; 12.8 instructions per update at 62 % issue, against
// 15.2 with horizontal tap pairs, a producer warp and 96 registers).  Measured
// on 512^3 x 720 x 768^2: 53.5 ms, before 60.1; on a tilted detector,
// 256^3 x 180 x 384^2, whose columns need a reciprocal per voxel: 3.0 ms,
// before 8.6 (absolute FP32 coordinates, three divisions a voxel and spilled
// sums).
// Every mbarrier wait is bounded (~2 s of %globaltimer by default; the
// pipeline waits take the limit as a kernel argument, so that a test can
// shorten it); a timeout sets the plan's error word, stops the CTA and drains
// the copies in flight, each drain wait with the full limit.
#include "ykb_internal.hpp"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>

namespace ykb {
namespace {

constexpr int TX = 16, TY = 32, ZT = 64;
constexpr int kZTail = 32;  // column length of a short last z tile
constexpr int NTHREADS = TX * TY;
constexpr int NWARPS = NTHREADS / 32;
constexpr int kMaxStages = 8;
constexpr int kSlots = 16;  // views whose box and terms are held: two rings' lengths
static_assert(NWARPS == 16 && kSlots >= 2 * kMaxStages && NWARPS >= kMaxStages, "turns of the warps");
constexpr unsigned long long kWaitNs = 2000000000ull;

// error word bits
constexpr int kErrTimeout = 1;
constexpr int kErrFootprint = 2;
constexpr int kErrAlign = 4;

// a TMA tile copy writes shared memory at 128-byte aligned addresses: each
// stage starts on a 128-byte boundary
__host__ __device__ constexpr int stage_stride_floats(int bw, int bh, bool pair)
{
    return (bw * bh * (pair ? 2 : 1) + 31) / 32 * 32;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
                 "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok) : "r"(smem_addr(bar)), "r"(parity) : "memory");
    return ok != 0;
}

// bounded wait: false after limit_ns
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity,
    unsigned long long limit_ns = kWaitNs)
{
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    while (!mbar_try_wait(bar, parity))
        if (global_ns() - t0 > limit_ns) return false;
    return true;
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar,
    int x, int y, int z)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_addr(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ double rcp64(double x)
{
    double r = static_cast<double>(__frcp_rn(static_cast<float>(x)));
    return r * (2.0 - x * r);
}

// Packed FP32 pairs (sm_100 f32x2 arithmetic): two z-voxels per instruction.
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
__device__ __forceinline__ f2 f2add(f2 a, f2 b)
{
    f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 f2sub(f2 a, f2 b)
{
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// rounded towards minus infinity
__device__ __forceinline__ f2 f2add_rm(f2 a, f2 b)
{
    f2 d;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
template <int OFF>
__device__ __forceinline__ float lds(uint32_t addr)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(addr), "n"(OFF));
    return v;
}
// one row pair (8-byte aligned)
template <int OFF>
__device__ __forceinline__ void lds2(uint32_t addr, float& lo, float& hi)
{
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2+%3];" : "=f"(lo), "=f"(hi) : "r"(addr), "n"(OFF));
}

// t = v + 1.5*2^23 rounded down holds floor(v) in its low mantissa bits for
// |v| < 2^22, and t - 1.5*2^23 is floor(v).  The map v -> t is monotonic.
constexpr float kFloorMagic = 12582912.0f;
constexpr uint32_t kFloorMagicBits = 0x4B400000u;
__device__ __forceinline__ int floor_row(float v)
{
    return static_cast<int>(__float_as_uint(__fadd_rd(v, kFloorMagic)) - kFloorMagicBits);
}

__device__ __forceinline__ float sqrt_approx(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Detector box of a voxel tile for one view: columns c0 .. c1 and rows
// r0 .. r1 hold the taps floor(u), floor(u) + 1 and the row pairs floor(v) of
// every voxel centre of the tile, with one pixel of margin each side.  The
// columns start at the TMA alignment (16 bytes: two row pairs, four floats).
// The pre-pass and the kernel evaluate the same corners with the same code
// (the map is projective and the tile convex: the corners bound it).
struct Box { int c0, c1, r0, r1; };

__device__ __forceinline__ void corner_uv(const FdkViewCoef& c, double X, double Y, double Z,
    double& u, double& v)
{
    const double den = fma(c.cd[2], Z, fma(c.cd[1], Y, fma(c.cd[0], X, c.cd[3])));
    const double r = rcp64(den);
    u = fma(c.cu[2], Z, fma(c.cu[1], Y, fma(c.cu[0], X, c.cu[3]))) * r;
    v = fma(c.cv[2], Z, fma(c.cv[1], Y, fma(c.cv[0], X, c.cv[3]))) * r;
}

__device__ __forceinline__ Box box_from_range(double umin, double umax, double vmin, double vmax,
    int align)
{
    umin = fmax(umin, -1e8); umax = fmin(umax, 1e8);
    vmin = fmax(vmin, -1e8); vmax = fmin(vmax, 1e8);
    Box b;
    b.c0 = (static_cast<int>(floor(umin)) - 1) & ~(align - 1);
    b.c1 = static_cast<int>(floor(umax)) + 2;
    b.r0 = static_cast<int>(floor(vmin)) - 1;
    b.r1 = static_cast<int>(floor(vmax)) + 1;
    return b;
}

struct TileGeom {
    double x0, x1, y0, y1, z0, z1;
    double xc, yc;  // centre of the nominal TX x TY tile (reference point of its column terms)
};

__device__ __forceinline__ TileGeom tile_geom(const VolumeGrid& g, int bx, int by, int za, int zc)
{
    TileGeom t;
    const int xa = bx * TX, ya = by * TY;
    t.x0 = g.ox + xa * g.vx;
    t.x1 = g.ox + min(xa + TX - 1, g.nx - 1) * g.vx;
    t.y0 = g.oy + ya * g.vy;
    t.y1 = g.oy + min(ya + TY - 1, g.ny - 1) * g.vy;
    t.z0 = g.oz + za * g.vz;
    t.z1 = g.oz + (za + zc - 1) * g.vz;  // all zc slices are evaluated
    t.xc = g.ox + (xa + 0.5 * (TX - 1)) * g.vx;
    t.yc = g.oy + (ya + 0.5 * (TY - 1)) * g.vy;
    return t;
}

// Pre-pass: largest box over all (tile, view) pairs: widths at both
// alignments and the rows of row pairs.
__global__ void box_extent_kernel(const FdkViewCoef* __restrict__ coef, int n_views, VolumeGrid g,
    int tiles_x, int tiles_y, int tiles_z, int* __restrict__ out)
{
    const long n = static_cast<long>(tiles_x) * tiles_y * tiles_z * n_views;
    int w2 = 0, w4 = 0, h = 0;
    for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long>(gridDim.x) * blockDim.x) {
        const int k = static_cast<int>(i % n_views);
        const long t = i / n_views;
        const int bx = static_cast<int>(t % tiles_x);
        const int by = static_cast<int>((t / tiles_x) % tiles_y);
        const int bz = static_cast<int>(t / (static_cast<long>(tiles_x) * tiles_y));
        const TileGeom tg = tile_geom(g, bx, by, bz * ZT, ZT);
        double umin = 1e300, umax = -1e300, vmin = 1e300, vmax = -1e300;
        for (int q = 0; q < 8; ++q) {
            double u, v;
            corner_uv(coef[k], (q & 1) ? tg.x1 : tg.x0, (q & 2) ? tg.y1 : tg.y0,
                (q & 4) ? tg.z1 : tg.z0, u, v);
            umin = fmin(umin, u); umax = fmax(umax, u);
            vmin = fmin(vmin, v); vmax = fmax(vmax, v);
        }
        const Box b2 = box_from_range(umin, umax, vmin, vmax, 2);
        const Box b4 = box_from_range(umin, umax, vmin, vmax, 4);
        w2 = max(w2, b2.c1 - b2.c0 + 1);
        w4 = max(w4, b4.c1 - b4.c0 + 1);
        h = max(h, b2.r1 - b2.r0 + 1);
    }
    atomicMax(out, w2);
    atomicMax(out + 1, w4);
    atomicMax(out + 2, h);
}

// Per-(tile, view) terms, FP64-derived once per tile and view and held beside
// the ring; each thread evaluates its column's terms from them in FP32.  With
// d = (X - xc, Y - yc) the column's offset from the tile centre and i the
// slice above the tile's first one:
//   den = dc + gd . d + i gd2                       (cd . P)
//   u   = uc + (hu . d + i hu2) / den      hu = (cu_x, cu_y) - u_c (cd_x, cd_y)
//   v   = vc + (hv . d + i hv2) / den      hv = (cv_x, cv_y) - v_c (cd_x, cd_y)
// exact rewrites of u = cu.P / cd.P and v = cv.P / cd.P about the tile
// centre's column (the numerators of u - u_c and v - v_c vanish there); on
// axial views gd2 = hu2 = 0.  u and v are relative to the staged box, so they
// stay below the box size and round to within 4e-6 px.  The weights:
//   FDK     w = wbase / dep^2, dep = pc + gp . d    (cr . P; cr_z is zero: the
//           depth is measured along a horizontal ray)
//   pseudo  w = kq |P - S| / den^3: on the ray through P the detector point is
//           at L = |P - S| plane / den, so the reference's k L^3 / |P - S|^2
//           is voxel volume x plane^2 |P - S| / (du dv den^3); P - S from the
//           tile centre's first voxel.
// Untilted columns of plain rows and of the pseudo-matched weight take
// ColumnTerms instead.
struct alignas(16) TileTerms {
    float uc, hu0, hu1, hu2;
    float vc, hv0, hv1, hv2;
    float dc, gd0, gd1, gd2;
    float p0, p1, p2, p3;  // FDK: pc, gp0, gp1, wbase; pseudo: P - S, kq
};

template <bool PSEUDO>
__device__ __forceinline__ TileTerms tile_terms(const FdkViewCoef& c, const PseudoViewCoef* pv,
    const TileGeom& tg, double vz, int c0, int r0)
{
    const double den = fma(c.cd[2], tg.z0, fma(c.cd[1], tg.yc, fma(c.cd[0], tg.xc, c.cd[3])));
    const double rd = 1.0 / den;
    const double uc = fma(c.cu[2], tg.z0, fma(c.cu[1], tg.yc, fma(c.cu[0], tg.xc, c.cu[3]))) * rd;
    const double vc = fma(c.cv[2], tg.z0, fma(c.cv[1], tg.yc, fma(c.cv[0], tg.xc, c.cv[3]))) * rd;
    TileTerms t;
    t.uc = static_cast<float>(uc - c0);
    t.hu0 = static_cast<float>(c.cu[0] - uc * c.cd[0]);
    t.hu1 = static_cast<float>(c.cu[1] - uc * c.cd[1]);
    t.hu2 = static_cast<float>((c.cu[2] - uc * c.cd[2]) * vz);
    t.vc = static_cast<float>(vc - r0);
    t.hv0 = static_cast<float>(c.cv[0] - vc * c.cd[0]);
    t.hv1 = static_cast<float>(c.cv[1] - vc * c.cd[1]);
    t.hv2 = static_cast<float>((c.cv[2] - vc * c.cd[2]) * vz);
    t.dc = static_cast<float>(den);
    t.gd0 = static_cast<float>(c.cd[0]);
    t.gd1 = static_cast<float>(c.cd[1]);
    t.gd2 = static_cast<float>(c.cd[2] * vz);
    if constexpr (PSEUDO) {
        t.p0 = static_cast<float>(tg.xc - pv->src[0]);
        t.p1 = static_cast<float>(tg.yc - pv->src[1]);
        t.p2 = static_cast<float>(tg.z0 - pv->src[2]);
        t.p3 = pv->kq;
    } else {
        t.p0 = static_cast<float>(fma(c.cr[1], tg.yc, fma(c.cr[0], tg.xc, c.cr[3])));
        t.p1 = static_cast<float>(c.cr[0]);
        t.p2 = static_cast<float>(c.cr[1]);
        t.p3 = static_cast<float>(c.wbase);
    }
    return t;
}

// Terms of an untilted column evaluated in FP64 and rounded once, u and v relative
// to the staged box: the plain-row and the pseudo-matched kernels, whose other
// arithmetic is accurate enough for the roundings of the tile terms to show.  Eight
// views of 64 x 48: 1.5e-7 of FP64 against 2.8e-7 from the tile terms; 256^3 x 360 x
// 384^2, pseudo-matched: 4.19 ms against 3.84, plain rows 5.24 against 4.93.
struct ColumnTerms {
    float u, vb, vs, w;  // v of slice i: vb + i vs
    float q2, rz0;       // pseudo: squared horizontal distance, height of slice 0
};

template <bool PSEUDO>
__device__ __forceinline__ ColumnTerms column_terms(const FdkViewCoef& c, const PseudoViewCoef* pv,
    double X, double Y, double Z, double vz, int c0, int r0)
{
    const double r = rcp64(fma(c.cd[2], Z, fma(c.cd[1], Y, fma(c.cd[0], X, c.cd[3]))));
    ColumnTerms t;
    t.u = static_cast<float>(fma(fma(c.cu[2], Z, fma(c.cu[1], Y, fma(c.cu[0], X, c.cu[3]))), r, -c0));
    t.vb = static_cast<float>(fma(fma(c.cv[2], Z, fma(c.cv[1], Y, fma(c.cv[0], X, c.cv[3]))), r, -r0));
    t.vs = static_cast<float>(c.cv[2] * vz * r);
    t.q2 = 1.f;
    t.rz0 = 0.f;
    if constexpr (PSEUDO) {
        const double dx = X - pv->src[0], dy = Y - pv->src[1];
        t.q2 = static_cast<float>(fma(dx, dx, dy * dy));
        t.rz0 = static_cast<float>(Z - pv->src[2]);
        t.w = static_cast<float>(pv->kq * r * r * r);
    } else {
        const double rp = rcp64(fma(c.cr[1], Y, fma(c.cr[0], X, c.cr[3])));
        t.w = static_cast<float>(c.wbase * rp * rp);
    }
    return t;
}

// Shared-memory ring budget of the one CTA of an SM.
constexpr size_t kRingBudget = 200 * 1024;

// Shared memory of the CTA: the ring of stages; per held view (slot) its
// terms and its copy (box column, box row, view, 1 or 0: nothing to copy);
// per stage its barrier and how many warps have finished with it so far.
struct BpSmem {
    float* ring;
    TileTerms* terms;   // [kSlots]
    int4* copies;       // [kSlots]
    uint64_t* full;     // [kMaxStages]
    uint32_t* done;     // [kMaxStages]
    int* abort_flag;
    int* issued;        // views issued so far (or withheld)
    int stage_floats;
};
constexpr size_t kBpTables = kSlots * (sizeof(TileTerms) + sizeof(int4)) +
    kMaxStages * (sizeof(uint64_t) + sizeof(uint32_t)) + 2 * sizeof(int);

__device__ __forceinline__ BpSmem bp_smem(int BW, int BH, bool pair, int stages)
{
    extern __shared__ unsigned char smem_raw[];
    // 128-byte aligned base (the launch requests 128 bytes of slack)
    unsigned char* smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
    BpSmem m;
    m.stage_floats = stage_stride_floats(BW, BH, pair);
    m.ring = reinterpret_cast<float*>(smem);
    m.terms = reinterpret_cast<TileTerms*>(
        smem + static_cast<size_t>(m.stage_floats) * sizeof(float) * stages);
    m.copies = reinterpret_cast<int4*>(m.terms + kSlots);
    m.full = reinterpret_cast<uint64_t*>(m.copies + kSlots);
    m.done = reinterpret_cast<uint32_t*>(m.full + kMaxStages);
    m.abort_flag = reinterpret_cast<int*>(m.done + kMaxStages);
    m.issued = m.abort_flag + 1;
    return m;
}

// The launch's jobs: job j is tile j % n_tiles over the views of split
// j / n_tiles.  Tiles in order: layers of TX x TY tiles (x fastest), the
// ZT-slice layers from slice 0, then at most one layer of kZTail-slice tiles
// (a short last part of the volume; it lies inside the ZT-slice layer of the
// box pre-pass, so its footprints fit the same box).
struct Schedule {
    int tiles_x, tiles_y, main_layers;
    long n_tiles, n_jobs;
    int n_views, splits;
    long part_floats;  // distance of one split's sums from the next split's
};

// A walk over the (job, view) pairs of one CTA.
struct Cursor {
    long job;
    int k, k1;  // view, and the first view past the job's
    int bx, by, za;
    bool main;
};

__device__ __forceinline__ void cursor_open(Cursor& c, const Schedule& sc)
{
    if (c.job >= sc.n_jobs) return;
    const int split = static_cast<int>(c.job / sc.n_tiles);
    const long t = c.job - split * sc.n_tiles;
    c.k = static_cast<int>(static_cast<long>(sc.n_views) * split / sc.splits);
    c.k1 = static_cast<int>(static_cast<long>(sc.n_views) * (split + 1) / sc.splits);
    const long per_layer = static_cast<long>(sc.tiles_x) * sc.tiles_y;
    const int bz = static_cast<int>(t / per_layer);
    const int rem = static_cast<int>(t - bz * per_layer);
    c.by = rem / sc.tiles_x;
    c.bx = rem - c.by * sc.tiles_x;
    c.main = bz < sc.main_layers;
    c.za = c.main ? bz * ZT : sc.main_layers * ZT + (bz - sc.main_layers) * kZTail;
}

__device__ __forceinline__ void cursor_next(Cursor& c, const Schedule& sc)
{
    if (c.job < sc.n_jobs && ++c.k == c.k1) {
        c.job += gridDim.x;
        cursor_open(c, sc);
    }
}

// The box and terms of the cursor's view into slot `slot` (one warp; lanes
// 0..7 project one tile corner each).
template <bool PAIR, bool PSEUDO>
__device__ __forceinline__ void hold_view(const BpSmem& sm, const Cursor& c, const Schedule& sc,
    const FdkViewCoef* __restrict__ coef, const PseudoViewCoef* __restrict__ pseudo,
    const VolumeGrid& g, int slot)
{
    const int lane = threadIdx.x & 31;
    if (c.job >= sc.n_jobs) {
        if (lane == 0) sm.copies[slot] = make_int4(0, 0, 0, 0);
        return;
    }
    const TileGeom tg = tile_geom(g, c.bx, c.by, c.za, c.main ? ZT : kZTail);
    double umin = 1e300, umax = -1e300, vmin = 1e300, vmax = -1e300;
    if (lane < 8) {
        corner_uv(coef[c.k], (lane & 1) ? tg.x1 : tg.x0, (lane & 2) ? tg.y1 : tg.y0,
            (lane & 4) ? tg.z1 : tg.z0, umin, vmin);
        umax = umin; vmax = vmin;
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        umin = fmin(umin, __shfl_xor_sync(0xffffffffu, umin, o));
        umax = fmax(umax, __shfl_xor_sync(0xffffffffu, umax, o));
        vmin = fmin(vmin, __shfl_xor_sync(0xffffffffu, vmin, o));
        vmax = fmax(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    }
    if (lane == 0) {
        const Box b = box_from_range(umin, umax, vmin, vmax, PAIR ? 2 : 4);
        sm.terms[slot] = tile_terms<PSEUDO>(coef[c.k], PSEUDO ? pseudo + c.k : nullptr, tg, g.vz,
            b.c0, b.r0);
        sm.copies[slot] = make_int4(b.c0, b.r0, c.k, 1);
    }
    __syncwarp();
}

// Issues the copy of slot `slot` into stage s (one thread).
template <bool PAIR>
__device__ __forceinline__ void issue_copy(const BpSmem& sm, const CUtensorMap* map, int slot,
    int s, uint32_t box_bytes, int withheld_view)
{
    const int4 b = sm.copies[slot];
    if (b.w == 0) return;
    ++*reinterpret_cast<volatile int*>(sm.issued);
    // test hook: no copy and no arrival for this view, so every wait for it
    // runs out
    if (b.z == withheld_view) return;
    mbar_arrive_expect_tx(&sm.full[s], box_bytes);
    // row pair (n, n + 1) is row n + 1 of the layout
    tma_load_3d(sm.ring + static_cast<size_t>(s) * sm.stage_floats, map, &sm.full[s], b.x,
        PAIR ? b.y + 1 : b.y, b.z);
}

// Taps of the row pair at address a: the left and right columns' values and
// their differences to the next row.
template <bool PAIR>
__device__ __forceinline__ void load_taps(uint32_t a, uint32_t row_bytes, float& ml, float& dl,
    float& mr, float& dr)
{
    if constexpr (PAIR) {
        lds2<0>(a, ml, dl);
        lds2<8>(a, mr, dr);
    } else {
        ml = lds<0>(a);
        mr = lds<4>(a);
        dl = lds<0>(a + row_bytes) - ml;
        dr = lds<4>(a + row_bytes) - mr;
    }
}

// The CTA's pipeline state: the view being consumed (stage, its phase, the
// count of views so far) and the cursor a ring's length ahead.
struct Pipe {
    int s;
    uint32_t phase;
    uint32_t q;
    Cursor ahead;
};

// One job: the tile and views at `cur`.  False when a wait ran out.
template <bool AXIAL, bool PAIR, bool PSEUDO, int ZC, bool ACC>
__device__ __forceinline__ bool bp_job(const BpSmem& sm, const CUtensorMap* map,
    const FdkViewCoef* __restrict__ coef, const PseudoViewCoef* __restrict__ pseudo,
    const VolumeGrid& g, const Schedule& sc, int BW, int BH, int stages, float* __restrict__ vol,
    int* __restrict__ err, const PipelineWait& pw, const Cursor& cur, Pipe& pipe)
{
    constexpr uint32_t ES = PAIR ? 8u : 4u;  // bytes per staged element
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t row_bytes = ES * static_cast<uint32_t>(BW);
    const uint32_t box_bytes = row_bytes * static_cast<uint32_t>(BH);
    const int rows = PAIR ? BH : BH - 1;  // row pairs of a stage
    // a warp covers an 8x4 block of columns, each half-warp a 4x4 block: the
    // detector footprint of 16 lanes then spans few columns, so the 16-lane
    // phases of 8-byte shared loads (and 32-lane 4-byte ones) rarely share
    // a bank
    const int lx = 8 * (warp & 1) + 4 * (lane >> 4) + (lane & 3);
    const int ly = 4 * (warp >> 1) + ((lane >> 2) & 3);
    const int x = cur.bx * TX + lx, y = cur.by * TY + ly;
    const bool active = x < g.nx && y < g.ny;
    // the column's offset from the tile centre (exact: a few voxel pitches)
    const float dx = static_cast<float>((lx - 0.5 * (TX - 1)) * g.vx);
    const float dy = static_cast<float>((ly - 0.5 * (TY - 1)) * g.vy);
    const float vz = static_cast<float>(g.vz);
    float acc[ZC];
#pragma unroll
    for (int i = 0; i < ZC; ++i) acc[i] = 0.f;
    bool bad = false;

    for (int k = cur.k; k < cur.k1; ++k) {
        const int s = pipe.s;
        // the warp leaves together: a lane whose wait ran out takes its whole
        // warp with it, so no lane is left waiting at a warp barrier below
        if (!__all_sync(0xffffffffu, mbar_wait(&sm.full[s], pipe.phase, pw.limit_ns))) {
            if (lane == 0) {
                atomicOr(err, kErrTimeout);
                *(volatile int*)sm.abort_flag = 1;
            }
            return false;
        }
        // this warp's turn to prepare the view that will refill the stage?
        // Its slot's last view is kSlots - stages >= stages views back, so every
        // warp has read it (they are at most a ring apart)
        const uint32_t next = (pipe.q + static_cast<uint32_t>(stages)) & (kSlots - 1);
        if (static_cast<uint32_t>(warp) == next)
            hold_view<PAIR, PSEUDO>(sm, pipe.ahead, sc, coef, pseudo, g, static_cast<int>(next));
        cursor_next(pipe.ahead, sc);

        constexpr bool COLUMN64 = AXIAL && (!PAIR || PSEUDO);
        const TileTerms& T = sm.terms[pipe.q & (kSlots - 1)];
        const float4 tu = *reinterpret_cast<const float4*>(&T.uc);
        const float4 tv = *reinterpret_cast<const float4*>(&T.vc);
        const float4 td = *reinterpret_cast<const float4*>(&T.dc);
        const float4 tp = *reinterpret_cast<const float4*>(&T.p0);
        const uint32_t S = smem_addr(sm.ring + static_cast<size_t>(s) * sm.stage_floats);
        const float den = fmaf(td.z, dy, fmaf(td.y, dx, td.x));
        const float nu0 = fmaf(tu.z, dy, tu.y * dx), nv0 = fmaf(tv.z, dy, tv.y * dx);
        float w;
        float q2 = 1.f, rz0 = 0.f;  // pseudo: squared horizontal distance, height of slice 0
        if constexpr (PSEUDO) {
            const float rx = dx + tp.x, ry = dy + tp.y;
            q2 = fmaf(rx, rx, ry * ry);
            rz0 = tp.z;
            w = tp.w;
        } else {
            const float rp = rcp_approx(fmaf(tp.z, dy, fmaf(tp.y, dx, tp.x)));
            w = tp.w * rp * rp;
        }
        const f2 M2 = f2pack(kFloorMagic, kFloorMagic);
        if constexpr (AXIAL) {
            float u, vb, vs;
            if constexpr (COLUMN64) {
                const int4 b = sm.copies[pipe.q & (kSlots - 1)];
                const ColumnTerms c = column_terms<PSEUDO>(coef[k], PSEUDO ? pseudo + k : nullptr,
                    g.ox + x * g.vx, g.oy + y * g.vy, g.oz + cur.za * g.vz, g.vz, b.x, b.y);
                u = c.u; vb = c.vb; vs = c.vs; w = c.w; q2 = c.q2; rz0 = c.rz0;
            } else {
                float rd = rcp_approx(den);
                rd = fmaf(rd, fmaf(-den, rd, 1.f), rd);  // one Newton step: vs walks ZC slices
                u = fmaf(nu0, rd, tu.x);
                vb = fmaf(nv0, rd, tv.x);
                vs = tv.w * rd;
            }
            const float fu = floorf(u);
            int col = static_cast<int>(fu);
            float au = u - fu;
            // every tap inside the staged box (it holds the detector's values,
            // zero outside the detector); |v| < 2^21 keeps the floor exact.
            // The rows lie between those of the column's ends (monotonic)
            const float ve = fmaf(static_cast<float>(ZC - 1), vs, vb);
            const int na = floor_row(vb), nb = floor_row(ve);
            const bool inside = fabsf(u) < 1e6f && fabsf(vb) < 1e6f && fabsf(vs) < 3e4f &&
                fabsf(w) < 1e30f && q2 > 0.f && col >= 0 && col <= BW - 2 && min(na, nb) >= 0 &&
                max(na, nb) < rows;
            if (!active || !inside) {
                if (active) bad = true;
                // no contribution; every read stays at the stage origin
                w = 0.f; au = 0.f; vs = 0.f; vb = 0.f;
                col = 0;
                q2 = 1.f; rz0 = 0.f;
            }
            // byte address of row pair n, column col: n row_bytes + base, n
            // from the floor word (wrapping 32-bit arithmetic)
            const uint32_t base = S + ES * static_cast<uint32_t>(col) - row_bytes * kFloorMagicBits;
            // the column's horizontal weights, with the view weight folded in
            const float w1 = w * au, w0 = w - w1;
#pragma unroll
            for (int j = 0; j < ZC / 2; ++j) {
                const f2 v2 = f2pack(fmaf(2.f * j, vs, vb), fmaf(2.f * j + 1.f, vs, vb));
                const f2 t2 = f2add_rm(v2, M2);
                float t[2], f[2];
                f2unpack(t2, t[0], t[1]);
                f2unpack(f2sub(v2, f2sub(t2, M2)), f[0], f[1]);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float ml, dl, mr, dr;
                    load_taps<PAIR>(__float_as_uint(t[e]) * row_bytes + base, row_bytes, ml, dl, mr, dr);
                    const float l = fmaf(f[e], dl, ml), r = fmaf(f[e], dr, mr);
                    float& a = acc[2 * j + e];
                    if constexpr (PSEUDO) {
                        const float rz = fmaf(2.f * j + e, vz, rz0);
                        a = fmaf(sqrt_approx(fmaf(rz, rz, q2)), fmaf(w1, r, w0 * l), a);
                    } else {
                        a = fmaf(w1, r, fmaf(w0, l, a));
                    }
                }
            }
        } else {
            // end points: u and v are monotonic along the column (den > 0); a
            // hundredth of a pixel covers the rounding between them
            const float dene = fmaf(static_cast<float>(ZC - 1), td.w, den);
            const float ra = rcp_approx(den), re = rcp_approx(dene);
            const float ua = fmaf(nu0, ra, tu.x), va = fmaf(nv0, ra, tv.x);
            const float ue = fmaf(fmaf(static_cast<float>(ZC - 1), tu.w, nu0), re, tu.x);
            const float ve = fmaf(fmaf(static_cast<float>(ZC - 1), tv.w, nv0), re, tv.x);
            const bool inside = den > 0.f && dene > 0.f && fminf(ua, ue) >= 0.01f &&
                fmaxf(ua, ue) <= static_cast<float>(BW - 1) - 0.01f && fminf(va, ve) >= 0.01f &&
                fmaxf(va, ve) <= static_cast<float>(rows) - 0.01f && fabsf(w) < 1e30f && q2 > 0.f;
            float d0 = den, d1 = td.w, u0 = nu0, u1 = tu.w, uc = tu.x, v0 = nv0, v1 = tv.w, vc = tv.x;
            if (!active || !inside) {
                if (active) bad = true;
                // no contribution; every read stays at the stage origin
                w = 0.f; d0 = 1.f; d1 = 0.f; u0 = u1 = uc = v0 = v1 = vc = 0.f;
                q2 = 1.f; rz0 = 0.f;
            }
            const uint32_t base = S - (row_bytes + ES) * kFloorMagicBits;
#pragma unroll
            for (int i = 0; i < ZC; ++i) {
                const float fi = static_cast<float>(i);
                const float di = fmaf(fi, d1, d0);
                float rd = rcp_approx(di);
                const f2 uv = f2pack(fmaf(fmaf(fi, u1, u0), rd, uc), fmaf(fmaf(fi, v1, v0), rd, vc));
                const f2 t2 = f2add_rm(uv, M2);
                float tu_, tv_, au, av;
                f2unpack(t2, tu_, tv_);
                f2unpack(f2sub(uv, f2sub(t2, M2)), au, av);
                float ml, dl, mr, dr;
                load_taps<PAIR>(__float_as_uint(tv_) * row_bytes + __float_as_uint(tu_) * ES + base,
                    row_bytes, ml, dl, mr, dr);
                const float l = fmaf(av, dl, ml), r = fmaf(av, dr, mr);
                float wi = w;
                if constexpr (PSEUDO) {
                    rd = fmaf(rd, fmaf(-di, rd, 1.f), rd);
                    const float rz = fmaf(fi, vz, rz0);
                    wi = w * sqrt_approx(fmaf(rz, rz, q2)) * (rd * rd * rd);
                }
                acc[i] = fmaf(wi, fmaf(au, r - l, l), acc[i]);
            }
        }
        // the last warp to finish with the stage refills it.  The count is
        // taken with acquire-release order after the whole warp's reads, and
        // the proxy fence orders them before the copy's writes
        __syncwarp();
        if (lane == 0) {
            uint32_t before;
            asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;"
                         : "=r"(before) : "r"(smem_addr(&sm.done[s])) : "memory");
            if ((before & (NWARPS - 1)) == NWARPS - 1) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                issue_copy<PAIR>(sm, map, static_cast<int>(next), s, box_bytes, pw.withheld_view);
            }
        }
        __syncwarp();
        ++pipe.q;
        if (++pipe.s == stages) { pipe.s = 0; pipe.phase ^= 1u; }
    }
    if (bad) atomicOr(err, kErrFootprint);
    if (!active) return true;
    const long plane = static_cast<long>(g.nx) * g.ny;
    float* dst = vol + (cur.job / sc.n_tiles) * sc.part_floats + static_cast<long>(y) * g.nx + x;
#pragma unroll
    for (int i = 0; i < ZC; ++i) {
        const int z = cur.za + i;
        if (z < g.nz) {
            // ACC: a reduction in L2 (each voxel has this one writer, so the
            // sum is the plain old + acc): no load round trip per value
            if constexpr (ACC) atomicAdd(dst + z * plane, acc[i]);
            else dst[z * plane] = acc[i];
        }
    }
    return true;
}

// Persistent: one CTA of 16 warps per SM walks jobs blockIdx.x, +gridDim.x,
// ...; the ring runs on across them, so a tile costs no pipeline fill of its
// own.
// ACC: add to the volume instead of writing it (a separate kernel, so that
// the write-only form's registers are not shaped by the reductions)
template <bool AXIAL, bool PAIR, bool PSEUDO, bool ACC>
__global__ void __launch_bounds__(NTHREADS, 1) fdk_bp_tma_kernel(const __grid_constant__ CUtensorMap map,
    const FdkViewCoef* __restrict__ coef, const __grid_constant__ VolumeGrid g, int BW, int BH,
    int stages, float* __restrict__ vol, int* __restrict__ err,
    const PseudoViewCoef* __restrict__ pseudo, const __grid_constant__ Schedule sc, PipelineWait pw)
{
    const BpSmem sm = bp_smem(BW, BH, PAIR, stages);
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) {
        *sm.abort_flag = 0;
        *sm.issued = 0;
        if ((smem_addr(sm.full) & 7u) != 0 || (smem_addr(sm.ring) & 127u) != 0) {
            atomicOr(err, kErrAlign);
            *sm.abort_flag = 1;
        }
        for (int s = 0; s < stages; ++s) {
            mbar_init(&sm.full[s], 1);
            sm.done[s] = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    Pipe pipe;
    pipe.s = 0;
    pipe.phase = 0;
    pipe.q = 0;
    pipe.ahead.job = blockIdx.x;
    cursor_open(pipe.ahead, sc);
    for (int i = 0; i < stages; ++i) {
        if (warp == i) hold_view<PAIR, PSEUDO>(sm, pipe.ahead, sc, coef, pseudo, g, i);
        cursor_next(pipe.ahead, sc);
    }
    __syncthreads();
    if (*sm.abort_flag) return;
    if (tid == 0) {
        const uint32_t box_bytes = static_cast<uint32_t>(BW * BH * (PAIR ? 8 : 4));
        for (int i = 0; i < stages; ++i)
            issue_copy<PAIR>(sm, &map, i, i, box_bytes, pw.withheld_view);
    }
    bool ok = true;
    for (Cursor cur{static_cast<long>(blockIdx.x), 0, 0, 0, 0, 0, false}; ok && cur.job < sc.n_jobs;
         cur.job += gridDim.x) {
        cursor_open(cur, sc);
        ok = cur.main
            ? bp_job<AXIAL, PAIR, PSEUDO, ZT, ACC>(sm, &map, coef, pseudo, g, sc, BW, BH, stages,
                  vol, err, pw, cur, pipe)
            : bp_job<AXIAL, PAIR, PSEUDO, kZTail, ACC>(sm, &map, coef, pseudo, g, sc, BW, BH,
                  stages, vol, err, pw, cur, pipe);
    }
    // after a timeout: every issued copy must land before the CTA exits
    __syncthreads();
    if (tid == 0 && *(volatile int*)sm.abort_flag) {
        const int issued = *(volatile int*)sm.issued;
        for (int q = max(0, issued - stages); q < issued; ++q)
            if (sm.copies[q & (kSlots - 1)].z != pw.withheld_view)
                mbar_wait(&sm.full[q % stages], static_cast<uint32_t>(q / stages) & 1u);
    }
}

// out[i] (+)= the sum of the splits' parts, in order (HBM and L2 traffic; the
// parts are `stride` floats apart, a multiple of 4; vec: out is 16-byte
// aligned).
__global__ void __launch_bounds__(256) sum_parts_kernel(const float* __restrict__ parts, int splits,
    long stride, long n, int vec, float* __restrict__ out, int accumulate)
{
    const long step = static_cast<long>(gridDim.x) * blockDim.x;
    const long first = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
    const long n4 = vec ? n / 4 : 0;
    for (long i = first; i < n4; i += step) {
        float4 a = accumulate ? reinterpret_cast<const float4*>(out)[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        for (int s = 0; s < splits; ++s) {
            const float4 b = __ldcs(reinterpret_cast<const float4*>(parts + s * stride) + i);
            a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
        }
        reinterpret_cast<float4*>(out)[i] = a;
    }
    for (long i = 4 * n4 + first; i < n; i += step) {
        float a = accumulate ? out[i] : 0.f;
        for (int s = 0; s < splits; ++s) a += __ldcs(parts + s * stride + i);
        out[i] = a;
    }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
    static std::once_flag once;
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
                cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// Staged box widths (elements): 8 mod 16, so a row of row pairs is 64 mod 128
// bytes: the 16 lanes of a half-warp, whose footprints span a few columns and
// at most a row or two, then rarely meet on one bank (a pitch of 32 mod 128
// bytes put rows n and n + 1 four elements apart on the same banks: 16 % more
// shared-memory wavefronts, measured).  Four narrower where that buys a third
// stage (1081 vs 1491 ms on the 1024^3 x 1440 workload when its 52-wide box
// had 3 stages or 56-wide 2).
int stages_of(int bw, int bh, bool pair)
{
    const size_t stage = static_cast<size_t>(stage_stride_floats(bw, bh, pair)) * sizeof(float);
    const int s = static_cast<int>(kRingBudget / std::max<size_t>(stage, 1));
    return s >= 2 ? std::min(s, kMaxStages) : 0;
}

int staged_width(int w, int bh, bool pair)
{
    const int wide = (w + 7) / 16 * 16 + 8;
    if (wide > 256 || bh > 256) return 0;
    if (wide - 4 >= w && stages_of(wide, bh, pair) < 3 && stages_of(wide - 4, bh, pair) >= 3)
        return wide - 4;
    return wide;
}

// z tiling: ZT-slice tiles, except that a remainder of at most kZTail
// slices becomes one kZTail-slice tile instead of a ZT-slice tile that is
// mostly outside the volume.
Schedule tile_schedule(const VolumeGrid& g, int n_views)
{
    const int rem = g.nz % ZT;
    const bool tail = rem > 0 && rem <= kZTail;
    Schedule sc{};
    sc.main_layers = tail ? g.nz / ZT : (g.nz + ZT - 1) / ZT;
    sc.tiles_x = (g.nx + TX - 1) / TX;
    sc.tiles_y = (g.ny + TY - 1) / TY;
    sc.n_tiles = static_cast<long>(sc.tiles_x) * sc.tiles_y * (sc.main_layers + (tail ? 1 : 0));
    sc.n_views = n_views;
    sc.splits = 1;
    sc.n_jobs = sc.n_tiles;
    return sc;
}

// floats of one split's sums: the volume's, to a multiple of four
size_t part_stride(const VolumeGrid& g)
{
    return (static_cast<size_t>(g.nx) * g.ny * g.nz + 3) / 4 * 4;
}

// Splits of the views that finish a launch soonest: jobs run in rounds of one
// per SM, a job takes its views plus about two views' time to fill the ring
// and write its sums, and the splits' sums cost a launch (4 us) and a write and
// a read (4 TB/s).  In units of a tile's view, 3 us.  64^3 x 60 views, 8 tiles:
// 20 us in 18 splits, 171 in one; 128^3 x 180, 64 tiles: 257 and 503 us;
// 256^3, 512 tiles, four rounds of 148 SMs for 3.5 rounds of work: 7 half
// rounds; from about 20 rounds on, one split.
int split_count(long n_tiles, int n_views, int sms, size_t floats, size_t part_floats)
{
    const long most = std::min<long>({static_cast<long>(part_floats / std::max<size_t>(floats, 1)),
        static_cast<long>(n_views), 64L});
    int best = 1;
    double best_cost = 0.0;
    for (int s = 1; s <= std::max(most, 1L); ++s) {
        const double rounds = static_cast<double>((n_tiles * s + sms - 1) / sms);
        double cost = rounds * ((n_views + s - 1) / s + 2.0);
        if (s > 1) cost += (4e-6 + 4.0 * (2 * s + 2) * static_cast<double>(floats) / 4e12) / 3e-6;
        if (s == 1 || cost < best_cost) {
            best = s;
            best_cost = cost;
        }
    }
    return best;
}

cudaError_t sm_count(int* sms)
{
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    return e != cudaSuccess ? e : cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, device);
}

template <bool AXIAL, bool PAIR, bool PSEUDO, bool ACC>
cudaError_t launch_form(const CUtensorMap& map, const FdkViewCoef* coef, const VolumeGrid& g,
    int bw, int bh, float* vol, int* err, const PseudoViewCoef* pseudo, const Schedule& sc, int sms,
    PipelineWait pw, cudaStream_t s)
{
    const int stages = stages_of(bw, bh, PAIR);
    if (stages == 0) return cudaErrorInvalidConfiguration;
    const size_t smem = 128 + kBpTables +
        static_cast<size_t>(stage_stride_floats(bw, bh, PAIR)) * sizeof(float) * stages;
    auto k = fdk_bp_tma_kernel<AXIAL, PAIR, PSEUDO, ACC>;
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
        static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    // one persistent CTA per SM (the ring takes most of its shared memory)
    const unsigned grid = static_cast<unsigned>(std::min<long>(sc.n_jobs, sms));
    k<<<grid, NTHREADS, smem, s>>>(map, coef, g, bw, bh, stages, vol, err, pseudo, sc, pw);
    return cudaGetLastError();
}

template <bool AXIAL, bool PAIR, bool PSEUDO>
cudaError_t launch_jobs(const CUtensorMap& map, const FdkViewCoef* coef, const VolumeGrid& g,
    int bw, int bh, float* vol, int accumulate, int* err, const PseudoViewCoef* pseudo, float* parts,
    size_t part_floats, Schedule sc, PipelineWait pw, cudaStream_t s)
{
    int sms = 0;
    cudaError_t e = sm_count(&sms);
    if (e != cudaSuccess) return e;
    const size_t floats = part_stride(g);
    sc.splits = split_count(sc.n_tiles, sc.n_views, sms, floats, parts ? part_floats : 0);
    sc.n_jobs = sc.n_tiles * sc.splits;
    if (sc.splits == 1)
        return accumulate
            ? launch_form<AXIAL, PAIR, PSEUDO, true>(map, coef, g, bw, bh, vol, err, pseudo, sc, sms, pw, s)
            : launch_form<AXIAL, PAIR, PSEUDO, false>(map, coef, g, bw, bh, vol, err, pseudo, sc, sms, pw, s);
    sc.part_floats = static_cast<long>(floats);
    e = launch_form<AXIAL, PAIR, PSEUDO, false>(map, coef, g, bw, bh, parts, err, pseudo, sc, sms, pw, s);
    if (e != cudaSuccess) return e;
    const int vec = reinterpret_cast<uintptr_t>(vol) % 16 == 0;
    const long n = static_cast<long>(g.nx) * g.ny * g.nz;
    sum_parts_kernel<<<static_cast<unsigned>(std::min<long>((floats / 4 + 255) / 256, sms * 8)), 256, 0, s>>>(
        parts, sc.splits, sc.part_floats, n, vec, vol, accumulate);
    return cudaGetLastError();
}

} // namespace

// Largest tile box over all views and tiles as row pairs and as plain rows (a
// width of 0: it does not fit the copy or the ring).
cudaError_t fdk_tma_box(const FdkViewCoef* coef, int n_views, const VolumeGrid& g, int* scratch3,
    FdkTmaBox* box, cudaStream_t s)
{
    *box = FdkTmaBox{};
    cudaError_t e = cudaMemsetAsync(scratch3, 0, 3 * sizeof(int), s);
    if (e != cudaSuccess) return e;
    const int tx = (g.nx + TX - 1) / TX, ty = (g.ny + TY - 1) / TY, tz = (g.nz + ZT - 1) / ZT;
    box_extent_kernel<<<1184, 256, 0, s>>>(coef, n_views, g, tx, ty, tz, scratch3);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    int host[3] = {0, 0, 0};
    if ((e = cudaMemcpyAsync(host, scratch3, sizeof host, cudaMemcpyDeviceToHost, s)) != cudaSuccess)
        return e;
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
    box->pair_h = host[2];
    box->row_h = host[2] + 1;
    const auto fit = [](int w, int h, bool pair) {
        const int bw = w > 256 ? 0 : staged_width(w, h, pair);
        return bw > 0 && stages_of(bw, h, pair) > 0 ? bw : 0;
    };
    box->pair_w = fit(host[0], box->pair_h, true);
    box->row_w = fit(host[1], box->row_h, false);
    return cudaSuccess;
}

int fdk_tma_z_tile() { return ZT; }

bool fdk_tma_available() { return encode_fn() != nullptr; }

size_t fdk_tma_part_floats(const VolumeGrid& g, int n_views)
{
    int sms = 0;
    if (sm_count(&sms) != cudaSuccess) return 0;
    const size_t floats = part_stride(g);
    const int splits = split_count(tile_schedule(g, n_views).n_tiles, n_views, sms, floats,
        (size_t(256) << 20) / sizeof(float));
    return splits > 1 ? floats * splits : 0;
}

cudaError_t launch_fdk_backproject_tma(const float* filtered, int layout, int ld,
    const FdkViewCoef* coef, int n_views, int nu, int nv, const VolumeGrid& g, bool axial,
    const FdkTmaBox& box, float* vol, int accumulate, int* err, float* parts, size_t part_floats,
    cudaStream_t s, const PseudoViewCoef* pseudo, PipelineWait pw)
{
    auto enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    const bool pair = layout == kFilteredPairs;
    const int bw = pair ? box.pair_w : box.row_w, bh = pair ? box.pair_h : box.row_h;
    if (bw == 0 || (pseudo && !pair)) return cudaErrorInvalidValue;
    const size_t esz = pair ? 8 : 4;  // a row pair's column moves as one 8-byte element
    const int rows = pair ? nv + 1 : nv;
    CUtensorMap map;
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(nu), static_cast<cuuint64_t>(rows),
                                static_cast<cuuint64_t>(n_views)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld) * esz,
                                   static_cast<cuuint64_t>(ld) * rows * esz};
    const cuuint32_t tile[3] = {static_cast<cuuint32_t>(bw), static_cast<cuuint32_t>(bh), 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = enc(&map,
        pair ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
        const_cast<float*>(filtered), dims, strides, tile, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    const Schedule sc = tile_schedule(g, n_views);
    const auto launch = pseudo ? (axial ? launch_jobs<true, true, true> : launch_jobs<false, true, true>)
        : pair ? (axial ? launch_jobs<true, true, false> : launch_jobs<false, true, false>)
               : (axial ? launch_jobs<true, false, false> : launch_jobs<false, false, false>);
    return launch(map, coef, g, bw, bh, vol, accumulate, err, pseudo, parts, part_floats, sc, pw, s);
}

// Plain rows [views][nv][ld_in] -> row pairs [views][nv + 1][ldp], the layout
// the filter epilogue writes directly: row r of a view holds
// (f[r - 1][u], f[r][u] - f[r - 1][u]), rows outside the detector zero.
__global__ void __launch_bounds__(256) pairify_kernel(const float* __restrict__ in, int ld_in,
    long views, int nu, int nv, float2* __restrict__ out, int ldp)
{
    const long rows = views * (nv + 1);
    for (long r = blockIdx.x; r < rows; r += gridDim.x) {
        const long view = r / (nv + 1);
        const int n = static_cast<int>(r - view * (nv + 1)) - 1;
        const float* row = in + (view * nv + n) * ld_in;
        for (int u = threadIdx.x; u < nu; u += blockDim.x) {
            const float a = n >= 0 ? row[u] : 0.f;
            const float b = n + 1 < nv ? row[ld_in + u] : 0.f;
            out[r * ldp + u] = make_float2(a, b - a);
        }
    }
}

cudaError_t launch_fdk_pairify(const float* in, int ld_in, long views, int nu, int nv, float* out,
    int ldp, cudaStream_t s)
{
    if (views <= 0) return cudaSuccess;
    const long rows = views * (nv + 1);
    pairify_kernel<<<static_cast<unsigned>(std::min<long>(rows, 148 * 64)), 256, 0, s>>>(in, ld_in,
        views, nu, nv, reinterpret_cast<float2*>(out), ldp);
    return cudaGetLastError();
}

} // namespace ykb
