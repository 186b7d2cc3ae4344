// ivr_march.cu -- the per-ray march: ray setup, slab test, sample lattice,
// trilinear reconstruction, transfer function, brick compositing, RGBA
// stores.  One thread per ray; a warp covers an 8x4 screen tile.
//
// Compiled with -fmad=false: every float multiply and add is rounded on its
// own, as in the reference's C, unless written as fmaf() here.  With IEEE
// division and square root (no fast-math) the REF preset reproduces the
// reference's arithmetic operation for operation.
#include <float.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>

#include "ivr_internal.h"

namespace ivr {
namespace {

constexpr int kBlockX = 16;  // pixels per block: 2x2 warps of 8x4
constexpr int kBlockY = 8;
constexpr int kThreads = 128;
// Samples of a ray that one loop iteration takes (K), all their loads in
// flight before the first is composited, and resident blocks per SM each
// kernel is compiled for (65,536 / (128 blocks) registers a thread).  A
// launch is bound by the latency of its longest rays as much as by its
// throughput, so loads in flight within a thread are worth more than warps
// beside it.  Measured on GB300 (us a frame at K = 2, 4, 6, 8 with 5 blocks,
// the start of the sweep K = 2 with 9 blocks): u16 learned 1024^3 at
// 1920x1080 462, 368, 341, 368 (556); u16 without skipping 266, 218, 198,
// 200 (368); u8 128^3 at 256x256 69, 56, 51, 51 (80); f32 (four registers a
// voxel pair) 512^3 at 1024x1024 392, 342, 357, 352 (395); with the edges
// clamped as they are now learned 328 and 356 at K = 6 and 8, f32 333 and 351
// at K = 4 and 6.  The batched
// kernel reads its frames from global memory and has no tail: there more
// warps win (32 f32 frames of a 512^3 volume: 3.67 ms at K = 2 with 8 blocks,
// 3.74 with 9, 3.92 with 7; 20 u16 frames 2.53 ms at K = 4 with 8, 3.06 with
// 7, 2.72 with 6, 2.88 at K = 2 with 9; u8 2.40, 2.37, 2.52, 2.59).
#ifndef IVR_K_INT
#define IVR_K_INT 6
#endif
#ifndef IVR_K_F32
#define IVR_K_F32 4
#endif
#ifndef IVR_CFG_BLOCKS_PER_SM
#define IVR_CFG_BLOCKS_PER_SM 5
#endif
template <int DT> __host__ __device__ constexpr int cfg_k() { return DT == IVR_F32 ? IVR_K_F32 : IVR_K_INT; }
constexpr int kCfgBlocksPerSm = IVR_CFG_BLOCKS_PER_SM;
// Launches without any grid take their samples in packed pairs, six at a time
// for every type (us a frame of a 301x260x223 volume, 4, 6, 8 samples: u16
// 853x479 202, 182, 194 against 186 unpacked; f32 1024x1024 560, 535, 553
// against 572; u8 1024x1024 472 against 497).  With a grid, packing loses: its
// pairs cost the run loop registers (u16 learned 341 -> 383, the batched
// kernel 3.85 -> 3.91 ms).
constexpr int kPlainK = 6;
template <int DT> __host__ __device__ constexpr int batch_k() { return DT == IVR_F32 ? 2 : 4; }
constexpr int kBatchBlocksPerSm = 8;
constexpr int kPeakBlocksPerSm = 9;  // the sampler alone (sample_peak_kernel)

template <int DT> struct VoxT;
template <> struct VoxT<IVR_U8> { using T = uint8_t; using V4 = uchar4; };
template <> struct VoxT<IVR_U16> { using T = uint16_t; using V4 = ushort4; };
template <> struct VoxT<IVR_F32> { using T = float; using V4 = float4; };

template <int DT>
__device__ __forceinline__ float vload(const void *p, long long i)
{
    return (float) __ldg(reinterpret_cast<const typename VoxT<DT>::T *>(p) + i);
}

// getrayintersect (ray.c:276-318).  All six planes are visited: once
// tin >= tout no later plane can make it a hit, so skipping the reference's
// early loop exit changes nothing.
// numer = d - n.o and denom = n.d for face p (normals of aabb.facenormals,
// main.c:611-613), evaluated as dot3f does.
__device__ __forceinline__ void plane_eval(int p, float dc, float ox, float oy, float oz, float dx, float dy,
                                           float dz, float &numer, float &denom)
{
    const int axis = p >> 1;
    const float nrm = (p & 1) ? 1.0f : -1.0f;
    const float nx = axis == 0 ? nrm : 0.0f, ny = axis == 1 ? nrm : 0.0f, nz = axis == 2 ? nrm : 0.0f;
    numer = dc - (nx * ox + ny * oy + nz * oz);
    denom = nx * dx + ny * dy + nz * dz;
}

__device__ __forceinline__ bool ray_box(const float *dc, float ox, float oy, float oz, float dx, float dy,
                                        float dz, float &tin, float &tout)
{
    tin = -FLT_MAX;
    tout = FLT_MAX;
#pragma unroll
    for (int p = 0; p < 6; p++) {
        float numer, denom;
        plane_eval(p, dc[p], ox, oy, oz, dx, dy, dz, numer, denom);
        if (tin < tout) {
            if (denom == 0.0f) {
                if (numer < 0.0f) tin = tout + 1.0f;
            } else {
                float thit = numer / denom;
                if (denom > 0.0f) tout = fminf(tout, thit);
                else tin = fmaxf(tin, thit);
            }
        }
    }
    return tin < tout && (tin > 0.0f || tout > 0.0f);
}

// The CONFIG slab test: ray_box's planes and visiting order, with each hit
// parameter taken as +-numer times the ray's reciprocal direction component
// (id*) instead of a division -- the CONFIG lattice's own definition; the
// REF preset keeps the reference's division.  For the axis-aligned normals
// numer = d -+ o and denom = +-d exactly, so only the rounding of the hit
// parameters differs from ray_box.
__device__ __forceinline__ bool ray_box_cfg(const float *dc, float ox, float oy, float oz, float dx, float dy,
                                            float dz, float idx, float idy, float idz, float &tin, float &tout)
{
    tin = -FLT_MAX;
    tout = FLT_MAX;
#pragma unroll
    for (int p = 0; p < 6; p++) {
        const int axis = p >> 1;
        const bool pos = (p & 1) != 0;
        const float o = axis == 0 ? ox : axis == 1 ? oy : oz;
        const float d = axis == 0 ? dx : axis == 1 ? dy : dz;
        const float id = axis == 0 ? idx : axis == 1 ? idy : idz;
        const float numer = pos ? dc[p] - o : dc[p] + o;
        if (tin < tout) {
            if (d == 0.0f) {
                if (numer < 0.0f) tin = tout + 1.0f;
            } else {
                const float thit = (pos ? numer : -numer) * id;
                if (pos ? d > 0.0f : d < 0.0f) tout = fminf(tout, thit);
                else tin = fmaxf(tin, thit);
            }
        }
    }
    return tin < tout && (tin > 0.0f || tout > 0.0f);
}

// getlinearsample (ray.c:87-181, non-BGQ branch), quirks included: the
// weights are scaled by the cell size squared, and the x weight blends the
// +1 row (y) neighbour.  x + fabs(min.x) is a double sum in the reference,
// which rounds to the same float as this float sum.
template <int DT>
__device__ __forceinline__ float sample_ref(const DevBrick &b, float x, float y, float z)
{
    const int vw = b.nx, vh = b.ny, vd = b.nz;
    float ratio = (x - b.bminx) / b.w;
    int j = (int) ((float) vw * ratio);
    ratio = (y - b.bminy) / b.h;
    int i = (int) ((float) vh * ratio);
    ratio = (z - b.bminz) / b.d;
    int k = (int) ((float) vd * ratio);
    i = min(i, vh - 2);
    j = min(j, vw - 2);
    k = min(k, vd - 2);
    i = max(i, 0);  // no lower clamp in the reference; guards memory only
    j = max(j, 0);
    k = max(k, 0);
    const long long row = vw, slab = (long long) vw * vh;
    const long long p = k * slab + i * row + j;
    float v000 = vload<DT>(b.data, p);
    float v100 = vload<DT>(b.data, p + row);
    float v010 = vload<DT>(b.data, p + 1);
    float v001 = vload<DT>(b.data, p + slab);
    float v101 = vload<DT>(b.data, p + row + slab);
    float v011 = vload<DT>(b.data, p + 1 + slab);
    float v110 = vload<DT>(b.data, p + row + 1);
    float v111 = vload<DT>(b.data, p + row + 1 + slab);
    float xp = x + fabsf(b.bminx), yp = y + fabsf(b.bminy), zp = z + fabsf(b.bminz);
    float x0 = ((float) j * b.w) / (float) vw;
    float y0 = ((float) i * b.h) / (float) vh;
    float z0 = ((float) k * b.d) / (float) vd;
    float xd = (fabsf(xp - x0) * b.w) / (float) vw;
    float yd = (fabsf(yp - y0) * b.h) / (float) vh;
    float zd = (fabsf(zp - z0) * b.d) / (float) vd;
    float c00 = v000 * (1.0f - xd) + v100 * xd;
    float c10 = v010 * (1.0f - xd) + v110 * xd;
    float c01 = v001 * (1.0f - xd) + v101 * xd;
    float c11 = v011 * (1.0f - xd) + v111 * xd;
    float c0 = c00 * (1.0f - yd) + c10 * yd;
    float c1 = c01 * (1.0f - yd) + c11 * yd;
    return c0 * (1.0f - zd) + c1 * zd;
}

// Two floats in one 64-bit register pair: sm_100's packed FP32 instructions
// do both operations in one issue slot.  The assembler contracts a packed
// product that only feeds a packed sum into one fma, whatever the rounding
// qualifiers and flags say (measured: 246,536 of 2^20 sums differ), so F2 has
// no product-then-sum: such steps stay scalar, where it does not.
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ void f2_split(F2 x, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

// x / c for a divisor fixed over a ray: h = 1/c rounded to nearest, l the
// rest of 1/c.  fmaf(x, h, x * l) is within one rounding of a relative 2^-46
// of the quotient, so it is one of its two float neighbours; the remainder of
// that is then exact in one fmaf, and adding it times h gives the quotient
// rounded to nearest (Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", 1990, theorem on the final division step;
// the two-word reciprocal is Brisebarre and Muller's, "Correctly rounded
// multiplication by arbitrary precision constants", 2008).  Both hold while
// nothing overflows, the quotient is normal and the remainder, a multiple of
// 2^-47 |x|, is no finer than floats are: for x = 0 and |x| in [2^-73, 2^98]
// with c in [2^-16, 2^40], which is what ref_fast lets through.
struct FixedDiv {
    F2 mc, h, l;  // -c, 1/c, the rest of 1/c, for both lanes
    __device__ __forceinline__ explicit FixedDiv(float d)
    {
        const float r = 1.0f / d;
        mc = f2(-d);
        h = f2(r);
        l = f2(fmaf(-d, r, 1.0f) * r);
    }
    __device__ __forceinline__ F2 operator()(F2 x) const
    {
        const F2 q = f2_fma(x, h, x * l);
        return f2_fma(f2_fma(q, mc, x), h, q);
    }
};

// Whether every division that sample_ref makes along the ray is one that
// FixedDiv rounds as IEEE division does.  The divisors are the brick's extents
// and dims.  The positions x = o + d t are compared with a brick edge and cell
// corners (at least 2^-32 where they are not 0); where the edge or o is at least
// 2^-30, the difference of two floats near each other is a multiple of the
// smaller one's last place, so it is 0 or at least 2^-57.  An edge at 0 (inner
// bricks) seen from o = 0 needs d t away from 0 as well.  The last division's
// dividend is such a difference times the extent: 2^-73 at least.  Positions are
// below 2^58 (t is at most 2^17), times an extent 2^98.
constexpr float kRefNear = 9.313225746154785e-10f, kRefFar = 1.099511627776e12f;  // 2^-30, 2^40
constexpr float kRefThin = 1.52587890625e-5f;                                     // 2^-16
constexpr int kRefDim = 1 << 16;
__device__ __forceinline__ bool ref_fast_axis(float o, float d, float bmin, float extent, int dim, float tin)
{
    if (!(fabsf(o) <= kRefFar && fabsf(d) <= kRefFar && extent >= kRefThin && extent <= kRefFar &&
          fabsf(bmin) <= kRefFar && dim <= kRefDim))
        return false;
    if (fabsf(bmin) >= kRefNear) return true;
    if (bmin != 0.0f) return false;
    if (fabsf(o) >= kRefNear) return true;
    return o == 0.0f && (d == 0.0f || (fabsf(d) >= kRefNear && tin >= 1.0e-6f));
}
__device__ __forceinline__ bool ref_fast(const FrameDesc &f, const DevBrick &b, float dx, float dy, float dz, float tin)
{
    return fabsf(tin) <= 65536.0f && ref_fast_axis(f.origx, dx, b.bminx, b.w, b.nx, tin) &&
           ref_fast_axis(f.origy, dy, b.bminy, b.h, b.ny, tin) && ref_fast_axis(f.origz, dz, b.bminz, b.d, b.nz, tin);
}

// A ray's REF sampler in one brick: sample_ref with its nine divisions, all
// by the brick's extents or dims, as FixedDivs, and (u8, u16) the eight
// voxels from the corner-packed copy in two loads.
struct RefSampler {
    FixedDiv w, h, d, nx, ny, nz;
    __device__ __forceinline__ explicit RefSampler(const DevBrick &b)
        : w(b.w), h(b.h), d(b.d), nx((float) b.nx), ny((float) b.ny), nz((float) b.nz)
    {
    }
};
// Two samples' cells and weights.
struct RefPos {
    int j[2], i[2], k[2];
    F2 xd, yd, zd;
};

// sample_ref's cell and weight along one axis, for two positions u: `inv` and
// `n` divide by the extent and the dim.  The weight's sign is left to the
// caller: rounding is symmetric, so its magnitude is the reference's.
__device__ __forceinline__ F2 ref_axis(F2 u, float bmin, float extent, int dim, const FixedDiv &inv, const FixedDiv &n,
                                       int (&cell)[2])
{
    float r0, r1;
    f2_split(f2((float) dim) * inv(u + f2(-bmin)), r0, r1);
    cell[0] = max(min((int) r0, dim - 2), 0);
    cell[1] = max(min((int) r1, dim - 2), 0);
    const F2 mu0 = n(f2((float) cell[0], (float) cell[1]) * f2(-extent));  // minus the cell's corner
    return n(((u + f2(fabsf(bmin))) + mu0) * f2(extent));
}

__device__ __forceinline__ RefPos ref_pos(const DevBrick &b, const RefSampler &r, F2 x, F2 y, F2 z)
{
    RefPos p;
    p.xd = ref_axis(x, b.bminx, b.w, b.nx, r.w, r.nx, p.j);
    p.yd = ref_axis(y, b.bminy, b.h, b.ny, r.h, r.ny, p.i);
    p.zd = ref_axis(z, b.bminz, b.d, b.nz, r.d, r.nz, p.k);
    return p;
}

// The cell's voxels as loaded: from the corner-packed copy (an f32 copy holds
// differences, which do not give the voxels back), or one by one.
template <int DT> struct RefCell {
    using E = typename VoxT<DT>::V4;
    E lo, hi;
};

template <int DT>
__device__ __forceinline__ RefCell<DT> ref_load(const DevBrick &b, int j, int i, int k)
{
    using V = typename VoxT<DT>::V4;
    using T = typename VoxT<DT>::T;
    RefCell<DT> c;
    if (DT != IVR_F32 && b.quad) {
        const unsigned qx = (unsigned) b.nx - 1u, qs = qx * ((unsigned) b.ny - 1u);
        const V *e = reinterpret_cast<const V *>(b.quad) + ((unsigned) k * qs + (unsigned) i * qx + (unsigned) j);
        c.lo = __ldg(e);
        c.hi = __ldg(e + qs);
    } else {
        const unsigned row = (unsigned) b.nx, slab = row * (unsigned) b.ny;
        const T *q = reinterpret_cast<const T *>(b.data) + ((unsigned) k * slab + (unsigned) i * row + (unsigned) j);
        c.lo.x = __ldg(q);
        c.lo.y = __ldg(q + 1);
        c.lo.z = __ldg(q + row);
        c.lo.w = __ldg(q + row + 1);
        c.hi.x = __ldg(q + slab);
        c.hi.y = __ldg(q + slab + 1);
        c.hi.z = __ldg(q + slab + row);
        c.hi.w = __ldg(q + slab + row + 1);
    }
    return c;
}

// sample_ref's blend, operation for operation (the x weight blends the +1
// row)
template <int DT>
__device__ __forceinline__ float ref_interp(const RefCell<DT> &c, float xd, float yd, float zd)
{
    const float v000 = (float) c.lo.x, v010 = (float) c.lo.y, v100 = (float) c.lo.z, v110 = (float) c.lo.w;
    const float v001 = (float) c.hi.x, v011 = (float) c.hi.y, v101 = (float) c.hi.z, v111 = (float) c.hi.w;
    const float xe = 1.0f - xd, ye = 1.0f - yd, ze = 1.0f - zd;
    const float c00 = v000 * xe + v100 * xd;
    const float c10 = v010 * xe + v110 * xd;
    const float c01 = v001 * xe + v101 * xd;
    const float c11 = v011 * xe + v111 * xd;
    const float c0 = c00 * ye + c10 * yd;
    const float c1 = c01 * ye + c11 * yd;
    return c0 * ze + c1 * zd;
}

__device__ __forceinline__ float lerpf(float a, float b, float t) { return fmaf(t, b - a, a); }

// CONFIG sampler: trilinear with voxel values at cell corners (the
// reference's index convention; the halo sits on the high side), clamp to
// edge, at a position (ux, uy, uz) in the brick's voxel coordinates (voxel
// (j, i, k) at u = (j, i, k)).  Split in two so that the march's macrocell
// check can use the cell coordinates of the sample it is about to take.
struct CellPos {
    int j, i, k;         // voxel cell, clamped to [0, n-2]
    float fx, fy, fz;    // position in it, [0, 1]
};

__device__ __forceinline__ CellPos cell_cfg(const DevBrick &b, float ux, float uy, float uz)
{
    const int nx = b.nx, ny = b.ny, nz = b.nz;
    // clamp to edge: the cell to [0, n-2] (the conversion takes what is
    // negative to 0), the fraction to [0, 1] by the subtraction's saturation.
    // u - floor(u) is exact, so this is the cell and the fraction of the
    // coordinate clamped to [0, n-1] first, without the clamps' six
    // instructions (f32 512^3 frame 347 -> 333 us, learned 1024^3 340 -> 328,
    // u8 128^3 26.4 -> 25.0).  n is at least 2.
    CellPos c;
    c.j = (int) min(__float2uint_rd(ux), (unsigned) (nx - 2));
    c.i = (int) min(__float2uint_rd(uy), (unsigned) (ny - 2));
    c.k = (int) min(__float2uint_rd(uz), (unsigned) (nz - 2));
    c.fx = __saturatef(ux - (float) c.j);
    c.fy = __saturatef(uy - (float) c.i);
    c.fz = __saturatef(uz - (float) c.k);
    return c;
}

// Packed integer voxels without conversion instructions (which run on a
// narrow pipe; eight per sample made the u8/u16 corner-packed sampler
// conversion-bound): a u8 or u16 lane placed in the low mantissa bits under
// the exponent of 2^23 is the float 2^23 + v, exactly.  lerp23 is lerpf on
// two such values: B - A is b - a and A - 2^23 is a, both exact, so the
// result is lerpf(a, b, t) bit for bit.  (For the brick's own voxels, one
// load each, the conversion is cheaper than the permute and the offset.)
__device__ __forceinline__ float off23(unsigned v, unsigned sel)
{
    return __int_as_float(__byte_perm(v, 0x4B000000u, sel));
}
__device__ __forceinline__ float lerp23(float A, float B, float t) { return fmaf(t, B - A, A - 8388608.0f); }
// byte_perm selectors: u8 lane n of a word, u16 half n of a word, each with
// 0x4B in the top byte and zeros between
constexpr unsigned kU8Lane0 = 0x7540u, kU8Lane1 = 0x7541u, kU8Lane2 = 0x7542u, kU8Lane3 = 0x7543u;
constexpr unsigned kU16Half0 = 0x7410u, kU16Half1 = 0x7432u;

template <int DT>
__device__ __forceinline__ float fetch_cfg(const DevBrick &b, const CellPos &c)
{
    const int nx = b.nx, ny = b.ny;
    const int j = c.j, i = c.i, k = c.k;
    const float fx = c.fx, fy = c.fy, fz = c.fz;
    float c00, c10, c01, c11;
    if (b.quad) {
        // corner-packed copy: the cell's 8 voxels in two vector loads
        using V = typename VoxT<DT>::V4;
        const unsigned qx = (unsigned) nx - 1u, qs = qx * ((unsigned) ny - 1u);
        const V *e = reinterpret_cast<const V *>(b.quad) + ((unsigned) k * qs + (unsigned) i * qx + (unsigned) j);
        if (DT == IVR_U8) {
            // one word per element: lanes (j, i), (j+1, i), (j, i+1), (j+1, i+1)
            const unsigned lo = __ldg(reinterpret_cast<const unsigned *>(e));
            const unsigned hi = __ldg(reinterpret_cast<const unsigned *>(e + qs));
            c00 = lerp23(off23(lo, kU8Lane0), off23(lo, kU8Lane1), fx);
            c10 = lerp23(off23(lo, kU8Lane2), off23(lo, kU8Lane3), fx);
            c01 = lerp23(off23(hi, kU8Lane0), off23(hi, kU8Lane1), fx);
            c11 = lerp23(off23(hi, kU8Lane2), off23(hi, kU8Lane3), fx);
        } else if (DT == IVR_U16) {
            // two words per element, two lanes each
            const uint2 lo = __ldg(reinterpret_cast<const uint2 *>(e));
            const uint2 hi = __ldg(reinterpret_cast<const uint2 *>(e + qs));
            c00 = lerp23(off23(lo.x, kU16Half0), off23(lo.x, kU16Half1), fx);
            c10 = lerp23(off23(lo.y, kU16Half0), off23(lo.y, kU16Half1), fx);
            c01 = lerp23(off23(hi.x, kU16Half0), off23(hi.x, kU16Half1), fx);
            c11 = lerp23(off23(hi.y, kU16Half0), off23(hi.y, kU16Half1), fx);
        } else if (kQuadDelta) {
            // (v0, v1 - v0) pairs: the x lerps without their subtraction
            const V lo = __ldg(e), hi = __ldg(e + qs);
            c00 = fmaf(fx, (float) lo.y, (float) lo.x);
            c10 = fmaf(fx, (float) lo.w, (float) lo.z);
            c01 = fmaf(fx, (float) hi.y, (float) hi.x);
            c11 = fmaf(fx, (float) hi.w, (float) hi.z);
        } else {
            const V lo = __ldg(e), hi = __ldg(e + qs);
            c00 = lerpf((float) lo.x, (float) lo.y, fx);
            c10 = lerpf((float) lo.z, (float) lo.w, fx);
            c01 = lerpf((float) hi.x, (float) hi.y, fx);
            c11 = lerpf((float) hi.z, (float) hi.w, fx);
        }
    } else {
        // one pointer to the cell's low corner (a brick holds fewer than
        // 2^32 voxels, checked at load, so its offset fits 32 bits); the
        // other corners are whole rows (nx) and slabs (nx*ny) away, the +1
        // neighbours an immediate offset
        using T = typename VoxT<DT>::T;
        const unsigned sz = (unsigned) nx * (unsigned) ny;
        const T *q0 = reinterpret_cast<const T *>(b.data) + ((unsigned) k * sz + (unsigned) i * (unsigned) nx + (unsigned) j);
        const T *q1 = q0 + nx, *q2 = q0 + sz, *q3 = q2 + nx;
        c00 = lerpf((float) __ldg(q0), (float) __ldg(q0 + 1), fx);
        c10 = lerpf((float) __ldg(q1), (float) __ldg(q1 + 1), fx);
        c01 = lerpf((float) __ldg(q2), (float) __ldg(q2 + 1), fx);
        c11 = lerpf((float) __ldg(q3), (float) __ldg(q3 + 1), fx);
    }
    float c0 = lerpf(c00, c10, fy);
    float c1 = lerpf(c01, c11, fy);
    return lerpf(c0, c1, fz);
}

template <int DT>
__device__ __forceinline__ float sample_cfg(const DevBrick &b, float ux, float uy, float uz)
{
    return fetch_cfg<DT>(b, cell_cfg(b, ux, uy, uz));
}

// One voxel cell of a corner-packed copy as loaded: the two elements (slab
// k and k+1), each holding the cell's four voxels of that slab.
template <int DT> struct QuadCell;
template <> struct QuadCell<IVR_U8> { unsigned lo, hi; };
template <> struct QuadCell<IVR_U16> { uint2 lo, hi; };
template <> struct QuadCell<IVR_F32> { float4 lo, hi; };

// element offset of cell c in the corner-packed copy (unique per cell)
__device__ __forceinline__ unsigned quad_key(const DevBrick &b, const CellPos &c)
{
    const unsigned qx = (unsigned) b.nx - 1u, qs = qx * ((unsigned) b.ny - 1u);
    return (unsigned) c.k * qs + (unsigned) c.i * qx + (unsigned) c.j;
}

template <int DT>
__device__ __forceinline__ QuadCell<DT> quad_load(const DevBrick &b, unsigned key)
{
    using E = decltype(QuadCell<DT>::lo);
    const unsigned qs = ((unsigned) b.nx - 1u) * ((unsigned) b.ny - 1u);
    const E *e = reinterpret_cast<const E *>(b.quad) + key;
    QuadCell<DT> q;
    q.lo = __ldg(e);
    q.hi = __ldg(e + qs);
    return q;
}

// fetch_cfg's corner-packed interpolation on a loaded cell
template <int DT>
__device__ __forceinline__ float quad_interp(const QuadCell<DT> &q, const CellPos &c)
{
    float c00, c10, c01, c11;
    if constexpr (DT == IVR_U8) {
        c00 = lerp23(off23(q.lo, kU8Lane0), off23(q.lo, kU8Lane1), c.fx);
        c10 = lerp23(off23(q.lo, kU8Lane2), off23(q.lo, kU8Lane3), c.fx);
        c01 = lerp23(off23(q.hi, kU8Lane0), off23(q.hi, kU8Lane1), c.fx);
        c11 = lerp23(off23(q.hi, kU8Lane2), off23(q.hi, kU8Lane3), c.fx);
    } else if constexpr (DT == IVR_U16) {
        c00 = lerp23(off23(q.lo.x, kU16Half0), off23(q.lo.x, kU16Half1), c.fx);
        c10 = lerp23(off23(q.lo.y, kU16Half0), off23(q.lo.y, kU16Half1), c.fx);
        c01 = lerp23(off23(q.hi.x, kU16Half0), off23(q.hi.x, kU16Half1), c.fx);
        c11 = lerp23(off23(q.hi.y, kU16Half0), off23(q.hi.y, kU16Half1), c.fx);
    } else if (kQuadDelta) {
        c00 = fmaf(c.fx, q.lo.y, q.lo.x);
        c10 = fmaf(c.fx, q.lo.w, q.lo.z);
        c01 = fmaf(c.fx, q.hi.y, q.hi.x);
        c11 = fmaf(c.fx, q.hi.w, q.hi.z);
    } else {
        c00 = lerpf(q.lo.x, q.lo.y, c.fx);
        c10 = lerpf(q.lo.z, q.lo.w, c.fx);
        c01 = lerpf(q.hi.x, q.hi.y, c.fx);
        c11 = lerpf(q.hi.z, q.hi.w, c.fx);
    }
    const float c0 = lerpf(c00, c10, c.fy);
    const float c1 = lerpf(c01, c11, c.fy);
    return lerpf(c0, c1, c.fz);
}

// Two samples' interpolation in packed FP32 instructions, each lane rounding
// as the scalar code above does: b - a is one fma by -1 (an exact product), so
// no product feeds a sum.
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) { return f2_fma(b, f2(-1.0f), a); }
__device__ __forceinline__ F2 f2_lerp(F2 a, F2 b, F2 t) { return f2_fma(t, f2_sub(b, a), a); }
__device__ __forceinline__ F2 f2_lerp23(F2 A, F2 B, F2 t) { return f2_fma(t, f2_sub(B, A), A + f2(-8388608.0f)); }

// quad_interp of two loaded cells
template <int DT>
__device__ __forceinline__ void quad_interp2(const QuadCell<DT> &p, const QuadCell<DT> &q, const CellPos &c,
                                             const CellPos &d, float &s0, float &s1)
{
    const F2 fx = f2(c.fx, d.fx), fy = f2(c.fy, d.fy), fz = f2(c.fz, d.fz);
    F2 c00, c10, c01, c11;
    if constexpr (DT == IVR_U8) {
        auto v = [](unsigned a, unsigned b, unsigned lane) { return f2(off23(a, lane), off23(b, lane)); };
        c00 = f2_lerp23(v(p.lo, q.lo, kU8Lane0), v(p.lo, q.lo, kU8Lane1), fx);
        c10 = f2_lerp23(v(p.lo, q.lo, kU8Lane2), v(p.lo, q.lo, kU8Lane3), fx);
        c01 = f2_lerp23(v(p.hi, q.hi, kU8Lane0), v(p.hi, q.hi, kU8Lane1), fx);
        c11 = f2_lerp23(v(p.hi, q.hi, kU8Lane2), v(p.hi, q.hi, kU8Lane3), fx);
    } else if constexpr (DT == IVR_U16) {
        auto v = [](unsigned a, unsigned b, unsigned half) { return f2(off23(a, half), off23(b, half)); };
        c00 = f2_lerp23(v(p.lo.x, q.lo.x, kU16Half0), v(p.lo.x, q.lo.x, kU16Half1), fx);
        c10 = f2_lerp23(v(p.lo.y, q.lo.y, kU16Half0), v(p.lo.y, q.lo.y, kU16Half1), fx);
        c01 = f2_lerp23(v(p.hi.x, q.hi.x, kU16Half0), v(p.hi.x, q.hi.x, kU16Half1), fx);
        c11 = f2_lerp23(v(p.hi.y, q.hi.y, kU16Half0), v(p.hi.y, q.hi.y, kU16Half1), fx);
    } else {
        auto x = [&](float a0, float b0, float a1, float b1) {
            return kQuadDelta ? f2(fmaf(c.fx, b0, a0), fmaf(d.fx, b1, a1))
                              : f2(lerpf(a0, b0, c.fx), lerpf(a1, b1, d.fx));
        };
        c00 = x(p.lo.x, p.lo.y, q.lo.x, q.lo.y);
        c10 = x(p.lo.z, p.lo.w, q.lo.z, q.lo.w);
        c01 = x(p.hi.x, p.hi.y, q.hi.x, q.hi.y);
        c11 = x(p.hi.z, p.hi.w, q.hi.z, q.hi.w);
    }
    f2_split(f2_lerp(f2_lerp(c00, c10, fy), f2_lerp(c01, c11, fy), fz), s0, s1);
}

// A ray's CONFIG lattice in a brick's voxel coordinates: lattice index i
// samples u_i = fmaf(i, s, base) per axis, with s = (d * ic) * dt and
// base = fmaf(d * ic, t0, (o - bmin) * ic) -- the point o + t_i d, t_i =
// t0 + i dt, mapped by the brick's world-to-voxel scaling ic.  Three fmaf
// per sample instead of the lattice parameter, the world point and its
// mapping.
struct VoxLattice {
    float sx, sy, sz;
    float bx, by, bz;
};

__device__ __forceinline__ VoxLattice vox_lattice(const DevBrick &b, float ox, float oy, float oz, float dx,
                                                  float dy, float dz, float t0, float dt)
{
    const float ux = dx * b.icx, uy = dy * b.icy, uz = dz * b.icz;
    VoxLattice L;
    L.sx = ux * dt;
    L.sy = uy * dt;
    L.sz = uz * dt;
    L.bx = fmaf(ux, t0, (ox - b.bminx) * b.icx);
    L.by = fmaf(uy, t0, (oy - b.bminy) * b.icy);
    L.bz = fmaf(uz, t0, (oz - b.bminz) * b.icz);
    return L;
}

__device__ __forceinline__ float4 lut_at(const FrameDesc &f, int idx)
{
    idx = min(max(idx, 0), f.lut_n - 1);
    return __ldg(f.lut + idx);
}

// One sample of a transfer function of transferfuncs.c:24-199, composited
// into c = (r, g, b, a).
template <int TF>
__device__ __forceinline__ void ref_composite(const FrameDesc &f, float s, const float4 &e, float4 &c)
{
    const float myalpha = f.alpha;
    if (TF == IVR_TF_MED) {  // transferfuncs.c:24-68
        c.z = ((double) e.z < 0.8) ? fmaxf(e.z, c.z) : c.z;
        c.y = ((double) e.y < 0.8) ? fmaxf(e.y, c.y) : c.y;
        c.x = ((double) e.x < 0.8) ? fmaxf(e.x, c.x) : c.x;
        c.w = e.w * myalpha;
    } else if (TF == IVR_TF_BLEND) {  // transferfuncs.c:70-83
        const float al = e.w;
        c.z = al * e.z + (1.0f - al) * c.z;
        c.y = al * e.y + (1.0f - al) * c.y;
        c.x = al * e.x + (1.0f - al) * c.x;
        c.w = al * myalpha;
    } else if (TF == IVR_TF_SEISMIC2 || TF == IVR_TF_CHEM) {  // transferfuncs.c:109-168
        const float al = e.w * myalpha;
        const float oma = 1.0f - al;
        c.z = oma * c.z + al * e.z;
        c.y = oma * c.y + al * e.y;
        c.x = oma * c.x + al * e.x;
        c.w = al + oma * c.w;
        if (c.w > 1.0f) c.w = 1.0f;
    } else if (TF == IVR_TF_RGBBLEND) {  // transferfuncs.c:170-200
        const unsigned u = __float_as_uint(s);
        const float r = 1.0f / 255.0f * (float) ((u >> 24) & 0xff);
        const float g = 1.0f / 255.0f * (float) ((u >> 16) & 0xff);
        const float bl = 1.0f / 255.0f * (float) ((u >> 8) & 0xff);
        const float al = myalpha;
        const float oma = 1.0f - al;
        c.z = oma * c.z + al * bl;
        c.y = oma * c.y + al * g;
        c.x = oma * c.x + al * r;
        c.w = al + oma * c.w;
        if (c.w > 1.0f) c.w = 1.0f;
    } else {  // IVR_TF_SEISMIC, transferfuncs.c:86-107
        c.z = ((double) e.z > 0.65 && e.z < 1.0f) ? 0.6f : c.z;
        c.y = ((double) e.y > 0.65 && e.y < 1.0f) ? 0.0f : c.y;
        c.x = ((double) e.x > 0.65 && e.x < 1.0f) ? 0.0f : c.x;
        c.z = ((double) e.z > 0.5 && e.z < 0.65f) ? 0.9f : c.z;
        c.y = ((double) e.y > 0.5 && e.y < 0.65f) ? 0.9f : c.y;
        c.x = ((double) e.x > 0.5 && e.x < 0.65f) ? 0.9f : c.x;
        c.z = ((double) e.z > 0.3 && e.z < 0.5f) ? 0.0f : c.z;
        c.y = ((double) e.y > 0.3 && e.y < 0.5f) ? 0.0f : c.y;
        c.x = ((double) e.x > 0.3 && e.x < 0.5f) ? 0.6f : c.x;
        c.w = 1.0f * myalpha;
    }
}

// raycast (ray.c:59-85) + getsamplesonray (ray.c:239-273) + one transfer
// function.  Samples are computed in the order the transfer function
// consumes them (ascending or descending) instead of being stored, kRefPairs
// pairs at a time with their loads in flight together.  Returns (r, g, b, a).
// Bound by instruction issue (68% of the slots, 202 M warp instructions for
// 128^3 u8 at 512x512): nine IEEE divisions a sample and up to 512 column
// increments a pixel took 425 us; FixedDivs and shared increments 271; the
// divisions of two samples packed, two pairs in flight, 254 (one pair 269).
// 4, 6 and 8 blocks per SM instead of 5: 260, 265, 299.
constexpr int kRefPairs = 2;        // pairs of samples per iteration
constexpr int kRefBlocksPerSm = 5;  // resident blocks it is compiled for
template <int TF> __device__ __forceinline__ constexpr bool ref_down()
{
    return TF == IVR_TF_SEISMIC2 || TF == IVR_TF_CHEM || TF == IVR_TF_RGBBLEND;
}

// the LUT entry of a sample: BLEND takes no lutoffset; lut_at clamps every
// index (as SEISMIC2 and CHEM do)
template <int TF>
__device__ __forceinline__ float4 ref_entry(const FrameDesc &f, float s)
{
    if (TF == IVR_TF_RGBBLEND) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    return lut_at(f, lut_index((int) s, TF == IVR_TF_BLEND ? 0 : f.lut_off));
}

// The ray's iend samples by sample_ref itself, one by one: rays on which
// FixedDiv might round otherwise (ref_fast).
template <int DT, int TF>
__device__ __noinline__ float4 raycast_ref_general(const FrameDesc &f, const DevBrick &b, float dx, float dy, float dz,
                                                   float tin, int iend)
{
    float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int n = 0; n < iend; n++) {
        const float t = tin + ((float) (ref_down<TF>() ? iend - 1 - n : n) * f.step);
        const float s = sample_ref<DT>(b, dx * t + f.origx, dy * t + f.origy, dz * t + f.origz);
        ref_composite<TF>(f, s, ref_entry<TF>(f, s), c);
    }
    return c;
}

template <int DT, int TF>
__device__ __forceinline__ float4 raycast_ref(const FrameDesc &f, const DevBrick &b, float dx, float dy, float dz,
                                              unsigned long long &nexec)
{
    float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float tin, tout;
    if (!ray_box(b.dconst, f.origx, f.origy, f.origz, dx, dy, dz, tin, tout)) return c;
    const float dt = f.step;
    int iend = (int) (1.0f + (tout - tin) / dt + 0.5f);
    if (f.max_samples > 0 && iend > f.max_samples) iend = f.max_samples;
    if (iend <= 0) return c;
    nexec += (unsigned long long) iend;
    if (!ref_fast(f, b, dx, dy, dz, tin)) return raycast_ref_general<DT, TF>(f, b, dx, dy, dz, tin, iend);
    const RefSampler rs(b);
    for (int n = 0; n < iend; n += 2 * kRefPairs) {
        RefPos p[kRefPairs];
        RefCell<DT> v[2 * kRefPairs];
#pragma unroll
        for (int k = 0; k < kRefPairs; k++) {
            // (past the last sample the last one again, not composited)
            const int a = min(n + 2 * k, iend - 1), e = min(n + 2 * k + 1, iend - 1);
            const float ta = tin + ((float) (ref_down<TF>() ? iend - 1 - a : a) * dt);
            const float te = tin + ((float) (ref_down<TF>() ? iend - 1 - e : e) * dt);
            p[k] = ref_pos(b, rs, f2(dx * ta + f.origx, dx * te + f.origx), f2(dy * ta + f.origy, dy * te + f.origy),
                           f2(dz * ta + f.origz, dz * te + f.origz));
#pragma unroll
            for (int q = 0; q < 2; q++) v[2 * k + q] = ref_load<DT>(b, p[k].j[q], p[k].i[q], p[k].k[q]);
        }
        float s[2 * kRefPairs];
        float4 e[2 * kRefPairs];
#pragma unroll
        for (int k = 0; k < kRefPairs; k++) {
            float xd[2], yd[2], zd[2];
            f2_split(p[k].xd, xd[0], xd[1]);
            f2_split(p[k].yd, yd[0], yd[1]);
            f2_split(p[k].zd, zd[0], zd[1]);
#pragma unroll
            for (int q = 0; q < 2; q++)
                s[2 * k + q] = ref_interp<DT>(v[2 * k + q], fabsf(xd[q]), fabsf(yd[q]), fabsf(zd[q]));
        }
#pragma unroll
        for (int k = 0; k < 2 * kRefPairs; k++) e[k] = ref_entry<TF>(f, s[k]);
#pragma unroll
        for (int k = 0; k < 2 * kRefPairs; k++) {
            if (n + k >= iend) break;
            ref_composite<TF>(f, s[k], e[k], c);
        }
    }
    return c;
}

// compositetiles (main.c:1206-1215): d = s + (1 - s.a) * d
__device__ __forceinline__ float4 over(float4 s, float4 d)
{
    d.z = s.z + (1.0f - s.w) * d.z;
    d.y = s.y + (1.0f - s.w) * d.y;
    d.x = s.x + (1.0f - s.w) * d.x;
    d.w = s.w + (1.0f - s.w) * d.w;
    return d;
}

// (uint8)(v*255 + 0.5) for v in [0,1], exact: for v = m * 2^(e-150) the
// value is floor((255 m + 2^(s-1)) / 2^s) with s = 150 - e.
__device__ __forceinline__ unsigned q8(float v)
{
    if (!(v > 0.0f)) return 0u;
    if (v >= 1.0f) return 255u;
    unsigned bits = __float_as_uint(v);
    int e = (int) (bits >> 23);
    if (e == 0) return 0u;  // subnormal: far below 1/510
    unsigned long long m = (bits & 0x7fffffu) | 0x800000u;
    int s = 150 - e;
    if (s >= 34) return 0u;
    return (unsigned) ((255ull * m + (1ull << (s - 1))) >> s);
}

__device__ __forceinline__ bool in_rect(const DevBrick &b, int i, int j)
{
    return i >= b.istrt && i < b.istop && j >= b.jstrt && j < b.jstop;
}

// CONFIG lattice: t_i = fmaf(i, dt, t0).
__device__ __forceinline__ float cfg_t(float t0, float dt, int i) { return fmaf((float) i, dt, t0); }
// First lattice index i >= 0 with t_i >= a.  The estimate is exact up to
// rounding, so the fix-up loops run a step or two; they are bounded anyway.
constexpr int kMaxLattice = 1 << 24;
__device__ __forceinline__ int cfg_first_ge(float t0, float dt, float idt, float a)
{
    if (!(a > t0)) return 0;
    float q = (a - t0) * idt;  // an estimate: the loops below make it exact
    int i = q < (float) kMaxLattice ? (int) q : kMaxLattice;
    for (int it = 0; it < 64 && i > 0 && cfg_t(t0, dt, i - 1) >= a; it++) i--;
    for (int it = 0; it < 64 && i < kMaxLattice && cfg_t(t0, dt, i) < a; it++) i++;
    return i;
}


// K consecutive samples of a ray from lattice index fi: every load is issued
// before the first interpolation.  Samples past the ray's run are harmless:
// cell_cfg clamps the cells.  PACK: in packed pairs (K even).
template <int DT, int K, bool PACK>
__device__ __forceinline__ void sample_run(const DevBrick &b, const VoxLattice &L, float fi, float (&s)[K])
{
    CellPos c[K];
    if constexpr (PACK) {
#pragma unroll
        for (int k = 0; k < K; k += 2) {
            const F2 fk = f2(fi + (float) k, fi + (float) (k + 1));
            float ux[2], uy[2], uz[2];
            f2_split(f2_fma(fk, f2(L.sx), f2(L.bx)), ux[0], ux[1]);
            f2_split(f2_fma(fk, f2(L.sy), f2(L.by)), uy[0], uy[1]);
            f2_split(f2_fma(fk, f2(L.sz), f2(L.bz)), uz[0], uz[1]);
            c[k] = cell_cfg(b, ux[0], uy[0], uz[0]);
            c[k + 1] = cell_cfg(b, ux[1], uy[1], uz[1]);
        }
    } else {
#pragma unroll
        for (int k = 0; k < K; k++) {
            const float fk = fi + (float) k;  // (float) (i + k): i < 2^24
            c[k] = cell_cfg(b, fmaf(fk, L.sx, L.bx), fmaf(fk, L.sy, L.by), fmaf(fk, L.sz, L.bz));
        }
    }
    if (b.quad) {
        // Every sample loads its own cell, also where two share one: a copy
        // of the neighbour's voxels would wait for that load, and its branch
        // holds up the loads behind it (u16 learned frame 523 -> 358 us, f32
        // unchanged).
        QuadCell<DT> q[K];
#pragma unroll
        for (int k = 0; k < K; k++) q[k] = quad_load<DT>(b, quad_key(b, c[k]));
#pragma unroll
        for (int k = 0; k < K; k += PACK ? 2 : 1) {
            if constexpr (PACK) quad_interp2<DT>(q[k], q[k + 1], c[k], c[k + 1], s[k], s[k + 1]);
            else s[k] = quad_interp<DT>(q[k], c[k]);
        }
    } else {
#pragma unroll
        for (int k = 0; k < K; k++) s[k] = fetch_cfg<DT>(b, c[k]);
    }
}

// The LUT entries of K samples, all loads issued before the first is
// composited, and the first n of them composited front to back into acc.
// True when the ray ended (alpha reached term).
template <int K>
__device__ __forceinline__ bool composite_run(const FrameDesc &f, const float (&s)[K], int n, float opac, float term,
                                              float4 &acc)
{
    float4 e[K];
#pragma unroll
    for (int k = 0; k < K; k++) e[k] = lut_at(f, lut_index((int) (s[k] * f.lut_scale), f.lut_off));
#pragma unroll
    for (int k = 0; k < K; k++) {
        if (k >= n) break;
        const float wgt = (1.0f - acc.w) * (e[k].w * opac);
        acc.x = fmaf(wgt, e[k].x, acc.x);
        acc.y = fmaf(wgt, e[k].y, acc.y);
        acc.z = fmaf(wgt, e[k].z, acc.z);
        acc.w = acc.w + wgt;
        if (acc.w >= term) return true;
    }
    return false;
}

// A ray in a brick's macrocell grid: looks up the cell of sample i.
// Returns true where the cell is opaque, with `next` one past the last sample
// (i at least) taken in it without another look; else false, with `next` the
// sample to look at after the leap over the transparent cube around it.
// isx, isy, isz: lattice steps per voxel (about 1 / L.s).
__device__ __forceinline__ bool look_cell(const DevBrick &b, const uint8_t *empty, const VoxLattice &L, float isx,
                                          float isy, float isz, int i, int &next)
{
    const float fi = (float) i;
    const CellPos c = cell_cfg(b, fmaf(fi, L.sx, L.bx), fmaf(fi, L.sy, L.by), fmaf(fi, L.sz, L.bz));
    // the sample's macrocell: its voxel cell (the sampler's own index
    // arithmetic) over the macrocell edge (cells are never negative: the
    // sampler clamps them)
    const int cs = b.cshift, edge = 1 << cs;
    const int cj = c.j >> cs, ci = c.i >> cs, ck = c.k >> cs;
    // r >= 1: the cube of cells within r-1 of this one is transparent
    const int r = empty[(ck * b.mcy + ci) * b.mcx + cj];
    const int rr = max(r, 1);
    // the voxel plane of the face through which the ray leaves that cube (or
    // this one opaque cell), per axis, and the lattice index of the exit;
    // approximate, the margins absorb its rounding
    const float fx = (float) ((L.sx > 0.0f ? cj + rr : cj - rr + 1) * edge);
    const float fy = (float) ((L.sy > 0.0f ? ci + rr : ci - rr + 1) * edge);
    const float fz = (float) ((L.sz > 0.0f ? ck + rr : ck - rr + 1) * edge);
    const float qx = L.sx != 0.0f ? (fx - L.bx) * isx : FLT_MAX;
    const float qy = L.sy != 0.0f ? (fy - L.by) * isy : FLT_MAX;
    const float qz = L.sz != 0.0f ? (fz - L.bz) * isz : FLT_MAX;
    const float q = fminf(fmaxf(fminf(qx, fminf(qy, qz)), 0.0f), (float) kMaxLattice);
    const int iexit = (int) q;  // last lattice index at or before the exit
    if (r == 0) {
        next = max(iexit, i) + 1;
        return true;
    }
    // Leap.  Sample positions are monotone in the lattice index along each
    // axis and sample i lies in the cube, so when the last one before the
    // exit (iexit) is still short of every exit face, so is every sample up
    // to it: all are in the transparent cube, and the march resumes just past
    // the exit.  Otherwise (rounding at a face) it resumes two samples
    // earlier, where the next look decides again.  Every leap moves forward.
    const float fe = (float) iexit;
    const float ex = fmaf(fe, L.sx, L.bx), ey = fmaf(fe, L.sy, L.by), ez = fmaf(fe, L.sz, L.bz);
    const bool inside = (L.sx > 0.0f ? ex < fx : L.sx < 0.0f ? ex >= fx : true) &&
                        (L.sy > 0.0f ? ey < fy : L.sy < 0.0f ? ey >= fy : true) &&
                        (L.sz > 0.0f ? ez < fz : L.sz < 0.0f ? ez >= fz : true);
    next = max(i, inside ? iexit : iexit - 2) + 1;  // iexit + 1 or iexit - 1
    return false;
}

// One brick of the CONFIG march without skipping: samples tin_k <= t_i <
// tout_k of the ray's lattice, front-to-back into acc, K per iteration.
template <int DT, int K, bool PACK>
__device__ __forceinline__ void march_plain(const FrameDesc &f, const DevBrick &b, float dx, float dy, float dz,
                                            float idx, float idy, float idz, float t0, float dt, float idt,
                                            float4 &acc, bool &done)
{
    float tin, tout;
    if (!ray_box_cfg(b.dconst, f.origx, f.origy, f.origz, dx, dy, dz, idx, idy, idz, tin, tout)) return;
    const int i1 = cfg_first_ge(t0, dt, idt, tout);
    const VoxLattice L = vox_lattice(b, f.origx, f.origy, f.origz, dx, dy, dz, t0, dt);
    for (int i = cfg_first_ge(t0, dt, idt, tin); i < i1; i += K) {
        float s[K];
        sample_run<DT, K, PACK>(b, L, (float) i, s);
        if (composite_run<K>(f, s, i1 - i, f.alpha, f.term_alpha, acc)) {
            done = true;
            return;
        }
    }
}

// The census of one brick (a diagnostic launch): the march's samples one by
// one, each counted and its macrocell marked.
template <int DT, bool SKIP>
__device__ void march_census(const FrameDesc &f, const DevBrick &b, const uint8_t *empty, float dx, float dy, float dz,
                             float idx, float idy, float idz, float t0, float dt, float idt, float4 &acc, bool &done,
                             unsigned long long &nexec, unsigned long long &nlat)
{
    float tin, tout;
    if (!ray_box_cfg(b.dconst, f.origx, f.origy, f.origz, dx, dy, dz, idx, idy, idz, tin, tout)) return;
    const int i0 = cfg_first_ge(t0, dt, idt, tin);
    const int i1 = cfg_first_ge(t0, dt, idt, tout);
    nlat += (unsigned long long) max(i1 - i0, 0);
    if (done) return;
    const VoxLattice L = vox_lattice(b, f.origx, f.origy, f.origz, dx, dy, dz, t0, dt);
    const float isx = idx * idt * b.vwx, isy = idy * idt * b.vwy, isz = idz * idt * b.vwz;
    int held = i0;  // samples i..held-1 lie in an opaque cell already looked up
    for (int i = i0; i < i1;) {
        if (SKIP && i >= held) {
            int next;
            if (!look_cell(b, empty, L, isx, isy, isz, i, next)) {
                i = next;
                continue;
            }
            held = next;
        }
        const float fi = (float) i;
        const CellPos c = cell_cfg(b, fmaf(fi, L.sx, L.bx), fmaf(fi, L.sy, L.by), fmaf(fi, L.sz, L.bz));
        nexec++;
        b.touched[((long long) (c.k >> b.cshift) * b.mcy + (c.i >> b.cshift)) * b.mcx + (c.j >> b.cshift)] = 1;
        const float s[1] = {fetch_cfg<DT>(b, c)};
        if (composite_run<1>(f, s, 1, f.alpha, f.term_alpha, acc)) {
            done = true;
            return;
        }
        i++;
    }
}

// Samples a lane looks ahead for (at most 255: a run's length has 8 bits),
// and runs it can hold.  Learned 1024^3 / f32 512^3 frames, us: 549 / 373 at
// 32 samples, 527 / 361 at 64, 518 / 356 at 128.
constexpr int kRunSamples = 128;
constexpr int kRunMax = 8;
constexpr unsigned kFullWarp = 0xffffffffu;
static_assert(kRunSamples < 256, "run lengths have 8 bits");

// A ray's direction, its reciprocals and the ray's lattice: in registers, or
// (PARK) in the lane's column of a [kRayWords][kThreads] shared array, read
// where they are used and out of the way while samples are taken.  The
// batched kernel, which has 64 registers, parks: kept in registers they pushed
// the sampling loop's own values into local memory, as many requests as all
// its other loads (f32, 32 frames: 3.85 -> 3.76 ms, u16 20 frames 2.62 ->
// 2.56).  The frame kernels have the registers and read what is uniform from
// the constant bank.
enum RayWord { kDx, kDy, kDz, kIdx, kIdy, kIdz, kT0, kDt, kIdt, kRayWords };
template <bool PARK> struct Ray {
    float v[kRayWords];
    __device__ __forceinline__ void set(RayWord k, float x) { v[k] = x; }
    __device__ __forceinline__ float operator[](RayWord k) const { return v[k]; }
};
template <> struct Ray<true> {
    volatile float *v;
    __device__ __forceinline__ void set(RayWord k, float x) { v[k * kThreads] = x; }
    __device__ __forceinline__ float operator[](RayWord k) const { return v[k * kThreads]; }
};

// One brick of the CONFIG march with a skipping grid, in two alternating
// steps.  (1) Each lane walks its ray over the macrocell grid and notes the
// runs of lattice indices that lie in opaque cells, until it has
// kRunSamples of them: transparent cubes are leapt over, runs of
// neighbouring opaque cells join.  (2) All lanes sample and composite their
// runs.  A warp whose lanes checked a cell wherever one of them left its
// last one ran that check (a dependent load and some 60 instructions) in
// nearly every iteration; here the lanes walk together and sample together,
// each with the same number of samples at hand.  The samples taken are the
// same as when every cell is checked as it is reached, and every sample is
// computed exactly as without skipping.  `runs` is the lane's column of a
// [kRunMax][kThreads] shared array: start in the low 24 bits, length above.
// Every lane of the warp calls this (`in` false: without a ray), and the
// loops are the warp's, so that lanes which leave a step early wait for the
// others instead of taking the next step on their own (that took twice the
// time).  Bound by the latency of the longest rays: of a 317 us launch (384^3
// f32, 2x2x2 bricks, 1024x1024) the SMs have work for 86%, and use 56% of
// their issue slots meanwhile.
template <int DT, int K, bool PARK>
__device__ __forceinline__ void march_runs(const FrameDesc &f, const DevBrick &b, const uint8_t *empty,
                                           unsigned *runs, bool in, const Ray<PARK> &ray, float4 &acc, bool &done)
{
    const float dx = ray[kDx], dy = ray[kDy], dz = ray[kDz], idx = ray[kIdx], idy = ray[kIdy], idz = ray[kIdz];
    const float t0 = ray[kT0], dt = ray[kDt], idt = ray[kIdt];
    float tin, tout;
    in = in && ray_box_cfg(b.dconst, f.origx, f.origy, f.origz, dx, dy, dz, idx, idy, idz, tin, tout);
    int i = in ? cfg_first_ge(t0, dt, idt, tin) : 0;  // the next lattice index to look at
    int i1 = in ? cfg_first_ge(t0, dt, idt, tout) : 0;
    const float opac = f.alpha, term = f.term_alpha;
    const VoxLattice L = vox_lattice(b, f.origx, f.origy, f.origz, dx, dy, dz, t0, dt);
    int held = i;  // indices i..held-1 lie in an opaque cell already checked
    while (__any_sync(kFullWarp, i < i1)) {
        const float isx = ray[kIdx] * ray[kIdt] * b.vwx, isy = ray[kIdy] * ray[kIdt] * b.vwy,
                    isz = ray[kIdz] * ray[kIdt] * b.vwz;
        int nr = 0, n = 0;       // runs noted, samples in them
        int start = 0, len = 0;  // the run being built
        bool walk = i < i1;
        while (__any_sync(kFullWarp, walk)) {
            if (!walk) continue;
            if (i >= held) {
                int next;
                if (look_cell(b, empty, L, isx, isy, isz, i, next)) held = next;
                else i = next;
            }
            if (i < held && i < i1) {
                const bool gap = len > 0 && start + len != i;
                if (gap && nr == kRunMax - 1) {
                    walk = false;  // no room for another run
                } else {
                    if (gap) {
                        runs[nr * kThreads] = (unsigned) start | (unsigned) len << 24;
                        nr++;
                        len = 0;
                    }
                    if (len == 0) start = i;
                    const int take = min(min(held, i1) - i, kRunSamples - n);
                    len += take;
                    n += take;
                    i += take;
                }
            }
            walk = walk && i < i1 && n < kRunSamples;
        }
        if (len > 0) {
            runs[nr * kThreads] = (unsigned) start | (unsigned) len << 24;
            nr++;
        }
        // the runs' samples, K at a time, their loads in flight before the
        // first is composited; those past a run's end are not composited
        // (cell_cfg clamps the cells, so computing them is always safe)
        len = 0;
        for (int r = 0;;) {
            if (len == 0 && r < nr) {
                const unsigned w = runs[r * kThreads];
                start = (int) (w & 0xffffffu);
                len = (int) (w >> 24);
                r++;
            }
            if (!__any_sync(kFullWarp, len > 0)) break;
            if (len == 0) continue;
            float s[K];
            sample_run<DT, K, false>(b, L, (float) start, s);
            if (composite_run<K>(f, s, len, opac, term, acc)) {
                done = true;
                nr = 0;
                len = 0;
                i = i1;
            } else {
                const int take = min(len, K);
                start += take;
                len -= take;
            }
        }
    }
}

__device__ __forceinline__ void count_exec(const FrameDesc &f, unsigned long long nexec,
                                           unsigned long long nlat = 0)
{
    if (f.counters == nullptr) return;
    // every lane of the warp reaches here (out-of-range pixels store
    // nothing but still count zero)
    for (int o = 16; o > 0; o >>= 1) {
        nexec += __shfl_xor_sync(0xffffffffu, nexec, o);
        nlat += __shfl_xor_sync(0xffffffffu, nlat, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(f.counters, nexec);
        if (nlat) atomicAdd(f.counters + 1, nlat);
    }
}

__device__ __forceinline__ void pixel_of(const FrameDesc &f, int &i, int &j, int &oi, int &oj)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    oj = blockIdx.x * kBlockX + (warp & 1) * 8 + (lane & 7);
    oi = blockIdx.y * kBlockY + (warp >> 1) * 4 + (lane >> 3);
    j = f.out_x + oj;
    i = f.out_y + oi;
}

template <int DT, int TF>
__global__ void __launch_bounds__(kThreads, kRefBlocksPerSm) march_ref_kernel(const __grid_constant__ FrameDesc f, float4 *out32,
                                                             uchar4 *out8)
{
    // Each brick casts its own ray with the sequential column increments of
    // createlocalimage (main.c:986-999): a chain of up to the window's width
    // of additions, each rounded, so nothing shorter gives its value.  Per
    // brick, row and component one lane walks the chain to the block's first
    // column (s_dir); the pixels add at most kBlockX more.
    __shared__ float s_dir[kMaxBricks][kBlockY][3];
    const int j0 = f.out_x + (int) blockIdx.x * kBlockX, i0 = f.out_y + (int) blockIdx.y * kBlockY;
    for (int q = threadIdx.x >> 5; q < f.nb; q += kThreads / 32) {
        const DevBrick &b = f.b[q];
        const int lane = threadIdx.x & 31, row = lane / 3, comp = lane - 3 * row;
        if (row >= kBlockY || (f.single >= 0 && q != f.single)) continue;
        if (j0 + kBlockX <= b.jstrt || j0 >= b.jstop || i0 + kBlockY <= b.istrt || i0 >= b.istop) continue;
        const float fi = (float) (i0 + row - b.istrt);
        float dir = comp == 0 ? b.dir0x + f.incrix * fi : comp == 1 ? b.dir0y + f.incriy * fi : b.dir0z + f.incriz * fi;
        const float incr = comp == 0 ? f.incrjx : comp == 1 ? f.incrjy : f.incrjz;
        for (int c = b.jstrt; c < j0; c++) dir += incr;
        s_dir[q][row][comp] = dir;
    }
    __syncthreads();
    int i, j, oi, oj;
    pixel_of(f, i, j, oi, oj);
    const bool inside = oj < f.out_w && oi < f.out_h;
    float4 d = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    unsigned long long nexec = 0;
    if (inside && i < f.vh && j < f.vw) {
        // far -> near over of per-brick colours
        for (int s = f.nb - 1; s >= 0; s--) {
            const int k = f.order[s];
            if (f.single >= 0 && k != f.single) continue;
            const DevBrick &b = f.b[k];
            if (!in_rect(b, i, j)) continue;
            const float *dir = s_dir[k][i - i0];
            float dx = dir[0], dy = dir[1], dz = dir[2];
            for (int c = max(b.jstrt, j0); c <= j; c++) {
                dx += f.incrjx;
                dy += f.incrjy;
                dz += f.incrjz;
            }
            float4 cs = raycast_ref<DT, TF>(f, b, dx, dy, dz, nexec);
            d = over(cs, d);
        }
    }
    if (inside) {
        const long long o = (long long) oi * f.out_w + oj;
        if (out32) out32[o] = d;
        if (out8) out8[o] = make_uchar4(q8(d.x), q8(d.y), q8(d.z), q8(d.w));
    }
    count_exec(f, nexec);
}

// One CONFIG ray per lane: pixel (i, j) of the viewport, all bricks front to
// back, skipping by the bricks' grids, or by the exact grids f.exact when
// exact.  Every lane of the warp calls it; one with `live` false has no ray.
template <int DT, bool SKIP, bool CENSUS, int K, bool PARK = false>
__device__ __forceinline__ float4 ray_cfg(const FrameDesc &f, int i, int j, bool live, unsigned long long &nexec,
                                          unsigned long long &nlat, unsigned *runs, bool exact = false,
                                          volatile float *park = nullptr)
{
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    bool any = false;
    for (int k = 0; k < f.nb; k++) any |= in_rect(f.b[k], i, j);
    live = live && any;
    if (!__any_sync(kFullWarp, live)) return acc;
    // ctm * (u, v, 5) at the pixel centre
    const float u = f.left + ((float) j + 0.5f) * f.du;
    const float v = f.bottom + ((float) i + 0.5f) * f.dv;
    const float dx = f.ctm[0] * u + f.ctm[1] * v + f.ctm[2] * f.eyen;
    const float dy = f.ctm[3] * u + f.ctm[4] * v + f.ctm[5] * f.eyen;
    const float dz = f.ctm[6] * u + f.ctm[7] * v + f.ctm[8] * f.eyen;
    const float idx = 1.0f / dx, idy = 1.0f / dy, idz = 1.0f / dz;
    float tin, tout;
    live = live && ray_box_cfg(f.gdconst, f.origx, f.origy, f.origz, dx, dy, dz, idx, idy, idz, tin, tout);
    const float t0 = live && tin > 0.0f ? tin : 0.0f;
    const float len = sqrtf(fmaf(dz, dz, fmaf(dy, dy, dx * dx)));
    const float dt = f.step / len;
    bool done = !live || !(dt > 0.0f);
    const float idt = 1.0f / dt;
    Ray<PARK> ray;
    if constexpr (PARK) ray.v = park;
    ray.set(kDx, dx);
    ray.set(kDy, dy);
    ray.set(kDz, dz);
    ray.set(kIdx, idx);
    ray.set(kIdy, idy);
    ray.set(kIdz, idz);
    ray.set(kT0, t0);
    ray.set(kDt, dt);
    ray.set(kIdt, idt);
    for (int s = 0; s < f.nb; s++) {
        const int k = f.order[s];
        if (f.single >= 0 && k != f.single) continue;
        const DevBrick &b = f.b[k];
        const bool in = (CENSUS ? live : !done) && in_rect(b, i, j);
        if (!__any_sync(kFullWarp, in)) continue;
        const uint8_t *empty = exact ? f.exact[k] : b.empty;
        if constexpr (CENSUS) {
            if (in && SKIP && empty != nullptr)
                march_census<DT, true>(f, b, empty, dx, dy, dz, idx, idy, idz, t0, dt, idt, acc, done, nexec, nlat);
            else if (in)
                march_census<DT, false>(f, b, empty, dx, dy, dz, idx, idy, idz, t0, dt, idt, acc, done, nexec, nlat);
        } else if (SKIP && empty != nullptr) {
            march_runs<DT, K, PARK>(f, b, empty, runs, in, ray, acc, done);
        } else if (in) {
            march_plain<DT, SKIP ? K : kPlainK, !SKIP>(f, b, ray[kDx], ray[kDy], ray[kDz], ray[kIdx], ray[kIdy], ray[kIdz], ray[kT0], ray[kDt],
                               ray[kIdt], acc, done);
        }
    }
    return acc;
}

// One pixel of the output window (ow, oh) = (oj, oi).
template <int DT, bool SKIP, bool CENSUS, int K, bool PARK>
__device__ __forceinline__ float4 pixel_cfg(const FrameDesc &f, int oi, int oj, float4 *out32, uchar4 *out8,
                                            unsigned long long &nexec, unsigned long long &nlat, unsigned *runs,
                                            volatile float *park)
{
    const bool in_window = oj < f.out_w && oi < f.out_h;
    const int j = f.out_x + oj, i = f.out_y + oi;
    const float4 acc = ray_cfg<DT, SKIP, CENSUS, K, PARK>(f, i, j, in_window && i < f.vh && j < f.vw, nexec, nlat,
                                                          runs, false, park);
    if (!in_window) return acc;
    const long long o = (long long) oi * f.out_w + oj;
    if (out32) out32[o] = acc;
    if (out8) out8[o] = make_uchar4(q8(acc.x), q8(acc.y), q8(acc.z), q8(acc.w));
    return acc;
}

// Estimated cost of one CONFIG ray, in samples: a walk over the bricks'
// macrocell grids front to back, cell by cell, with no volume reads.  A
// transparent cube (the grid's distance field) costs one step, as the
// march's leap over it does; an opaque cell costs the lattice points it
// holds, and its mean LUT opacity (b.opac) lowers the ray's estimated
// transmittance, so that the walk stops about where early termination
// would.  Only the order of tiles depends on it, never a pixel.
__device__ float ray_cost(const FrameDesc &f, int i, int j)
{
    bool any = false;
    for (int k = 0; k < f.nb; k++) any |= in_rect(f.b[k], i, j);
    if (!any) return 0.0f;
    const float u = f.left + ((float) j + 0.5f) * f.du;
    const float v = f.bottom + ((float) i + 0.5f) * f.dv;
    const float dx = f.ctm[0] * u + f.ctm[1] * v + f.ctm[2] * f.eyen;
    const float dy = f.ctm[3] * u + f.ctm[4] * v + f.ctm[5] * f.eyen;
    const float dz = f.ctm[6] * u + f.ctm[7] * v + f.ctm[8] * f.eyen;
    const float idx = 1.0f / dx, idy = 1.0f / dy, idz = 1.0f / dz;
    float tin, tout;
    if (!ray_box_cfg(f.gdconst, f.origx, f.origy, f.origz, dx, dy, dz, idx, idy, idz, tin, tout)) return 0.0f;
    const float t0 = tin > 0.0f ? tin : 0.0f;
    const float dt = f.step / sqrtf(fmaf(dz, dz, fmaf(dy, dy, dx * dx)));
    if (!(dt > 0.0f)) return 0.0f;
    const float idt = 1.0f / dt;
    const float ox = f.origx, oy = f.origy, oz = f.origz;
    // log2 of the transmittance where the march stops
    const float lstop = f.term_alpha < 1.0f ? __log2f(1.0f - f.term_alpha) : -FLT_MAX;
    float lt = 0.0f, cost = 0.0f;
    for (int s = 0; s < f.nb; s++) {
        const int k = f.order[s];
        if (f.single >= 0 && k != f.single) continue;
        const DevBrick &b = f.b[k];
        if (!in_rect(b, i, j)) continue;
        float ta, tb;
        if (!ray_box_cfg(b.dconst, ox, oy, oz, dx, dy, dz, idx, idy, idz, ta, tb)) continue;
        float t = fmaxf(ta, t0);
        if (b.empty == nullptr || b.opac == nullptr) {
            cost += fmaxf(tb - t, 0.0f) * idt;
            continue;
        }
        for (int it = 0; it < 4096 && t < tb; it++) {
            // the cell a quarter step past t (the march's index arithmetic)
            const float tm = fmaf(0.25f, dt, t);
            const int cj = min(max((int) floorf((fmaf(dx, tm, ox) - b.bminx) * b.icx), 0), b.nx - 2) >> b.cshift;
            const int ci = min(max((int) floorf((fmaf(dy, tm, oy) - b.bminy) * b.icy), 0), b.ny - 2) >> b.cshift;
            const int ck = min(max((int) floorf((fmaf(dz, tm, oz) - b.bminz) * b.icz), 0), b.nz - 2) >> b.cshift;
            const long long c = ((long long) ck * b.mcy + ci) * b.mcx + cj;
            const int r = b.empty[c];
            const int oq = b.opac[c];
            const int rr = max(r, 1);
            const float tx = dx > 0.0f ? (fmaf((float) (cj + rr), b.mcwx, b.bminx) - ox) * idx
                             : dx < 0.0f ? (fmaf((float) (cj - rr + 1), b.mcwx, b.bminx) - ox) * idx : FLT_MAX;
            const float ty = dy > 0.0f ? (fmaf((float) (ci + rr), b.mcwy, b.bminy) - oy) * idy
                             : dy < 0.0f ? (fmaf((float) (ci - rr + 1), b.mcwy, b.bminy) - oy) * idy : FLT_MAX;
            const float tz = dz > 0.0f ? (fmaf((float) (ck + rr), b.mcwz, b.bminz) - oz) * idz
                             : dz < 0.0f ? (fmaf((float) (ck - rr + 1), b.mcwz, b.bminz) - oz) * idz : FLT_MAX;
            float te = fminf(fminf(tx, ty), fminf(tz, tb));
            if (!(te > t)) te = t + dt;
            if (r != 0) {
                cost += 1.0f;
            } else {
                const float n = (te - t) * idt;
                const float a = (float) (oq * oq) * (1.0f / 65025.0f) * f.alpha;
                if (a > 0.0f) {
                    const float la = __log2f(1.0f - fminf(a, 0.999f));  // per sample, < 0
                    const float need = (lstop - lt) / la;
                    if (need <= n) return cost + need;
                    lt = fmaf(n, la, lt);
                }
                cost += n;
            }
            t = te;
        }
    }
    return cost;
}

constexpr int kCostKeys = 64;  // quarter-octave buckets of the tile cost

// Tile costs: kCostRays threads per 8x4 tile walk rays of it (its centre,
// two opposite corners, or all four); the tile's key is the quarter-octave
// of the largest, counted per key in counts[0..63].
#ifndef IVR_COST_RAYS
#define IVR_COST_RAYS 4
#endif
constexpr int kCostRays = IVR_COST_RAYS;
static_assert(kCostRays == 1 || kCostRays == 2 || kCostRays == 4, "rays per tile: 1, 2 or 4");
__global__ void tile_cost_kernel(const __grid_constant__ FrameDesc f, uint8_t *key, int *counts, long long ntiles)
{
    __shared__ int hist[kCostKeys];
    for (int t = threadIdx.x; t < kCostKeys; t += blockDim.x) hist[t] = 0;
    __syncthreads();
    const long long g = (long long) blockIdx.x * blockDim.x + threadIdx.x;
    const long long tile = g / kCostRays;
    const int r = (int) (g % kCostRays);
    const int tiles_x = (f.out_w + 7) >> 3;
    float cost = 0.0f;
    if (tile < ntiles) {
        const int di = kCostRays == 1 ? 2 : kCostRays == 2 ? 3 * r : 3 * (r >> 1);
        const int dj = kCostRays == 1 ? 4 : kCostRays == 2 ? 7 * r : 7 * (r & 1);
        const int oi = min((int) (tile / tiles_x) * 4 + di, f.out_h - 1);
        const int oj = min((int) (tile % tiles_x) * 8 + dj, f.out_w - 1);
        const int i = f.out_y + oi, j = f.out_x + oj;
        if (i < f.vh && j < f.vw) cost = ray_cost(f, i, j);
    }
    for (int o = 1; o < kCostRays; o <<= 1) cost = fmaxf(cost, __shfl_xor_sync(0xffffffffu, cost, o));
    if (tile < ntiles && r == 0) {
        const int kq = min(max((int) (__log2f(cost + 1.0f) * 4.0f), 0), kCostKeys - 1);
        key[tile] = (uint8_t) kq;
        atomicAdd(&hist[kq], 1);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < kCostKeys; t += blockDim.x)
        if (hist[t]) atomicAdd(&counts[t], hist[t]);
}

// The permutation, costliest key first: perm[start(key) + n] = tile, with
// start(key) the number of tiles of larger keys.  counts[64..127] are the
// per-key cursors (zero on entry); ties go in block order.
__global__ void tile_scatter_kernel(const uint8_t *key, int *counts, int *perm, long long ntiles)
{
    __shared__ int start[kCostKeys], loc[kCostKeys], base[kCostKeys];
    if (threadIdx.x < kCostKeys) loc[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int k = kCostKeys - 1; k >= 0; k--) {
            start[k] = acc;
            acc += counts[k];
        }
    }
    __syncthreads();
    const long long tile = (long long) blockIdx.x * blockDim.x + threadIdx.x;
    int kq = 0, rank = 0;
    if (tile < ntiles) {
        kq = key[tile];
        rank = atomicAdd(&loc[kq], 1);
    }
    __syncthreads();
    if (threadIdx.x < kCostKeys && loc[threadIdx.x] > 0)
        base[threadIdx.x] = atomicAdd(&counts[kCostKeys + threadIdx.x], loc[threadIdx.x]);
    __syncthreads();
    if (tile < ntiles) {
        const long long pos = (long long) start[kq] + base[kq] + rank;
        if (pos < ntiles) perm[pos] = (int) tile;
    }
}

// What the judge's verdict needs (from the frame descriptor).
struct JudgeArgs {
    JudgeWords *judge;
    int *judge_reject;
    int *learned_bad;
    int judge_tol;
};

// End of a judge launch for one block: the largest difference and pixel
// count of its warps go into the judge words (one set of atomics per block,
// not per warp: thousands of warps updating the same words would serialise
// on them); the launch's last block sets the verdict (fail = largest
// difference > tolerance), adds it to the totals, marks the learned grid
// wrong on failure and clears the per-frame words.  A grid already marked
// wrong was not used (the frame marched with the exact grid): nothing is
// judged and the frame counts as an exact one.  Every thread of the block
// calls it.
__device__ __forceinline__ void judge_finish(const JudgeArgs &a, int worst, unsigned judged, bool known_bad)
{
    __shared__ int b_worst;
    __shared__ unsigned b_judged;
    if (threadIdx.x == 0) {
        b_worst = 0;
        b_judged = 0;
    }
    __syncthreads();
    for (int o = 16; o > 0; o >>= 1) {
        worst = max(worst, __shfl_xor_sync(0xffffffffu, worst, o));
        judged += __shfl_xor_sync(0xffffffffu, judged, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (worst > 0) atomicMax_block(&b_worst, worst);
        if (judged) atomicAdd_block(&b_judged, judged);
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    JudgeWords *jw = a.judge;
    if (b_worst > 0) atomicMax(&jw->maxdiff, b_worst);
    if (b_judged) atomicAdd(&jw->pixels, (unsigned long long) b_judged);
    __threadfence();
    if (atomicAdd(&jw->warps_done, 1) != (int) gridDim.x - 1) return;  // counts blocks
    __threadfence();
    const int m = atomicAdd(&jw->maxdiff, 0);
    const int failed = m > a.judge_tol;
    jw->fail = failed;
    if (known_bad) {
        jw->exact_frames += 1;
    } else {
        jw->frames += 1;
        jw->fallbacks += (unsigned long long) failed;
        if (m > jw->worst) jw->worst = m;
    }
    if (failed) {
        *a.learned_bad = 1;
        *(volatile int *) a.judge_reject = 1;
        __threadfence_system();
    }
    jw->maxdiff = 0;
    jw->warps_done = 0;
}

// Tiles judged in a frame: judge_phase, judge_phase + judge_stride, ...
__host__ __device__ inline long long judged_tiles(long long ntiles, int stride, int phase)
{
    return ntiles > phase ? (ntiles - phase + stride - 1) / stride : 0;
}

// Tickets a launch of `total` tiles on `nwarps` warps takes: each tile after
// the warps' first ones, and one failed take per warp; none when the warps'
// first tiles are all.
__host__ __device__ inline long long launch_tickets(long long total, long long nwarps)
{
    return total > nwarps ? total : 0;
}

// Programmatic launches: a launch may begin while the one before it on its
// stream ends.  Until it has waited here it reads only what no launch in
// flight writes and stores nothing (a plain frame marches each warp's first
// tile; judged and gated launches read verdicts and wait at once); the launch
// after it may begin once all its blocks have waited.  Frames of 256x256 in a
// row: 47 -> 25 us each.
__device__ __forceinline__ void after_previous()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// CONFIG kernel, persistent: every warp takes one 8x4 pixel tile by its rank
// and then tiles from the view's ticket counter until none are left, so warps
// that drew short rays pick up more work instead of idling while the grid's
// last blocks finish.  Taken from the counter too, the first (costliest)
// tiles went four to a block to the SMs that started first: a 256x256 frame
// took 86 us, with the busiest SM at 55% and the mean at 7%, and takes 75 by
// rank.  With f.perm the n-th tile is perm[n] (costliest first).
// A gated launch (f.gate set) renders only if *f.gate != 0; otherwise it
// takes its share of tickets (launch_tickets) and leaves.
// JUDGE (learned skipping): the first tickets re-march the judged tiles
// (judge_phase modulo judge_stride) with the exact grids into f.judge8,
// each on its own warp, so that a judged heavy tile does not double the
// launch's longest warp; the rest render every tile.  A learned grid
// already marked wrong (*learned_bad) is not used: the tiles march with the
// exact grids and nothing is re-marched.  judge_compare_kernel gives the
// verdict afterwards.
template <int DT, bool SKIP, bool CENSUS, bool JUDGE>
__global__ void __launch_bounds__(kThreads, kCfgBlocksPerSm)
    march_cfg_kernel(const __grid_constant__ FrameDesc f, float4 *out32, uchar4 *out8)
{
    __shared__ unsigned s_runs[SKIP && !CENSUS ? kRunMax * kThreads : 1];
    unsigned long long nexec = 0, nlat = 0;
    const int lane = threadIdx.x & 31;
    const int tiles_x = (f.out_w + 7) >> 3;
    const long long ntiles = (long long) tiles_x * ((f.out_h + 3) >> 2);
    const long long njudged = JUDGE ? judged_tiles(ntiles, f.judge_stride, f.judge_phase) : 0;
    const long long total = ntiles + njudged, nwarps = (long long) gridDim.x * (kThreads / 32);
    if (JUDGE || CENSUS || f.gate != nullptr) after_previous();
    if (f.gate != nullptr && *f.gate == 0) {
        // no fallback: the launch's share of tickets in one add
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(f.tickets, (unsigned long long) launch_tickets(total, nwarps));
        return;
    }
    const bool exact = JUDGE && *(volatile const int *) f.learned_bad != 0;
    // the warp's first tile is its rank among the launch's warps, counted
    // across the blocks: the costliest tiles spread over the SMs, one each
    // before any has two
    long long q = (long long) (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    for (bool first = true;; first = false) {
        if (!first) {
            after_previous();
            if (total <= nwarps) break;
            unsigned long long ticket = 0;
            if (lane == 0) ticket = atomicAdd(f.tickets, 1ull);
            q = nwarps + (long long) (__shfl_sync(0xffffffffu, ticket, 0) - f.ticket_base);
            if (q >= total) break;
        } else if (q >= total) {
            continue;
        }
        // a judged tile (re-marched with the exact grids into judge8) or a
        // render tile, through one copy of the march
        const bool judge = JUDGE && q < njudged;
        if (judge && exact) continue;
        long long tile;
        if (judge) {
            tile = q * f.judge_stride + f.judge_phase;
        } else {
            tile = q - njudged;
            if (f.perm != nullptr) {
                const long long p = f.perm[tile];
                if (p >= 0 && p < ntiles) tile = p;  // a permutation by construction; never leave the window
            }
        }
        const int oi = (int) (tile / tiles_x) * 4 + (lane >> 3), oj = (int) (tile % tiles_x) * 8 + (lane & 7);
        const bool in_window = oi < f.out_h && oj < f.out_w;
        const int i = f.out_y + oi, j = f.out_x + oj;
        const float4 acc =
            ray_cfg<DT, SKIP, CENSUS, cfg_k<DT>()>(
                f, i, j, in_window && i < f.vh && j < f.vw, nexec, nlat, s_runs + threadIdx.x, judge || exact);
        const uchar4 a8 = make_uchar4(q8(acc.x), q8(acc.y), q8(acc.z), q8(acc.w));
        if (first) after_previous();
        if (judge) {
            f.judge8[q * 32 + lane] = a8;
        } else if (in_window) {
            const long long o = (long long) oi * f.out_w + oj;
            if (out32) out32[o] = acc;
            if (out8) out8[o] = a8;
        }
    }
    if (CENSUS) count_exec(f, nexec, nlat);
}

// The verdict of a learned-skip frame: each warp compares one judged tile's
// exact re-march (judge8) with the stored frame (out8, or out32 quantised).
__global__ void judge_compare_kernel(JudgeArgs a, const uchar4 *judge8, const uchar4 *out8, const float4 *out32,
                                     int out_x, int out_y, int out_w, int out_h, int vw, int vh, int stride,
                                     int phase)
{
    const int lane = threadIdx.x & 31;
    const int tiles_x = (out_w + 7) >> 3;
    const long long njudged = judged_tiles((long long) tiles_x * ((out_h + 3) >> 2), stride, phase);
    const bool known_bad = *(volatile const int *) a.learned_bad != 0;
    int worst = 0;
    unsigned judged = 0;
    if (!known_bad)
        for (long long q = (long long) blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); q < njudged;
             q += (long long) gridDim.x * (blockDim.x >> 5)) {
            const long long tile = q * stride + phase;
            const int oi = (int) (tile / tiles_x) * 4 + (lane >> 3), oj = (int) (tile % tiles_x) * 8 + (lane & 7);
            if (oi < out_h && oj < out_w && out_y + oi < vh && out_x + oj < vw) {
                const uchar4 e = judge8[q * 32 + lane];
                const long long o = (long long) oi * out_w + oj;
                uchar4 v;
                if (out8) {
                    v = out8[o];
                } else {
                    const float4 c = out32[o];
                    v = make_uchar4(q8(c.x), q8(c.y), q8(c.z), q8(c.w));
                }
                const int d = max(max(abs((int) v.x - (int) e.x), abs((int) v.y - (int) e.y)),
                                  max(abs((int) v.z - (int) e.z), abs((int) v.w - (int) e.w)));
                worst = max(worst, d);
                judged++;
            }
        }
    judge_finish(a, worst, judged, known_bad);
}

// Sample-rate roofline: the CONFIG sampler (trilinear reconstruction, LUT
// fetch, front-to-back blend) with nothing else -- no ray set-up, skipping,
// termination or divergence -- over a brick small enough to stay in L1/L2.
// Each thread marches its own ray of `steps` samples, 0.5 voxel apart, from
// a start that neighbouring lanes share up to a voxel, as in an 8x4 tile.
// One sample of the roofline's brick through a sampler layout: the
// march's own sampler (corner-packed copy, or the brick itself when b.quad
// is null), or a 3D texture of the brick -- eight point fetches blended as
// fetch_cfg does (the same value, bit for bit), or one hardware-filtered
// fetch (fixed-point weights).
template <int DT, int LAYOUT>
__device__ __forceinline__ float sample_layout(const DevBrick &b, const SamplerTex &t, float ux, float uy, float uz)
{
    if (LAYOUT == IVR_SAMPLER_QUADS || LAYOUT == IVR_SAMPLER_BRICKS) return sample_cfg<DT>(b, ux, uy, uz);
    const CellPos c = cell_cfg(b, ux, uy, uz);
    if (LAYOUT == IVR_SAMPLER_TEX_LINEAR)
        return tex3D<float>(t.linear, (float) c.j + c.fx + 0.5f, (float) c.i + c.fy + 0.5f,
                            (float) c.k + c.fz + 0.5f) * t.scale;
    using T = typename VoxT<DT>::T;
    const float x0 = (float) c.j + 0.5f, y0 = (float) c.i + 0.5f, z0 = (float) c.k + 0.5f;
    const float x1 = x0 + 1.0f, y1 = y0 + 1.0f, z1 = z0 + 1.0f;
    const float c00 = lerpf((float) tex3D<T>(t.point, x0, y0, z0), (float) tex3D<T>(t.point, x1, y0, z0), c.fx);
    const float c10 = lerpf((float) tex3D<T>(t.point, x0, y1, z0), (float) tex3D<T>(t.point, x1, y1, z0), c.fx);
    const float c01 = lerpf((float) tex3D<T>(t.point, x0, y0, z1), (float) tex3D<T>(t.point, x1, y0, z1), c.fx);
    const float c11 = lerpf((float) tex3D<T>(t.point, x0, y1, z1), (float) tex3D<T>(t.point, x1, y1, z1), c.fx);
    return lerpf(lerpf(c00, c10, c.fy), lerpf(c01, c11, c.fy), c.fz);
}

template <int DT, int LAYOUT>
__global__ void __launch_bounds__(kThreads, kPeakBlocksPerSm) sample_peak_kernel(const __grid_constant__ FrameDesc f,
                                                                                SamplerTex tex, int steps,
                                                                                float4 *out)
{
    const DevBrick &b = f.b[0];
    const unsigned gid = blockIdx.x * blockDim.x + threadIdx.x;
    // the warp's 8x4 tile of starts, one voxel apart, at a hashed place
    const unsigned w = gid >> 5, lane = gid & 31;
    const unsigned h = w * 2654435761u;
    // positions in the brick's voxel coordinates, as the march samples
    const float sx = (float) (b.nx - 2), sy = (float) (b.ny - 2), sz = (float) (b.nz - 2);
    float x = 2.0f + (float) (h % 997u) / 997.0f * (sx - 12.0f) + (float) (lane & 7);
    float y = 2.0f + (float) ((h >> 10) % 991u) / 991.0f * (sy - 8.0f) + (float) (lane >> 3);
    float z = 2.0f + (float) ((h >> 20) % 983u) / 983.0f * (sz - 4.0f);
    // half a voxel per step along a direction fixed per warp
    const float dx = (w & 1) ? 0.3f : -0.3f, dy = (w & 2) ? 0.2f : -0.2f, dz = (w & 4) ? 0.35f : -0.35f;
    const float lox = 1.0f, hix = sx - 1.0f;
    const float loy = 1.0f, hiy = sy - 1.0f;
    const float loz = 1.0f, hiz = sz - 1.0f;
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int i = 0; i < steps; i++) {
        const float s = sample_layout<DT, LAYOUT>(b, tex, x, y, z);
        const float4 e = lut_at(f, lut_index((int) (s * f.lut_scale), f.lut_off));
        const float wgt = (1.0f - acc.w) * (e.w * f.alpha);
        acc.x = fmaf(wgt, e.x, acc.x);
        acc.y = fmaf(wgt, e.y, acc.y);
        acc.z = fmaf(wgt, e.z, acc.z);
        acc.w = acc.w * 0.5f + wgt;  // stays below 1: no termination
        x += dx;
        y += dy;
        z += dz;
        // reflect at the faces so the ray stays inside the brick
        x = x < lox ? 2.0f * lox - x : (x > hix ? 2.0f * hix - x : x);
        y = y < loy ? 2.0f * loy - y : (y > hiy ? 2.0f * hiy - y : y);
        z = z < loz ? 2.0f * loz - z : (z > hiz ? 2.0f * hiz - z : z);
    }
    out[gid] = acc;
}

// The largest |layout sample - exact trilinear sample (the brick itself)|
// over npos hashed positions of the brick, as float bits into *err.
template <int DT, int LAYOUT>
__global__ void sample_err_kernel(const __grid_constant__ FrameDesc f, SamplerTex tex, int npos, unsigned *err)
{
    const DevBrick &b = f.b[0];
    DevBrick ref = b;
    ref.quad = nullptr;
    float worst = 0.0f;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npos; p += gridDim.x * blockDim.x) {
        unsigned h = (unsigned) p * 2654435761u + 12345u;
        const float ux = (float) ((h = h * 1664525u + 1013904223u) >> 8) / 16777216.0f * (float) (b.nx - 1);
        const float uy = (float) ((h = h * 1664525u + 1013904223u) >> 8) / 16777216.0f * (float) (b.ny - 1);
        const float uz = (float) ((h = h * 1664525u + 1013904223u) >> 8) / 16777216.0f * (float) (b.nz - 1);
        worst = fmaxf(worst, fabsf(sample_layout<DT, LAYOUT>(b, tex, ux, uy, uz) - sample_cfg<DT>(ref, ux, uy, uz)));
    }
    atomicMax(err, __float_as_uint(worst));  // non-negative floats order as their bits
}

// SM count of the current device, looked up once per device
int sm_count()
{
    static std::atomic<int> count[64];
    int dev = 0;
    cudaGetDevice(&dev);
    int sms = dev >= 0 && dev < 64 ? count[dev].load(std::memory_order_relaxed) : 0;
    if (sms == 0) {
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (dev >= 0 && dev < 64) count[dev].store(sms, std::memory_order_relaxed);
    }
    return sms;
}

template <typename K>
int persistent_grid(K kernel, size_t smem)
{
    const int sms = sm_count();
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, smem);
    return sms * (per_sm > 0 ? per_sm : 1);
}

template <int DT>
cudaError_t launch_dt(const FrameDesc &f, float4 *o32, uchar4 *o8, cudaStream_t s, long long *warps_launched,
                      bool early)
{
    dim3 grid((f.out_w + kBlockX - 1) / kBlockX, (f.out_h + kBlockY - 1) / kBlockY);
    if (f.preset == IVR_PRESET_CONFIG) {
        bool skip = false;
        for (int k = 0; k < f.nb; k++) skip |= f.b[k].empty != nullptr;
        const bool judge = f.judge != nullptr;
        if (judge && (!skip || f.census || !f.judge8 || f.judge_stride < 1 || f.judge_phase < 0 ||
                      f.judge_phase >= f.judge_stride))
            return cudaErrorInvalidValue;
        auto kern = f.census ? (skip ? march_cfg_kernel<DT, true, true, false> : march_cfg_kernel<DT, false, true, false>)
                    : judge  ? march_cfg_kernel<DT, true, false, true>
                    : skip   ? march_cfg_kernel<DT, true, false, false>
                             : march_cfg_kernel<DT, false, false, false>;
        const long long ntiles = (long long) ((f.out_w + 7) >> 3) * ((f.out_h + 3) >> 2);
        const long long total = ntiles + (judge ? judged_tiles(ntiles, f.judge_stride, f.judge_phase) : 0);
        constexpr int kWarps = kThreads / 32;
        const int blocks = (int) std::min((long long) persistent_grid(kern, 0), (total + kWarps - 1) / kWarps);
        if (warps_launched) *warps_launched = launch_tickets(total, (long long) blocks * kWarps);
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned) blocks);
        cfg.blockDim = dim3(kThreads);
        cfg.stream = s;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr.val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = early ? 1 : 0;
        return cudaLaunchKernelEx(&cfg, kern, f, o32, o8);
    }
    if (warps_launched) *warps_launched = 0;
    switch (f.tf_mode) {
    case IVR_TF_SEISMIC: march_ref_kernel<DT, IVR_TF_SEISMIC><<<grid, kThreads, 0, s>>>(f, o32, o8); break;
    case IVR_TF_MED: march_ref_kernel<DT, IVR_TF_MED><<<grid, kThreads, 0, s>>>(f, o32, o8); break;
    case IVR_TF_SEISMIC2: march_ref_kernel<DT, IVR_TF_SEISMIC2><<<grid, kThreads, 0, s>>>(f, o32, o8); break;
    case IVR_TF_CHEM: march_ref_kernel<DT, IVR_TF_CHEM><<<grid, kThreads, 0, s>>>(f, o32, o8); break;
    case IVR_TF_BLEND: march_ref_kernel<DT, IVR_TF_BLEND><<<grid, kThreads, 0, s>>>(f, o32, o8); break;
    case IVR_TF_RGBBLEND: march_ref_kernel<DT, IVR_TF_RGBBLEND><<<grid, kThreads, 0, s>>>(f, o32, o8); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// Batched CONFIG kernel: the tiles of every frame of a batch in one
// persistent launch.  Frame descriptors are in device memory (uploaded with
// the batch); a warp's ticket is a global tile number, mapped to its frame by
// a binary search over the frames' first tiles.  Warp tiles are TW x (32/TW)
// pixels; PAIR takes batch_k samples per loop iteration, else one.
template <int DT, int TW, bool PAIR>
__global__ void __launch_bounds__(kThreads, kBatchBlocksPerSm)
    march_batch_kernel(const BatchHeader *__restrict__ hdr, const BatchItem *__restrict__ items,
                       unsigned long long *ticket)
{
    constexpr int TH = 32 / TW;
    __shared__ unsigned s_runs[kRunMax * kThreads];
    __shared__ float s_ray[kRayWords * kThreads];
    const int lane = threadIdx.x & 31;
    const int n = hdr->nitems;
    const long long total = hdr->total_tiles;
    unsigned long long nexec = 0, nlat = 0;
    for (;;) {
        unsigned long long t = 0;
        if (lane == 0) t = atomicAdd(ticket, 1ull);
        const long long g = (long long) __shfl_sync(0xffffffffu, t, 0);
        if (g >= total) break;
        int lo = 0, hi = n - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (items[mid].tile0 <= g) lo = mid;
            else hi = mid - 1;
        }
        const BatchItem &it = items[lo];
        const long long tile = g - it.tile0;
        pixel_cfg<DT, true, false, PAIR ? batch_k<DT>() : 1, true>(it.f, (int) (tile / it.tiles_x) * TH + lane / TW,
                                        (int) (tile % it.tiles_x) * TW + lane % TW, it.out32, it.out8, nexec, nlat,
                                        s_runs + threadIdx.x, s_ray + threadIdx.x);
    }
}

template <int DT, int TW, bool PAIR>
cudaError_t launch_batch_v(const BatchHeader *hdr, const BatchItem *items, unsigned long long *ticket,
                           cudaStream_t s)
{
    auto kern = march_batch_kernel<DT, TW, PAIR>;
    // shared memory for the resident blocks (1 KB each is the system's) and
    // the rest of the 256 KB to L1, which bounds the kernel: the driver's own
    // choice, 100 KB, takes 3672 us for 32 f32 frames, this 3623 (20 u16 frames
    // 2528 and 2493, u8 2397 and 2365).
    // The frame kernels measured the same at 12 to 25%.
    constexpr int kSmem = kBatchBlocksPerSm * (int) (sizeof(float) * kThreads * (kRunMax + kRayWords) + 1024);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         (100 * kSmem + 228 * 1024 - 1) / (228 * 1024));
    if (e != cudaSuccess) return e;
    kern<<<persistent_grid(kern, 0), kThreads, 0, s>>>(hdr, items, ticket);
    return cudaGetLastError();
}

template <int DT>
cudaError_t launch_batch_dt(int variant, const BatchHeader *hdr, const BatchItem *items, unsigned long long *ticket,
                            cudaStream_t s)
{
    switch (variant) {
    case 0: return launch_batch_v<DT, 8, true>(hdr, items, ticket, s);
    case 1: return launch_batch_v<DT, 8, false>(hdr, items, ticket, s);
    case 2: return launch_batch_v<DT, 4, true>(hdr, items, ticket, s);
    case 3: return launch_batch_v<DT, 4, false>(hdr, items, ticket, s);
    case 4: return launch_batch_v<DT, 16, true>(hdr, items, ticket, s);
    case 5: return launch_batch_v<DT, 16, false>(hdr, items, ticket, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

int batch_variant_tile_w(int variant) { return variant < 2 ? 8 : variant < 4 ? 4 : 16; }

cudaError_t launch_batch(int dtype, int variant, const BatchHeader *hdr, const BatchItem *items,
                         unsigned long long *ticket, cudaStream_t s)
{
    switch (dtype) {
    case IVR_U8: return launch_batch_dt<IVR_U8>(variant, hdr, items, ticket, s);
    case IVR_U16: return launch_batch_dt<IVR_U16>(variant, hdr, items, ticket, s);
    case IVR_F32: return launch_batch_dt<IVR_F32>(variant, hdr, items, ticket, s);
    default: return cudaErrorInvalidValue;
    }
}

template <int DT, int LAYOUT>
cudaError_t launch_sample_layout(const FrameDesc &f, const SamplerTex &tex, int steps, float4 *out,
                                 long long *samples, unsigned *err, cudaStream_t s)
{
    auto kern = sample_peak_kernel<DT, LAYOUT>;
    const int blocks = persistent_grid(kern, 0);
    if (out) {
        kern<<<blocks, kThreads, 0, s>>>(f, tex, steps, out);
        *samples = (long long) blocks * kThreads * steps;
    }
    if (err) sample_err_kernel<DT, LAYOUT><<<256, 256, 0, s>>>(f, tex, 1 << 20, err);
    return cudaGetLastError();
}

template <int DT>
cudaError_t launch_sample_dt(const FrameDesc &f, int layout, const SamplerTex &tex, int steps, float4 *out,
                             long long *samples, unsigned *err, cudaStream_t s)
{
    switch (layout) {
    case IVR_SAMPLER_QUADS: return launch_sample_layout<DT, IVR_SAMPLER_QUADS>(f, tex, steps, out, samples, err, s);
    case IVR_SAMPLER_BRICKS: return launch_sample_layout<DT, IVR_SAMPLER_BRICKS>(f, tex, steps, out, samples, err, s);
    case IVR_SAMPLER_TEX_POINT:
        return launch_sample_layout<DT, IVR_SAMPLER_TEX_POINT>(f, tex, steps, out, samples, err, s);
    case IVR_SAMPLER_TEX_LINEAR:
        return launch_sample_layout<DT, IVR_SAMPLER_TEX_LINEAR>(f, tex, steps, out, samples, err, s);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_sample_peak(const FrameDesc &f, int layout, const SamplerTex &tex, int steps, float4 *out,
                               long long *samples, unsigned *err, cudaStream_t s)
{
    switch (f.dtype) {
    case IVR_U8: return launch_sample_dt<IVR_U8>(f, layout, tex, steps, out, samples, err, s);
    case IVR_U16: return launch_sample_dt<IVR_U16>(f, layout, tex, steps, out, samples, err, s);
    case IVR_F32: return launch_sample_dt<IVR_F32>(f, layout, tex, steps, out, samples, err, s);
    default: return cudaErrorInvalidValue;
    }
}

int sample_peak_threads()
{
    return persistent_grid(sample_peak_kernel<IVR_F32, IVR_SAMPLER_QUADS>, 0) * kThreads;
}

cudaError_t launch_judge_compare(const FrameDesc &f, const uchar4 *out8, const float4 *out32, cudaStream_t s)
{
    const long long ntiles = (long long) ((f.out_w + 7) >> 3) * ((f.out_h + 3) >> 2);
    const long long nj = judged_tiles(ntiles, f.judge_stride, f.judge_phase);
    const long long blocks = nj > 0 ? (nj + 7) / 8 : 1;  // a warp per judged tile
    JudgeArgs a{f.judge, f.judge_reject, f.learned_bad, f.judge_tol};
    judge_compare_kernel<<<(unsigned) (blocks < 152 * 16 ? blocks : 152 * 16), 256, 0, s>>>(
        a, f.judge8, out8, out32, f.out_x, f.out_y, f.out_w, f.out_h, f.vw, f.vh, f.judge_stride, f.judge_phase);
    return cudaGetLastError();
}

// The order shortens the end of a launch whose warps draw several tiles each;
// below that the next frame's launch, which may begin in row order while this
// one ends (launch_march's early), fills it better.  us a frame, cost / row
// order: 2048 tiles 52 / 25, 9600 164 / 160, 15000 107 / 100, 32768 304 / 317,
// 64800 333 / 354; for one frame alone the row order is 10 to 25 us faster up
// to 15000 tiles and equal above.
bool tile_order_pays(const FrameDesc &f)
{
    constexpr long long kTilesPerWarp = 8;
    const long long ntiles = (long long) ((f.out_w + 7) >> 3) * ((f.out_h + 3) >> 2);
    return ntiles >= kTilesPerWarp * sm_count() * kCfgBlocksPerSm * (kThreads / 32);
}

cudaError_t launch_tile_order(const FrameDesc &f, uint8_t *key, int *counts, int *perm, cudaStream_t s)
{
    const long long ntiles = (long long) ((f.out_w + 7) >> 3) * ((f.out_h + 3) >> 2);
    if (ntiles <= 0) return cudaSuccess;
    if (ntiles > (1ll << 30)) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(counts, 0, sizeof(int) * 2 * kCostKeys, s);
    if (e != cudaSuccess) return e;
    tile_cost_kernel<<<(unsigned) ((ntiles * kCostRays + 127) / 128), 128, 0, s>>>(f, key, counts, ntiles);
    tile_scatter_kernel<<<(unsigned) ((ntiles + 255) / 256), 256, 0, s>>>(key, counts, perm, ntiles);
    return cudaGetLastError();
}

long long judge_scratch_bytes(const FrameDesc &f)
{
    const long long ntiles = (long long) ((f.out_w + 7) >> 3) * ((f.out_h + 3) >> 2);
    return judged_tiles(ntiles, f.judge_stride, f.judge_phase) * 32 * (long long) sizeof(uchar4);
}

cudaError_t launch_march(const FrameDesc &f, float4 *out32, uchar4 *out8, cudaStream_t s, long long *warps, bool early)
{
    if (warps) *warps = 0;
    if (f.out_w <= 0 || f.out_h <= 0) return cudaSuccess;
    switch (f.dtype) {
    case IVR_U8: return launch_dt<IVR_U8>(f, out32, out8, s, warps, early);
    case IVR_U16: return launch_dt<IVR_U16>(f, out32, out8, s, warps, early);
    case IVR_F32: return launch_dt<IVR_F32>(f, out32, out8, s, warps, early);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace ivr
