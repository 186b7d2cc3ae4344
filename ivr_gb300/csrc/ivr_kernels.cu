// ivr_kernels.cu -- the kernels around the march: byte swap, brick gather,
// min/max + histogram (initvolluts), macrocell min/max and per-TF empty
// flags, sort-last compositing (compositetiles) and RGBA8 quantisation.
// Compiled with -fmad=false like the march.
#include <float.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "ivr_internal.h"
#include "ivr_mlp.h"

namespace ivr {
namespace {

constexpr int kSms = 152;

int grid_for(long long n, int threads, int per_sm = 8)
{
    long long g = (n + threads - 1) / threads;
    long long cap = (long long) kSms * per_sm;
    return (int) (g < cap ? (g < 1 ? 1 : g) : cap);
}

__global__ void byteswap16_kernel(uint16_t *p, long long n)
{
    for (long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < n; i += (long long) gridDim.x * blockDim.x)
        p[i] = (uint16_t) ((p[i] >> 8) | (p[i] << 8));
}

// BYTESWAP_FP (sysutil.h:121-133): byte order reversed
__global__ void byteswap32_kernel(uint32_t *p, long long n)
{
    for (long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < n; i += (long long) gridDim.x * blockDim.x)
        p[i] = __byte_perm(p[i], 0, 0x0123);
}

// readfromfile (main.c:1254-1265): brick [sz..sz+ld) x [sy..sy+lh) x
// [sx..sx+lw) of the global volume into a dense [ld][lh][lw] array.
// A warp copies whole rows, four 32-voxel pieces in flight; HBM-bound.
template <typename T>
__global__ void __launch_bounds__(256) gather_kernel(const T *__restrict__ src, int gw, int gh, T *__restrict__ dst,
                                                     int sx, int sy, int sz, int lw, int lh, long long rows)
{
    const int lane = threadIdx.x & 31;
    const long long r = (long long) blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (r >= rows) return;
    const int y = (int) (r % lh), z = (int) (r / lh);
    const T *p = src + ((long long) (sz + z) * gh + (sy + y)) * gw + sx;
    T *q = dst + r * lw;
    for (int x = lane; x < lw; x += 128) {
        T v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = x + 32 * u < lw ? __ldg(p + x + 32 * u) : T(0);
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (x + 32 * u < lw) q[x + 32 * u] = v[u];
    }
}

// 16 bytes of voxels at a time: the passes over a whole volume (min/max,
// histogram) read it with aligned vector loads; the volume's own array is a
// device allocation, so its base is aligned for every dtype, and the last
// n % kVec voxels are read one by one.
template <typename T> constexpr int kVec = 16 / (int) sizeof(T);

template <typename T> __device__ __forceinline__ T vox_of(const uint4 &q, int e)
{
    const unsigned w = (&q.x)[e * (int) sizeof(T) / 4];
    if constexpr (sizeof(T) == 4) return __uint_as_float(w);
    else return (T) (w >> (8 * ((e * (int) sizeof(T)) & 3)));
}

// Min and max of the volume, one pair per block.  Bound by HBM.  Each thread
// keeps four 16-byte loads in flight; integer voxels are compared as packed
// lanes and converted once at the end (the conversion is exact and
// monotone), floats with fminf/fmaxf, which pass over NaNs.
template <typename T> struct MinMaxAcc {
    // packed lanes of a 32-bit word
    unsigned lo = 0xffffffffu, hi = 0u;
    __device__ __forceinline__ void word(unsigned w)
    {
        if constexpr (sizeof(T) == 1) {
            lo = __vminu4(lo, w);
            hi = __vmaxu4(hi, w);
        } else {
            lo = __vminu2(lo, w);
            hi = __vmaxu2(hi, w);
        }
    }
    __device__ __forceinline__ void one(T v)
    {
        unsigned w = v;
        for (int b = 8 * (int) sizeof(T); b < 32; b *= 2) w |= w << b;
        word(w);
    }
    __device__ __forceinline__ void get(float &l, float &h) const
    {
        unsigned a = 0xffffffffu, b = 0u;
        for (int e = 0; e < 4 / (int) sizeof(T); e++) {
            a = min(a, (unsigned) (T) (lo >> (8 * (int) sizeof(T) * e)));
            b = max(b, (unsigned) (T) (hi >> (8 * (int) sizeof(T) * e)));
        }
        l = (float) a;
        h = (float) b;
    }
};
template <> struct MinMaxAcc<float> {
    float lo = FLT_MAX, hi = -FLT_MAX;
    __device__ __forceinline__ void one(float v)
    {
        lo = fminf(lo, v);
        hi = fmaxf(hi, v);
    }
    __device__ __forceinline__ void word(unsigned w) { one(__uint_as_float(w)); }
    __device__ __forceinline__ void get(float &l, float &h) const
    {
        l = lo;
        h = hi;
    }
};

template <typename T>
__global__ void minmax_kernel(const T *__restrict__ data, long long n, float *partial)
{
    MinMaxAcc<T> acc;
    const long long nv = n / kVec<T>, stride = (long long) gridDim.x * blockDim.x;
    const long long t = blockIdx.x * (long long) blockDim.x + threadIdx.x;
    const uint4 *q = reinterpret_cast<const uint4 *>(data);
    long long i = t;
    bool any = false;
    for (; i + 3 * stride < nv; i += 4 * stride) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = __ldcs(q + i + u * stride);
#pragma unroll
        for (int u = 0; u < 4; u++) {
            acc.word(v[u].x);
            acc.word(v[u].y);
            acc.word(v[u].z);
            acc.word(v[u].w);
        }
        any = true;
    }
    for (; i < nv; i += stride) {
        const uint4 v = __ldcs(q + i);
        acc.word(v.x);
        acc.word(v.y);
        acc.word(v.z);
        acc.word(v.w);
        any = true;
    }
    if (t < n - nv * kVec<T>) {
        acc.one(__ldg(data + nv * kVec<T> + t));
        any = true;
    }
    float lo = FLT_MAX, hi = -FLT_MAX;
    if (any) acc.get(lo, hi);
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    __shared__ float slo[32], shi[32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { slo[w] = lo; shi[w] = hi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < (int) (blockDim.x >> 5); k++) { lo = fminf(lo, slo[k]); hi = fmaxf(hi, shi[k]); }
        partial[2 * blockIdx.x] = lo;
        partial[2 * blockIdx.x + 1] = hi;
    }
}

// The value range as a kernel argument: known to the host, or still in
// device memory (the allocation-free histogram).
struct MinArg {
    float v;
    const float *dev;
};

// histogram (mathutil.c:459-467): bin (int)(v - min).  Bound by the atomics:
// one shared-memory counter per voxel, and background voxels that all want
// the same one.  (One global atomic per voxel above 12,288 bins took 65.7 ms
// for 512^3 u16 voxels with 70% background; with its result copied to the
// host this takes 0.16 ms.  Adding the blocks' counters up over clusters of 2, 4
// or 8 first: 0.16, 0.17, 0.21.)
// - The bins are cut into `gridDim.y` ranges of `nb` that fit a block's
//   shared memory (65,536 bins take two ranges of 128 KB: 256 KB do not fit
//   an SM); every range's blocks read the whole volume, the second reader
//   mostly from L2.
// - A range with room to spare keeps 2^rep copies of each counter, the copy
//   by lane, so that equal neighbours in a warp do not wait for each other.
// - Each thread counts bin 0 (the minimum: the background) in a register, and
//   16 bytes of one value (background, saturated regions) as one addition.
//   (Runs carried from voxel to voxel instead took two branches a voxel: 183
//   us for 512^3 u16 voxels against 120.)
template <typename T>
__global__ void __launch_bounds__(1024) hist_kernel(const T *__restrict__ data, long long n, MinArg mn, int hsize,
                                                    int nb, int rep, int *hist)
{
    extern __shared__ int sh[];
    const int first = (int) blockIdx.y * nb, bins = min(nb, hsize - first);
    for (int b = threadIdx.x; b < bins << rep; b += blockDim.x) sh[b] = 0;
    __syncthreads();
    const float fmin = mn.dev ? __ldg(mn.dev) : mn.v;
    // integer voxels: their minimum is an integer too, and the float
    // difference the rule takes is exact, so the bin is the integer difference
    const int imin = sizeof(T) < 4 ? (int) fmin : 0;
    const int copy = threadIdx.x & ((1 << rep) - 1);
    int zero = 0;
    auto add = [&](T v, int count) {
        const int b = (int) ((unsigned) (sizeof(T) < 4 ? (int) v - imin : (int) ((float) v - fmin)) - (unsigned) first);
        if (b == 0) zero += count;
        else if ((unsigned) b < (unsigned) bins) atomicAdd(&sh[(b << rep) + copy], count);
    };
    auto add16 = [&](const uint4 &q) {
        const unsigned w = q.x;
        bool same = q.y == w && q.z == w && q.w == w;
        if (sizeof(T) < 4) same = same && w == __byte_perm(w, 0, sizeof(T) == 1 ? 0x0000 : 0x1010);
        if (same) {
            add(vox_of<T>(q, 0), kVec<T>);
        } else {
#pragma unroll
            for (int e = 0; e < kVec<T>; e++) add(vox_of<T>(q, e), 1);
        }
    };
    const long long nv = n / kVec<T>, stride = (long long) gridDim.x * blockDim.x;
    const long long t = blockIdx.x * (long long) blockDim.x + threadIdx.x;
    const uint4 *q = reinterpret_cast<const uint4 *>(data);
    long long i = t;
    for (; i + 3 * stride < nv; i += 4 * stride) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = __ldg(q + i + u * stride);
#pragma unroll
        for (int u = 0; u < 4; u++) add16(v[u]);
    }
    for (; i < nv; i += stride) add16(__ldg(q + i));
    if (t < n - nv * kVec<T>) add(__ldg(data + nv * kVec<T> + t), 1);
    zero = __reduce_add_sync(0xffffffffu, zero);
    if ((threadIdx.x & 31) == 0 && zero) atomicAdd(&sh[0], zero);
    __syncthreads();
    // neighbouring blocks start at different bins, so that their additions
    // to the result do not meet
    const int turn = (int) ((long long) blockIdx.x * bins / gridDim.x);
    for (int k = threadIdx.x; k < bins; k += blockDim.x) {
        const int b = k + turn < bins ? k + turn : k + turn - bins;
        int c = 0;
        for (int r = 0; r < 1 << rep; r++) c += sh[(b << rep) + ((r + threadIdx.x) & ((1 << rep) - 1))];
        if (c) atomicAdd(&hist[first + b], c);
    }
}

// The same for volumes of few voxels and as many bins as a block's static
// shared memory has counters: a counter a bin, a voxel a step, small blocks.
// What bounds it are the launch and the counters' clearing and adding up, which
// hist_kernel's large blocks, copies and vectors only make longer.  Kernel
// alone, this and hist_kernel: 32^3 u8, 256 bins 2.1 and 3.9 us, 116^3 f32, 256
// bins 3.4 and 5.7, 160^3 u16, 4096 bins 10.4 and 8.7.
constexpr int kHistFewBins = 12288;
template <typename T>
__global__ void __launch_bounds__(512) hist_few_kernel(const T *__restrict__ data, long long n, MinArg mn, int hsize,
                                                       int *hist)
{
    __shared__ int sh[kHistFewBins];
    for (int b = threadIdx.x; b < hsize; b += blockDim.x) sh[b] = 0;
    __syncthreads();
    const float fmin = mn.dev ? __ldg(mn.dev) : mn.v;
    for (long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < n; i += (long long) gridDim.x * blockDim.x) {
        const int b = (int) ((float) __ldg(data + i) - fmin);
        if ((unsigned) b < (unsigned) hsize) atomicAdd(&sh[b], 1);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < hsize; b += blockDim.x)
        if (sh[b]) atomicAdd(&hist[b], sh[b]);
}

// The same with the counters in global memory: for more bins than two ranges
// hold (float volumes of a wide range), and for volumes too small to pay for
// clearing and adding up the shared counters of more bins than hist_few_kernel
// takes.
template <typename T>
__global__ void hist_global_kernel(const T *__restrict__ data, long long n, MinArg mn, int hsize, int *hist)
{
    const float fmin = mn.dev ? __ldg(mn.dev) : mn.v;
    int zero = 0, cur = -1, run = 0;
    for (long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < n; i += (long long) gridDim.x * blockDim.x) {
        const int b = (int) ((float) __ldg(data + i) - fmin);
        if (b == 0) {
            zero++;
        } else {
            if (b != cur) {
                if ((unsigned) cur < (unsigned) hsize) atomicAdd(&hist[cur], run);
                cur = b;
                run = 0;
            }
            run++;
        }
    }
    if ((unsigned) cur < (unsigned) hsize) atomicAdd(&hist[cur], run);
    zero = __reduce_add_sync(0xffffffffu, zero);
    if ((threadIdx.x & 31) == 0 && zero) atomicAdd(&hist[0], zero);
}

// Macrocell min/max: with edge c = 2^cs, cell (cx,cy,cz) spans voxels
// [c*cx, min(c*cx+c, n-1)] per axis -- its voxel cells plus the +1 layer a
// trilinear sample in the cell also reads.  HBM-bound: the volume is read
// once, (c+1)^2/c^2 of it with the layers that neighbouring cells share
// (those mostly from L2).  A block takes the cells over a segment of kCols
// columns: its 8 warps share the (c+1)^2 rows of the segment, each lane
// keeping the min and max of its columns over its warp's rows, and the rows'
// results meet in shared memory.  One block per cell with two divisions per
// voxel took 3.5 ms for 1024^3 u16 voxels (0.6 TB/s).
// VEC: rows start on 16 bytes and a lane's columns are one 16-byte load,
// integer voxels compared as packed lanes; otherwise they are 4 columns 32
// apart.
constexpr int kMcWarps = 8;
template <typename T, bool VEC> struct McTile {
    static constexpr int kPer = VEC ? kVec<T> : 4;  // columns a lane
    static constexpr int kCols = 32 * kPer;
    T lo[kMcWarps][kCols], hi[kMcWarps][kCols];
    T xlo[kMcWarps], xhi[kMcWarps];  // the column after the segment
};
template <typename T> __device__ __forceinline__ T vmin_of(T a, T b) { return a < b ? a : b; }
template <typename T> __device__ __forceinline__ T vmax_of(T a, T b) { return a > b ? a : b; }
template <> __device__ __forceinline__ float vmin_of(float a, float b) { return fminf(a, b); }
template <> __device__ __forceinline__ float vmax_of(float a, float b) { return fmaxf(a, b); }
template <typename T> __device__ __forceinline__ T vtop() { return (T) ~(T) 0; }
template <> __device__ __forceinline__ float vtop<float>() { return FLT_MAX; }
template <typename T> __device__ __forceinline__ T vbottom() { return 0; }
template <> __device__ __forceinline__ float vbottom<float>() { return -FLT_MAX; }

template <typename T, bool VEC>
__global__ void __launch_bounds__(32 * kMcWarps) macrocell_kernel(const T *__restrict__ data, int nx, int ny, int nz,
                                                                  int cs, float *mc, int mcx, int mcy, int nseg)
{
    using Tile = McTile<T, VEC>;
    constexpr int kPer = Tile::kPer, kCols = Tile::kCols;
    __shared__ __align__(16) Tile s;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = 1 << cs;
    const unsigned seg = blockIdx.x % nseg, rest = blockIdx.x / nseg;
    const int cy = (int) (rest % mcy), cz = (int) (rest / mcy), xb = (int) seg * kCols;
    const int y0 = cy << cs, z0 = cz << cs;
    const int ey = min(y0 + c, ny - 1) - y0 + 1, ez = min(z0 + c, nz - 1) - z0 + 1, rows = ey * ez;
    auto row = [&](int r) { return data + ((long long) (z0 + r / ey) * ny + (y0 + r % ey)) * nx; };
    // this lane's columns over the warp's rows
    MinMaxAcc<T> acc[4];           // VEC: one per 32-bit word of the load
    T lo[kPer], hi[kPer];
#pragma unroll
    for (int u = 0; u < kPer; u++) {
        lo[u] = vtop<T>();
        hi[u] = vbottom<T>();
    }
    if constexpr (VEC) {
        const int x = xb + lane * kPer;  // nx is a multiple of kPer
        if (x < nx) {
            for (int r = warp; r < rows; r += 4 * kMcWarps) {
                uint4 v[4];
#pragma unroll
                for (int u = 0; u < 4; u++)  // past the last row: the last one again
                    v[u] = __ldg(reinterpret_cast<const uint4 *>(row(min(r + u * kMcWarps, rows - 1)) + x));
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    acc[0].word(v[u].x);
                    acc[1].word(v[u].y);
                    acc[2].word(v[u].z);
                    acc[3].word(v[u].w);
                }
            }
        }
        uint4 l, h;
        if constexpr (sizeof(T) == 4) {
            l = make_uint4(__float_as_uint(acc[0].lo), __float_as_uint(acc[1].lo), __float_as_uint(acc[2].lo), __float_as_uint(acc[3].lo));
            h = make_uint4(__float_as_uint(acc[0].hi), __float_as_uint(acc[1].hi), __float_as_uint(acc[2].hi), __float_as_uint(acc[3].hi));
        } else {
            l = make_uint4(acc[0].lo, acc[1].lo, acc[2].lo, acc[3].lo);
            h = make_uint4(acc[0].hi, acc[1].hi, acc[2].hi, acc[3].hi);
        }
        *reinterpret_cast<uint4 *>(&s.lo[warp][lane * kPer]) = l;
        *reinterpret_cast<uint4 *>(&s.hi[warp][lane * kPer]) = h;
    } else {
        for (int r = warp; r < rows; r += 2 * kMcWarps) {
            const T *p = row(r), *q = row(min(r + kMcWarps, rows - 1));
            T v[2][kPer];
#pragma unroll
            for (int u = 0; u < kPer; u++) {  // past the last column: the last one again
                const int x = min(xb + lane + 32 * u, nx - 1);
                v[0][u] = __ldg(p + x);
                v[1][u] = __ldg(q + x);
            }
#pragma unroll
            for (int u = 0; u < kPer; u++) {
                lo[u] = vmin_of(lo[u], vmin_of(v[0][u], v[1][u]));
                hi[u] = vmax_of(hi[u], vmax_of(v[0][u], v[1][u]));
            }
        }
#pragma unroll
        for (int u = 0; u < kPer; u++) {
            s.lo[warp][lane + 32 * u] = lo[u];
            s.hi[warp][lane + 32 * u] = hi[u];
        }
    }
    T xl = vtop<T>(), xh = vbottom<T>();
    if (xb + kCols < nx)
        for (int r = warp + lane * kMcWarps; r < rows; r += 32 * kMcWarps) {
            const T v = __ldg(row(r) + xb + kCols);
            xl = vmin_of(xl, v);
            xh = vmax_of(xh, v);
        }
    for (int o = 16; o > 0; o >>= 1) {
        xl = vmin_of(xl, (T) __shfl_xor_sync(0xffffffffu, xl, o));
        xh = vmax_of(xh, (T) __shfl_xor_sync(0xffffffffu, xh, o));
    }
    if (lane == 0) {
        s.xlo[warp] = xl;
        s.xhi[warp] = xh;
    }
    __syncthreads();
    // the warps' rows together: thread t owns columns t, t + 256, ...
    for (int x = threadIdx.x; x < kCols; x += 32 * kMcWarps) {
        T l = s.lo[0][x], h = s.hi[0][x];
#pragma unroll
        for (int w = 1; w < kMcWarps; w++) {
            l = vmin_of(l, s.lo[w][x]);
            h = vmax_of(h, s.hi[w][x]);
        }
        s.lo[0][x] = l;
        s.hi[0][x] = h;
    }
    if (threadIdx.x == 0)
        for (int w = 1; w < kMcWarps; w++) {
            s.xlo[0] = vmin_of(s.xlo[0], s.xlo[w]);
            s.xhi[0] = vmax_of(s.xhi[0], s.xhi[w]);
        }
    __syncthreads();
    // a cell's c columns (c divides 32) and the next one
    for (int x = threadIdx.x; x < kCols; x += 32 * kMcWarps) {
        T l = s.lo[0][x], h = s.hi[0][x];
        for (int o = c >> 1; o > 0; o >>= 1) {
            l = vmin_of(l, (T) __shfl_xor_sync(0xffffffffu, l, o));
            h = vmax_of(h, (T) __shfl_xor_sync(0xffffffffu, h, o));
        }
        const int cx = (xb + x) >> cs;
        if ((x & (c - 1)) == 0 && cx < mcx) {
            const bool last = x + c == kCols;
            l = vmin_of(l, last ? s.xlo[0] : s.lo[0][x + c]);
            h = vmax_of(h, last ? s.xhi[0] : s.hi[0][x + c]);
            float *o = mc + 2 * (((long long) cz * mcy + cy) * mcx + cx);
            *reinterpret_cast<float2 *>(o) = make_float2((float) l, (float) h);
        }
    }
}

template <typename T>
cudaError_t macrocells_dt(const T *data, int nx, int ny, int nz, int cell, float *mc, int mcx, int mcy, int mcz,
                          cudaStream_t s)
{
    int cs = 0;
    while ((1 << cs) < cell) cs++;
    const bool vec = (long long) nx * sizeof(T) % 16 == 0 && reinterpret_cast<uintptr_t>(data) % 16 == 0;
    const int cols = vec ? McTile<T, true>::kCols : McTile<T, false>::kCols;
    const int nseg = (mcx * cell + cols - 1) / cols;
    const unsigned grid = (unsigned) ((long long) nseg * mcy * mcz);
    if (vec) macrocell_kernel<T, true><<<grid, 32 * kMcWarps, 0, s>>>(data, nx, ny, nz, cs, mc, mcx, mcy, nseg);
    else macrocell_kernel<T, false><<<grid, 32 * kMcWarps, 0, s>>>(data, nx, ny, nz, cs, mc, mcx, mcy, nseg);
    return cudaGetLastError();
}

// A cell is transparent when no LUT entry its samples can index (lut_range)
// has non-zero opacity.
// nzprefix[i] = number of entries in [0, i) with non-zero opacity.
// Writes kDistCap for a transparent cell and 0 for the others.  In the same
// pass (opac non-null), the tile cost estimate's input: 255 sqrt(mean LUT
// opacity over the entries the cell's voxel range [min, max] indexes); the
// square root keeps small opacities apart; aprefix[i] = sum of the
// opacities of entries [0, i).
__global__ void empty_kernel(const float *mc, int ncell, const int *nzprefix, const double *aprefix, int lut_n,
                             int lut_off, float lut_scale, uint8_t *dist, uint8_t *opac)
{
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncell; c += gridDim.x * blockDim.x) {
        const int x0 = __float2int_rz(mc[2 * c] * lut_scale), x1 = __float2int_rz(mc[2 * c + 1] * lut_scale);
        const LutRange r = lut_range(x0, x1, lut_off, lut_n);
        dist[c] = (nzprefix[r.hi + 1] - nzprefix[r.lo]) == 0 ? (uint8_t) kDistCap : 0;
        if (opac) {
            const int a = min(max(lut_index(x0, lut_off), 0), lut_n - 1);
            const int b = min(max(lut_index(x1, lut_off), a), lut_n - 1);
            const double mean = (aprefix[b + 1] - aprefix[a]) / (double) (b - a + 1);
            const float q = sqrtf(fminf(fmaxf((float) mean, 0.0f), 1.0f)) * 255.0f + 0.5f;
            opac[c] = (uint8_t) min((int) q, 255);
        }
    }
}

// The Chebyshev distance (in cells) from each transparent cell to the
// nearest opaque one, capped: d = min(cap, max(|dx|, |dy|, |dz|) to the
// nearest cell with flag 0), 0 for opaque cells; cells outside the grid are
// not opaque (a ray there has left the brick).  Every cell within d-1 of a
// cell with d >= 1 is then transparent.  The L-infinity distance separates
// by axis: with g0 = 0 (opaque) or cap (transparent) and, along each axis
// in turn, g(p) = min over |k| <= cap of max(|k|, g(p + k)), three passes
// give the distance exactly (a minimum over the cells of the window of the
// largest per-axis offset; anything farther than the cap is the cap).
//
// One pass over the lines along `axis` (0 = x, 1 = y, 2 = z), in place: a
// block takes `lines` neighbouring lines whole (32, fewer for very long
// lines; neighbours along x for the y and z passes, along y for the x
// pass), so that its loads and stores coalesce, stages them in shared
// memory and writes them back once all are read.
constexpr int kDistLines = 32;
__global__ void dist_axis_kernel(uint8_t *dist, int mcx, int mcy, int mcz, int axis, int lines)
{
    extern __shared__ uint8_t tile[];  // [L][lines + 1]
    const int P = lines + 1;
    const int L = axis == 0 ? mcx : axis == 1 ? mcy : mcz;
    const long long slab = (long long) mcx * mcy;
    const long long stride = axis == 0 ? 1 : axis == 1 ? mcx : slab;
    // this block's group of lines: the first line's base and the distance
    // between neighbouring lines; nl lines are in the grid
    const int across = axis == 0 ? mcy : mcx;  // lines of a group run along this dimension
    const int groups_across = (across + lines - 1) / lines;
    const long long g = blockIdx.x;
    const int outer = (int) (g / groups_across), first = (int) (g % groups_across) * lines;
    const int nl = min(lines, across - first);
    long long base;
    long long step;
    if (axis == 0) {  // rows (y, z): outer = z, lines along y
        base = ((long long) outer * mcy + first) * mcx;
        step = mcx;
    } else if (axis == 1) {  // columns (x, z): outer = z, lines along x
        base = (long long) outer * slab + first;
        step = 1;
    } else {  // pillars (x, y): outer = y, lines along x
        base = (long long) outer * mcx + first;
        step = 1;
    }
    const int n = L * nl;
    // element e of the group: line l, position p (the x pass walks a row's
    // bytes with neighbouring threads, the others neighbouring lines); four
    // loads in flight per thread before their stores
    constexpr int U = 4;
    for (int e0 = threadIdx.x; e0 < n; e0 += U * blockDim.x) {
        uint8_t v[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int e = e0 + u * blockDim.x;
            const int l = axis == 0 ? e / L : e % nl, p = axis == 0 ? e % L : e / nl;
            v[u] = e < n ? dist[base + l * step + p * stride] : 0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int e = e0 + u * blockDim.x;
            const int l = axis == 0 ? e / L : e % nl, p = axis == 0 ? e % L : e / nl;
            if (e < n) tile[p * P + l] = v[u];
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        const int l = axis == 0 ? e / L : e % nl, p = axis == 0 ? e % L : e / nl;
        int m = tile[p * P + l];
        for (int k = 1; k < m; k++) {  // only offsets below the current minimum can lower it
            if (p - k >= 0) m = min(m, max(k, (int) tile[(p - k) * P + l]));
            if (p + k < L) m = min(m, max(k, (int) tile[(p + k) * P + l]));
        }
        dist[base + l * step + p * stride] = (uint8_t) m;
    }
}

// compositetiles (main.c:1203-1218)
__global__ void composite_kernel(float4 *dst, const float4 *__restrict__ src, int num, long long npix)
{
    for (long long p = blockIdx.x * (long long) blockDim.x + threadIdx.x; p < npix; p += (long long) gridDim.x * blockDim.x) {
        float4 d = dst[p];
        for (int k = num - 1; k >= 0; k--) {
            float4 s = __ldg(src + (long long) k * npix + p);
            d.z = s.z + (1.0f - s.w) * d.z;
            d.y = s.y + (1.0f - s.w) * d.y;
            d.x = s.x + (1.0f - s.w) * d.x;
            d.w = s.w + (1.0f - s.w) * d.w;
        }
        dst[p] = d;
    }
}

// (uint8)(v*255 + 0.5) for v clamped to [0,1], computed exactly in integers
// (see q8 in ivr_march.cu).
__device__ __forceinline__ unsigned q8k(float v)
{
    if (!(v > 0.0f)) return 0u;
    if (v >= 1.0f) return 255u;
    unsigned bits = __float_as_uint(v);
    int e = (int) (bits >> 23);
    if (e == 0) return 0u;
    unsigned long long m = (bits & 0x7fffffu) | 0x800000u;
    int s = 150 - e;
    if (s >= 34) return 0u;
    return (unsigned) ((255ull * m + (1ull << (s - 1))) >> s);
}

// Four floats in, one 32-bit word out per step where the buffers allow it, two
// steps in flight.  Bound by HBM and by q8k's 64-bit integers, each about half:
// 1920x1080 RGBA in 12.4 us (3.3 TB/s, issue slots 66% full); a float a thread
// with single-byte stores took 17.7.
__global__ void __launch_bounds__(256) quantize4_kernel(const float4 *__restrict__ in, uchar4 *__restrict__ out,
                                                        long long n4, int rest)
{
    const long long stride = (long long) gridDim.x * blockDim.x;
    for (long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < n4; i += 2 * stride) {
        const bool two = i + stride < n4;
        const float4 a = __ldg(in + i), b = two ? __ldg(in + i + stride) : a;
        out[i] = make_uchar4(q8k(a.x), q8k(a.y), q8k(a.z), q8k(a.w));
        if (two) out[i + stride] = make_uchar4(q8k(b.x), q8k(b.y), q8k(b.z), q8k(b.w));
    }
    if (blockIdx.x == 0 && threadIdx.x < rest)  // the last n % 4 floats
        reinterpret_cast<uint8_t *>(out + n4)[threadIdx.x] =
            (uint8_t) q8k(reinterpret_cast<const float *>(in + n4)[threadIdx.x]);
}

// unaligned buffers
__global__ void quantize_kernel(const float *__restrict__ in, uint8_t *__restrict__ out, long long n)
{
    for (long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x; i < n; i += (long long) gridDim.x * blockDim.x)
        out[i] = (uint8_t) q8k(in[i]);
}

// ---- allocation-free histogram ---------------------------------------------
// Scratch of ivr_volume_histogram_noalloc: min/max partials, the reduced
// min/max and up to kNoAllocMaxBins bins, in one static device array that
// every GPU loading this library holds until the process exits.
struct NoAllocScratch {
    float partial[2 * kSms * 4];
    float minmax[2];
    int hist[kNoAllocMaxBins];
};
static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(NoAllocScratch)];

__global__ void minmax_final_kernel(const float *partial, int nparts, float *minmax)
{
    float lo = FLT_MAX, hi = -FLT_MAX;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
        lo = fminf(lo, partial[2 * i]);
        hi = fmaxf(hi, partial[2 * i + 1]);
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    __shared__ float slo[32], shi[32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { slo[w] = lo; shi[w] = hi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < (int) (blockDim.x >> 5); k++) { lo = fminf(lo, slo[k]); hi = fmaxf(hi, shi[k]); }
        minmax[0] = lo;
        minmax[1] = hi;
    }
}

constexpr int kHistBlocks = kSms;           // one block an SM
constexpr int kHistSmem = 224 * 1024;       // shared memory a block may ask for
constexpr int kHistBins = kHistSmem / 4;    // counters in it
constexpr int kHistRanges = 2;              // ranges before the counters move to global memory:
                                            // at four (229,375 bins, 256^3 f32 voxels) a call
                                            // took 130 us against 88 in global memory, at two
                                            // (65,536 bins, 256^3 u16) 75 against 87
constexpr long long kHistFew = 8192LL * 2 * kHistBlocks;  // voxels from which hist_kernel's blocks have
                                                         // work for the time their counters take
constexpr int kHistSmall = 128;             // voxels per bin below which global counters win, of more
                                            // bins than hist_few_kernel takes: 65,536 bins, u16: 160^3
                                            // (62 a bin) 52 us a call shared and 47 global, 256^3 (256)
                                            // 75 and 87.  (With fewer bins they lose: voxels that crowd
                                            // in one wait for each other.  80^3 u16 voxels, 60% of one
                                            // value, 4096 bins: 151 us global, 4.2 in hist_few_kernel.)

template <typename T>
cudaError_t hist_launch(const T *data, long long n, MinArg mn, int hsize, int *hist, cudaStream_t s)
{
    static std::atomic<unsigned long long> attr{0};
    cudaError_t e = set_dynamic_smem_once(hist_kernel<T>, kHistSmem, attr);
    if (e != cudaSuccess) return e;
    const int ranges = (hsize + kHistBins - 1) / kHistBins;
    const int nb = (hsize + ranges - 1) / ranges;
    int rep = 0;
    while (rep < 5 && (nb << (rep + 1)) <= kHistBins / 2) rep++;  // 112 KB: two blocks an SM
    const size_t smem = sizeof(int) * ((size_t) nb << rep);
    const int per_sm = smem <= kHistSmem / 2 ? 2 : 1;
    // 8192 voxels a block at least: clearing and adding up the counters costs
    // about that much
    const long long most = n / 8192 + 1, wave = (long long) kHistBlocks * per_sm / ranges;
    const dim3 grid((unsigned) (wave < most ? wave : most), ranges);
    hist_kernel<T><<<grid, 1024, smem, s>>>(data, n, mn, hsize, nb, rep, hist);
    return cudaGetLastError();
}

template <typename T>
cudaError_t hist_dt(const T *data, long long n, MinArg mn, int hsize, int *hist, cudaStream_t s)
{
    if (sizeof(T) < 4) hsize = std::min(hsize, 65536);  // integer voxels: the bins above stay empty
    if (hsize <= kHistFewBins && n < kHistFew) {
        hist_few_kernel<<<grid_for(n, 512, 2), 512, 0, s>>>(data, n, mn, hsize, hist);
        return cudaGetLastError();
    }
    if (hsize > kHistRanges * kHistBins || (hsize > kHistFewBins && n < (long long) kHistSmall * hsize)) {
        hist_global_kernel<<<grid_for(n, 256), 256, 0, s>>>(data, n, mn, hsize, hist);
        return cudaGetLastError();
    }
    return hist_launch(data, n, mn, hsize, hist, s);
}

cudaError_t hist_any(const void *data, int dtype, long long n, MinArg mn, int hsize, int *hist, cudaStream_t s)
{
    switch (dtype) {
    case IVR_U8: return hist_dt((const uint8_t *) data, n, mn, hsize, hist, s);
    case IVR_U16: return hist_dt((const uint16_t *) data, n, mn, hsize, hist, s);
    default: return hist_dt((const float *) data, n, mn, hsize, hist, s);
    }
}

cudaError_t minmax_any(const void *data, int dtype, long long n, float *partial, int nparts, cudaStream_t s)
{
    switch (dtype) {
    case IVR_U8: minmax_kernel<<<nparts, 256, 0, s>>>((const uint8_t *) data, n, partial); break;
    case IVR_U16: minmax_kernel<<<nparts, 256, 0, s>>>((const uint16_t *) data, n, partial); break;
    default: minmax_kernel<<<nparts, 256, 0, s>>>((const float *) data, n, partial); break;
    }
    return cudaGetLastError();
}

}  // namespace

// Device address of the static scratch on the current device.  Resolved
// once per device with cudaGetSymbolAddress (the first call on a device
// loads this module there if it is not loaded yet).
static cudaError_t noalloc_scratch(NoAllocScratch **out)
{
    static std::mutex mu;
    static void *ptrs[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(mu);
    if (!ptrs[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        ptrs[dev] = p;
    }
    *out = static_cast<NoAllocScratch *>(ptrs[dev]);
    return cudaSuccess;
}

cudaError_t noalloc_histogram(const void *data, int dtype, long long n, int hsize, int *hist_host,
                              float *minmax_host, cudaStream_t s)
{
    NoAllocScratch *sc = nullptr;
    cudaError_t e = noalloc_scratch(&sc);
    if (e != cudaSuccess) return e;
    const int parts = kSms * 4;
    if ((e = minmax_any(data, dtype, n, sc->partial, parts, s)) != cudaSuccess) return e;
    minmax_final_kernel<<<1, 1024, 0, s>>>(sc->partial, parts, sc->minmax);
    if ((e = cudaMemsetAsync(sc->hist, 0, sizeof(int) * (size_t) hsize, s)) != cudaSuccess) return e;
    if ((e = hist_any(data, dtype, n, MinArg{0.0f, sc->minmax}, hsize, sc->hist, s)) != cudaSuccess) return e;
    if ((e = cudaMemcpyAsync(hist_host, sc->hist, sizeof(int) * (size_t) hsize, cudaMemcpyDeviceToHost, s)) !=
        cudaSuccess)
        return e;
    if ((e = cudaMemcpyAsync(minmax_host, sc->minmax, 2 * sizeof(float), cudaMemcpyDeviceToHost, s)) != cudaSuccess)
        return e;
    return cudaStreamSynchronize(s);
}

size_t dtype_size(int dtype) { return dtype == IVR_U8 ? 1 : dtype == IVR_U16 ? 2 : 4; }

int minmax_parts() { return kSms * 4; }

cudaError_t launch_byteswap(void *data, long long n, int elem, cudaStream_t s)
{
    if (n <= 0 || elem == 1) return cudaSuccess;
    if (elem == 2) byteswap16_kernel<<<grid_for(n, 256), 256, 0, s>>>((uint16_t *) data, n);
    else byteswap32_kernel<<<grid_for(n, 256), 256, 0, s>>>((uint32_t *) data, n);
    return cudaGetLastError();
}

cudaError_t launch_gather_brick(const void *src, int gw, int gh, int gd, void *dst, int sx, int sy, int sz, int lw,
                                int lh, int ld, int elem, cudaStream_t s)
{
    (void) gd;
    const long long rows = (long long) lh * ld;
    const unsigned g = (unsigned) ((rows + 7) / 8);
    if (elem == 1) gather_kernel<<<g, 256, 0, s>>>((const uint8_t *) src, gw, gh, (uint8_t *) dst, sx, sy, sz, lw, lh, rows);
    else if (elem == 2) gather_kernel<<<g, 256, 0, s>>>((const uint16_t *) src, gw, gh, (uint16_t *) dst, sx, sy, sz, lw, lh, rows);
    else gather_kernel<<<g, 256, 0, s>>>((const uint32_t *) src, gw, gh, (uint32_t *) dst, sx, sy, sz, lw, lh, rows);
    return cudaGetLastError();
}

cudaError_t launch_minmax(const void *data, int dtype, long long n, float *partial, int nparts, cudaStream_t s)
{
    return minmax_any(data, dtype, n, partial, nparts, s);
}

cudaError_t launch_histogram(const void *data, int dtype, long long n, float mn, int hsize, int *hist, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(hist, 0, sizeof(int) * (size_t) hsize, s);
    if (e != cudaSuccess) return e;
    return hist_any(data, dtype, n, MinArg{mn, nullptr}, hsize, hist, s);
}

cudaError_t launch_macrocells(const void *data, int dtype, int nx, int ny, int nz, int cell, float *mc, int mcx,
                              int mcy, int mcz, cudaStream_t s)
{
    switch (dtype) {
    case IVR_U8: return macrocells_dt((const uint8_t *) data, nx, ny, nz, cell, mc, mcx, mcy, mcz, s);
    case IVR_U16: return macrocells_dt((const uint16_t *) data, nx, ny, nz, cell, mc, mcx, mcy, mcz, s);
    default: return macrocells_dt((const float *) data, nx, ny, nz, cell, mc, mcx, mcy, mcz, s);
    }
}

cudaError_t launch_empty_flags(const float *mc, int mcx, int mcy, int mcz, const int *nzprefix, const double *aprefix,
                               int lut_n, int lut_off, float lut_scale, uint8_t *empty, uint8_t *opac, cudaStream_t s)
{
    const int ncell = mcx * mcy * mcz;
    empty_kernel<<<grid_for(ncell, 256), 256, 0, s>>>(mc, ncell, nzprefix, aprefix, lut_n, lut_off, lut_scale, empty,
                                                      opac);
    return launch_dist_transform(empty, mcx, mcy, mcz, s);
}

cudaError_t launch_dist_transform(uint8_t *dist, int mcx, int mcy, int mcz, cudaStream_t s)
{
    if (mcx <= 0 || mcy <= 0 || mcz <= 0) return cudaSuccess;
    const int dims[3] = {mcx, mcy, mcz};
    for (int axis = 0; axis < 3; axis++) {
        const int L = dims[axis];
        if (L == 1) continue;  // a line of one cell keeps its flag
        // 32 lines a block up to 1489 cells a line, fewer above
        const int lines = std::min(kDistLines, 48 * 1024 / L - 1);
        if (lines < 1) return cudaErrorInvalidValue;  // a line of more than 24576 macrocells
        const size_t smem = (size_t) L * (lines + 1);
        const int across = axis == 0 ? mcy : mcx, outer = axis == 2 ? mcy : mcz;
        const long long groups = (long long) outer * ((across + lines - 1) / lines);
        dist_axis_kernel<<<(unsigned) groups, 256, smem, s>>>(dist, mcx, mcy, mcz, axis, lines);
    }
    return cudaGetLastError();
}

// The smallest power of two that is n or more.
unsigned pow2_from(unsigned n)
{
    unsigned p = 1;
    while (p < n) p *= 2;
    return p;
}

// A block of up to 256 threads over columns, groups of rows and slabs of a
// volume: whole warps of columns up to `columns`, or what a narrower row has,
// and the rest of the threads on further groups, then on further slabs, so that
// lanes are not left without a column or a row.
dim3 slab_block(int w, int groups, unsigned columns)
{
    const unsigned tx = w >= 32 ? std::min(columns, (unsigned) (w + 31) / 32 * 32) : pow2_from((unsigned) w);
    const unsigned ty = std::min(256 / tx, pow2_from((unsigned) groups));
    return dim3(tx, ty, std::min(64u, 256 / (tx * ty)));
}

// Per-voxel gradient (gradient3d, restated as intended): per axis a halved
// central difference inside and a halved one-sided difference on the
// faces, times the unit spacing; w = |(x, y, z)| as mag3f computes it.
// HBM-bound: the volume read once, 16 bytes written per voxel.  A thread
// walks kGradRows rows down its column with the rows around it in registers;
// the x and z neighbours come from L1 and L2.  512x512x384 f32 voxels: 560 us
// with three 64-bit divisions per voxel; 332 us (6.1 TB/s) with 4 rows of 128
// or 256 columns; 1, 2, 8 rows 461, 376, 340; 16 voxels up a z column instead,
// whose stores touch 16 slabs at a time, 490.  Narrow rows and low slabs share
// a block (slab_block): 2x2048x2048 voxels (x, y, z) 49 us, with a warp a row
// 285; 2x2x4,000,000 56 and 2352.
constexpr int kGradRows = 4, kGradColumns = 128;
template <typename T>
__global__ void __launch_bounds__(256) gradient_kernel(const T *__restrict__ vol, int w, int h, int d,
                                                       float4 *__restrict__ out, unsigned bx, unsigned by)
{
    const unsigned r = blockIdx.x / bx;
    const int j = (int) (blockIdx.x % bx * blockDim.x + threadIdx.x);
    const int i0 = (int) (r % by * blockDim.y + threadIdx.y) * kGradRows, i1 = min(i0 + kGradRows, h);
    const int k = (int) (r / by * blockDim.z + threadIdx.z);
    if (j >= w || i0 >= h || k >= d) return;
    const long long slab = (long long) w * h;
    const T *p = vol + k * slab + (long long) i0 * w + j;
    float4 *q = out + k * slab + (long long) i0 * w + j;
    // offsets of the neighbours each difference takes
    const int xl = j > 0 ? -1 : 0, xh = j < w - 1 ? 1 : 0;
    const long long zl = k > 0 ? -slab : 0, zh = k < d - 1 ? slab : 0;
    float below = (float) __ldg(i0 > 0 ? p - w : p), here = (float) __ldg(p);
#pragma unroll
    for (int u = 0; u < kGradRows; u++, p += w, q += w) {
        if (i0 + u >= i1) break;
        const float above = i0 + u < h - 1 ? (float) __ldg(p + w) : here;
        const float x = ((float) __ldg(p + xh) - (float) __ldg(p + xl)) / 2.0f;
        const float y = (above - below) / 2.0f;
        const float z = ((float) __ldg(p + zh) - (float) __ldg(p + zl)) / 2.0f;
        *q = make_float4(x, y, z, sqrtf(x * x + y * y + z * z));
        below = here;
        here = above;
    }
}

cudaError_t launch_gradient(const void *data, int dtype, int w, int h, int d, float4 *out, cudaStream_t s)
{
    const dim3 block = slab_block(w, (h + kGradRows - 1) / kGradRows, kGradColumns);
    const unsigned bx = (w + block.x - 1) / block.x, by = (h + block.y * kGradRows - 1) / (block.y * kGradRows);
    const unsigned grid = (unsigned) ((unsigned long long) bx * by * ((d + block.z - 1) / block.z));
    switch (dtype) {
    case IVR_U8: gradient_kernel<<<grid, block, 0, s>>>((const uint8_t *) data, w, h, d, out, bx, by); break;
    case IVR_U16: gradient_kernel<<<grid, block, 0, s>>>((const uint16_t *) data, w, h, d, out, bx, by); break;
    case IVR_F32: gradient_kernel<<<grid, block, 0, s>>>((const float *) data, w, h, d, out, bx, by); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// Corner-packed copy; bound by its stores (4x the brick).  A thread walks
// kQuadRows rows down its column (slab_block), each voxel row loaded once for
// the two element rows it belongs to.  With a 64-bit division per index and
// an element a thread it took 4.9 ms for 1024^3 u16 voxels (2.2 TB/s).  Narrow
// bricks, u16, so, in whole warps a row and an element a thread: 8x1024x1024
// voxels (x, y, z) 14, 45 and 26 us, 2x2048x2048 18, 173 and 16.
constexpr int kQuadRows = 4;
template <typename T, typename V>
__global__ void __launch_bounds__(256) quad_kernel(const T *__restrict__ src, int nx, int ny, int nz,
                                                   V *__restrict__ dst, unsigned bx, unsigned by)
{
    const int qx = nx - 1, qy = ny - 1;
    const unsigned r = blockIdx.x / bx;
    const int j = (int) (blockIdx.x % bx * blockDim.x + threadIdx.x);
    const int i0 = (int) (r % by * blockDim.y + threadIdx.y) * kQuadRows;
    const long long k = r / by * blockDim.z + threadIdx.z;
    if (j >= qx || i0 >= qy || k >= nz) return;
    const T *p = src + (k * ny + i0) * nx + j;
    V *q = dst + (k * qy + i0) * qx + j;
    T a[kQuadRows + 1], b[kQuadRows + 1];
#pragma unroll
    for (int u = 0; u <= kQuadRows; u++) {
        const T *row = p + (long long) u * nx;
        const bool in = i0 + u <= qy;
        a[u] = in ? __ldg(row) : T(0);
        b[u] = in ? __ldg(row + 1) : T(0);
    }
#pragma unroll
    for (int u = 0; u < kQuadRows; u++) {
        if (i0 + u >= qy) break;
        V v;
        v.x = a[u];
        v.y = b[u];
        v.z = a[u + 1];
        v.w = b[u + 1];
        if constexpr (sizeof(T) == sizeof(float)) {
            if (kQuadDelta) {  // the sampler's x-lerp differences, rounded as it rounds them
                v.y = b[u] - a[u];
                v.w = b[u + 1] - a[u + 1];
            }
        }
        q[(long long) u * qx] = v;
    }
}

size_t quad_bytes(int dtype, int nx, int ny, int nz)
{
    return (size_t) (nx - 1) * (ny - 1) * nz * 4 * dtype_size(dtype);
}

cudaError_t launch_quads(const void *data, int dtype, int nx, int ny, int nz, void *quad, cudaStream_t s)
{
    const dim3 block = slab_block(nx - 1, (ny - 1 + kQuadRows - 1) / kQuadRows, 32);
    const unsigned bx = (nx - 1 + block.x - 1) / block.x, by = (ny - 1 + block.y * kQuadRows - 1) / (block.y * kQuadRows);
    const unsigned grid = (unsigned) ((unsigned long long) bx * by * ((nz + block.z - 1) / block.z));
    switch (dtype) {
    case IVR_U8: quad_kernel<<<grid, block, 0, s>>>((const uint8_t *) data, nx, ny, nz, (uchar4 *) quad, bx, by); break;
    case IVR_U16: quad_kernel<<<grid, block, 0, s>>>((const uint16_t *) data, nx, ny, nz, (ushort4 *) quad, bx, by); break;
    case IVR_F32: quad_kernel<<<grid, block, 0, s>>>((const float *) data, nx, ny, nz, (float4 *) quad, bx, by); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_composite(float *dst, const float *src, int num, long long npix, cudaStream_t s)
{
    composite_kernel<<<grid_for(npix, 256), 256, 0, s>>>((float4 *) dst, (const float4 *) src, num, npix);
    return cudaGetLastError();
}

cudaError_t launch_quantize(const float *in, uint8_t *out, long long n, cudaStream_t s)
{
    const bool vec = reinterpret_cast<uintptr_t>(in) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 4 == 0;
    if (vec)
        quantize4_kernel<<<grid_for((n + 3) / 4, 256), 256, 0, s>>>((const float4 *) in, (uchar4 *) out, n / 4,
                                                                     (int) (n % 4));
    else quantize_kernel<<<grid_for(n, 256), 256, 0, s>>>(in, out, n);
    return cudaGetLastError();
}

}  // namespace ivr
