// qt_resize.cu — BILINEAR downsampling of RGBA8 textures for mip chains
// (qt_resize_bilinear_device in include/quicktex_cuda.h).
//
// quicktex builds each mip level with Pillow: image_utils.resize_no_premultiply
// (quicktex/image_utils.py:40-52) resizes the RGB bands and the alpha band
// separately with Image.resize(size, Image.BILINEAR), and dds.encode
// (quicktex/dds.py:275-280) resizes the ORIGINAL image to every level. Pillow's
// resampler treats each band alike, so the result equals resizing all four
// channels of the RGBA8 texture independently, which is what this file does.
//
// The arithmetic restates Pillow 12.2.0's separable fixed-point resampler
// (src/libImaging/Resample.c: precompute_coeffs, normalize_coeffs_8bpc,
// ImagingResampleHorizontal_8bpc / ImagingResampleVertical_8bpc,
// ImagingResampleInner), a third-party dependency of quicktex:
//   - per output coordinate: scale = in/out, filterscale = max(scale, 1),
//     support = filterscale (the triangle filter's support is 1), centre
//     (x + 0.5)*scale, taps [xmin, xmin + n) with xmin = (int)(centre - support
//     + 0.5) clamped to 0 and end (int)(centre + support + 0.5) clamped to the
//     input size; weight of tap t = tri((t + xmin - centre + 0.5)/filterscale),
//     tri(d) = max(0, 1 - |d|), each divided by their sum (in tap order) when
//     the sum is non-zero, all in double;
//   - weights to fixed point with 22 fraction bits, rounded half away from zero;
//   - each output value = clamp((2^21 + sum(value * weight)) >> 22, 0, 255), 32-bit;
//   - a horizontal pass over the source rows the vertical pass needs, to 8-bit
//     values, then a vertical pass; a pass whose size does not change is skipped.
// The weights are computed on the device in double, operation by operation as Pillow does (-fmad=false: no
// contraction): on the host they took 27-88 us of every call (470 us of a 2048^2 chain's 730), more than the resampling.

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "qt_internal.h"

namespace {

constexpr int kPrecisionBits = 22;  // 32 - 8 - 2

// Size of one dimension's resampling: the widest output's tap count, and an output's first and one-past-last tap
struct Scale {
    int in_size, out_size, ksize;
    double scale, support;
    Scale(int in, int out) : in_size(in), out_size(out) {
        scale = (double)(float)in / out;
        support = 1.0 * (scale < 1.0 ? 1.0 : scale);
        ksize = (int)std::ceil(support) * 2 + 1;
    }
    __host__ __device__ int2 bounds(int xx, double &center) const {
        center = 0.0 + (xx + 0.5) * scale;
        int xmin = (int)(center - support + 0.5);
        if (xmin < 0) xmin = 0;
        int xmax = (int)(center + support + 0.5);
        if (xmax > in_size) xmax = in_size;
        return make_int2(xmin, xmax);
    }
};

__device__ __forceinline__ double tri(double x) {
    if (x < 0.0) x = -x;
    return x < 1.0 ? 1.0 - x : 0.0;
}

__device__ __forceinline__ double fixed_point(double k) { return k < 0 ? -0.5 + k * (1 << kPrecisionBits) : 0.5 + k * (1 << kPrecisionBits); }

// One output's fixed-point weights by a warp, into row[0 .. taps); returns its first tap and tap count. Pillow adds the
// weights in tap order, a chain of dependent additions (~20 cycles a tap with the exchanges: 1078 x 169 -> 1 x 80 took 36 us, two
// thirds of it this sum). Here the lanes add every 32nd weight and their sums meet in a tree, which is another rounding of the same sum: of n
// weights, none negative, any two orders differ by less than (n + 8) * 2^-52 of the sum. A fixed-point weight is the same for
// both unless that much moves its quotient across an integer; a warp that meets such a weight (about one
// output in 10^5) does the sum again in tap order. For power-of-two scales (the halving chains of power-of-two
// textures) every weight is a multiple of 1 / (2 scale), so the sum is exact in any order.
__device__ __forceinline__ int2 output_taps(const Scale &S, int o, int32_t *row) {
    const int lane = threadIdx.x & 31;
    double center;
    const int2 b = S.bounds(o, center);
    const int xmin = b.x, n = b.y - b.x;
    const double ss = 1.0 / S.support;
    const bool pow2 = S.scale >= 1.0 && (__double_as_longlong(S.scale) & 0xFFFFFFFFFFFFFll) == 0;
    double ww = 0.0;
#pragma unroll 4
    for (int x = lane; x < n; x += 32) ww += tri((x + xmin - center + 0.5) * ss);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) ww += __shfl_xor_sync(0xffffffffu, ww, d);
    const double slack = (n + 8) * 0x1p-52;
    bool near = false;
#pragma unroll 4
    for (int x = lane; x < n; x += 32) {
        double k = tri((x + xmin - center + 0.5) * ss);
        if (ww != 0.0) k /= ww;
        const double v = fixed_point(k), d = v * slack;
        row[x] = (int32_t)v;
        near |= (int32_t)(v - d) != (int32_t)(v + d);
    }
    if (!pow2 && __any_sync(0xffffffffu, near)) {
        ww = 0.0;
        for (int x0 = 0; x0 < n; x0 += 32) {
            const int x = x0 + lane;
            const double w = x < n ? tri((x + xmin - center + 0.5) * ss) : 0.0;
#pragma unroll
            for (int i = 0; i < 32; i++) ww += __shfl_sync(0xffffffffu, w, i);  // past the last tap: + 0.0
        }
        for (int x = lane; x < n; x += 32) {
            double k = tri((x + xmin - center + 0.5) * ss);
            if (ww != 0.0) k /= ww;
            row[x] = (int32_t)fixed_point(k);
        }
    }
    return make_int2(xmin, n);
}

// The tap tables of both dimensions, one warp per output coordinate: per output its first tap and tap count, and ksize
// weights
__global__ void __launch_bounds__(256) k_taps(Scale h, Scale v, int2 *__restrict__ bounds_h, int32_t *__restrict__ kk_h,
                                              int2 *__restrict__ bounds_v, int32_t *__restrict__ kk_v, int y_first) {
    const long o = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (o >= (long)h.out_size + v.out_size) return;
    const bool vertical = o >= h.out_size;
    const int i = (int)(vertical ? o - h.out_size : o);
    const int2 b = vertical ? output_taps(v, i, kk_v + (size_t)i * v.ksize) : output_taps(h, i, kk_h + (size_t)i * h.ksize);
    // the vertical pass reads the horizontal pass's rows, the first of them y_first
    if ((threadIdx.x & 31) == 0) (vertical ? bounds_v : bounds_h)[i] = make_int2(vertical ? b.x - y_first : b.x, b.y);
}

__device__ __forceinline__ uint32_t clip8(int v) {
    v >>= kPrecisionBits;
    return (uint32_t)(v < 0 ? 0 : (v > 255 ? 255 : v));
}

__device__ __forceinline__ uint32_t weighted(int s0, int s1, int s2, int s3) {
    return clip8(s0) | (clip8(s1) << 8) | (clip8(s2) << 16) | (clip8(s3) << 24);
}

__device__ __forceinline__ void add_tap(int s[4], uint32_t p, int c) {
    s[0] += (int)(p & 0xFF) * c;
    s[1] += (int)((p >> 8) & 0xFF) * c;
    s[2] += (int)((p >> 16) & 0xFF) * c;
    s[3] += (int)(p >> 24) * c;
}

// Horizontal pass: rows [y0, y0 + rows) of src (width w) -> rows [0, rows) of dst (width dw). G lanes share an output's
// taps, G half the scale's power of two, so that neighbouring lanes read neighbouring texels at deep levels (one
// output per lane strides by the scale); each lane sums them for four rows at once, which keeps four loads in flight
// and reads each weight once. The 4 x 4 sums are exact integers; they meet by exchanging halves, so that lane bits
// 0 and 1 end up with one row each and bits 2 and 3 with one channel each. Work is (row quad, output) pairs in
// one sequence, so few outputs leave no lanes idle. A call from 2048^2 to 1024^2 took 89 us, to 256^2 108, to 32^2 38;
// with this and the taps on the device 27, 24 and 22.
template <int G>
__global__ void __launch_bounds__(256) k_resample_h(const uint32_t *__restrict__ src, int w, int y0, int rows,
                                                    uint32_t *__restrict__ dst, int dw, const int2 *__restrict__ bounds,
                                                    const int32_t *__restrict__ kk, int ksize) {
    const int sub = threadIdx.x & (G - 1);
    const long quads = (rows + 3) / 4, groups = quads * dw, stride = (long)gridDim.x * (256 / G);
    // a warp's lanes stay together: every lane of it runs the same number of iterations
    for (long g0 = ((long)blockIdx.x * 256 + (threadIdx.x & ~31)) / G; g0 < groups; g0 += stride) {
        const long go = g0 + (threadIdx.x & 31) / G;
        const bool have = go < groups;
        const long g = have ? go : groups - 1;  // lanes past the end take part in the exchanges
        const int x = (int)(g % dw), y = 4 * (int)(g / dw);
        const int2 b = bounds[x];
        const int32_t *k = kk + (size_t)x * ksize;
        const uint32_t *row[4];
#pragma unroll
        for (int r = 0; r < 4; r++) row[r] = src + (size_t)(y0 + (y + r < rows ? y + r : rows - 1)) * w + b.x;
        int s[4][4] = {};
#pragma unroll 4
        for (int t = sub; t < b.y; t += G) {
            const int c = __ldg(k + t);
#pragma unroll
            for (int r = 0; r < 4; r++) add_tap(s[r], __ldg(row[r] + t), c);
        }
        int v[16];
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = s[i >> 2][i & 3];
        int n = 16;
#pragma unroll
        for (int bit = 1; bit < G && bit < 16; bit <<= 1) {
            n >>= 1;
            const bool hi = sub & bit;
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (j < n) {
                    const int send = hi ? v[j] : v[j + n], keep = hi ? v[j + n] : v[j];
                    v[j] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
                }
        }
        if (G == 32) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 16);
        constexpr int kRows = G >= 4 ? 1 : 4 / G, kChannels = G >= 16 ? 1 : G >= 8 ? 2 : 4;
        const int r0 = (G >= 2 ? (sub & 1) * 2 : 0) + (G >= 4 ? (sub >> 1) & 1 : 0);
        const int c0 = (G >= 8 ? ((sub >> 2) & 1) * 2 : 0) + (G >= 16 ? (sub >> 3) & 1 : 0);
#pragma unroll
        for (int r = 0; r < kRows; r++) {
            uint32_t p = 0;
#pragma unroll
            for (int c = 0; c < kChannels; c++) p |= clip8(v[r * kChannels + c] + (1 << (kPrecisionBits - 1))) << (8 * (c0 + c));
            if (G >= 8) p |= __shfl_xor_sync(0xffffffffu, p, 4);
            if (G >= 16) p |= __shfl_xor_sync(0xffffffffu, p, 8);
            if (have && (sub >> 2) == 0 && y + r0 + r < rows) dst[(size_t)(y + r0 + r) * dw + x] = p;
        }
    }
}

// Vertical pass: src (width w, rows indexed by the bounds) -> dst (w x dh). A CTA takes TX columns of one output row and
// splits the taps over its 256 / TX groups of threads, whose sums meet in shared memory: few columns with
// thousands of taps each (the deep levels) have as many threads to themselves as many columns with a few.
template <int TX>
__global__ void __launch_bounds__(256) k_resample_v(const uint32_t *__restrict__ src, int w, uint32_t *__restrict__ dst,
                                                    int dh, const int2 *__restrict__ bounds,
                                                    const int32_t *__restrict__ kk, int ksize) {
    constexpr int TY = 256 / TX;
    __shared__ int4 part[TY > 1 ? 256 : 1];
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX, xo = blockIdx.x * TX + tx, x = xo < w ? xo : w - 1;
    if (TY == 1 && xo >= w) return;
    for (int yy = blockIdx.y; yy < dh; yy += gridDim.y) {
        const int2 b = bounds[yy];
        const int32_t *k = kk + (size_t)yy * ksize;
        int s[4] = {};
#pragma unroll 4
        for (int t = ty; t < b.y; t += TY) add_tap(s, __ldg(src + (size_t)(b.x + t) * w + x), __ldg(k + t));
        if (TY > 1) {
            part[threadIdx.x] = make_int4(s[0], s[1], s[2], s[3]);
            __syncthreads();
#pragma unroll
            for (int d = 128; d >= TX; d >>= 1) {
                if (threadIdx.x < d) {
                    const int4 o = part[threadIdx.x + d];
                    int4 &a = part[threadIdx.x];
                    a = make_int4(a.x + o.x, a.y + o.y, a.z + o.z, a.w + o.w);
                }
                __syncthreads();
            }
            const int4 a = part[tx];
            s[0] = a.x; s[1] = a.y; s[2] = a.z; s[3] = a.w;
            __syncthreads();  // the next row's sums overwrite part
        }
        const int half = 1 << (kPrecisionBits - 1);
        if (ty == 0 && xo < w) dst[(size_t)yy * w + x] = weighted(s[0] + half, s[1] + half, s[2] + half, s[3] + half);
    }
}

// One output's weights by one thread (few taps)
__device__ __forceinline__ int2 output_taps_thread(const Scale &S, int o, int32_t *row) {
    double center;
    const int2 b = S.bounds(o, center);
    const int xmin = b.x, n = b.y - b.x;
    const double ss = 1.0 / S.support;
    double ww = 0.0;
    for (int x = 0; x < n; x++) ww += tri((x + xmin - center + 0.5) * ss);
    for (int x = 0; x < n; x++) {
        double k = tri((x + xmin - center + 0.5) * ss);
        if (ww != 0.0) k /= ww;
        row[x] = (int32_t)fixed_point(k);
    }
    return make_int2(xmin, n);
}

// Both passes of a small texture in one kernel: a cluster of 8 CTAs per output row, which splits the source rows that it
// needs. Each CTA computes the taps (few: a thread per output, many: a warp), the horizontal pass of its rows and
// their share of the vertical sums, all in shared memory; the CTAs then add the shares, each for some of the columns. A
// row of the horizontal pass is computed by the ~2 output rows that need it; for that the call is one launch without
// scratch memory: three launches and the allocation take 22 us of host time, one 11, and a chain's small levels have
// nothing else. G as in k_resample_h. Five CTAs per SM: with the four that 50 registers leave, 85 rows wait for a second wave (23 x 156 ->
// 2 x 85 12.5 us, with five 8.4).
constexpr int kSplit = 8;
struct SmallLayout {  // word offsets in shared memory
    int kk_v, bounds_h, kk_h, rows, share, words;
    SmallLayout(const Scale &h, const Scale &v) {
        const int nv = v.in_size == v.out_size ? 1 : std::min(v.ksize, v.in_size);
        kk_v = 0;
        bounds_h = (v.ksize + 1) / 2 * 2;
        kk_h = bounds_h + 2 * h.out_size;
        rows = kk_h + h.out_size * h.ksize;
        share = (rows + (nv + kSplit - 1) / kSplit * h.out_size + 3) / 4 * 4;
        words = share + 4 * h.out_size;
    }
};

template <int G>
__global__ void __cluster_dims__(kSplit, 1, 1) __launch_bounds__(256, 5) k_resize_small(const uint32_t *__restrict__ src, Scale h, Scale v, uint32_t *__restrict__ dst, SmallLayout L) {
    extern __shared__ __align__(16) int32_t sm[];  // share is read as int4
    __shared__ int2 bv;
    const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    int2 *const bounds_h = reinterpret_cast<int2 *>(sm + L.bounds_h);
    uint32_t *const mid = reinterpret_cast<uint32_t *>(sm + L.rows);
    int4 *const share = reinterpret_cast<int4 *>(sm + L.share);
    const int rank = (int)cluster.block_rank(), yy = blockIdx.x / kSplit;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, w = h.in_size, dw = h.out_size;
    const bool need_h = w != dw, need_v = v.in_size != v.out_size;
    const int half = 1 << (kPrecisionBits - 1);
    if (warp == 7) {
        const int2 b = need_v ? output_taps(v, yy, sm + L.kk_v) : make_int2(yy, 1);
        if (lane == 0) bv = b;
    }
    if (need_h && h.ksize <= 32) {
        for (int x = threadIdx.x; x < dw; x += 256) bounds_h[x] = output_taps_thread(h, x, sm + L.kk_h + x * h.ksize);
    } else if (need_h) {
        for (int x = warp; x < dw; x += 8) {
            const int2 b = output_taps(h, x, sm + L.kk_h + x * h.ksize);
            if (lane == 0) bounds_h[x] = b;
        }
    }
    __syncthreads();
    // horizontal: source rows bv.x + rank, + 8, ... -> mid, G lanes an output
    const int rows = bv.y > rank ? (bv.y - rank + kSplit - 1) / kSplit : 0, items = rows * dw, sub = lane & (G - 1);
    for (int i0 = (threadIdx.x & ~31) / G; i0 < items; i0 += 256 / G) {
        const int io = i0 + lane / G, i = io < items ? io : items - 1;
        const int r = i / dw, x = i - r * dw;
        const uint32_t *row = src + (size_t)(bv.x + rank + r * kSplit) * w;
        uint32_t p;
        if (need_h) {
            const int2 b = bounds_h[x];
            const int32_t *k = sm + L.kk_h + x * h.ksize;
            int s[4] = {};
#pragma unroll 4
            for (int t = sub; t < b.y; t += G) add_tap(s, __ldg(row + b.x + t), k[t]);
#pragma unroll
            for (int d = 1; d < G; d <<= 1)
#pragma unroll
                for (int c = 0; c < 4; c++) s[c] += __shfl_xor_sync(0xffffffffu, s[c], d);
            p = weighted(s[0] + half, s[1] + half, s[2] + half, s[3] + half);
        } else {
            p = __ldg(row + x);
        }
        if (io < items && sub == 0) mid[io] = p;
    }
    __syncthreads();
    // vertical: this CTA's rows' share of every column's sums, then the columns' sums over the CTAs
    if (need_v)
        for (int x = threadIdx.x; x < dw; x += 256) {
            int s[4] = {};
            for (int r = 0; r < rows; r++) add_tap(s, mid[r * dw + x], sm[L.kk_v + rank + r * kSplit]);
            share[x] = make_int4(s[0], s[1], s[2], s[3]);
        }
    cluster.sync();
    for (int x = rank + kSplit * threadIdx.x; x < dw; x += kSplit * 256) {
        uint32_t p;
        if (need_v) {
            int4 a = make_int4(half, half, half, half);
#pragma unroll
            for (int c = 0; c < kSplit; c++) {
                const int4 o = cluster.map_shared_rank(share, c)[x];
                a = make_int4(a.x + o.x, a.y + o.y, a.z + o.z, a.w + o.w);
            }
            p = weighted(a.x, a.y, a.z, a.w);
        } else {
            p = cluster.map_shared_rank(mid, 0)[x];  // the one row is rank 0's
        }
        dst[(size_t)yy * dw + x] = p;
    }
    cluster.sync();  // the others' reads of this CTA's shared memory
}

// Which resizes run as one launch: between separate buffers only (its CTAs read the source while others write the result,
// where the two passes of the general path have read all of it before the first write), and where the clusters have little to do.
// Each computes the horizontal taps for itself, and every source row is read by the clusters of the ~2 output rows that need
// it, so many rows or columns cost more than three launches: up to 128 rows (8 CTAs each: little over a wave), 20480
// texels of result and 70 K source texels a cluster, which only 8 SMs read; a single texel's launch saves more than that. Measured, one
// launch / general path: 128^2 -> 64^2 6.7 / 13.0 us, 256^2 -> 64^2 8.0 / 12.6, 500^2 -> 125^2 14.6 / 12.6, 512^2 -> 256^2 28.9 / 12.6,
// 500^2 -> 1000^2 205 / 17, 300^2 -> 1024^2 214 / 17; 915 x 77 -> 19 x 2 (70,455 texels a cluster) 12.5 / 15.6, 510 x 334 -> 7 x 5 (68,850)
// 16.6 / 16.6, 500^2 -> 7^2 (72,500) 18.7 / 16.6, 1086 x 109 -> 66 x 1 (118,374) 33 / 14.7; 512^2 -> 1 16.6 / 20.8.
constexpr long kSmallTexels = 512L * 512, kSmallRows = 128, kSmallResult = 20480, kSmallRead = 71680;

// The result's size first: with it bounded, the layout's and the launch's 32-bit products are in range.
bool small_resize(const Scale &h, const Scale &v) {
    if ((long)h.in_size * v.in_size > kSmallTexels || v.out_size > kSmallRows || (long)h.out_size * v.out_size > kSmallResult) return false;
    const long rows = v.in_size == v.out_size ? 1 : std::min(v.ksize, v.in_size);
    return (rows * h.in_size <= kSmallRead || h.out_size * v.out_size == 1) && (long)SmallLayout(h, v).words * 4 <= 46 * 1024;
}

template <int G> void resize_small_g(const uint32_t *in, const Scale &h, const Scale &v, uint32_t *out, cudaStream_t s) {
    const SmallLayout L(h, v);
    k_resize_small<G><<<(unsigned)v.out_size * kSplit, 256, (size_t)L.words * 4, s>>>(in, h, v, out, L);
}

void resize_small(const uint32_t *in, const Scale &h, const Scale &v, uint32_t *out, cudaStream_t s) {
    const int scale = h.in_size / h.out_size / 2;
    if (scale >= 32) resize_small_g<32>(in, h, v, out, s);
    else if (scale >= 8) resize_small_g<8>(in, h, v, out, s);
    else if (scale >= 2) resize_small_g<2>(in, h, v, out, s);
    else resize_small_g<1>(in, h, v, out, s);
}

template <int G>
void resample_h_g(const uint32_t *in, int w, int y0, int rows, uint32_t *out, int dw, const int2 *b, const int32_t *k, int ksize, cudaStream_t s) {
    const long ctas = std::min<long>(((long)dw * ((rows + 3) / 4) * G + 255) / 256, 148L * 64);
    k_resample_h<G><<<(unsigned)ctas, 256, 0, s>>>(in, w, y0, rows, out, dw, b, k, ksize);
}

void resample_h(const uint32_t *in, int w, int y0, int rows, uint32_t *out, int dw, const int2 *b, const int32_t *k,
                int ksize, cudaStream_t s) {
    const int scale = w / dw / 2;  // lanes per output: half the scale's power of two
    if (scale >= 32) resample_h_g<32>(in, w, y0, rows, out, dw, b, k, ksize, s);
    else if (scale >= 16) resample_h_g<16>(in, w, y0, rows, out, dw, b, k, ksize, s);
    else if (scale >= 8) resample_h_g<8>(in, w, y0, rows, out, dw, b, k, ksize, s);
    else if (scale >= 4) resample_h_g<4>(in, w, y0, rows, out, dw, b, k, ksize, s);
    else if (scale >= 2) resample_h_g<2>(in, w, y0, rows, out, dw, b, k, ksize, s);
    else resample_h_g<1>(in, w, y0, rows, out, dw, b, k, ksize, s);
}

template <int TX>
void resample_v_x(const uint32_t *in, int w, uint32_t *out, int dh, const int2 *b, const int32_t *k, int ksize, cudaStream_t s) {
    k_resample_v<TX><<<dim3((unsigned)((w + TX - 1) / TX), (unsigned)std::min(dh, 65535)), 256, 0, s>>>(in, w, out, dh, b, k, ksize);
}

void resample_v(const uint32_t *in, int w, uint32_t *out, int dh, const int2 *b, const int32_t *k, int ksize,
                cudaStream_t s) {
    if (ksize <= 16) resample_v_x<256>(in, w, out, dh, b, k, ksize, s);
    else if (ksize <= 128) resample_v_x<32>(in, w, out, dh, b, k, ksize, s);
    else if (w >= 64 || (w >= 8 && ksize <= 1024)) resample_v_x<8>(in, w, out, dh, b, k, ksize, s);
    else resample_v_x<1>(in, w, out, dh, b, k, ksize, s);
}

}  // namespace

extern "C" int qtk_resize_is_small(int w, int h, int dw, int dh) { return small_resize(Scale(w, dw), Scale(h, dh)); }

extern "C" int qt_resize_bilinear_device(const uint8_t *src, int w, int h, uint8_t *dst, int dw, int dh, void *stream) {
    if (!src || !dst) return qtk::set_error(QT_ERR_ARG, "NULL buffer");
    if (w <= 0 || h <= 0 || dw <= 0 || dh <= 0) return qtk::set_error(QT_ERR_ARG, "Texture sizes must be greater than 0");
    if ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 3)
        return qtk::set_error(QT_ERR_ARG, "resize: buffers must be 4-byte aligned");
    if (int rc = qtk::ensure_current_device(nullptr)) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e;
    if (dw == w && dh == h) {  // Image.resize to the same size returns a copy
        e = cudaMemcpyAsync(dst, src, (size_t)w * h * 4, cudaMemcpyDeviceToDevice, s);
        return e == cudaSuccess ? QT_OK : qtk::cuda_error((int)e, "resize copy");
    }
    const bool need_h = dw != w, need_v = dh != h;
    const Scale sh(w, dw), sv(h, dh);
    const bool shared = src < dst + (size_t)dw * dh * 4 && dst < src + (size_t)w * h * 4;
    if (!shared && small_resize(sh, sv)) {
        resize_small(reinterpret_cast<const uint32_t *>(src), sh, sv, reinterpret_cast<uint32_t *>(dst), s);
        e = cudaGetLastError();
        return e == cudaSuccess ? QT_OK : qtk::cuda_error((int)e, "resize");
    }
    double centre;
    const int y_first = sv.bounds(0, centre).x, tmp_rows = sv.bounds(dh - 1, centre).y - y_first;

    // one stream-ordered block for both tap tables and the horizontal pass's rows; every part starts on a 16-byte
    // boundary (the bounds are read as 8-byte int2)
    const auto al = [](size_t n) { return (n + 15) / 16 * 16; };
    const size_t o_kh = al((size_t)dw * sizeof(int2)), o_bv = o_kh + al((size_t)dw * sh.ksize * sizeof(int32_t));
    const size_t o_kv = o_bv + al((size_t)dh * sizeof(int2)), o_tmp = o_kv + al((size_t)dh * sv.ksize * sizeof(int32_t));
    uint8_t *d_taps = nullptr;
    if ((e = qtk::scratch_alloc((void **)&d_taps, o_tmp + (need_h && need_v ? (size_t)dw * tmp_rows * 4 : 0), s)) != cudaSuccess)
        return qtk::cuda_error((int)e, "resize scratch");
    uint32_t *const d_tmp = reinterpret_cast<uint32_t *>(d_taps + o_tmp);
    k_taps<<<(unsigned)(((long)dw + dh + 7) / 8), 256, 0, s>>>(sh, sv, reinterpret_cast<int2 *>(d_taps), reinterpret_cast<int32_t *>(d_taps + o_kh),
                                                              reinterpret_cast<int2 *>(d_taps + o_bv), reinterpret_cast<int32_t *>(d_taps + o_kv),
                                                              need_h ? y_first : 0);
    e = cudaGetLastError();
    if (e == cudaSuccess) {
        const int2 *b_h = reinterpret_cast<const int2 *>(d_taps);
        const int32_t *k_h = reinterpret_cast<const int32_t *>(d_taps + o_kh);
        const int2 *b_v = reinterpret_cast<const int2 *>(d_taps + o_bv);
        const int32_t *k_v = reinterpret_cast<const int32_t *>(d_taps + o_kv);
        const uint32_t *in = reinterpret_cast<const uint32_t *>(src);
        uint32_t *out = reinterpret_cast<uint32_t *>(dst);
        if (need_h && need_v) {
            resample_h(in, w, y_first, tmp_rows, d_tmp, dw, b_h, k_h, sh.ksize, s);
            resample_v(d_tmp, dw, out, dh, b_v, k_v, sv.ksize, s);
        } else if (need_h) {
            resample_h(in, w, 0, h, out, dw, b_h, k_h, sh.ksize, s);
        } else {
            resample_v(in, w, out, dh, b_v, k_v, sv.ksize, s);
        }
        e = cudaGetLastError();
    }
    qtk::scratch_free(d_taps, s);
    return e == cudaSuccess ? QT_OK : qtk::cuda_error((int)e, "resize");
}

// ---------------------------------------------------------------------------
// Vertical flip and the BC3nm swizzle of the command-line encoder
// (quicktex/cli/encode.py:52-58: image.transpose(FLIP_TOP_BOTTOM), then
// Image.merge('RGBA', (255, band c1, band c1, band c0))), one texel per thread.
// ---------------------------------------------------------------------------
namespace {

__global__ void __launch_bounds__(256) k_flip_swizzle(const uint32_t *__restrict__ src, int w, int h,
                                                      uint32_t *__restrict__ dst, int flip, int c0, int c1) {
    const long n = (long)w * h;
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const int y = (int)(i / w), x = (int)(i - (long)y * w);
        uint32_t v = __ldg(src + (size_t)(flip ? h - 1 - y : y) * w + x);
        if (c0 >= 0) {
            const uint32_t a = (v >> (8 * c0)) & 0xFF, g = (v >> (8 * c1)) & 0xFF;
            v = 0xFFu | (g << 8) | (g << 16) | (a << 24);
        }
        dst[i] = v;
    }
}

}  // namespace

extern "C" int qt_flip_swizzle_device(const uint8_t *src, int w, int h, uint8_t *dst, int flip, int c0, int c1,
                                      void *stream) {
    if (!src || !dst) return qtk::set_error(QT_ERR_ARG, "NULL buffer");
    if (w <= 0 || h <= 0) return qtk::set_error(QT_ERR_ARG, "Texture sizes must be greater than 0");
    if ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 3)
        return qtk::set_error(QT_ERR_ARG, "flip/swizzle: buffers must be 4-byte aligned");
    if (c0 >= 0 && (c0 > 3 || c1 < 0 || c1 > 3)) return qtk::set_error(QT_ERR_ARG, "Channel out of range");
    const size_t bytes = (size_t)w * h * 4;
    if (src < dst + bytes && dst < src + bytes) return qtk::set_error(QT_ERR_ARG, "flip/swizzle: buffers overlap");
    if (int rc = qtk::ensure_current_device(nullptr)) return rc;
    const long n = (long)w * h;
    long blocks = (n + 255) / 256;
    if (blocks > 148L * 64) blocks = 148L * 64;
    k_flip_swizzle<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(reinterpret_cast<const uint32_t *>(src), w, h,
                                                                     reinterpret_cast<uint32_t *>(dst), flip != 0,
                                                                     c0 >= 0 ? c0 : -1, c1);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? QT_OK : qtk::cuda_error((int)e, "flip/swizzle");
}
