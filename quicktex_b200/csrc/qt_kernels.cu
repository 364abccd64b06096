// qt_kernels.cu — sm_100a kernels of the S3TC encode/decode path and their
// launchers.
//
// Mapping. Every kernel runs one 4x4 block per thread. BC1 (and the colour
// half of BC3) runs the reference encoder (BC1Encoder::EncodeBlock,
// BC1Encoder.cpp:261-342) sequentially per thread, in its order; those
// kernels are in qt_bc1_thread.cuh, included below. The reference's
// FindSelectors early exits never change an accepted result (every exit bound
// is >= the later acceptance bound), so full errors are computed instead.
//
// Floating point. Every operation whose rounding matters is written with an
// explicit round-to-nearest intrinsic (__fadd_rn, __fmul_rn, __fdiv_rn), in
// the reference's operation order; the compiler never contracts these into
// FMAs. Plain float arithmetic (and fmaf) is used only where every operand and
// result is an integer below 2^24, i.e. exact.
//
// BC4/BC5 encode and all decoders are HBM-bound: one thread per block,
// 16-byte row loads/stores where the texture is 4-aligned, 32-bit words elsewhere.
// The persistent batch kernels (k_batch: any mix; k_batch_fast: BC1/BC3 without a
// search) run tiles from a device work queue. The cooperative encoder of levels
// 13-19 is in qt_coop.cu.

#include <cuda_pipeline.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <type_traits>

#include "qt_coop.h"
#include "qt_device.cuh"

namespace qtk {

// One thread per block. Idx is uint32_t whenever the block count and the grid fit
// 31 bits (the common case: no 64-bit division per block), else uint64_t. BC5 is held to
// 40 registers (6 CTAs of 256 threads per SM instead of 5 at its natural 44): its loads
// need the extra warps in flight (measured 0.83 -> 0.88 of HBM at 16384^2, bit-identical).
// BC4 gives no minimum (0), where the compiler settles at 32 registers; an explicit
// minimum of 1 to 4 CTAs lets it take 52-56 and costs BC4 a tenth of its bandwidth.
//
// BC4: one block per thread. BC5 (two channels' arithmetic per texel) was latency-bound, so its
// grid is persistent (the SMs filled at the kernel's occupancy) and each thread's next block
// arrives by cp.async into shared memory while it encodes the current one: the rows are
// transposed there ([buffer][texel row][thread], 16 bytes each), so a warp's copies and reads
// are conflict-free, and the block in flight holds no registers (0.88 -> 0.905 of HBM; the same
// for BC4 measured 0.97 -> 0.91, so BC4 keeps the plain loop). Edge blocks of a texture whose
// width is not a multiple of 4 (or an unaligned base) are loaded directly, with the wrap rule.
template <bool BC5, typename Idx, bool STAGED = BC5>
__global__ void __launch_bounds__(256, BC5 ? 6 : 0) k_bc4_encode(const uint8_t *__restrict__ rgba, int w, int h, Idx bw, Idx b_begin,
                                                    Idx nblocks, int c0, int c1, int aligned, uint8_t *__restrict__ out) {
    if constexpr (!STAGED) {
        for (Idx b = b_begin + (Idx)blockIdx.x * blockDim.x + threadIdx.x; b < nblocks; b += (Idx)gridDim.x * blockDim.x) {
            const int by = (int)(b / bw), bx = (int)(b - (Idx)by * bw);
            uint32_t px[16];
            load_block_any(rgba, w, h, bx, by, aligned && (bx * 4 + 4 <= w) && (by * 4 + 4 <= h), px);
            if constexpr (BC5) reinterpret_cast<uint4 *>(out)[b] = bc5_block_thread(px, c0, c1);
            else reinterpret_cast<uint2 *>(out)[b] = bc4_block_thread(px, c0);
        }
        return;
    }
    __shared__ uint4 stage[2][4][256];
    const Idx stride = (Idx)gridDim.x * blockDim.x;
    // the row copies of block bb into buffer buf, when it is an aligned interior block
    auto prefetch = [&](Idx bb, int buf) -> bool {
        if (bb >= nblocks) return false;
        const int by = (int)(bb / bw), bx = (int)(bb - (Idx)by * bw);
        if (!(aligned && (bx * 4 + 4 <= w) && (by * 4 + 4 <= h))) return false;
#pragma unroll
        for (int y = 0; y < 4; y++)
            __pipeline_memcpy_async(&stage[buf][y][threadIdx.x], rgba + ((size_t)(by * 4 + y) * w + bx * 4) * 4, 16);
        return true;
    };
    Idx b = b_begin + (Idx)blockIdx.x * blockDim.x + threadIdx.x;
    bool staged = prefetch(b, 0);
    __pipeline_commit();
    for (int buf = 0; b < nblocks; b += stride, buf ^= 1) {
        const bool next = prefetch(b + stride, buf ^ 1);
        __pipeline_commit();
        __pipeline_wait_prior(1);  // this block's copies (the group before the newest) have landed
        uint32_t px[16];
        if (staged) {
#pragma unroll
            for (int y = 0; y < 4; y++) {
                const uint4 q = stage[buf][y][threadIdx.x];
                px[4 * y] = q.x; px[4 * y + 1] = q.y; px[4 * y + 2] = q.z; px[4 * y + 3] = q.w;
            }
        } else {
            const int by = (int)(b / bw), bx = (int)(b - (Idx)by * bw);
            load_block_thread(rgba, w, h, bx, by, false, px);
        }
        reinterpret_cast<uint4 *>(out)[b] = bc5_block_thread(px, c0, c1);
        staged = next;
    }
    __pipeline_wait_prior(0);
}

// BC1 palette for decoding: Interpolator::Interpolate565BC1 (Interpolator.cpp:52-55)
template <int IT>
__device__ __forceinline__ void bc1_palette(uint32_t c0, uint32_t c1, bool allow3, bool write_alpha, uint32_t col[4]) {
    const int lo = (int)c0, hi = (int)c1;  // packed 5:6:5 == eppack layout
    const bool three = allow3 && (c1 >= c0);
    const Pal P = make_pal<IT>(lo, hi, three);
    // back to BC1 index order: colors[0]=c0, [1]=c1, [2], [3]
    uint32_t a3 = three ? 0u : 255u;
    if (!write_alpha) a3 = 255u;
    col[0] = (uint32_t)P.r0 | ((uint32_t)P.g0 << 8) | ((uint32_t)P.b0 << 16) | 0xFF000000u;
    col[2] = (uint32_t)P.r1 | ((uint32_t)P.g1 << 8) | ((uint32_t)P.b1 << 16) | 0xFF000000u;
    if (!three) {
        col[3] = (uint32_t)P.r2 | ((uint32_t)P.g2 << 8) | ((uint32_t)P.b2 << 16) | 0xFF000000u;
        col[1] = (uint32_t)P.r3 | ((uint32_t)P.g3 << 8) | ((uint32_t)P.b3 << 16) | 0xFF000000u;
    } else {
        col[1] = (uint32_t)P.r2 | ((uint32_t)P.g2 << 8) | ((uint32_t)P.b2 << 16) | 0xFF000000u;
        col[3] = (uint32_t)P.r3 | ((uint32_t)P.g3 << 8) | ((uint32_t)P.b3 << 16) | (a3 << 24);
    }
}

// BC4Block::GetValues (BC4Block.cpp:44-64), the 8 values as bytes: lo = values 0..3, hi = 4..7
__device__ __forceinline__ uint2 bc4_value_bytes(uint32_t a0, uint32_t a1) {
    uint32_t v2, v3, v4, v5, v6, v7;
    if (a0 <= a1) {  // GetValues6 (BC4Block.cpp:44-53)
        v2 = (a0 * 4 + a1) / 5; v3 = (a0 * 3 + a1 * 2) / 5; v4 = (a0 * 2 + a1 * 3) / 5; v5 = (a0 + a1 * 4) / 5;
        v6 = 0; v7 = 255;
    } else {  // GetValues8 (:55-64)
        v2 = (a0 * 6 + a1) / 7; v3 = (a0 * 5 + a1 * 2) / 7; v4 = (a0 * 4 + a1 * 3) / 7;
        v5 = (a0 * 3 + a1 * 4) / 7; v6 = (a0 * 2 + a1 * 5) / 7; v7 = (a0 + a1 * 6) / 7;
    }
    return make_uint2(a0 | (a1 << 8) | (v2 << 16) | (v3 << 24), v4 | (v5 << 8) | (v6 << 16) | (v7 << 24));
}

// Four 2-bit (BC1) or 3-bit (BC4) indices of one texel row, one per nibble: a PRMT selector.
__device__ __forceinline__ uint32_t nibbles2(uint32_t x) {
    x = (x & 0x0Fu) | ((x & 0xF0u) << 4);
    return (x & 0x0303u) | ((x & 0x0C0Cu) << 2);
}
__device__ __forceinline__ uint32_t nibbles3(uint32_t x) {
    return (x & 0x7u) | ((x & 0x38u) << 1) | ((x & 0x1C0u) << 2) | ((x & 0xE00u) << 3);
}

// The BC4 values of texel row y (4 texels), one byte each, from the 48 selector bits
__device__ __forceinline__ uint32_t bc4_row(uint2 vals, uint32_t sel_lo, uint32_t sel_hi, int y) {
    const uint32_t x = y == 0 ? sel_lo : y == 1 ? (sel_lo >> 12) : y == 2 ? __funnelshift_r(sel_lo, sel_hi, 24) : (sel_hi >> 4);
    return __byte_perm(vals.x, vals.y, nibbles3(x & 0xFFFu));
}

// Decode of one block into px[16] (RGBA8 words), for FMT 1 (BC1Decoder.cpp:33-55),
// 3 (BC3Decoder.cpp:26-31: BC1 colours without 3-colour mode, then BC4 into alpha),
// 4 (BC4Decoder.cpp:29-43 into channel c0 of (0,0,0,255)) and
// 5 (BC5Decoder.cpp:25-30: c0, then c1).
template <int FMT, int IT>
__device__ __forceinline__ void decode_texels(const uint8_t *__restrict__ blocks, size_t b, int write_alpha, int c0,
                                              int c1, uint32_t px[16]) {
    if (FMT == 1 || FMT == 3) {
        uint2 cb, ab = make_uint2(0u, 0u);
        if (FMT == 1) {
            cb = __ldg(reinterpret_cast<const uint2 *>(blocks) + b);
        } else {
            const uint4 q = __ldg(reinterpret_cast<const uint4 *>(blocks) + b);
            ab = make_uint2(q.x, q.y);
            cb = make_uint2(q.z, q.w);
        }
        uint32_t col[4];
        bc1_palette<IT>(cb.x & 0xFFFF, cb.x >> 16, FMT == 1, FMT == 1 && write_alpha, col);
        // channel planes: byte k of each = that channel of col[k]
        const uint32_t A = __byte_perm(col[0], col[1], 0x5140), B = __byte_perm(col[2], col[3], 0x5140);
        const uint32_t C = __byte_perm(col[0], col[1], 0x7362), D = __byte_perm(col[2], col[3], 0x7362);
        const uint32_t Rp = __byte_perm(A, B, 0x5410), Gp = __byte_perm(A, B, 0x7632);
        const uint32_t Bp = __byte_perm(C, D, 0x5410), Ap = __byte_perm(C, D, 0x7632);
        uint2 av = make_uint2(0u, 0u);
        uint32_t slo = 0u, shi = 0u;
        if (FMT == 3) {
            av = bc4_value_bytes(ab.x & 0xFF, (ab.x >> 8) & 0xFF);
            slo = (ab.x >> 16) | (ab.y << 16);
            shi = ab.y >> 16;
        }
#pragma unroll
        for (int y = 0; y < 4; y++) {
            const uint32_t S = nibbles2((cb.y >> (8 * y)) & 0xFFu);
            const uint32_t Rr = __byte_perm(Rp, 0u, S), Gr = __byte_perm(Gp, 0u, S), Br = __byte_perm(Bp, 0u, S);
            const uint32_t Ar = FMT == 3 ? bc4_row(av, slo, shi, y) : __byte_perm(Ap, 0u, S);
            const uint32_t X = __byte_perm(Rr, Gr, 0x5140), Y = __byte_perm(Br, Ar, 0x5140);
            const uint32_t X2 = __byte_perm(Rr, Gr, 0x7362), Y2 = __byte_perm(Br, Ar, 0x7362);
            px[4 * y + 0] = __byte_perm(X, Y, 0x5410);
            px[4 * y + 1] = __byte_perm(X, Y, 0x7632);
            px[4 * y + 2] = __byte_perm(X2, Y2, 0x5410);
            px[4 * y + 3] = __byte_perm(X2, Y2, 0x7632);
        }
    } else {
        uint2 q0, q1 = make_uint2(0u, 0u);
        if (FMT == 4) {
            q0 = __ldg(reinterpret_cast<const uint2 *>(blocks) + b);
        } else {
            const uint4 q = __ldg(reinterpret_cast<const uint4 *>(blocks) + b);
            q0 = make_uint2(q.x, q.y);
            q1 = make_uint2(q.z, q.w);
        }
        // texel k of a row: byte c0 <- value k, other bytes of (0,0,0,255); BC5 then byte c1 <- value k
        const uint32_t base0 = 0x7444u & ~(0xFu << (4 * c0));
        const uint32_t base1 = 0x3210u & ~(0xFu << (4 * c1));
        const uint2 v0 = bc4_value_bytes(q0.x & 0xFF, (q0.x >> 8) & 0xFF);
        const uint32_t lo0 = (q0.x >> 16) | (q0.y << 16), hi0 = q0.y >> 16;
        uint2 v1 = make_uint2(0u, 0u);
        uint32_t lo1 = 0u, hi1 = 0u;
        if (FMT == 5) {
            v1 = bc4_value_bytes(q1.x & 0xFF, (q1.x >> 8) & 0xFF);
            lo1 = (q1.x >> 16) | (q1.y << 16);
            hi1 = q1.y >> 16;
        }
#pragma unroll
        for (int y = 0; y < 4; y++) {
            const uint32_t W0 = bc4_row(v0, lo0, hi0, y);
            const uint32_t W1 = FMT == 5 ? bc4_row(v1, lo1, hi1, y) : 0u;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                uint32_t t = __byte_perm(W0, 0xFF000000u, base0 | ((uint32_t)k << (4 * c0)));
                if (FMT == 5) t = __byte_perm(t, W1, base1 | ((uint32_t)(4 + k) << (4 * c1)));
                px[4 * y + k] = t;
            }
        }
    }
}

// Store of a decoded block. Every texel of every block is decoded, and a texel
// is stored only if no later block (in the reference's by, bx, x, y write
// order) writes the same wrapped position: source (px, py) is final iff
// px + w >= 4*bw and py + h >= 4*bh (RawTexture::SetBlock, Texture.h:114-134).
// An interior block of a texture whose rows are off the 16-byte grid stores its texels one by one at fixed offsets. The
// wrapped form took all blocks of such a texture, two divisions a texel: BC1 8191 x 8190 162 -> 71 us, BC5 176 -> 73; aligned
// words formed by shuffles across lanes: 83.
__device__ __forceinline__ void store_block(const uint32_t px[16], int w, int h, int bw, int bh, int bx, int by,
                                            bool aligned, uint8_t *__restrict__ rgba) {
    if (bx > 0 && by > 0 && bx * 4 + 4 <= w && by * 4 + 4 <= h) {
        uint32_t *at = reinterpret_cast<uint32_t *>(rgba) + (size_t)(by * 4) * w + bx * 4;
#pragma unroll
        for (int y = 0; y < 4; y++, at += w) {
            if (aligned) {
                *reinterpret_cast<uint4 *>(at) = make_uint4(px[4 * y], px[4 * y + 1], px[4 * y + 2], px[4 * y + 3]);
            } else {
#pragma unroll
                for (int x = 0; x < 4; x++) at[x] = px[4 * y + x];
            }
        }
    } else {
#pragma unroll
        for (int y = 0; y < 4; y++)
#pragma unroll
            for (int x = 0; x < 4; x++) {
                const int sx = bx * 4 + x, sy = by * 4 + y;
                if (sx + w >= 4 * bw && sy + h >= 4 * bh)
                    *reinterpret_cast<uint32_t *>(rgba + ((size_t)wrapped(sy, h) * w + wrapped(sx, w)) * 4) = px[4 * y + x];
            }
    }
}

template <int FMT, int IT>
__device__ __forceinline__ void decode_block_fmt(const uint8_t *__restrict__ blocks, int w, int h, int bw, int bh,
                                                 size_t b, int bx, int by, int write_alpha, int c0, int c1,
                                                 bool aligned, uint8_t *__restrict__ rgba) {
    uint32_t px[16];
    decode_texels<FMT, IT>(blocks, b, write_alpha, c0, c1, px);
    store_block(px, w, h, bw, bh, bx, by, aligned, rgba);
}

// Runtime-format decode of block b (the batch kernel's entry).
template <int IT>
__device__ __forceinline__ void decode_block(const uint8_t *__restrict__ blocks, int w, int h, int bw, int bh, long b,
                                             int fmt, int write_alpha, int c0, int c1, int aligned,
                                             uint8_t *__restrict__ rgba) {
    const int by = (int)(b / bw), bx = (int)(b - (long)by * bw);
    switch (fmt) {
        case 1: decode_block_fmt<1, IT>(blocks, w, h, bw, bh, (size_t)b, bx, by, write_alpha, c0, c1, aligned, rgba); break;
        case 3: decode_block_fmt<3, IT>(blocks, w, h, bw, bh, (size_t)b, bx, by, write_alpha, c0, c1, aligned, rgba); break;
        case 4: decode_block_fmt<4, IT>(blocks, w, h, bw, bh, (size_t)b, bx, by, write_alpha, c0, c1, aligned, rgba); break;
        default: decode_block_fmt<5, IT>(blocks, w, h, bw, bh, (size_t)b, bx, by, write_alpha, c0, c1, aligned, rgba); break;
    }
}

// One thread per block; Idx as in k_bc4_encode.
template <int FMT, int IT, typename Idx>
__global__ void __launch_bounds__(256) k_decode(const uint8_t *__restrict__ blocks, int w, int h, Idx bw, int bh,
                                                Idx b_begin, Idx nblocks, int write_alpha, int c0, int c1, int aligned,
                                                uint8_t *__restrict__ rgba) {
    for (Idx b = b_begin + (Idx)blockIdx.x * blockDim.x + threadIdx.x; b < nblocks; b += (Idx)gridDim.x * blockDim.x) {
        const int by = (int)(b / bw), bx = (int)(b - (Idx)by * bw);
        decode_block_fmt<FMT, IT>(blocks, w, h, (int)bw, bh, (size_t)b, bx, by, write_alpha, c0, c1, aligned != 0, rgba);
    }
}

#include "qt_bc1_thread.cuh"

// ---------------------------------------------------------------------------
// persistent batch kernel: many textures, any format / op / level, one launch.
// A warp claims one tile (consecutive blocks of one texture) at a time; its
// lanes take the tile's blocks, one block per thread.
// ---------------------------------------------------------------------------
template <int IT> __device__ __noinline__ uint2 encode_bc1_batch(const qt_bc1_params *p, int color_mode, int pp) {
    return tpb::encode_block<IT>(*p, color_mode, pp);
}

__device__ __forceinline__ void batch_block(const BatchItemDev &__restrict__ I, long b) {
    const bool aligned = ((I.w & 3) == 0) && ((reinterpret_cast<uintptr_t>(I.op == QT_OP_ENCODE ? I.src : I.dst) & 15) == 0);
    if (I.op == QT_OP_DECODE) {
        switch (I.interp) {
            case IT_IDEAL: decode_block<IT_IDEAL>(I.src, I.w, I.h, I.bw, I.bh, b, I.fmt, I.write_alpha, I.c0, I.c1, aligned, I.dst); break;
            case IT_ROUND: decode_block<IT_ROUND>(I.src, I.w, I.h, I.bw, I.bh, b, I.fmt, I.write_alpha, I.c0, I.c1, aligned, I.dst); break;
            case IT_NVIDIA: decode_block<IT_NVIDIA>(I.src, I.w, I.h, I.bw, I.bh, b, I.fmt, I.write_alpha, I.c0, I.c1, aligned, I.dst); break;
            default: decode_block<IT_AMD>(I.src, I.w, I.h, I.bw, I.bh, b, I.fmt, I.write_alpha, I.c0, I.c1, aligned, I.dst); break;
        }
        return;
    }
    const int by = (int)(b / I.bw), bx = (int)(b - (long)by * I.bw);
    uint32_t v[16];
    load_block_thread(I.src, I.w, I.h, bx, by, aligned && (bx * 4 + 4 <= I.w) && (by * 4 + 4 <= I.h), v);
    if (I.fmt == 4 || I.fmt == 5) {
        if (I.fmt == 5) reinterpret_cast<uint4 *>(I.dst)[b] = bc5_block_thread(v, I.c0, I.c1);
        else reinterpret_cast<uint2 *>(I.dst)[b] = bc4_block_thread(v, I.c0);
        return;
    }
    int pp = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        tpb::t_px[i][threadIdx.x] = v[i];
        const uint32_t u = v[i] & 0x00FFFFFFu;
        pp += (int)__dp4a(u, u, 0u);
    }
    const int cm = I.fmt == 3 ? CM_FOUR : I.p.color_mode;  // BC3Encoder.h:39-40
    uint2 blk;
    switch (I.p.interpolator) {
        case IT_IDEAL: blk = encode_bc1_batch<IT_IDEAL>(&I.p, cm, pp); break;
        case IT_ROUND: blk = encode_bc1_batch<IT_ROUND>(&I.p, cm, pp); break;
        case IT_NVIDIA: blk = encode_bc1_batch<IT_NVIDIA>(&I.p, cm, pp); break;
        default: blk = encode_bc1_batch<IT_AMD>(&I.p, cm, pp); break;
    }
    if (I.fmt == 3) {
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = tpb::t_px[i][threadIdx.x];
        const uint2 a = bc4_block_thread(v, 3);
        reinterpret_cast<uint4 *>(I.dst)[b] = make_uint4(a.x, a.y, blk.x, blk.y);
    } else {
        reinterpret_cast<uint2 *>(I.dst)[b] = blk;
    }
}

// ctl[0] is the queue head (atomically advanced by each warp), ctl[1] the number of tiles.
__global__ void __launch_bounds__(tpb::kThreads, 4) k_batch(const BatchItemDev *__restrict__ items,
                                                            const TileDev *__restrict__ tiles, uint32_t *__restrict__ ctl) {
    for (int i = threadIdx.x; i < 64; i += blockDim.x) {
        if (i < 32) s_mid5[i] = c_mid5[i];
        s_mid6[i] = c_mid6[i];
        if (i < 16) s_vox[i] = c_voxels[i];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint32_t ntiles = ctl[1];
    while (true) {
        uint32_t t = 0;
        if (lane == 0) t = atomicAdd(&ctl[0], 1u);
        t = __shfl_sync(0xFFFFFFFFu, t, 0);
        if (t >= ntiles) break;
        const TileDev T = tiles[t];
        // the descriptor stays in (L1-cached) global memory: copying it to registers spills
        const BatchItemDev &I = items[T.item];
        for (uint32_t k = lane; k < T.count; k += 32) batch_block(I, (long)T.start + k);
        __syncwarp();
    }
}

// The batch's tiles of BC1/BC3 textures at settings without EndpointSearch and with the Faster or Check2 error mode (levels
// 0-3 and 5-12), one kernel per interpolator, error mode and colour mode, specialised as k_bc1_fast is:
// tiles[.. ctl[1]) through the counter ctl[0]. k_batch's generic body (phases called, kinds chosen at run time) costs
// about twice the instructions at levels 0-10 and, where a batch is small, 34 cycles an instruction: the eight levels of a
// 128^2 chain at level 5 took it 183 us. 400 mixed textures up to 1024^2: 977 -> 754 us; 64^2 chain, level 5: 212 -> 157.
template <int IT, int K4, int CM>
__global__ void __launch_bounds__(tpb::kThreads, K4 == K_F4_FASTER ? 6 : 4) k_batch_fast(const BatchItemDev *__restrict__ items,
                                                                                        const TileDev *__restrict__ tiles, uint32_t *__restrict__ ctl) {
    for (int i = threadIdx.x; i < 64; i += blockDim.x) {
        if (i < 32) s_mid5[i] = c_mid5[i];
        s_mid6[i] = c_mid6[i];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint32_t ntiles = ctl[1];
    while (true) {
        uint32_t t = 0;
        if (lane == 0) t = atomicAdd(&ctl[0], 1u);
        t = __shfl_sync(0xFFFFFFFFu, t, 0);
        if (t >= ntiles) break;
        const TileDev T = tiles[t];
        const BatchItemDev &I = items[T.item];
        const qt_bc1_params p = I.p;
        const int bc3 = I.fmt == 3, w = I.w, h = I.h, bw = I.bw;
        const int aligned = ((w & 3) == 0) && ((reinterpret_cast<uintptr_t>(I.src) & 15) == 0);
        for (uint32_t j = lane; j < T.count; j += 32) {
            const long b = (long)T.start + j;
            uint32_t v[16];
            const int pp = stage_block(I.src, w, h, bw, b, aligned, v);
            const uint2 blk = tpb::encode_block<IT, K4, true, false>(p, CM, pp);
            if (bc3) {
#pragma unroll
                for (int i = 0; i < 16; i++) v[i] = tpb::t_px[i][threadIdx.x];
                const uint2 a = bc4_block_thread(v, 3);
                reinterpret_cast<uint4 *>(I.dst)[b] = make_uint4(a.x, a.y, blk.x, blk.y);
            } else {
                reinterpret_cast<uint2 *>(I.dst)[b] = blk;
            }
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// host-side launchers
// ---------------------------------------------------------------------------
int num_sms() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    return sms;
}

static int grid_for(long work, int per_cta) {
    const long need = (work + per_cta - 1) / per_cta;
    const long cap = (long)num_sms() * 64;
    return (int)(need < cap ? (need > 0 ? need : 1) : cap);
}

int upload_tables(int device) {
    int prev = 0;
    cudaGetDevice(&prev);
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_tab, &host_tables(), sizeof(DevTables));
    if (e == cudaSuccess) e = upload_coop_tables();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    cudaSetDevice(prev);
    return (int)e;
}

// below this many blocks the split pass costs more than idle solid lanes do
constexpr long kSplitMinBlocks = 16384;

long defer_min_blocks() { return 2L * num_sms() * 4 * tpb::kThreads; }

// the four-colour cluster fit runs twice (EncodeBlock, BC1Encoder.cpp:299-302); exactly then
// encode_block, given a Deferred, stops blocks before the second pass
static bool cf2_pass(const qt_bc1_params &p) {
    return p.two_cf_passes && (p.exhaustive || p.orderings3 > 0 || p.orderings4 > 0);
}

// The specialised encoder (k_bc1_fast) for a setting without EndpointSearch: its four-colour
// selector kind is the error mode (every setting has cluster-fit orderings, so it needs block
// errors: BC1Encoder.cpp:267-276); its colour mode is the setting's, four-colour for BC3. With
// list/count the blocks are the listed ones.
template <int IT, int K4>
static void launch_fast_k(int g, cudaStream_t s, const uint8_t *rgba, int w, int h, int bw, long b0, long b1,
                          const qt_bc1_params &p, uint8_t *out, bool bc3, int aligned, const uint32_t *list,
                          const uint32_t *count) {
    const int cm = bc3 ? CM_FOUR : p.color_mode;  // BC3Encoder.h:39-40
    if (cm == CM_FOUR)
        k_bc1_fast<IT, K4, CM_FOUR><<<g, tpb::kThreads, 0, s>>>(rgba, w, h, bw, b0, b1, p, out, bc3, aligned, list, count);
    else if (cm == CM_THREE)
        k_bc1_fast<IT, K4, CM_THREE><<<g, tpb::kThreads, 0, s>>>(rgba, w, h, bw, b0, b1, p, out, bc3, aligned, list, count);
    else
        k_bc1_fast<IT, K4, CM_TB><<<g, tpb::kThreads, 0, s>>>(rgba, w, h, bw, b0, b1, p, out, bc3, aligned, list, count);
}

template <int IT>
static void launch_fast_it(int g, cudaStream_t s, const uint8_t *rgba, int w, int h, int bw, long b0, long b1,
                           const qt_bc1_params &p, uint8_t *out, bool bc3, int aligned, const uint32_t *list,
                           const uint32_t *count) {
    switch (p.error_mode) {
        case EM_NONE: launch_fast_k<IT, K_F4_NONE>(g, s, rgba, w, h, bw, b0, b1, p, out, bc3, aligned, list, count); break;
        case EM_FASTER: launch_fast_k<IT, K_F4_FASTER>(g, s, rgba, w, h, bw, b0, b1, p, out, bc3, aligned, list, count); break;
        case EM_CHECK2: launch_fast_k<IT, K_F4_CHECK2>(g, s, rgba, w, h, bw, b0, b1, p, out, bc3, aligned, list, count); break;
        default: launch_fast_k<IT, K_F4_FULL>(g, s, rgba, w, h, bw, b0, b1, p, out, bc3, aligned, list, count); break;
    }
}

static void launch_fast(int g, cudaStream_t s, const uint8_t *rgba, int w, int h, int bw, long b0, long b1,
                        const qt_bc1_params &p, uint8_t *out, bool bc3, int aligned, const uint32_t *list,
                        const uint32_t *count) {
    switch (p.interpolator) {
        case IT_IDEAL: launch_fast_it<IT_IDEAL>(g, s, rgba, w, h, bw, b0, b1, p, out, bc3, aligned, list, count); break;
        case IT_ROUND: launch_fast_it<IT_ROUND>(g, s, rgba, w, h, bw, b0, b1, p, out, bc3, aligned, list, count); break;
        case IT_NVIDIA: launch_fast_it<IT_NVIDIA>(g, s, rgba, w, h, bw, b0, b1, p, out, bc3, aligned, list, count); break;
        default: launch_fast_it<IT_AMD>(g, s, rgba, w, h, bw, b0, b1, p, out, bc3, aligned, list, count); break;
    }
}

template <typename F>
static void by_interp(int interpolator, F &&f) {
    switch (interpolator) {
        case IT_IDEAL: f(std::integral_constant<int, IT_IDEAL>()); break;
        case IT_ROUND: f(std::integral_constant<int, IT_ROUND>()); break;
        case IT_NVIDIA: f(std::integral_constant<int, IT_NVIDIA>()); break;
        default: f(std::integral_constant<int, IT_AMD>()); break;
    }
}

// Scratch of the deferred path over n blocks, in 32-bit words: a 64-word header (word 0 the
// list count, 1-3 the search queues' counts, 4-6 their heads, 8-9 the second-pass queue's
// counts, 16 the finish queue's count, 32-63 the list counts of a texture encoded in parts),
// the list of non-solid blocks, the three search queues (5 arrays each), the finish queue (3
// arrays) and, with the second cluster-fit pass, its queue (6 arrays).
constexpr int kPartCount0 = 32, kMaxParts = 32;
static size_t defer_words(long n, bool cf2) { return 64 + 19 * (size_t)n + (cf2 ? 6 * (size_t)n : 0); }

static DeferQueues defer_layout(uint32_t *scratch, long n, bool cf2) {
    DeferQueues d{};
    uint32_t *qb = scratch + 64 + n;
    d.q.count = scratch + 1;
    d.q.head = scratch + 4;
    d.q.cap = n;
    d.q.b = qb;
    d.q.lohi = qb + 3 * (size_t)n;
    d.q.err = qb + 6 * (size_t)n;
    d.q.sel = qb + 9 * (size_t)n;
    d.q.mode = qb + 12 * (size_t)n;
    d.fq.count = scratch + 16;  // searches that moved the endpoints
    d.fq.b = qb + 15 * (size_t)n;
    d.fq.lohi = d.fq.b + (size_t)n;
    d.fq.mode = d.fq.b + 2 * (size_t)n;
    if (cf2) {
        uint32_t *cb = qb + 18 * (size_t)n;
        d.c.count = scratch + 8;
        d.c.b = cb;
        d.c.lohi = cb + (size_t)n;
        d.c.err = cb + 2 * (size_t)n;
        d.c.sel = cb + 3 * (size_t)n;
        d.c.mode = cb + 4 * (size_t)n;
        d.c.orig = cb + 5 * (size_t)n;
        d.c.cap = n;
    }
    return d;
}

template <int IT>
static void launch_split(cudaStream_t s, const uint8_t *rgba, int w, int h, long b0, long b1, uint8_t *out, bool bc3, int aligned, uint32_t *list,
                         uint32_t *count) {
    k_bc1_split<IT><<<grid_for(b1 - b0, kSplitThreads), kSplitThreads, 0, s>>>(rgba, w, h, (w + 3) / 4, b0, b1, out, bc3, aligned, list, count);
}

// The deferred path's first passes over the blocks [b0, b1): the split pass lists the
// non-solid blocks in list/count, the encoder runs each to its first cluster-fit pass and
// queues what remains (second pass, 3-colour trials, EndpointSearch) in d.
template <int I>
static void defer_front(const uint8_t *rgba, int w, int h, const qt_bc1_params &p, uint8_t *out, bool bc3, int aligned,
                        const DeferQueues &d, bool coop, uint32_t *list, uint32_t *count, long b0, long b1, cudaStream_t s) {
    const int bw = (w + 3) / 4;
    const long n = b1 - b0;
    launch_split<I>(s, rgba, w, h, b0, b1, out, bc3, aligned, list, count);
    if (coop) {
        coop_defer(rgba, w, h, p, out, bc3, aligned, n, list, count, d, s);
        return;
    }
    k_bc1_defer<I><<<grid_for(n, tpb::kThreads), tpb::kThreads, 0, s>>>(rgba, w, h, bw, p, out, bc3, aligned, list,
                                                                          count, d.q, d.c);
}

// ... and its passes over the queues: second cluster-fit pass and 3-colour trials (cf2),
// EndpointSearch with lane refill, and the selectors of the searches that moved.
template <int I>
static void defer_back(const uint8_t *rgba, int w, int h, const qt_bc1_params &p, uint8_t *out, bool bc3, int aligned,
                       const DeferQueues &d, bool cf2, bool coop, cudaStream_t s) {
    const int bw = (w + 3) / 4;
    const int gsearch = num_sms() * 4;
    if (coop) {
        coop_defer_rest(rgba, w, h, p, out, bc3, aligned, d, cf2, s);
        k_bc1_finish<I><<<gsearch, tpb::kThreads, 0, s>>>(rgba, w, h, bw, p, out, bc3, aligned, d.fq);
        return;
    }
    if (cf2) k_bc1_cf2<I><<<gsearch, tpb::kThreads, 0, s>>>(rgba, w, h, bw, p, out, bc3, aligned, d.c, d.q);
    k_bc1_search<I><<<gsearch, tpb::kThreads, 0, s>>>(rgba, w, h, bw, p, out, bc3, aligned, d.q, d.fq);
    k_bc1_finish<I><<<gsearch, tpb::kThreads, 0, s>>>(rgba, w, h, bw, p, out, bc3, aligned, d.fq);
}

static int texel_aligned(const uint8_t *rgba, int w) {
    return ((w & 3) == 0) && ((reinterpret_cast<uintptr_t>(rgba) & 15) == 0);
}

bool bc1_parts_eligible(long nblocks, const qt_bc1_params &p) {
    return p.search_rounds > 0 && nblocks >= defer_min_blocks() && nblocks <= 0xFFFFFFFFL;
}

int bc1_parts_begin(Bc1Parts &ps, long nblocks, const qt_bc1_params &p, void *stream) {
    cudaStream_t s = (cudaStream_t)stream;
    ps = Bc1Parts{};
    if (!bc1_parts_eligible(nblocks, p)) return (int)cudaErrorInvalidValue;
    ps.n = nblocks;
    ps.cf2 = cf2_pass(p);
    cudaError_t e = scratch_alloc((void **)&ps.scratch, defer_words(nblocks, ps.cf2) * sizeof(uint32_t), s);
    if (e != cudaSuccess) {
        ps.scratch = nullptr;
        return (int)e;
    }
    e = cudaMemsetAsync(ps.scratch, 0, 64 * sizeof(uint32_t), s);
    return (int)e;
}

int bc1_parts_add(Bc1Parts &ps, const uint8_t *rgba, int w, int h, const qt_bc1_params &p, uint8_t *out, bool bc3,
                  long b_begin, long b_end, void *stream) {
    if (!ps.scratch || ps.parts >= kMaxParts || b_begin < 0 || b_end > ps.n || b_end <= b_begin)
        return (int)cudaErrorInvalidValue;
    // part k lists its non-solid blocks in its own slice of the list (at most b_end - b_begin
    // of them) and counts them in header word 32 + k; the queues are shared
    uint32_t *list = ps.scratch + 64 + b_begin, *count = ps.scratch + kPartCount0 + ps.parts++;
    const DeferQueues d = defer_layout(ps.scratch, ps.n, ps.cf2);
    cudaStream_t s = (cudaStream_t)stream;
    by_interp(p.interpolator, [&](auto I) {
        defer_front<decltype(I)::value>(rgba, w, h, p, out, bc3, texel_aligned(rgba, w), d, coop_setting(p, ps.n), list, count, b_begin, b_end, s);
    });
    return (int)cudaGetLastError();
}

int bc1_parts_end(Bc1Parts &ps, const uint8_t *rgba, int w, int h, const qt_bc1_params &p, uint8_t *out, bool bc3,
                  void *stream) {
    if (!ps.scratch) return (int)cudaErrorInvalidValue;
    const DeferQueues d = defer_layout(ps.scratch, ps.n, ps.cf2);
    cudaStream_t s = (cudaStream_t)stream;
    by_interp(p.interpolator, [&](auto I) {
        defer_back<decltype(I)::value>(rgba, w, h, p, out, bc3, texel_aligned(rgba, w), d, ps.cf2, coop_setting(p, ps.n), s);
    });
    const cudaError_t e = cudaGetLastError();
    bc1_parts_free(ps, stream);
    return (int)e;
}

void bc1_parts_free(Bc1Parts &ps, void *stream) {
    if (ps.scratch) scratch_free(ps.scratch, (cudaStream_t)stream);
    ps.scratch = nullptr;
}

int launch_bc1_encode_range(const uint8_t *rgba, int w, int h, const qt_bc1_params &p, uint8_t *out, bool bc3,
                            long b_begin, long b_end, void *stream) {
    const int bw = (w + 3) / 4;
    const long n = b_end - b_begin;
    if (n <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    {
        const int aligned = texel_aligned(rgba, w);
        const int g = grid_for(n, tpb::kThreads);
        if ((n < kSplitMinBlocks || n > 0xFFFFFFFFL) && p.search_rounds == 0) {
            launch_fast(g, s, rgba, w, h, bw, b_begin, b_end, p, out, bc3, aligned, nullptr, nullptr);
            return (int)cudaGetLastError();
        }
        if ((n < kSplitMinBlocks || n > 0xFFFFFFFFL) && coop_setting(p, n)) {
            return (int)coop_encode(rgba, w, h, b_begin, n, p, out, bc3, aligned, nullptr, nullptr, s);
        }
        if (n < kSplitMinBlocks || n > 0xFFFFFFFFL) {
            switch (p.interpolator) {
                case IT_IDEAL: k_bc1_thread<IT_IDEAL, false><<<g, tpb::kThreads, 0, s>>>(rgba, w, h, bw, b_begin, b_end, p, out, bc3, aligned, nullptr, nullptr); break;
                case IT_ROUND: k_bc1_thread<IT_ROUND, false><<<g, tpb::kThreads, 0, s>>>(rgba, w, h, bw, b_begin, b_end, p, out, bc3, aligned, nullptr, nullptr); break;
                case IT_NVIDIA: k_bc1_thread<IT_NVIDIA, false><<<g, tpb::kThreads, 0, s>>>(rgba, w, h, bw, b_begin, b_end, p, out, bc3, aligned, nullptr, nullptr); break;
                default: k_bc1_thread<IT_AMD, false><<<g, tpb::kThreads, 0, s>>>(rgba, w, h, bw, b_begin, b_end, p, out, bc3, aligned, nullptr, nullptr); break;
            }
            return (int)cudaGetLastError();
        }
        // solid blocks first, then the encoder over the rest (list + count, stream-ordered scratch);
        // with EndpointSearch, the encoder queues the searches and k_bc1_search runs them
        // deferred only when the queue holds at least two searches per resident lane of the
        // search kernel: below that no lane gets a second entry to refill from, and the extra
        // pass costs more than it saves (measured at L18: -5% at 1024^2, +10% at 2048^2)
        const bool defer = p.search_rounds > 0 && n >= defer_min_blocks();
        // and the second four-colour cluster-fit pass, when there is one, runs in its own pass
        // for the blocks where it can change the result
        const bool cf2 = defer && cf2_pass(p);
        const size_t words = defer ? defer_words(n, cf2) : 64 + (size_t)n;
        uint32_t *scratch = nullptr;
        cudaError_t e = scratch_alloc((void **)&scratch, words * sizeof(uint32_t), s);
        if (e != cudaSuccess) return (int)e;
        uint32_t *count = scratch, *list = scratch + 64;
        e = cudaMemsetAsync(scratch, 0, 64 * sizeof(uint32_t), s);  // list count, queue counts and heads
        if (e == cudaSuccess && defer) {
            const DeferQueues d = defer_layout(scratch, n, cf2);
            by_interp(p.interpolator, [&](auto I) {
                defer_front<decltype(I)::value>(rgba, w, h, p, out, bc3, aligned, d, coop_setting(p, n), list, count, b_begin, b_end, s);
                defer_back<decltype(I)::value>(rgba, w, h, p, out, bc3, aligned, d, cf2, coop_setting(p, n), s);
            });
            e = cudaGetLastError();
        } else if (e == cudaSuccess && p.search_rounds == 0) {
            switch (p.interpolator) {
                case IT_IDEAL: launch_split<IT_IDEAL>(s, rgba, w, h, b_begin, b_end, out, bc3, aligned, list, count); break;
                case IT_ROUND: launch_split<IT_ROUND>(s, rgba, w, h, b_begin, b_end, out, bc3, aligned, list, count); break;
                case IT_NVIDIA: launch_split<IT_NVIDIA>(s, rgba, w, h, b_begin, b_end, out, bc3, aligned, list, count); break;
                default: launch_split<IT_AMD>(s, rgba, w, h, b_begin, b_end, out, bc3, aligned, list, count); break;
            }
            launch_fast(g, s, rgba, w, h, bw, 0, 0, p, out, bc3, aligned, list, count);
            e = cudaGetLastError();
        } else if (e == cudaSuccess && coop_setting(p, n)) {
            by_interp(p.interpolator, [&](auto I) {
                constexpr int IT = decltype(I)::value;
                launch_split<IT>(s, rgba, w, h, b_begin, b_end, out, bc3, aligned, list, count);
            });
            e = coop_encode(rgba, w, h, 0, n, p, out, bc3, aligned, list, count, s);
        } else if (e == cudaSuccess) {
            switch (p.interpolator) {
                case IT_IDEAL:
                    launch_split<IT_IDEAL>(s, rgba, w, h, b_begin, b_end, out, bc3, aligned, list, count);
                    k_bc1_thread<IT_IDEAL, true><<<g, tpb::kThreads, 0, s>>>(rgba, w, h, bw, 0, 0, p, out, bc3, aligned, list, count);
                    break;
                case IT_ROUND:
                    launch_split<IT_ROUND>(s, rgba, w, h, b_begin, b_end, out, bc3, aligned, list, count);
                    k_bc1_thread<IT_ROUND, true><<<g, tpb::kThreads, 0, s>>>(rgba, w, h, bw, 0, 0, p, out, bc3, aligned, list, count);
                    break;
                case IT_NVIDIA:
                    launch_split<IT_NVIDIA>(s, rgba, w, h, b_begin, b_end, out, bc3, aligned, list, count);
                    k_bc1_thread<IT_NVIDIA, true><<<g, tpb::kThreads, 0, s>>>(rgba, w, h, bw, 0, 0, p, out, bc3, aligned, list, count);
                    break;
                default:
                    launch_split<IT_AMD>(s, rgba, w, h, b_begin, b_end, out, bc3, aligned, list, count);
                    k_bc1_thread<IT_AMD, true><<<g, tpb::kThreads, 0, s>>>(rgba, w, h, bw, 0, 0, p, out, bc3, aligned, list, count);
                    break;
            }
            e = cudaGetLastError();
        }
        scratch_free(scratch, s);
        return (int)e;
    }
}

int bc1_encode_kernels(long n, const qt_bc1_params &p) {
    if (n <= 0) return 0;
    if (n < kSplitMinBlocks || n > 0xFFFFFFFFL) return 1;
    if (p.search_rounds == 0 || n < defer_min_blocks()) return 2;
    return cf2_pass(p) ? 5 : 4;  // split, encoder, (second cluster-fit pass,) search, finish
}

int launch_bc1_encode(const uint8_t *rgba, int w, int h, const qt_bc1_params &p, uint8_t *out, bool bc3, void *stream) {
    return launch_bc1_encode_range(rgba, w, h, p, out, bc3, 0, (long)((w + 3) / 4) * ((h + 3) / 4), stream);
}

int batch_sms() { return num_sms(); }

static int batch_ctas_per_sm_at(int threads) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_batch, threads, 0) != cudaSuccess || n <= 0) n = 1;
    return n;
}

// kinds 2..25 of a batch's kernels (qt_internal.h): interpolator, Faster or Check2, colour mode
template <int IT, int K4> static const void *batch_fast_cm(int cm) {
    return cm == 0 ? (const void *)k_batch_fast<IT, K4, CM_FOUR> : cm == 1 ? (const void *)k_batch_fast<IT, K4, CM_THREE> : (const void *)k_batch_fast<IT, K4, CM_TB>;
}
template <int IT> static const void *batch_fast_it(int k) { return k < 3 ? batch_fast_cm<IT, K_F4_FASTER>(k) : batch_fast_cm<IT, K_F4_CHECK2>(k - 3); }

int batch_kind(int op, int fmt, const qt_bc1_params &p) {
    if (op != QT_OP_ENCODE || (fmt != 1 && fmt != 3)) return 0;
    if (coop_batch_setting(p)) return 1;
    if (p.search_rounds != 0 || (p.error_mode != EM_FASTER && p.error_mode != EM_CHECK2)) return 0;
    const int cm = (fmt == 3 || p.color_mode == CM_FOUR) ? 0 : p.color_mode == CM_THREE ? 1 : 2;  // BC3Encoder.h:39-40
    return 2 + p.interpolator * 6 + (p.error_mode == EM_CHECK2 ? 3 : 0) + cm;
}

// A grid below k_batch's occupancy limit (ctas_per_sm * threads) leaves the rest of the SMs to other work: then every kernel of
// the batch has that many warps per SM and no more (batch_limited: the kernels also run one after the other). Without one the kernels
// other than k_batch launch what they keep resident, with the CTA size they were tuned at.
bool batch_limited(int ctas_per_sm, int threads) {
    return ctas_per_sm > 0 && ctas_per_sm * threads < batch_ctas_per_sm_at(tpb::kThreads) * tpb::kThreads;
}

int batch_launch(int kind, int ctas_per_sm, int threads, BatchLaunch *l) {
    *l = BatchLaunch{};
    if (threads != 32 && threads != 64 && threads != tpb::kThreads) return (int)cudaErrorInvalidValue;
    if (kind == 0) {
        l->func = (const void *)k_batch;
        l->threads = threads;
        l->grid = num_sms() * (ctas_per_sm > 0 ? ctas_per_sm : batch_ctas_per_sm_at(threads));
        return 0;
    }
    int resident = 5;  // CTAs per SM: 5 to 6 by the instance's registers
    if (kind == 1) {
        if (const int rc = batch_coop_launch(l, &resident)) return rc;
    } else {
        const int k = (kind - 2) % 6, it = (kind - 2) / 6;
        l->func = it == IT_IDEAL ? batch_fast_it<IT_IDEAL>(k) : it == IT_ROUND ? batch_fast_it<IT_ROUND>(k) : it == IT_NVIDIA ? batch_fast_it<IT_NVIDIA>(k) : batch_fast_it<IT_AMD>(k);
    }
    l->threads = tpb::kThreads;
    if (batch_limited(ctas_per_sm, threads)) {  // the same warps in the largest CTAs that divide them
        const int lanes = ctas_per_sm * threads;
        l->threads = lanes % tpb::kThreads == 0 ? tpb::kThreads : lanes % 64 == 0 ? 64 : 32;
        resident = std::min(resident, lanes / l->threads);
    }
    l->grid = num_sms() * resident;
    return 0;
}

int launch_batch(const BatchItemDev *items, const TileDev *tiles, uint32_t *ctl, int grid, int threads, void *stream) {
    // the kernel's shared-memory columns hold tpb::kThreads threads; smaller CTAs use a prefix
    if (threads != 32 && threads != 64 && threads != tpb::kThreads) return (int)cudaErrorInvalidValue;
    if (grid <= 0) grid = num_sms() * batch_ctas_per_sm_at(threads);
    k_batch<<<grid, threads, 0, (cudaStream_t)stream>>>(items, tiles, ctl);
    return (int)cudaGetLastError();
}

int launch_batch(const BatchItemDev *items, const TileDev *tiles, uint32_t *ctl, int grid, void *stream) {
    return launch_batch(items, tiles, ctl, grid, tpb::kThreads, stream);
}

// Grid of one thread per block when it fits (uint32_t indices), else a
// grid-stride loop over 64-bit indices.
static bool small_index(long n, int *grid) {
    const long ctas = (n + 255) / 256;
    if (n <= 0x7FFFFFFFL && ctas <= 0x7FFFFFFFL / 256) {
        *grid = (int)(ctas > 0 ? ctas : 1);
        return true;
    }
    *grid = num_sms() * 64;
    return false;
}

int launch_bc4_encode_range(const uint8_t *rgba, int w, int h, int c0, int c1, bool bc5, uint8_t *out, long b_begin,
                            long b_end, void *stream) {
    const int bw = (w + 3) / 4;
    if (b_end <= b_begin) return 0;
    const int aligned = ((w & 3) == 0) && ((reinterpret_cast<uintptr_t>(rgba) & 15) == 0);
    cudaStream_t s = (cudaStream_t)stream;
    int grid = 0;
    if (small_index(b_end, &grid)) {
        grid = (int)((b_end - b_begin + 255) / 256);
        if (bc5 && aligned) {  // persistent: at most the CTAs the SMs hold at once (each thread then loops,
                    // its next block's copies in flight while it encodes)
            static int resident = 0;
            if (resident <= 0) {  // 32 KB of staging per CTA: the shared-memory carveout that fits 6
                int per_sm = 0;
                const void *k = (const void *)k_bc4_encode<true, uint32_t>;
                cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
                const cudaError_t oe = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 256, 0);
                cudaGetLastError();
                resident = num_sms() * (oe == cudaSuccess && per_sm > 0 ? per_sm : 1);
            }
            grid = std::min(grid, resident);
        }
        const uint32_t ubw = (uint32_t)bw, u0 = (uint32_t)b_begin, un = (uint32_t)b_end;
        // rows off the 16-byte grid have nothing to stage: one block per thread (8190 x 8191: 66 us, persistent 85)
        if (bc5 && !aligned) k_bc4_encode<true, uint32_t, false><<<grid, 256, 0, s>>>(rgba, w, h, ubw, u0, un, c0, c1, 0, out);
        else if (bc5) k_bc4_encode<true, uint32_t><<<grid, 256, 0, s>>>(rgba, w, h, ubw, u0, un, c0, c1, aligned, out);
        else k_bc4_encode<false, uint32_t><<<grid, 256, 0, s>>>(rgba, w, h, ubw, u0, un, c0, c1, aligned, out);
    } else {
        const uint64_t ubw = (uint64_t)bw, u0 = (uint64_t)b_begin, un = (uint64_t)b_end;
        if (bc5) k_bc4_encode<true, uint64_t><<<grid, 256, 0, s>>>(rgba, w, h, ubw, u0, un, c0, c1, aligned, out);
        else k_bc4_encode<false, uint64_t><<<grid, 256, 0, s>>>(rgba, w, h, ubw, u0, un, c0, c1, aligned, out);
    }
    return (int)cudaGetLastError();
}

int launch_bc4_encode(const uint8_t *rgba, int w, int h, int c0, int c1, bool bc5, uint8_t *out, void *stream) {
    return launch_bc4_encode_range(rgba, w, h, c0, c1, bc5, out, 0, (long)((w + 3) / 4) * ((h + 3) / 4), stream);
}

template <int FMT, int IT, typename Idx>
static void launch_decode_t(int grid, cudaStream_t s, const uint8_t *blocks, int w, int h, int bw, int bh, long b0,
                            long n, int write_alpha, int c0, int c1, int aligned, uint8_t *rgba) {
    k_decode<FMT, IT, Idx><<<grid, 256, 0, s>>>(blocks, w, h, (Idx)bw, bh, (Idx)b0, (Idx)n, write_alpha, c0, c1, aligned, rgba);
}

template <typename Idx>
static void launch_decode_idx(int fmt, int interp, int grid, cudaStream_t s, const uint8_t *blocks, int w, int h,
                              int bw, int bh, long b0, long n, int write_alpha, int c0, int c1, int aligned, uint8_t *rgba) {
#define QT_DEC(F, I) launch_decode_t<F, I, Idx>(grid, s, blocks, w, h, bw, bh, b0, n, write_alpha, c0, c1, aligned, rgba)
    if (fmt == 4) { QT_DEC(4, IT_IDEAL); return; }
    if (fmt == 5) { QT_DEC(5, IT_IDEAL); return; }
    if (fmt == 1) {
        switch (interp) {
            case IT_IDEAL: QT_DEC(1, IT_IDEAL); break;
            case IT_ROUND: QT_DEC(1, IT_ROUND); break;
            case IT_NVIDIA: QT_DEC(1, IT_NVIDIA); break;
            default: QT_DEC(1, IT_AMD); break;
        }
        return;
    }
    switch (interp) {
        case IT_IDEAL: QT_DEC(3, IT_IDEAL); break;
        case IT_ROUND: QT_DEC(3, IT_ROUND); break;
        case IT_NVIDIA: QT_DEC(3, IT_NVIDIA); break;
        default: QT_DEC(3, IT_AMD); break;
    }
#undef QT_DEC
}

int launch_decode_range(int fmt, const uint8_t *blocks, int w, int h, int interp, int write_alpha, int c0, int c1,
                        uint8_t *rgba, long b_begin, long b_end, void *stream) {
    const int bw = (w + 3) / 4, bh = (h + 3) / 4;
    if (b_end <= b_begin) return 0;
    const int aligned = ((w & 3) == 0) && ((reinterpret_cast<uintptr_t>(rgba) & 15) == 0);
    int grid = 0;
    if (small_index(b_end, &grid)) {
        grid = (int)((b_end - b_begin + 255) / 256);
        launch_decode_idx<uint32_t>(fmt, interp, grid, (cudaStream_t)stream, blocks, w, h, bw, bh, b_begin, b_end, write_alpha, c0, c1, aligned, rgba);
    } else {
        launch_decode_idx<uint64_t>(fmt, interp, grid, (cudaStream_t)stream, blocks, w, h, bw, bh, b_begin, b_end, write_alpha, c0, c1, aligned, rgba);
    }
    return (int)cudaGetLastError();
}

int launch_decode(int fmt, const uint8_t *blocks, int w, int h, int interp, int write_alpha, int c0, int c1,
                  uint8_t *rgba, void *stream) {
    return launch_decode_range(fmt, blocks, w, h, interp, write_alpha, c0, c1, rgba, 0,
                               (long)((w + 3) / 4) * ((h + 3) / 4), stream);
}

}  // namespace qtk
