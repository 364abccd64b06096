// qt_device.cuh — device code shared by the kernel translation units (qt_kernels.cu, qt_coop.cu): the constant
// tables, the reference's scalar helpers (util.h, Color.cpp, Interpolator.cpp), the block writers and the
// thread-per-block BC4/BC5 encoders. Each unit has its own copy of the tables (upload_tables fills all of them).
//
// Floating point. Every operation whose rounding matters is written with an
// explicit round-to-nearest intrinsic (__fadd_rn, __fmul_rn, __fdiv_rn), in
// the reference's operation order; the compiler never contracts these into
// FMAs. Plain float arithmetic (and fmaf) is used only where every operand and
// result is an integer below 2^24, i.e. exact.
#pragma once

#include <cuda_runtime.h>

#include <cfloat>
#include <climits>
#include <cstddef>
#include <cstdint>

#include "qt_internal.h"

namespace qtk {

// ---------------------------------------------------------------------------
// constant tables
// ---------------------------------------------------------------------------
struct DevTables {
    uint16_t best4[969 * 128];
    uint16_t best3[153 * 32];
    uint16_t hash4[4096];
    uint16_t hash3[256];
    float4 factors4[969];
    float4 factors3[153];
    uint32_t orders4[969];
    uint32_t orders3[153];
    uint32_t match5[4][256];
    uint32_t match6[4][256];
    uint4 ord4[969];
    uint4 ord3[153];
    uint16_t coop4[969 * 128];
    uint16_t coop3[153 * 32];
};
static_assert(sizeof(DevTables) == sizeof(HostTables) && offsetof(DevTables, ord4) == offsetof(HostTables, ord4) &&
                  offsetof(DevTables, coop3) == offsetof(HostTables, coop3),
              "device and host table images must match");

static __device__ DevTables g_tab;

// Color::PreciseRound565 rounding points (Color.h:87-95); the values must be
// these exact floats for the rounding to match.
static __constant__ float c_mid5[32] = {.015686f, .047059f, .078431f, .111765f, .145098f, .176471f, .207843f, .241176f,
                                 .274510f, .305882f, .337255f, .370588f, .403922f, .435294f, .466667f, .5f,
                                 .533333f, .564706f, .596078f, .629412f, .662745f, .694118f, .725490f, .758824f,
                                 .792157f, .823529f, .854902f, .888235f, .921569f, .952941f, .984314f, 1e+37f};
static __constant__ float c_mid6[64] = {
    .007843f, .023529f, .039216f, .054902f, .070588f, .086275f, .101961f, .117647f, .133333f, .149020f, .164706f,
    .180392f, .196078f, .211765f, .227451f, .245098f, .262745f, .278431f, .294118f, .309804f, .325490f, .341176f,
    .356863f, .372549f, .388235f, .403922f, .419608f, .435294f, .450980f, .466667f, .482353f, .500000f, .517647f,
    .533333f, .549020f, .564706f, .580392f, .596078f, .611765f, .627451f, .643137f, .658824f, .674510f, .690196f,
    .705882f, .721569f, .737255f, .754902f, .772549f, .788235f, .803922f, .819608f, .835294f, .850980f, .866667f,
    .882353f, .898039f, .913725f, .929412f, .945098f, .960784f, .976471f, .992157f, 1e+37f};

// EndpointSearch voxel steps (BC1Encoder.cpp:933-950): dr, dg, db in 2-bit
// two's complement fields (bits 0-1, 2-3, 4-5) and the opposite step's index
// in bits 8-11.
static __constant__ uint16_t c_voxels[16] = {
    0x301, 0x404, 0x510, 0x003, 0x10C, 0x230, 0x905, 0xA11, 0xB14, 0x60F, 0x733, 0x83C, 0xD07, 0xC0D, 0xF1C, 0xE34};

constexpr int CM_INCOMPLETE = 0x00, CM_THREE = 0x03, CM_FOUR = 0x04, CM_TB = 0x13;
constexpr int EM_NONE = 0, EM_FASTER = 1, EM_CHECK2 = 2, EM_FULL = 3;
constexpr int EP_LS = 0, EP_BB = 1, EP_BBINT = 2, EP_PCA = 3;
constexpr int IT_IDEAL = 0, IT_ROUND = 1, IT_NVIDIA = 2, IT_AMD = 3;


// ---------------------------------------------------------------------------
// scalar helpers (util.h:110-154, Color.cpp)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int s8to5(int v) { int v2 = v * 31 + 128; return (v2 + (v2 >> 8)) >> 8; }
__device__ __forceinline__ int s8to6(int v) { int v2 = v * 63 + 128; return (v2 + (v2 >> 8)) >> 8; }
__device__ __forceinline__ int s5to8(int v) { return (v << 3) | (v >> 2); }
__device__ __forceinline__ int s6to8(int v) { return (v << 2) | (v >> 4); }
__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }
__device__ __forceinline__ int clamp255(int i) { return ((unsigned)i & 0xFFFFFF00u) ? ((~(i >> 31)) & 0xFF) : i; }
// float -> int with x86 cvttss2si semantics (INT_MIN when out of range or NaN)
__device__ __forceinline__ int f2i_x86(float v) {
    return (v > -2147483904.0f && v < 2147483648.0f) ? __float2int_rz(v) : INT_MIN;
}
// 5:6:5 endpoint packed as Pack565Unscaled (Color.cpp:41-46)
__device__ __forceinline__ int epr(int e) { return e >> 11; }
__device__ __forceinline__ int epg(int e) { return (e >> 5) & 63; }
__device__ __forceinline__ int epb(int e) { return e & 31; }
__device__ __forceinline__ int eppack(int r, int g, int b) { return (r << 11) | (g << 5) | b; }
__device__ __forceinline__ unsigned sq3(int a, int b, int c) { return (unsigned)(a * a + b * b + c * c); }

// Color::PreciseRound565 (Color.cpp:66-86)
__device__ __forceinline__ int precise_round565(float v0, float v1, float v2, const float *mid5, const float *mid6) {
    int r = clampi(f2i_x86(__fmul_rn(v0, 31.0f)), 0, 31);
    int g = clampi(f2i_x86(__fmul_rn(v1, 63.0f)), 0, 63);
    int b = clampi(f2i_x86(__fmul_rn(v2, 31.0f)), 0, 31);
    r += v0 > mid5[r];
    g += v1 > mid6[g];
    b += v2 > mid5[b];
    return eppack(r, g, b);
}

// PreciseRound565 of a cluster-fit trial's endpoint. The trial endpoints are table factors
// times sums of at most 3 * 16 * 255: over the factor tables |v| * 63 < 9500, finite and far
// inside int range, so truncation needs no x86 out-of-range case; the unsigned conversion
// saturates negatives to 0, which is the lower clamp.
__device__ __forceinline__ int precise_round565_cf(float v0, float v1, float v2, const float *mid5, const float *mid6) {
    int r = (int)min(__float2uint_rz(__fmul_rn(v0, 31.0f)), 31u);
    int g = (int)min(__float2uint_rz(__fmul_rn(v1, 63.0f)), 63u);
    int b = (int)min(__float2uint_rz(__fmul_rn(v2, 31.0f)), 31u);
    r += v0 > mid5[r];
    g += v1 > mid6[g];
    b += v2 > mid5[b];
    return eppack(r, g, b);
}

// ---------------------------------------------------------------------------
// interpolators (Interpolator.cpp:47-138)
// ---------------------------------------------------------------------------
// a, b are channel values (non-negative), so unsigned division gives the same quotients
template <int IT> __device__ __forceinline__ int i8(int a, int b) {
    const unsigned ua = (unsigned)a, ub = (unsigned)b;
    if (IT == IT_ROUND) return (int)((ua * 2 + ub + 1) / 3);
    if (IT == IT_AMD) return (int)((ua * 43 + ub * 21 + 32) >> 6);
    return (int)((ua * 2 + ub) / 3);
}
template <int IT> __device__ __forceinline__ int h8(int a, int b) {
    return (int)(IT == IT_AMD ? (((unsigned)a + (unsigned)b + 1) >> 1) : (((unsigned)a + (unsigned)b) / 2));
}
__device__ __forceinline__ int nv5(int a, int b) { return (int)((((unsigned)a * 2 + (unsigned)b) * 22) / 8); }
__device__ __forceinline__ int nv6(int a, int b) { int gd = b - a; return (256 * a + (gd / 4) + 128 + gd * 80) >> 8; }
__device__ __forceinline__ int nvh5(int a, int b) { return (int)((((unsigned)a + (unsigned)b) * 33) / 8); }
__device__ __forceinline__ int nvh6(int a, int b) { int gd = b - a; return (256 * a + gd / 4 + 128 + gd * 128) >> 8; }

// Palette in FindSelectors' internal selector order (BC1Encoder.cpp:684-693):
// four colours {c0, c2, c3, c1}, three colours {c0, c2, c1, c3=black}.
struct Pal {
    int r0, g0, b0, r1, g1, b1, r2, g2, b2, r3, g3, b3;
};

template <int IT> __device__ __forceinline__ Pal make_pal(int lo, int hi, bool three) {
    const int lr = epr(lo), lg = epg(lo), lb = epb(lo), hr = epr(hi), hg = epg(hi), hb = epb(hi);
    const int ar = s5to8(lr), ag = s6to8(lg), ab = s5to8(lb);  // colors[0]
    const int br = s5to8(hr), bg = s6to8(hg), bb = s5to8(hb);  // colors[1]
    int cr, cg, cb, dr, dg, db;                                // colors[2], colors[3]
    if (IT == IT_NVIDIA) {
        if (!three) {
            cr = nv5(lr, hr); cg = nv6(lg, hg); cb = nv5(lb, hb);
            dr = nv5(hr, lr); dg = nv6(hg, lg); db = nv5(hb, lb);
        } else {
            cr = nvh5(lr, hr); cg = nvh6(lg, hg); cb = nvh5(lb, hb);
            dr = dg = db = 0;
        }
    } else if (three) {
        cr = h8<IT>(ar, br); cg = h8<IT>(ag, bg); cb = h8<IT>(ab, bb);
        dr = dg = db = 0;
    } else {
        cr = i8<IT>(ar, br); cg = i8<IT>(ag, bg); cb = i8<IT>(ab, bb);
        dr = i8<IT>(br, ar); dg = i8<IT>(bg, ag); db = i8<IT>(bb, ab);
    }
    Pal p;
    p.r0 = ar; p.g0 = ag; p.b0 = ab;
    p.r1 = cr; p.g1 = cg; p.b1 = cb;
    if (!three) {
        p.r2 = dr; p.g2 = dg; p.b2 = db;
        p.r3 = br; p.g3 = bg; p.b3 = bb;
    } else {
        p.r2 = br; p.g2 = bg; p.b2 = bb;
        p.r3 = dr; p.g3 = dg; p.b3 = db;
    }
    return p;
}

// ---------------------------------------------------------------------------
// per-CTA shared copies of small constant tables (read by every BC1 kernel)
// ---------------------------------------------------------------------------
__shared__ float s_mid5[32], s_mid6[64];
__shared__ uint16_t s_vox[16];

// Selector-search kinds: the (colour mode, error mode) pairs FindSelectors is
// ever called with. Three-colour searches are always ErrorMode::Full
// (BC1Encoder.cpp:313-333, 978-984).
constexpr int K_F4_NONE = 0, K_F4_FASTER = 1, K_F4_CHECK2 = 2, K_F4_FULL = 3, K_T3 = 4, K_TB = 5;
__host__ __device__ constexpr bool kind_three(int k) { return k >= K_T3; }
__host__ __device__ constexpr int kind_mode(int k) { return k == K_T3 ? CM_THREE : (k == K_TB ? CM_TB : CM_FOUR); }
__device__ __forceinline__ int kind_for(int M, int em) { return M == CM_THREE ? K_T3 : (M == CM_TB ? K_TB : em); }

// Vector4::Dot (Vector4.h:53-57) in the reference's rounding: sum from 0, left to right
__device__ __forceinline__ float fdot4_rn(float a0, float a1, float a2, float a3, float b0, float b1, float b2, float b3) {
    float s = __fadd_rn(0.0f, __fmul_rn(a0, b0));
    s = __fadd_rn(s, __fmul_rn(a1, b1));
    s = __fadd_rn(s, __fmul_rn(a2, b2));
    return __fadd_rn(s, __fmul_rn(a3, b3));
}

__device__ __forceinline__ bool is_single_hash(bool four, int h) {
    return four ? (h == 15 || h == 700 || h == 753 || h == 515) : (h == 12 || h == 15 || h == 89);
}

// ---------------------------------------------------------------------------
// block writers (BC1Encoder.cpp:345-441, BC1Block.h:66-80)
// ---------------------------------------------------------------------------
template <int IT> __device__ __forceinline__ uint2 write_block_solid(uint32_t c) {
    const int cr = c & 0xFF, cg = (c >> 8) & 0xFF, cb = (c >> 16) & 0xFF;
    uint32_t mask = 0xAA;
    int mn, mx;
    if ((cr | cg | cb) == 0) {
        mn = 0; mx = 1; mask = 0x55;
    } else {
        // FindEndpointsSingleColor(color); the 3-colour tables equal the 4-colour
        // ones (SingleColorTable.h: N unused), so the 3-colour trial never wins.
        const uint32_t mr = g_tab.match5[IT][cr], mg = g_tab.match6[IT][cg], mb = g_tab.match5[IT][cb];
        mn = eppack((mr >> 8) & 0xFF, (mg >> 8) & 0xFF, (mb >> 8) & 0xFF);
        mx = eppack(mr & 0xFF, mg & 0xFF, mb & 0xFF);
        if (mn == mx) {
            if (mn > 0) { mn--; mask = 0; }
            else { mx = 1; mn = 0; mask = 0x55; }
        } else if (mx < mn) {
            const int t = mn; mn = mx; mx = t;
            mask = 0xFF;
        }
    }
    return make_uint2((uint32_t)mx | ((uint32_t)mn << 16), mask * 0x01010101u);
}

// WriteBlock of an EncodeResults (BC1Encoder.h:147-153): endpoints packed 5:6:5, sel the 16
// 2-bit internal selectors (texel i at bits 2i), mode its colour mode
__device__ __forceinline__ uint2 write_block(int lo, int hi, uint32_t sel_in, int mode) {
    int ep1 = lo, ep0 = hi;
    uint32_t lut;  // 4 x 2-bit entries
    if (mode & CM_FOUR) {
        lut = 1 | (3 << 2) | (2 << 4) | (0 << 6);
        if (ep1 > ep0) {
            const int t = ep1; ep1 = ep0; ep0 = t;
            lut = 0 | (2 << 2) | (3 << 4) | (1 << 6);
        } else if (ep1 == ep0) {
            if (ep1 > 0) { ep1--; lut = 0; }
            else { ep0 = 1; ep1 = 0; lut = 0x55; }
        }
    } else {
        lut = 1 | (2 << 2) | (0 << 4) | (3 << 6);
        if (ep1 < ep0) {
            const int t = ep1; ep1 = ep0; ep0 = t;
            lut = 0 | (2 << 2) | (1 << 4) | (3 << 6);
        }
    }
    uint32_t sel = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) sel |= ((lut >> (2 * ((sel_in >> (2 * i)) & 3))) & 3) << (2 * i);
    return make_uint2((uint32_t)ep0 | ((uint32_t)ep1 << 16), sel);
}

// ---------------------------------------------------------------------------
// thread-per-block kernels: BC4/BC5 encode, all decoders
//
// These move 72-80 bytes of HBM traffic per block, so at full bandwidth an SM
// has ~400 thread-instructions per block to spend. The per-block work is kept
// well under that: byte selection with PRMT (__byte_perm), one multiply-high
// per texel for the BC4 level, 32-bit block indices where they fit, and one
// kernel instantiation per format so nothing branches on it per block.
// ---------------------------------------------------------------------------
// s % n for 0 <= s < n + 3: a block's texel wraps at most once unless the texture is smaller than a block
__device__ __forceinline__ int wrapped(int s, int n) { return n >= 4 ? (s < n ? s : s - n) : s % n; }

// The block's texels: 16-byte rows with `fast` (an interior block, rows on the 16-byte grid), else texel by texel, at fixed
// offsets in an interior block. Rows off the grid took load_block_thread's wrapped form throughout, two divisions a texel: BC4
// 8190 x 8191 68 -> 55 us, BC5 93 -> 66; 16-byte words shifted across lanes by shuffles: 76 and 89, with the
// channel's bytes taken out first 66 and 87 (379 instructions a block against 230).
__device__ __forceinline__ void load_block_any(const uint8_t *__restrict__ rgba, int w, int h, int bx, int by,
                                                  bool fast, uint32_t px[16]) {
    if (fast) {
#pragma unroll
        for (int y = 0; y < 4; y++) {
            const uint4 q = __ldg(reinterpret_cast<const uint4 *>(rgba + ((size_t)(by * 4 + y) * w + bx * 4) * 4));
            px[4 * y] = q.x; px[4 * y + 1] = q.y; px[4 * y + 2] = q.z; px[4 * y + 3] = q.w;
        }
    } else if (bx * 4 + 4 <= w && by * 4 + 4 <= h) {
        const uint32_t *at = reinterpret_cast<const uint32_t *>(rgba) + (size_t)(by * 4) * w + bx * 4;
#pragma unroll
        for (int y = 0; y < 4; y++, at += w)
#pragma unroll
            for (int x = 0; x < 4; x++) px[4 * y + x] = __ldg(at + x);
    } else {
#pragma unroll
        for (int y = 0; y < 4; y++)
#pragma unroll
            for (int x = 0; x < 4; x++)
                px[4 * y + x] = __ldg(reinterpret_cast<const uint32_t *>(rgba) + (size_t)wrapped(by * 4 + y, h) * w + wrapped(bx * 4 + x, w));
    }
}

// The same for the BC1 encoders, which are not bound by their loads: with load_block_any they ran 3-8% slower (level 0 2048 x 2048
// 57 -> 59 us, 2047 x 2049 58 -> 64).
__device__ __forceinline__ void load_block_thread(const uint8_t *__restrict__ rgba, int w, int h, int bx, int by,
                                                  bool fast, uint32_t px[16]) {
    if (fast) {
#pragma unroll
        for (int y = 0; y < 4; y++) {
            const uint4 q = __ldg(reinterpret_cast<const uint4 *>(rgba + ((size_t)(by * 4 + y) * w + bx * 4) * 4));
            px[4 * y] = q.x; px[4 * y + 1] = q.y; px[4 * y + 2] = q.z; px[4 * y + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int y = 0; y < 4; y++)
#pragma unroll
            for (int x = 0; x < 4; x++) {
                const int sx = (bx * 4 + x) % w, sy = (by * 4 + y) % h;
                px[4 * y + x] = __ldg(reinterpret_cast<const uint32_t *>(rgba + ((size_t)sy * w + sx) * 4));
            }
    }
}

// The Levels table of BC4Encoder.cpp:45 ({1,7,6,5,4,3,2,0}: threshold count -> selector) as bytes for PRMT.
constexpr uint32_t kBC4MapLo = 1u | (7u << 8) | (6u << 16) | (5u << 24);
constexpr uint32_t kBC4MapHi = 4u | (3u << 8) | (2u << 16) | (0u << 24);

// Exact division of n < 4096 by d = 2*delta (delta 1..255) as __umulhi(n, M[delta]):
// M = (floor(2^(12+l) / d) + 1) << (20 - l), l = ceil(log2 d) (Granlund & Montgomery,
// "Division by invariant integers using multiplication", 1994, Thm 4.2, N = 12 bits).
struct BC4Magic {
    uint32_t m[256];
};
constexpr BC4Magic make_bc4_magic() {
    BC4Magic t{};
    for (int delta = 1; delta < 256; delta++) {
        const uint32_t d = 2u * (uint32_t)delta;
        int l = 0;
        while ((1u << l) < d) l++;
        const uint64_t m = (1ull << (12 + l)) / d + 1;
        t.m[delta] = (uint32_t)(m << (20 - l));
    }
    return t;
}
static __device__ const BC4Magic g_bc4_magic = make_bc4_magic();

// Selector packing shared by the BC4 and BC5 encoders. A level q (0..9, see below) indexes
// the Levels table with one PTX prmt.b32: a selector nibble 0..7 copies byte q of
// {kBC4MapHi:kBC4MapLo}, and 8 or 9 copies the sign of byte 0 or 1 (map 1 and 7: sign 0), i.e. 0,
// which is map[7], the selector of every level >= 7. So no clamp and no mask are needed: the
// other result bytes hold map[0] = 1 (selector nibble 0), a known constant. Selector words are then
// accumulated with IMAD, acc += word << 3j, and that constant's contribution is subtracted once at
// the end (the arithmetic is exact modulo 2^32 and the 3-bit fields never overlap).
// (CUDA's __byte_perm takes only the low 3 bits of each nibble, so it would map 8 and 9 to
// map[0] and map[1]; the lookup needs the PTX instruction's sign-replicate mode.)
__device__ __forceinline__ uint32_t prmt_levels(uint32_t selector) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(kBC4MapLo), "r"(kBC4MapHi), "r"(selector));
    return d;
}
constexpr uint32_t kPermOnes = 0x01010100u;  // prmt result bytes 1..3 for a selector < 16
template <int N>
__host__ __device__ constexpr uint32_t perm_garbage(uint32_t word) {  // sum of word << 3j, j < N
    uint32_t c = 0;
    for (int j = 0; j < N; j++) c += word << (3 * j);
    return c;
}

// BC4Encoder::EncodeBlock (BC4Encoder.cpp:30-71) on channel ch. The reference
// counts the thresholds delta*(1+2c) - bias (c = 0..6) that 14*value reaches;
// for min <= value <= max that count is exactly
// min(7, floor((14*(value - min) + 4 + delta) / (2*delta))), and the division is
// a multiply-high by g_bc4_magic (exact for numerators below 4096; both facts
// checked for every (min, max, value)). The level itself, floor(...), is at most 9
// (delta >= 1), so the prmt table lookup above takes it unclamped.
__device__ __forceinline__ uint2 bc4_block_thread(const uint32_t px[16], int ch) {
    const uint32_t sel = 0x4440u | (uint32_t)ch;  // byte ch of the texel, zeros above
    uint32_t v[16];
    uint32_t mn = 255u, mx = 0u;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        v[i] = __byte_perm(px[i], 0u, sel);
        mn = min(mn, v[i]);
        mx = max(mx, v[i]);
    }
    if (mn == mx) return make_uint2(mn | (mn << 8), 0u);  // BC4Block(min): solid
    const uint32_t delta = mx - mn;
    const uint32_t M = __ldg(&g_bc4_magic.m[delta]);
    const uint32_t K = 4u + delta - 14u * mn;  // 14*value + K == 14*(value - min) + 4 + delta (mod 2^32)
    uint32_t a0 = 0u, a1 = 0u;                 // texels 0..9 (30 bits), 10..15 (18 bits)
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const uint32_t q = __umulhi(14u * v[i] + K, M);
        const uint32_t word = prmt_levels(q);  // selector in byte 0
        if (i < 10) a0 += word << (3 * i);
        else a1 += word << (3 * (i - 10));
    }
    a0 -= perm_garbage<10>(kPermOnes);
    a1 -= perm_garbage<6>(kPermOnes);
    const uint32_t lo = a0 | (a1 << 30), hi = a1 >> 2;  // selector bits 0..31 and 32..47
    return make_uint2(mx | (mn << 8) | (lo << 16), (lo >> 16) | (hi << 16));
}

__device__ __forceinline__ uint32_t min_u16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("min.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("max.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

// BC5Encoder::EncodeBlock (BC5Encoder.cpp:25-30): BC4 of channel c0, then of c1,
// with the two channels carried side by side in 16-bit halves. One packed
// min/max per texel covers both channels, and one IMAD forms both numerators
// 14*value + K: a negative low-half K borrows one from the high half, which its
// high constant pre-compensates, so each half holds its channel's exact value.
// Both levels then index the Levels table in one prmt (selector nibbles 0 and 2),
// which puts channel c0's selector in byte 0 and c1's in byte 2 of one word; five
// texels' words accumulate into one register (two 15-bit fields, 3 bits per
// texel), as in bc4_block_thread.
__device__ __forceinline__ uint4 bc5_block_thread(const uint32_t px[16], int c0, int c1) {
    const uint32_t sel = 0x4040u | (uint32_t)c0 | ((uint32_t)c1 << 8);  // byte c0 -> bits 0..7, byte c1 -> bits 16..23
    uint32_t v[16];
    uint32_t mn = 0x00FF00FFu, mx = 0u;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        v[i] = __byte_perm(px[i], 0u, sel);
        mn = min_u16x2(mn, v[i]);
        mx = max_u16x2(mx, v[i]);
    }
    const uint32_t mn0 = mn & 0xFFFFu, mn1 = mn >> 16, d0 = (mx & 0xFFFFu) - mn0, d1 = (mx >> 16) - mn1;
    const uint32_t M0 = __ldg(&g_bc4_magic.m[d0]), M1 = __ldg(&g_bc4_magic.m[d1]);  // m[0] = 0: solid, fixed below
    const int K0 = 4 + (int)d0 - 14 * (int)mn0, K1 = 4 + (int)d1 - 14 * (int)mn1;
    const uint32_t Kp = ((uint32_t)K0 & 0xFFFFu) + ((uint32_t)(K1 - (K0 < 0 ? 1 : 0)) << 16);
    uint32_t g[4] = {0u, 0u, 0u, 0u};  // texels 0-4, 5-9, 10-14, 15: c0 fields in bits 0..14, c1 in 16..30
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const uint32_t num = 14u * v[i] + Kp;
        const uint32_t q0 = __umulhi(num & 0xFFFFu, M0), q1 = __umulhi(num >> 16, M1);  // levels 0..9
        const uint32_t word = prmt_levels(q0 + (q1 << 8));  // selectors in bytes 0, 2
        g[i / 5] += word << (3 * (i % 5));
    }
    constexpr uint32_t kOnes2 = 0x01000100u;  // prmt result bytes 1 and 3 (selector nibbles 1, 3 = 0)
    g[0] -= perm_garbage<5>(kOnes2);
    g[1] -= perm_garbage<5>(kOnes2);
    g[2] -= perm_garbage<5>(kOnes2);
    g[3] -= perm_garbage<1>(kOnes2);
    // channel fields: 15 + 15 + 15 + 3 bits -> selector bits 0..31 (lo) and 32..47 (hi)
    const uint32_t f00 = g[0] & 0xFFFFu, f01 = g[1] & 0xFFFFu, f02 = g[2] & 0xFFFFu, f03 = g[3] & 0xFFFFu;
    const uint32_t f10 = g[0] >> 16, f11 = g[1] >> 16, f12 = g[2] >> 16, f13 = g[3] >> 16;
    const uint32_t lo0 = f00 | (f01 << 15) | (f02 << 30), hi0 = (f02 >> 2) | (f03 << 13);
    const uint32_t lo1 = f10 | (f11 << 15) | (f12 << 30), hi1 = (f12 >> 2) | (f13 << 13);
    const uint32_t mx0 = mn0 + d0, mx1 = mn1 + d1;
    uint4 r;
    r.x = d0 ? (mx0 | (mn0 << 8) | (lo0 << 16)) : (mn0 | (mn0 << 8));  // BC4Block(min) when solid
    r.y = d0 ? ((lo0 >> 16) | (hi0 << 16)) : 0u;
    r.z = d1 ? (mx1 | (mn1 << 8) | (lo1 << 16)) : (mn1 | (mn1 << 8));
    r.w = d1 ? ((lo1 >> 16) | (hi1 << 16)) : 0u;
    return r;
}

}  // namespace qtk
