// qt_bc1_coop.cuh — warp-cooperative cluster fit and EndpointSearch of the BC1/BC3 encoder, for the
// Full error mode (levels 13-19). Included by qt_coop.cu after qt_bc1_thread.cuh.
//
// The phases of EncodeBlock that are sequential per block (metrics, FindEndpoints, FindSelectors,
// RefineBlockLS, the cluster fit's sort) run one block per lane, as in qt_bc1_thread.cuh. The trials of
// RefineBlockCF (BC1Encoder.cpp:905-927) and of EndpointSearch (:930-996) are independent given
// their start, so there the warp turns to one of its blocks at a time and every lane takes one trial: 32
// orderings (or 32 candidate steps) at once. All lanes share the block's texels, so the errors of the 32
// trials are a matrix product, palettes (32 x 3 per colour) by texels (3 x 16), and run on the
// tensor cores; the reference's "first strictly better trial" is an argmin over (error, index).
//
// Errors by mma. With |p - c|^2 = |p|^2 + (|c|^2 - 2 p.c), a trial's total is sum |p|^2 plus the sum over texels of
// the least of its colours' |c|^2 - 2 p.c. One mma.m16n8k8 (halves, float accumulators) gives that for one colour of
// 16 trials x 8 texels: a trial's row holds r, g, b and |c|^2 in two halves, the texel's column -2r, -2g, -2b, 1 and 256.
// Every entry is an integer that a half holds exactly and every sum is below 2^24, so the result is exact in any order
// (tests/test_coop_palette.py checks the arithmetic).
//
// What bounds it: a step of 32 trials issues 235 instructions a warp (93 of them the errors) and takes 345 cycles a
// scheduler; with one block per lane 32 trials take 427 instructions and ~550 cycles. The 16 mma hold the scheduler
// ~8 cycles each (the legacy tensor path: 93 instructions without any other work take 209 cycles), so they come to no
// more errors a cycle than dp4a; what the step saves is the rest of the loop, and above all the chain: a block's 128
// trials are 4 steps instead of 128. The step also moves 64 shared-memory wavefronts, 32 of them the rows. An
// integer mma (u8) with |c|^2 in the accumulators took 287 instructions and 484 cycles; 5 CTAs per SM (96
// registers) the same cycles a block as 4.

namespace coop {

constexpr int kWarps = tpb::kThreads / 32;

struct Work {  // per CTA: what every cooperative kernel needs
    uint4 pal[kWarps][4][32];    // [colour][row]: 8 halves a trial, rows placed by stage_row()
};
struct FitWork {  // the cluster fit's on top
    uint2 pre[kWarps][32][17];   // prefix sums of a lane's block in rank order: r | g << 16, b
    uint2 rnd5[32], rnd6[64];    // PreciseRound565: midpoint, then bytes: 8-bit values of r and r + 1, 0x66
    uint4 ord4[969], ord3[153];  // per ordering: LS factors x, y (= z), w and the byte offsets of its three prefix sums
};
constexpr size_t kSearchSmem = sizeof(Work), kFitSmem = sizeof(Work) + sizeof(FitWork);

extern __shared__ uint4 c_dyn[];
__device__ __forceinline__ Work &work() { return *reinterpret_cast<Work *>(c_dyn); }
__device__ __forceinline__ FitWork &fit() { return *reinterpret_cast<FitWork *>(reinterpret_cast<char *>(c_dyn) + sizeof(Work)); }
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// fills the CTA's tables (every thread calls it; ends with a barrier)
__device__ __forceinline__ void load_fit_tables(bool three) {
    FitWork &F = fit();
    for (int i = threadIdx.x; i < 969; i += blockDim.x) F.ord4[i] = g_tab.ord4[i];
    if (three)
        for (int i = threadIdx.x; i < 153; i += blockDim.x) F.ord3[i] = g_tab.ord3[i];
    for (int i = threadIdx.x; i < 64; i += blockDim.x) {
        if (i < 32) F.rnd5[i] = make_uint2(__float_as_uint(c_mid5[i]), (uint32_t)(s5to8(i) | ((s5to8(i + 1) & 0xFF) << 8)) | 0x660000u);
        F.rnd6[i] = make_uint2(__float_as_uint(c_mid6[i]), (uint32_t)(s6to8(i) | ((s6to8(i + 1) & 0xFF) << 8)) | 0x660000u);
    }
    __syncthreads();
}

__device__ __forceinline__ void mma_f16(float d[4], uint32_t a0, uint32_t a1, uint32_t b) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(b), "f"(0.0f));
}

__device__ __forceinline__ uint32_t h2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }
__device__ __forceinline__ uint32_t fma_h2(uint32_t a, uint32_t b, uint32_t c) { return as_u32(__hfma2(as_h2(a), as_h2(b), as_h2(c))); }
__device__ __forceinline__ uint32_t add_h2(uint32_t a, uint32_t b) { return as_u32(__hadd2(as_h2(a), as_h2(b))); }

// The texels of one block as B fragments: texels lane / 4 and lane / 4 + 8 of the block in shared-memory column `col`.
// A quad's lane t holds the factors of word t of a trial's row: (-2 r, -2 g), (-2 b, 0) or (0, -2 b) for a row whose
// blue is in the high half, (1, 256), (sum of r g b, -257).
struct Texels {
    uint32_t lo[2], hi[2];
};
// What a lane multiplies and adds to turn a texel into its words: the halves (1536 + x, 1536 + y) of two of its
// channels, or (1024 + r + g + b, ..) in lane 3 of a quad.
struct TexelForm {
    uint32_t sel, mul_lo, add_lo, mul_hi, add_hi;
    __device__ __forceinline__ TexelForm() {
        const int t = threadIdx.x & 3;
        sel = t == 0 ? 0x4140u : 0x4242u;
        mul_lo = t == 0 ? 0xC000C000u : t == 1 ? 0x0000C000u : t == 2 ? 0u : 0x00003C00u;                   // -2, -2 | -2, 0 | 0, 0 | 1, 0
        add_lo = t == 0 ? 0x6A006A00u : t == 1 ? 0x00006A00u : t == 2 ? 0x5C003C00u : 0xDC04E400u;          // 3072, 3072 | 3072, 0 | 1, 256 | -1024, -257
        mul_hi = t == 1 ? 0xC0000000u : mul_lo;
        add_hi = t == 1 ? 0x6A000000u : add_lo;
    }
    __device__ __forceinline__ void words(uint32_t p, uint32_t &lo, uint32_t &hi) const {
        const uint32_t sum = __dp4a(p, 0x00010101u, 0x6400u), v = (threadIdx.x & 3) == 3 ? sum : __byte_perm(p, 0x66u, sel);
        lo = fma_h2(v, mul_lo, add_lo);
        hi = fma_h2(v, mul_hi, add_hi);
    }
};
__device__ __forceinline__ Texels load_texels(int col, const TexelForm &f) {
    const int g = (threadIdx.x & 31) >> 2;
    Texels x;
    f.words(tpb::t_px[g][col], x.lo[0], x.hi[0]);
    f.words(tpb::t_px[g + 8][col], x.lo[1], x.hi[1]);
    return x;
}

// Row of a lane's trial in the A matrix: lane 4g + t takes row g + 8t, the row whose total the quad reduction below
// leaves in that lane. Where row g + 8t is kept in pal[]: rotated within its group of eight, so that a
// quarter-warp's 16-byte stores and ldmatrix's reads both hit all banks once.
__device__ __forceinline__ int stage_row(int g, int t) { return 8 * t + ((g + 2 * t) & 7); }

// A trial's palette as A rows. Values 0..255 are kept as the half 1536 + v (0x6600 | v), which needs no conversion:
// rg = (1536 + r, 1536 + g), b = (1536 + b of this colour, or of the other one, in either half) and n =
// (1024 + |c|^2 mod 256, 1024 + |c|^2 / 256). The offsets' share of the product, -3072 (r + g + b) + 1024 * 257,
// depends on the texel alone and is taken back by the fourth word, (3072, 1024) times (r + g + b, -257).
struct Rows {
    uint32_t rg[4], b[4], n[4];
};
constexpr uint32_t kRowEnd = 0x64006A00u;  // the halves 3072, 1024

// |c|^2 of the colour whose bytes are byte 0 and 2 of rg and byte `blue` of b, as the row's third word
template <int BLUE> __device__ __forceinline__ uint32_t norm_word(uint32_t rg, uint32_t b) {
    const uint32_t c = __byte_perm(rg, b, 0x1020 | ((4 + BLUE) << 8));  // r, g, b, 0x66
    const uint32_t n = __dp4a(c, c, 0x640000u - 0x66u * 0x66u);
    return __byte_perm(n, 0x64u, 0x2140);
}

// the rows of a colour given as an RGB0 word
__device__ __forceinline__ void colour_row(uint32_t c, uint32_t &rg, uint32_t &b, uint32_t &n) {
    rg = __byte_perm(c, 0x66u, 0x4140);
    b = __byte_perm(c, 0x66u, 0x4342);
    n = __byte_perm(__dp4a(c, c, 0x640000u), 0x64u, 0x2140);
}

__device__ __forceinline__ float min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Sum over a block's 16 texels of min over NC colours of (|c|^2 - 2 p.c), for this lane's own trial: over the texels x in
// the lanes whose rows are 0-15 (lane & 2 clear), y in the others. HIGH: bit k set where colour k's blue is in the high
// half. Every lane of the warp calls it.
template <int NC, int HIGH> __device__ __forceinline__ float trial_error(const Rows &w, const Texels &x, const Texels &y) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    Work &W = work();
    const int row = stage_row(g, t);
#pragma unroll
    for (int k = 0; k < NC; k++) W.pal[warp][k][row] = make_uint4(w.rg[k], w.b[k], w.n[k], kRowEnd);
    __syncwarp();
    uint32_t a[NC][4];
    const uint32_t from = smem_addr(&W.pal[warp][0][stage_row(lane & 7, lane >> 3)]);
#pragma unroll
    for (int k = 0; k < NC; k++)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(a[k][0]), "=r"(a[k][1]), "=r"(a[k][2]), "=r"(a[k][3])
                     : "r"(from + k * 512u));
    __syncwarp();  // the next call overwrites pal
    float s[4];
#pragma unroll
    for (int h = 0; h < 2; h++) {  // rows 16h .. 16h + 15
        float m[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; nt++) {
            float d[NC][4];
#pragma unroll
            for (int k = 0; k < NC; k++) {
                const Texels &z = h == 0 ? x : y;
                mma_f16(d[k], a[k][2 * h], a[k][2 * h + 1], (HIGH >> k) & 1 ? z.hi[nt] : z.lo[nt]);
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                m[nt][i] = min3(d[0][i], d[1][i], d[2][i]);
                if (NC > 3) m[nt][i] = fminf(m[nt][i], d[NC - 1][i]);
            }
        }
        s[2 * h] = (m[0][0] + m[0][1]) + (m[1][0] + m[1][1]);  // integers below 2^24: exact
        s[2 * h + 1] = (m[0][2] + m[0][3]) + (m[1][2] + m[1][3]);
    }
    // lane t of the quad keeps the total of row g + 8t
    const bool hi2 = t & 2, hi1 = t & 1;
    const float u0 = (hi2 ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, hi2 ? s[0] : s[2], 2);
    const float u1 = (hi2 ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, hi2 ? s[1] : s[3], 2);
    return (hi1 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, hi1 ? u0 : u1, 1);
}

__device__ __forceinline__ uint32_t rgb0(int r, int g, int b) { return (uint32_t)(r | (g << 8) | (b << 16)); }

__device__ __forceinline__ float add_sat(float a, float b) {
    float d;
    asm("add.rn.sat.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}

// two rounded channels as the halves (1536 + x, 1536 + y)
__device__ __forceinline__ uint32_t pair(uint32_t wx, bool ux, uint32_t wy, bool uy) {
    uint32_t sel = ux ? 0x6421u : 0x6420u;
    if (uy) sel += 0x100u;
    return __byte_perm(wx, wy, sel);
}

// Interpolated values of halves (1536 + a) towards (1536 + b), two channels at a time, again as 1536 + v:
// Ideal floor((2a + b) / 3), IdealRound floor((2a + b + 1) / 3), AMD (43a + 21b + 32) >> 6; three colours: (a + b) / 2,
// AMD (a + b + 1) / 2. In halves, t = 2a + b <= 765 is exact, and t / 3 rounded to an integer by adding
// 1536 (unit spacing up to 2048) gives floor((t + 1) / 3), so floor(t / 3) starts from t - 1; a third as a half is
// low by 8.2e-5, which moves t / 3 by at most 0.063, less than the 1/6 to the next rounding boundary.
template <int IT, bool THREE> __device__ __forceinline__ uint32_t mid_pair(uint32_t a, uint32_t b) {
    if (THREE) {
        const uint32_t s = (a & 0x00FF00FFu) + (b & 0x00FF00FFu) + (IT == IT_AMD ? 0x00010001u : 0u);
        return ((s >> 1) & 0x00FF00FFu) | 0x66006600u;
    }
    if (IT == IT_AMD) {
        const uint32_t s = 43u * (a & 0x00FF00FFu) + 21u * (b & 0x00FF00FFu) + 0x00200020u;  // fields of at most 16352
        return ((s >> 6) & 0x00FF00FFu) | 0x66006600u;
    }
    const uint32_t a0 = add_h2(a, 0xE600E600u);                                          // a - 1536
    const uint32_t b0 = add_h2(b, IT == IT_ROUND ? 0xE600E600u : 0xE601E601u);           // b - 1536 (- 1)
    return fma_h2(fma_h2(a0, 0x40004000u, b0), 0x35553555u, 0x66006600u);
}

// The rows of the palette between the endpoints whose channels round_channel gave (w, up: low r, g, b, high r, g, b).
// Colour order {low, mid, mid, high}; three colours {low, mid, high}. kHighBlue has bit k set where colour k's blue is
// in the high half of its word.
template <int IT, bool THREE> struct Palette {
    static constexpr int kHighBlue = IT == IT_NVIDIA ? 0 : (THREE ? 4 : 12);
    static __device__ __forceinline__ Rows rows(const uint32_t w[6], const bool up[6]) {
        Rows x;
        if constexpr (IT == IT_NVIDIA) {
            int v8[6], v5[6];
#pragma unroll
            for (int i = 0; i < 6; i++) {
                v8[i] = (int)__byte_perm(w[i], 0u, up[i] ? 0x4441u : 0x4440u);
                v5[i] = v8[i] >> (i % 3 == 1 ? 2 : 3);  // the expansion keeps the value in its high bits
            }
            colour_row(rgb0(v8[0], v8[1], v8[2]), x.rg[0], x.b[0], x.n[0]);
            if (THREE) {
                colour_row(rgb0(nvh5(v5[0], v5[3]), nvh6(v5[1], v5[4]), nvh5(v5[2], v5[5])), x.rg[1], x.b[1], x.n[1]);
                colour_row(rgb0(v8[3], v8[4], v8[5]), x.rg[2], x.b[2], x.n[2]);
            } else {
                colour_row(rgb0(nv5(v5[0], v5[3]), nv6(v5[1], v5[4]), nv5(v5[2], v5[5])), x.rg[1], x.b[1], x.n[1]);
                colour_row(rgb0(nv5(v5[3], v5[0]), nv6(v5[4], v5[1]), nv5(v5[5], v5[2])), x.rg[2], x.b[2], x.n[2]);
                colour_row(rgb0(v8[3], v8[4], v8[5]), x.rg[3], x.b[3], x.n[3]);
            }
        } else {
            x = from_pairs(pair(w[0], up[0], w[1], up[1]), pair(w[3], up[3], w[4], up[4]), pair(w[2], up[2], w[5], up[5]));
        }
        return x;
    }
    // (not Nvidia) from the halves a = (low r, low g), b = (high r, high g) and ab = (low b, high b), each 1536 + v
    static __device__ __forceinline__ Rows from_pairs(uint32_t a, uint32_t b, uint32_t ab) {
        Rows x;
        {
            const uint32_t ba = __byte_perm(ab, 0u, 0x1032);
            const uint32_t q = mid_pair<IT, THREE>(ab, ba);  // blues of the mids, (towards high, towards low)
            x.rg[0] = a;
            x.b[0] = ab;
            x.n[0] = norm_word<0>(a, ab);
            x.rg[1] = mid_pair<IT, THREE>(a, b);
            x.b[1] = q;
            x.n[1] = norm_word<0>(x.rg[1], q);
            if (THREE) {
                x.rg[2] = b;
                x.b[2] = ab;
                x.n[2] = norm_word<2>(b, ab);
            } else {
                x.rg[2] = mid_pair<IT, THREE>(b, a);
                x.b[2] = q;
                x.n[2] = norm_word<2>(x.rg[2], q);
                x.rg[3] = b;
                x.b[3] = ab;
                x.n[3] = norm_word<2>(b, ab);
            }
        }
        return x;
    }
};

// RefineBlockCF<K> (BC1Encoder.cpp:877-928), `passes` times, for the lanes' blocks with `run` (K_F4_FULL or K_T3). A
// second pass that repeats the first one's trials is skipped (tpb::cf_same_trials). With `split` only the first pass
// runs, and *again receives whether a second one can change the result.
template <int IT, int K>
__device__ __noinline__ void cluster_fit(const qt_bc1_params &p, bool run, tpb::R &r, const tpb::M &m, int pp_sum, int passes, bool *again) {
    constexpr bool four = !kind_three(K);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, col0 = threadIdx.x - lane;
    const bool exhaustive = p.exhaustive != 0;
    const unsigned total = exhaustive ? (four ? 969u : 153u) : (four ? p.orderings4 : p.orderings3);
    FitWork &F = fit();
    const uint4 *ord = four ? F.ord4 : F.ord3;
    const uint32_t tab5 = smem_addr(F.rnd5) - 8u * 0x4B000000u, tab6 = smem_addr(F.rnd6) - 8u * 0x4B000000u;
    int prev_start = -1;
    uint64_t prev_order = 0;
    for (int pass = 0; pass < passes; pass++) {
        int start = 0;
        tpb::R sc = tpb::rinit();
        if (run) {
            sc = tpb::single_color<IT>(r.lo, r.hi, m.av[0], m.av[1], m.av[2], !four);
            sc.mode = kind_mode(K);
            // a repeated pass changes nothing: its trials are the last pass's, whose minimum r already is, and its
            // single-colour trial, the only one that depends on r's endpoints, is no better
            if (pass > 0 && sc.err >= r.err && (r.err == 0 || tpb::cf_same_trials(four, r, prev_start, prev_order))) run = false;
        }
        if (run) {
            start = tpb::cf_start_hash(four, r.sel);
            const int axr = s5to8(epr(r.hi)) - s5to8(epr(r.lo)), axg = s6to8(epg(r.hi)) - s6to8(epg(r.lo)), axb = s5to8(epb(r.hi)) - s5to8(epb(r.lo));
            uint32_t key[16];
#pragma unroll
            for (int i = 0; i < 16; i++) key[i] = tpb::cf_key(tpb::px(i), axr, axg, axb, i);
            tpb::sort16(key);
            uint64_t order = 0;
            uint32_t arg = 0, ab = 0;
            F.pre[warp][lane][0] = make_uint2(0u, 0u);
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const int i = (int)(key[k] & 15);
                const uint32_t v = tpb::px(i);
                arg += (uint32_t)tpb::cr(v) | ((uint32_t)tpb::cg(v) << 16);
                ab += (uint32_t)tpb::cb(v);
                F.pre[warp][lane][k + 1] = make_uint2(arg, ab);
                if (passes > 1 || again) order |= (uint64_t)i << (4 * k);
            }
            prev_start = start;
            prev_order = order;
        }
        __syncwarp();
        const TexelForm form;
        bool won = false;
        unsigned won_q = 0;
        uint32_t won_err = 0;
        for (uint32_t todo = __ballot_sync(0xffffffffu, run); todo; todo &= todo - 1) {
            const int j = __ffs((int)todo) - 1;  // the block of lane j, with all lanes
            const int jstart = __shfl_sync(0xffffffffu, start, j), jpp = __shfl_sync(0xffffffffu, pp_sum, j);
            const uint32_t jerr = __shfl_sync(0xffffffffu, r.err, j), jsc = __shfl_sync(0xffffffffu, sc.err, j);
            const Texels x = load_texels(col0 + j, form);
            const uint32_t pre = smem_addr(&F.pre[warp][j][0]);
            const uint2 tt = F.pre[warp][j][16];
            // the selector total times 3 (2), less the trial's sums: on top of 2^23, as the sums' conversion below gives them
            const float denom = four ? 3.0f : 2.0f;
            const float t3r = (float)(tt.x & 0xFFFF) * denom + 8388608.0f, t3g = (float)(tt.x >> 16) * denom + 8388608.0f, t3b = (float)tt.y * denom + 8388608.0f;
            const uint16_t *row = (four ? g_tab.coop4 + jstart * 128 : g_tab.coop3 + jstart * 32) + lane;
            float best = INFINITY;
            unsigned best_q = 0;
            // a step's entry is loaded a step ahead
            auto entry = [&](unsigned q0) -> unsigned {
                const unsigned q = q0 + lane;
                if (!exhaustive) return q0 < total ? (unsigned)row[q0] : 0u;
                return (q < total ? q : 0u) | (is_single_hash(four, (int)q) ? 0x400u : 0u) | ((unsigned)lane << 11);
            };
            unsigned next = entry(0);
            for (unsigned q0 = 0; q0 < total; q0 += 32) {
                const unsigned raw = next;
                next = entry(q0 + 32);
                const uint4 o = ord[raw & 0x3FFu];
                uint32_t q0x, q0y, q1x, q1y, q2x = 0u, q2y = 0u;
                asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(q0x), "=r"(q0y) : "r"(pre + __byte_perm(o.w, 0u, 0x4440)));
                asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(q1x), "=r"(q1y) : "r"(pre + __byte_perm(o.w, 0u, 0x4441)));
                if (four) asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(q2x), "=r"(q2y) : "r"(pre + __byte_perm(o.w, 0u, 0x4442)));
                const uint32_t qrg = q0x + q1x + q2x, qb = q0y + q1y + q2y;
                // integers below 2^24, exact: 2^23 + n as a float, then 2^23 off
                const float kr = __uint_as_float(__byte_perm(qrg, 0x4B000000u, 0x7610)), kg = __uint_as_float(__byte_perm(qrg, 0x4B000000u, 0x7632)), kb = __uint_as_float(qb | 0x4B000000u);
                const float fr = __fadd_rn(kr, -8388608.0f), fg = __fadd_rn(kg, -8388608.0f), fb = __fadd_rn(kb, -8388608.0f);
                const float gr = __fsub_rn(t3r, kr), gg = __fsub_rn(t3g, kg), gb = __fsub_rn(t3b, kb);
                const float fx = __uint_as_float(o.x), fy = __uint_as_float(o.y), fw = __uint_as_float(o.z);
                const float v[6] = {add_sat(__fmul_rn(fx, gr), __fmul_rn(fy, fr)), add_sat(__fmul_rn(fx, gg), __fmul_rn(fy, fg)), add_sat(__fmul_rn(fx, gb), __fmul_rn(fy, fb)),
                                    add_sat(__fmul_rn(fy, gr), __fmul_rn(fw, fr)), add_sat(__fmul_rn(fy, gg), __fmul_rn(fw, fg)), add_sat(__fmul_rn(fy, gb), __fmul_rn(fw, fb))};
                // PreciseRound565 of the six channels as precise_round565_cf: v is clamped to [0, 1] already, which
                // changes neither the truncated product's clamp nor the midpoint test, and trunc(v * scale) is in the
                // mantissa after a round-towards-zero addition of 2^23
                uint32_t cw[6];
                bool up[6];
#pragma unroll
                for (int i = 0; i < 6; i++) {
                    const float cell = __fadd_rz(__fmul_rn(v[i], i % 3 == 1 ? 63.0f : 31.0f), 8388608.0f);
                    uint32_t mid;
                    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(mid), "=r"(cw[i]) : "r"((i % 3 == 1 ? tab6 : tab5) + __float_as_uint(cell) * 8u));
                    up[i] = v[i] > __uint_as_float(mid);
                }
                float err = trial_error<four ? 4 : 3, Palette<IT, !four>::kHighBlue>(Palette<IT, !four>::rows(cw, up), x, x);
                if (raw & 0x400u) err = (float)((int)jsc - jpp);  // a single-colour ordering
                const unsigned q = q0 + (raw >> 11);
                if (q < total && err < best) {
                    best = err;
                    best_q = q;
                }
            }
            // the first of the best trials; kept if strictly better than the block's result so far
            const int least = __float2int_rz(best), low = __reduce_min_sync(0xffffffffu, least);
            const uint32_t err = (uint32_t)(jpp + low);
            if (err < jerr) {
                const unsigned bq = __reduce_min_sync(0xffffffffu, least == low ? best_q : 0xffffffffu);
                if (lane == j) {
                    won = true;
                    won_q = bq;
                    won_err = err;
                }
            }
        }
        __syncwarp();
        if (won) {  // the winning trial's endpoints and selectors
            const int raw = exhaustive ? (int)won_q : (int)(four ? g_tab.best4[start * 128 + won_q] : g_tab.best3[start * 32 + won_q]), th = raw & 0x7FFF;
            if (exhaustive ? is_single_hash(four, th) : raw >= 0x8000) {
                r = sc;
            } else {
                const uint4 o = ord[th];
                const uint2 *pre = F.pre[warp][lane];
                const uint2 s1 = pre[(o.w & 0xFF) >> 3], s2 = pre[((o.w >> 8) & 0xFF) >> 3], s3 = four ? pre[((o.w >> 16) & 0xFF) >> 3] : make_uint2(0u, 0u);
                const uint32_t qrg = s1.x + s2.x + s3.x, qb = s1.y + s2.y + s3.y;
                const uint2 tt = pre[16];
                const float denom = four ? 3.0f : 2.0f, fr = (float)(qrg & 0xFFFF), fg = (float)(qrg >> 16), fb = (float)qb;
                const float gr = (float)(tt.x & 0xFFFF) * denom - fr, gg = (float)(tt.x >> 16) * denom - fg, gb = (float)tt.y * denom - fb;
                const float fx = __uint_as_float(o.x), fy = __uint_as_float(o.y), fw = __uint_as_float(o.z);
                r.lo = precise_round565_cf(__fadd_rn(__fmul_rn(fx, gr), __fmul_rn(fy, fr)), __fadd_rn(__fmul_rn(fx, gg), __fmul_rn(fy, fg)),
                                           __fadd_rn(__fmul_rn(fx, gb), __fmul_rn(fy, fb)), s_mid5, s_mid6);
                r.hi = precise_round565_cf(__fadd_rn(__fmul_rn(fy, gr), __fmul_rn(fw, fr)), __fadd_rn(__fmul_rn(fy, gg), __fmul_rn(fw, fg)),
                                           __fadd_rn(__fmul_rn(fy, gb), __fmul_rn(fw, fb)), s_mid5, s_mid6);
                r.err = won_err;
                r.mode = kind_mode(K);
                r.sel = tpb::find_selectors<IT, K>(r.lo, r.hi).x;
            }
        }
    }
    if (again) *again = run && r.err > 0 && !(tpb::cf_same_trials(four, r, prev_start, prev_order) &&
                                             tpb::single_color<IT>(r.lo, r.hi, m.av[0], m.av[1], m.av[2], !four).err >= r.err);
}

// EndpointSearch (BC1Encoder.cpp:930-996) of the lanes' blocks in `todo` (shared-memory columns col0 + lane, all of
// kind K), one block at a time: the 32 candidates that follow the last improvement at once, and the first that improves,
// in the order of the rounds, is accepted. The reference stops 32 rounds after its last improvement, and a candidate
// repeats every 32 rounds, so a window without an improvement ends the search. A block's lane receives its endpoints
// and whether they moved.
//
// The endpoints are kept as the halves that the rows are made from (1536 + v: red and green in one word, blue in
// another), so a window forms only its own candidate.
template <int IT, int K>
__device__ __forceinline__ void search_blocks(uint32_t todo, int col0, unsigned rounds, int pp_sum, tpb::R &res, bool &res_moved) {
    static_assert(IT != IT_NVIDIA, "search_blocks_nvidia");
    constexpr bool three = kind_three(K);
    const int lane = threadIdx.x & 31;
    const TexelForm form;
    // lane l always takes the candidates of the rounds congruent to l
    const uint16_t vx = s_vox[lane & 15];
    const int ddr = ((int)((unsigned)vx << 30)) >> 30, ddg = ((int)((unsigned)vx << 28)) >> 30, ddb = ((int)((unsigned)vx << 26)) >> 30;
    const int opposite = ((vx >> 8) & 15) | (lane & 16);
    const bool low = (lane & 16) != 0;
    auto halves = [](int e, uint32_t &rg, uint32_t &bb) {
        rg = (uint32_t)s5to8(epr(e)) + ((uint32_t)s6to8(epg(e)) << 16) + 0x66006600u;
        bb = (uint32_t)s5to8(epb(e)) + 0x6600u;
    };
    for (; todo; todo &= todo - 1) {
        const int j = __ffs((int)todo) - 1;
        int lo = __shfl_sync(0xffffffffu, res.lo, j), hi = __shfl_sync(0xffffffffu, res.hi, j);
        uint32_t err = __shfl_sync(0xffffffffu, res.err, j);
        const int pp = __shfl_sync(0xffffffffu, pp_sum, j);
        const Texels x = load_texels(col0 + j, form);
        uint32_t lo_rg, lo_b, hi_rg, hi_b;
        halves(lo, lo_rg, lo_b);
        halves(hi, hi_rg, hi_b);
        int forbidden = -1;
        bool moved = false;
        for (unsigned first = 0; first < rounds;) {
            const unsigned i = first + ((lane - first) & 31u);
            const int e = low ? lo : hi;
            const int n = eppack(__viaddmin_s32_relu(epr(e), ddr, 31), __viaddmin_s32_relu(epg(e), ddg, 63), __viaddmin_s32_relu(epb(e), ddb, 31));
            uint32_t rg, bb;
            halves(n, rg, bb);
            const uint32_t ab = __byte_perm(low ? bb : lo_b, low ? hi_b : bb, 0x5410);
            Rows w = Palette<IT, three>::from_pairs(low ? rg : lo_rg, low ? hi_rg : rg, ab);
            if (K == K_TB) colour_row(0u, w.rg[3], w.b[3], w.n[3]);  // black
            const uint32_t ne = (uint32_t)(pp + __float2int_rz(trial_error<K == K_T3 ? 3 : 4, Palette<IT, three>::kHighBlue>(w, x, x)));
            uint32_t better = __ballot_sync(0xffffffffu, i < rounds && lane != forbidden && ne < err);
            if (!better) break;
            better = __funnelshift_r(better, better, first);  // in the order of the rounds
            const unsigned at = first + (unsigned)__ffs((int)better) - 1u;
            const int f = (int)(at & 31);
            const int fn = __shfl_sync(0xffffffffu, n, f);
            rg = __shfl_sync(0xffffffffu, rg, f);
            bb = __shfl_sync(0xffffffffu, bb, f);
            err = __shfl_sync(0xffffffffu, ne, f);
            forbidden = __shfl_sync(0xffffffffu, opposite, f);
            if (f & 16) lo = fn, lo_rg = rg, lo_b = bb;
            else hi = fn, hi_rg = rg, hi_b = bb;
            first = at + 1;
            moved = true;
        }
        if (lane == j && moved) {
            res.lo = lo;
            res.hi = hi;
            res_moved = true;
        }
    }
}

// The same with Nvidia's interpolation, two blocks at a time: each half of the warp (lane & 2) takes the 16 candidates
// that follow its block's last improvement, and two windows without one end a search. An improvement throws the rest of
// its window away, and Nvidia's searches improve every few rounds (~13 times a block at level 17, against 0.5
// with Ideal), so half the candidates on twice the blocks is the better use of a window: level 18 at 512^2
// 253 -> 177 us, at 1024^2 560 -> 440 us. Where improvements are rare one block at a time is (level 18
// at 128^2: 45 us against 55).
template <int K>
__device__ __forceinline__ void search_blocks_nvidia(uint32_t todo, int col0, unsigned rounds, int pp_sum, tpb::R &res, bool &res_moved) {
    const int lane = threadIdx.x & 31, half = lane & 2;
    const TexelForm form;
    const int k = 2 * (lane >> 2) + (lane & 1);  // this lane takes the rounds congruent to k modulo 16
    const uint16_t vx = s_vox[k];
    const int ddr = ((int)((unsigned)vx << 30)) >> 30, ddg = ((int)((unsigned)vx << 28)) >> 30, ddb = ((int)((unsigned)vx << 26)) >> 30;
    const int opposite = (vx >> 8) & 15;
    Texels x[2] = {};
    int block[2] = {-1, -1};  // the halves' blocks
    // this lane's half's search
    int lo = 0, hi = 0, pp = 0, forbidden = -1, quiet = 0;
    uint32_t err = 0;
    unsigned first = 0;
    bool moved = false, done = true;
    for (;;) {
        const uint32_t idle = __ballot_sync(0xffffffffu, done);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (!((idle >> (2 * h)) & 1u)) continue;
            if (block[h] >= 0) {
                const int flo = __shfl_sync(0xffffffffu, lo, 2 * h), fhi = __shfl_sync(0xffffffffu, hi, 2 * h);
                const bool fm = (__ballot_sync(0xffffffffu, moved) >> (2 * h)) & 1u;
                if (lane == block[h] && fm) {
                    res.lo = flo;
                    res.hi = fhi;
                    res_moved = true;
                }
                block[h] = -1;
            }
            if (!todo) continue;
            const int j = __ffs((int)todo) - 1;
            todo &= todo - 1;
            block[h] = j;
            x[h] = load_texels(col0 + j, form);
            const int jlo = __shfl_sync(0xffffffffu, res.lo, j), jhi = __shfl_sync(0xffffffffu, res.hi, j), jpp = __shfl_sync(0xffffffffu, pp_sum, j);
            const uint32_t jerr = __shfl_sync(0xffffffffu, res.err, j);
            if (half == 2 * h) {
                lo = jlo;
                hi = jhi;
                pp = jpp;
                err = jerr;
                forbidden = -1;
                quiet = 0;
                first = 0;
                moved = false;
                done = false;
            }
        }
        if (block[0] < 0 && block[1] < 0) break;
        const unsigned i = first + ((k - first) & 15u);
        const bool low = (i & 16) != 0;
        const int e = low ? lo : hi;
        const int n = eppack(__viaddmin_s32_relu(epr(e), ddr, 31), __viaddmin_s32_relu(epg(e), ddg, 63), __viaddmin_s32_relu(epb(e), ddb, 31));
        const Pal P = make_pal<IT_NVIDIA>(low ? n : lo, low ? hi : n, kind_three(K));
        Rows w;
        colour_row(rgb0(P.r0, P.g0, P.b0), w.rg[0], w.b[0], w.n[0]);
        colour_row(rgb0(P.r1, P.g1, P.b1), w.rg[1], w.b[1], w.n[1]);
        colour_row(rgb0(P.r2, P.g2, P.b2), w.rg[2], w.b[2], w.n[2]);
        if (K != K_T3) colour_row(rgb0(P.r3, P.g3, P.b3), w.rg[3], w.b[3], w.n[3]);
        const uint32_t ne = (uint32_t)(pp + __float2int_rz(trial_error<K == K_T3 ? 3 : 4, 0>(w, x[0], x[1])));
        // the half's improving lanes: their bits are in the order of k, from the window's first round on, then around
        const uint32_t better = __ballot_sync(0xffffffffu, !done && i < rounds && (int)(i & 31) != forbidden && ne < err) & (0x33333333u << half);
        const unsigned s = first & 15u, at = (4u * (s >> 1) + (s & 1u)) + half;
        const uint32_t later = better & (0xffffffffu << at);
        const int f = better ? __ffs((int)(later ? later : better)) - 1 : lane;
        const int fn = __shfl_sync(0xffffffffu, n, f), fop = __shfl_sync(0xffffffffu, opposite, f);
        const uint32_t fe = __shfl_sync(0xffffffffu, ne, f);
        const unsigned fi = __shfl_sync(0xffffffffu, i, f);
        if (better) {
            if (fi & 16) lo = fn;
            else hi = fn;
            err = fe;
            forbidden = fop | (int)(fi & 16);
            first = fi + 1;
            quiet = 0;
            moved = true;
        } else {
            first += 16;
            quiet++;
        }
        done |= quiet == 2 || first >= rounds;
    }
}

// the searches of the lanes with `run`; returns whether this lane's moved
template <int IT> __device__ __forceinline__ bool search(bool run, unsigned rounds, int pp_sum, tpb::R &r) {
    const int col0 = threadIdx.x & ~31;
    bool moved = false;
    const uint32_t three = __ballot_sync(0xffffffffu, run && r.mode == CM_THREE), black = __ballot_sync(0xffffffffu, run && r.mode == CM_TB);
    const uint32_t four = __ballot_sync(0xffffffffu, run) & ~(three | black);
    if constexpr (IT == IT_NVIDIA) {
        if (four) search_blocks_nvidia<K_F4_FULL>(four, col0, rounds, pp_sum, r, moved);
        if (three) search_blocks_nvidia<K_T3>(three, col0, rounds, pp_sum, r, moved);
        if (black) search_blocks_nvidia<K_TB>(black, col0, rounds, pp_sum, r, moved);
    } else {
        if (four) search_blocks<IT, K_F4_FULL>(four, col0, rounds, pp_sum, r, moved);
        if (three) search_blocks<IT, K_T3>(three, col0, rounds, pp_sum, r, moved);
        if (black) search_blocks<IT, K_TB>(black, col0, rounds, pp_sum, r, moved);
    }
    return moved;
}

__device__ __forceinline__ int search_kind(const tpb::R &r) { return r.mode == CM_THREE ? K_T3 : (r.mode == CM_TB ? K_TB : K_F4_FULL); }

// EncodeBlock up to the four-colour cluster fit (BC1Encoder.cpp:264-297), one block per lane
template <int IT> __device__ __forceinline__ void front(const qt_bc1_params &p, const tpb::M &m, tpb::R &res, tpb::R &orig) {
    const int ep_passes = p.two_ep_passes ? 2 : 1;
    for (int round = 0; round < ep_passes; round++) {
        const int2 ep = tpb::find_endpoints(m, round == 1 ? EP_BB : p.endpoint_mode, false, (int)p.power_iterations);
        tpb::R to = tpb::rinit();
        to.lo = ep.x;
        to.hi = ep.y;
        tpb::R tr = to;
        const uint2 se = tpb::find_selectors<IT, K_F4_FULL>(tr.lo, tr.hi);
        tr.sel = se.x;
        tr.err = se.y;
        tr.mode = CM_FOUR;
        tr = tpb::refine_ls<IT, K_F4_FULL>(tr, m, p.two_ls_passes ? 2 : 1);
        if (tr.err < res.err) {
            res = tr;
            orig = to;
        }
    }
}

// ... and from the 3-colour trials to before EndpointSearch (:305-336). Every lane of the warp calls it; `run` marks
// the lanes that hold a block.
template <int IT>
__device__ __forceinline__ void three_colour(const qt_bc1_params &p, int color_mode, bool run, const tpb::M &m, int pp_sum, tpb::R &res, const tpb::R &orig) {
    if (!(color_mode & CM_THREE)) return;
    const int ls_passes = p.two_ls_passes ? 2 : 1;
    const bool three = run && res.err > 0;
    tpb::R t = orig;
    if (three) {
        const uint2 se = tpb::find_selectors<IT, K_T3>(t.lo, t.hi);
        t.sel = se.x;
        t.err = se.y;
        t.mode = CM_THREE;
        t = tpb::refine_ls<IT, K_T3>(t, m, ls_passes);
    }
    cluster_fit<IT, K_T3>(p, three && t.err > 0, t, m, pp_sum, p.two_cf_passes ? 2 : 1, nullptr);
    if (three && t.err < res.err) res = t;
    if (run && res.err > 0 && color_mode == CM_TB && m.has_black && !((m.mx[0] | m.mx[1] | m.mx[2]) < 4)) {
        const tpb::M mnb = tpb::metrics(true);
        const int2 ep = tpb::find_endpoints(mnb, EP_PCA, true, (int)p.power_iterations);
        tpb::R b = tpb::rinit();
        b.lo = ep.x;
        b.hi = ep.y;
        const uint2 se = tpb::find_selectors<IT, K_TB>(b.lo, b.hi);
        b.sel = se.x;
        b.err = se.y;
        b.mode = CM_TB;
        b = tpb::refine_ls<IT, K_TB>(b, mnb, ls_passes);
        if (b.err < res.err) res = b;
    }
}

// EncodeBlock of the blocks staged in the warp's shared-memory columns, one per lane with `have`
template <int IT> __device__ __forceinline__ uint2 encode_warp(const qt_bc1_params &p, int color_mode, bool have, int pp_sum) {
    uint2 blk = make_uint2(0u, 0u);
    bool run = have;
    if (have) {
        const uint32_t c0 = tpb::px(0);
        bool solid = true;
        for (int i = 1; i < 16; i++) solid &= tpb::px(i) == c0;
        if (solid) {
            blk = write_block_solid<IT>(c0);
            run = false;
        }
    }
    tpb::M m;
    tpb::R res = tpb::rinit(), orig = tpb::rinit();
    if (run) {
        m = tpb::metrics(false);
        front<IT>(p, m, res, orig);
    }
    cluster_fit<IT, K_F4_FULL>(p, run && res.err > 0, res, m, pp_sum, p.two_cf_passes ? 2 : 1, nullptr);
    three_colour<IT>(p, color_mode, run, m, pp_sum, res, orig);
    if (search<IT>(run && res.err > 0, p.search_rounds, pp_sum, res)) res.sel = tpb::fs_any<IT>(search_kind(res), res.lo, res.hi).x;
    if (run) blk = tpb::write(res);
    return blk;
}

__device__ __forceinline__ void write_out(uint8_t *out, int bc3, long b, uint2 blk) {
    if (bc3) {
        uint32_t v[16];
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = tpb::t_px[k][threadIdx.x];
        const uint2 a = bc4_block_thread(v, 3);
        reinterpret_cast<uint4 *>(out)[b] = make_uint4(a.x, a.y, blk.x, blk.y);
    } else {
        reinterpret_cast<uint2 *>(out)[b] = blk;
    }
}

}  // namespace coop

// EncodeBlock of the whole texture (or, with `list`, of its listed blocks). A warp takes `per_warp` (1 to 32) blocks at
// a time: fewer than 32 where the texture would otherwise leave warps without work (the cooperative phases, which
// are most of the work, need no full lanes).
template <int IT>
__global__ void __launch_bounds__(tpb::kThreads, 4) k_bc1_coop(const uint8_t *__restrict__ rgba, int w, int h, int bw, long b_begin, long nblocks,
                                                                qt_bc1_params p, uint8_t *__restrict__ out, int bc3, int aligned,
                                                                const uint32_t *__restrict__ list, const uint32_t *__restrict__ count, int per_warp) {
    load_tables_smem();
    const int color_mode = bc3 ? CM_FOUR : p.color_mode;  // BC3Encoder.h:39-40
    coop::load_fit_tables(color_mode != CM_FOUR);
    const int lane = threadIdx.x & 31;
    const long end = list ? (long)*count : nblocks, stride = (long)gridDim.x * coop::kWarps * per_warp;
    for (long wb = (list ? 0 : b_begin) + ((long)blockIdx.x * coop::kWarps + (threadIdx.x >> 5)) * per_warp; wb < end; wb += stride) {
        const bool have = lane < per_warp && wb + lane < end;
        long b = 0;
        int pp = 0;
        if (have) {
            b = list ? (long)list[wb + lane] : wb + lane;
            uint32_t v[16];
            pp = stage_block(rgba, w, h, bw, b, aligned, v);
        }
        __syncwarp();
        const uint2 blk = coop::encode_warp<IT>(p, color_mode, have, pp);
        if (have) coop::write_out(out, bc3, b, blk);
        __syncwarp();
    }
}

// The passes of a large texture (the counterparts of k_bc1_defer, k_bc1_cf2 and k_bc1_search, with the same queues).
// First pass: every listed block through its first four-colour cluster-fit pass; what remains is queued.
template <int IT>
__global__ void __launch_bounds__(tpb::kThreads, 4) k_bc1_coop_defer(const uint8_t *__restrict__ rgba, int w, int h, int bw, qt_bc1_params p,
                                                                      uint8_t *__restrict__ out, int bc3, int aligned,
                                                                      const uint32_t *__restrict__ list, const uint32_t *__restrict__ count,
                                                                      SearchQueues q, Cf2Queue c) {
    load_tables_smem();
    const int color_mode = bc3 ? CM_FOUR : p.color_mode;  // BC3Encoder.h:39-40
    coop::load_fit_tables(color_mode != CM_FOUR);
    const int lane = threadIdx.x & 31;
    const long end = (long)*count, stride = (long)gridDim.x * blockDim.x;
    for (long wb = (long)blockIdx.x * blockDim.x + threadIdx.x - lane; wb < end; wb += stride) {
        const bool have = wb + lane < end;
        tpb::Deferred d;
        d.need = d.cf2 = d.pass2 = false;
        d.queue = 0;
        long b = 0;
        int pp = 0;
        tpb::M m;
        tpb::R res = tpb::rinit(), orig = tpb::rinit();
        if (have) {
            b = (long)list[wb + lane];
            uint32_t v[16];
            pp = stage_block(rgba, w, h, bw, b, aligned, v);
            m = tpb::metrics(false);
            coop::front<IT>(p, m, res, orig);
        }
        __syncwarp();
        const bool run = have && res.err > 0;
        if (p.two_cf_passes) {
            bool again = false;
            coop::cluster_fit<IT, K_F4_FULL>(p, run, res, m, pp, 1, &again);
            if (have && (again || (res.err > 0 && (color_mode & CM_THREE)))) {
                d.cf2 = true;
                d.pass2 = again;
                d.r = res;
                d.orig = orig;
            }
        } else {
            coop::cluster_fit<IT, K_F4_FULL>(p, run, res, m, pp, 1, nullptr);
            coop::three_colour<IT>(p, color_mode, have, m, pp, res, orig);
        }
        if (have && !d.cf2 && res.err > 0) {
            d.need = true;
            d.queue = res.mode == CM_THREE ? 1 : (res.mode == CM_TB ? 2 : 0);
            d.r = res;
        }
        if (have) {  // for BC3 the alpha half now; a queued block's colour half is written by a later pass
            const uint2 blk = tpb::write(res);
            if (bc3 || (!d.need && !d.cf2)) coop::write_out(out, bc3, b, blk);
        }
        push_searches(q, d, b, lane);
        push_cf2(c, d, b, lane);
        __syncwarp();
    }
}

// Second pass: the queued blocks' second four-colour cluster-fit pass, for the entries that need it, and the 3-colour
// trials. The queue holds the second-pass entries from the front and the others from the back.
template <int IT>
__global__ void __launch_bounds__(tpb::kThreads, 4) k_bc1_coop_cf2(const uint8_t *__restrict__ rgba, int w, int h, int bw, qt_bc1_params p,
                                                                    uint8_t *__restrict__ out, int bc3, int aligned, Cf2Queue c, SearchQueues q) {
    load_tables_smem();
    const int color_mode = bc3 ? CM_FOUR : p.color_mode;
    coop::load_fit_tables(color_mode != CM_FOUR);
    const int lane = threadIdx.x & 31;
    const long n2 = (long)c.count[0], end = n2 + (long)c.count[1], stride = (long)gridDim.x * blockDim.x;
    for (long wb = (long)blockIdx.x * blockDim.x + threadIdx.x - lane; wb < end; wb += stride) {
        const long idx = wb + lane;
        const bool have = idx < end, pass2 = idx < n2;
        tpb::Deferred d;
        d.need = d.cf2 = d.pass2 = false;
        d.queue = 0;
        long b = 0;
        int pp = 0;
        tpb::M m;
        tpb::R res = tpb::rinit(), orig = tpb::rinit();
        if (have) {
            const long i = pass2 ? idx : c.cap - 1 - (idx - n2);
            b = (long)c.b[i];
            uint32_t v[16];
            pp = stage_block(rgba, w, h, bw, b, aligned, v);
            m = tpb::metrics(false);
            const uint32_t lh = c.lohi[i], ol = c.orig[i];
            res.lo = (int)(lh & 0xFFFF);
            res.hi = (int)(lh >> 16);
            res.err = c.err[i];
            res.sel = c.sel[i];
            res.mode = (int)c.mode[i];
            orig.lo = (int)(ol & 0xFFFF);
            orig.hi = (int)(ol >> 16);
        }
        __syncwarp();
        coop::cluster_fit<IT, K_F4_FULL>(p, have && pass2, res, m, pp, 1, nullptr);
        coop::three_colour<IT>(p, color_mode, have, m, pp, res, orig);
        if (have) {
            if (res.err > 0) {
                d.need = true;
                d.queue = res.mode == CM_THREE ? 1 : (res.mode == CM_TB ? 2 : 0);
                d.r = res;
            } else {
                const uint2 blk = tpb::write(res);
                if (bc3) reinterpret_cast<uint2 *>(out)[2 * b + 1] = blk;  // the colour half of the 16-byte block
                else reinterpret_cast<uint2 *>(out)[b] = blk;
            }
        }
        push_searches(q, d, b, lane);
        __syncwarp();
    }
}

// One queue of searches: a warp takes 32 entries, stages their texels, and searches them one after the other. Those that moved go to the finish queue, the others are written.
template <int IT, int K>
__device__ __forceinline__ void coop_search_queue(int qq, const uint8_t *__restrict__ rgba, int w, int h, int bw, unsigned rounds,
                                                  uint8_t *__restrict__ out, int bc3, int aligned, const SearchQueues &q, const FinishQueue &f) {
    const int lane = threadIdx.x & 31, col0 = threadIdx.x - lane;
    const long total = (long)q.count[qq], stride = (long)gridDim.x * blockDim.x;
    for (long wb = (long)blockIdx.x * blockDim.x + threadIdx.x - lane; wb < total; wb += stride) {
        const int n = (int)(total - wb < 32 ? total - wb : 32);
        long b = 0;
        int pp = 0;
        tpb::R r = tpb::rinit();
        if (lane < n) {
            const long slot = (long)qq * q.cap + wb + lane;
            b = (long)q.b[slot];
            const uint32_t lh = q.lohi[slot];
            r.lo = (int)(lh & 0xFFFF);
            r.hi = (int)(lh >> 16);
            r.err = q.err[slot];
            r.sel = q.sel[slot];
            r.mode = (int)q.mode[slot];
            uint32_t v[16];
            pp = stage_block(rgba, w, h, bw, b, aligned, v);
        }
        __syncwarp();
        bool moved = false;
        coop::search_blocks<IT, K>(__ballot_sync(0xffffffffu, lane < n), col0, rounds, pp, r, moved);
        const uint32_t fin = __ballot_sync(0xffffffffu, moved);
        uint32_t fbase = 0;
        if (lane == 0 && fin) fbase = atomicAdd(f.count, (uint32_t)__popc(fin));
        fbase = __shfl_sync(0xffffffffu, fbase, 0);
        if (moved) {
            const uint32_t slot = fbase + __popc(fin & ((1u << lane) - 1));
            f.b[slot] = (uint32_t)b;
            f.lohi[slot] = pack_lohi(r);
            f.mode[slot] = (uint32_t)r.mode;
        } else if (lane < n) {  // the queued selectors belong to these endpoints
            const uint2 blk = tpb::write(r);
            if (bc3) reinterpret_cast<uint2 *>(out)[2 * b + 1] = blk;
            else reinterpret_cast<uint2 *>(out)[b] = blk;
        }
        __syncwarp();
    }
}

constexpr int kCoopSearchCtas = 5;
template <int IT>
__global__ void __launch_bounds__(tpb::kThreads, kCoopSearchCtas) k_bc1_coop_search(const uint8_t *__restrict__ rgba, int w, int h, int bw, qt_bc1_params p,
                                                                       uint8_t *__restrict__ out, int bc3, int aligned, SearchQueues q, FinishQueue f) {
    load_tables_smem();
    coop_search_queue<IT, K_F4_FULL>(0, rgba, w, h, bw, p.search_rounds, out, bc3, aligned, q, f);
    coop_search_queue<IT, K_T3>(1, rgba, w, h, bw, p.search_rounds, out, bc3, aligned, q, f);
    coop_search_queue<IT, K_TB>(2, rgba, w, h, bw, p.search_rounds, out, bc3, aligned, q, f);
}

// The batch's tiles whose textures run cooperatively (coop_batch_setting): tiles[.. ctl[1]), claimed through ctl[0] as k_batch
// claims the others. One texture per tile, so a warp's settings are uniform.
template <int IT> __device__ __noinline__ uint2 encode_warp_batch(const qt_bc1_params &p, int color_mode, bool have, int pp) {
    return coop::encode_warp<IT>(p, color_mode, have, pp);
}

__global__ void __launch_bounds__(tpb::kThreads, 4) k_batch_coop(const BatchItemDev *__restrict__ items, const TileDev *__restrict__ tiles,
                                                                 uint32_t *__restrict__ ctl) {
    load_tables_smem();
    coop::load_fit_tables(true);
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
        const int bc3 = I.fmt == 3, w = I.w, h = I.h, cm = bc3 ? CM_FOUR : p.color_mode;  // BC3Encoder.h:39-40
        const int aligned = ((w & 3) == 0) && ((reinterpret_cast<uintptr_t>(I.src) & 15) == 0);
        for (uint32_t k = 0; k < T.count; k += 32) {
            const bool have = k + lane < T.count;
            const long b = (long)T.start + k + lane;
            int pp = 0;
            if (have) {
                uint32_t v[16];
                pp = stage_block(I.src, w, h, I.bw, b, aligned, v);
            }
            __syncwarp();
            uint2 blk;
            switch (p.interpolator) {
                case IT_IDEAL: blk = encode_warp_batch<IT_IDEAL>(p, cm, have, pp); break;
                case IT_ROUND: blk = encode_warp_batch<IT_ROUND>(p, cm, have, pp); break;
                case IT_NVIDIA: blk = encode_warp_batch<IT_NVIDIA>(p, cm, have, pp); break;
                default: blk = encode_warp_batch<IT_AMD>(p, cm, have, pp); break;
            }
            if (have) coop::write_out(I.dst, bc3, b, blk);
            __syncwarp();
        }
    }
}
