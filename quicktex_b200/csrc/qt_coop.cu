// qt_coop.cu — the warp-cooperative BC1/BC3 encoder's kernels (qt_bc1_coop.cuh) and launchers. A unit of its own: its texel
// rows are a bank apart, which the one-block-per-lane kernels do without (level 0 at 4096^2 measured 188 us against 200
// with them).
#define QT_TEXEL_PAD 1
#define QT_PHASE static

#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "qt_coop.h"
#include "qt_device.cuh"

namespace qtk {

#include "qt_bc1_thread.cuh"
#include "qt_bc1_coop.cuh"

// Whether a texture of n blocks runs the warp-cooperative cluster fit and search (qt_bc1_coop.cuh): only settings with
// the Full error mode and EndpointSearch (levels 13-19), and by what one block per lane would make of the
// texture. Below ~75k blocks (a lane each) that mapping takes the time of one block's chain of trials whatever
// n is, and the cooperative one is faster the longer the chain: four-colour Ideal, level 13 at 128^2 44 -> 25 us, 256^2 43 -> 41,
// 384^2 44 -> 46; level 15 at 256^2 60 -> 43, 512^2 69 -> 68, 768^2 80 -> 99; level 18 at 128^2 228 -> 46, 512^2 245 -> 106. On full lanes
// it wins where a pass has enough trials to pay for a block's fixed part (~110 warp instructions a pass): level 16 at 1536^2
// 435 -> 363 us, 2048^2 753 -> 746 (three-colour), 3000^2 1123 -> 1195; level 17 at 2048^2 792 -> 642, 3000^2 1704 -> 1744
// (three-colour + black, AMD); level 18 at 4096^2 3693 -> 3226. Nvidia's palettes cost more to form and its searches
// improve more often, so its lines lie lower: level 17 at 512^2 186 -> 157, 768^2 231 -> 257; level 18 at 768^2 316 -> 289, 1536^2 1345 ->
// 1343 (three-colour + black), 3000^2 2179 -> 2231.
// The deferred path (defer_min blocks and more) has no cooperative kernels for Nvidia: its first line, whatever the device's size.
extern "C" int qtk_coop_rule(const qt_bc1_params *p, long n, long defer_min) {
    if (p->error_mode != EM_FULL || p->search_rounds == 0) return false;
    const unsigned trials = (p->exhaustive ? 969u : p->orderings4) * (p->two_cf_passes ? 2u : 1u);
    const bool nvidia = p->interpolator == IT_NVIDIA;
    if (nvidia && n >= defer_min) return false;
    if (trials >= 200) return true;
    if (trials >= 100) return n <= (nvidia ? 20000 : 400000);
    if (trials >= 72) return nvidia ? n <= 16384 : n < defer_min;
    if (trials >= 48) return n <= (nvidia ? 9216 : 16384);
    return n <= (nvidia ? 3000 : 5000);
}
bool coop_setting(const qt_bc1_params &p, long n) { return qtk_coop_rule(&p, n, defer_min_blocks()); }

// The same for a texture of a batch, which shares full lanes with the others, and whose alternative (k_batch) runs the
// second pass and the search on the lanes that need them.
bool coop_batch_setting(const qt_bc1_params &p) {
    if (p.error_mode != EM_FULL || p.search_rounds == 0) return false;
    const unsigned trials = (p.exhaustive ? 969u : p.orderings4) * (p.two_cf_passes ? 2u : 1u);
    return trials >= (p.interpolator == IT_NVIDIA ? 200u : 72u);
}

// Lets a cooperative kernel have its dynamic shared memory (above 48 KB with the static part); once per
// kernel and device.
template <typename K> static cudaError_t allow_smem(K kernel, size_t bytes, std::atomic<uint64_t> &done) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return e;
}

constexpr int kCoopCtas = 4;  // resident CTAs per SM (launch bounds; 51 KB of shared memory each)

// as many blocks per warp as leave every resident warp the same share
template <int IT>
static cudaError_t launch_coop(cudaStream_t s, const uint8_t *rgba, int w, int h, long b0, long n, const qt_bc1_params &p, uint8_t *out, bool bc3,
                               int aligned, const uint32_t *list, const uint32_t *count) {
    static std::atomic<uint64_t> done{0};
    const cudaError_t e = allow_smem(k_bc1_coop<IT>, coop::kFitSmem, done);
    if (e != cudaSuccess) return e;
    const long resident = (long)num_sms() * kCoopCtas * coop::kWarps;
    const long rounds = (n + resident * 32 - 1) / (resident * 32);
    const int per = (int)std::min<long>(32, (n + resident * rounds - 1) / (resident * rounds));
    const long ctas = (n + (long)per * coop::kWarps - 1) / ((long)per * coop::kWarps);
    const int g = (int)std::min<long>(ctas, resident / coop::kWarps);
    k_bc1_coop<IT><<<g, tpb::kThreads, coop::kFitSmem, s>>>(rgba, w, h, (w + 3) / 4, b0, b0 + n, p, out, bc3, aligned, list, count, per);
    return cudaGetLastError();
}

cudaError_t coop_encode(const uint8_t *rgba, int w, int h, long b0, long n, const qt_bc1_params &p, uint8_t *out, bool bc3, int aligned,
                        const uint32_t *list, const uint32_t *count, cudaStream_t s) {
    switch (p.interpolator) {
        case IT_IDEAL: return launch_coop<IT_IDEAL>(s, rgba, w, h, b0, n, p, out, bc3, aligned, list, count);
        case IT_ROUND: return launch_coop<IT_ROUND>(s, rgba, w, h, b0, n, p, out, bc3, aligned, list, count);
        case IT_NVIDIA: return launch_coop<IT_NVIDIA>(s, rgba, w, h, b0, n, p, out, bc3, aligned, list, count);
        default: return launch_coop<IT_AMD>(s, rgba, w, h, b0, n, p, out, bc3, aligned, list, count);
    }
}

// (never Nvidia: qtk_coop_rule)
template <typename F> static void by_coop_interp(int interpolator, F &&f) {
    switch (interpolator) {
        case IT_IDEAL: f(std::integral_constant<int, IT_IDEAL>()); break;
        case IT_ROUND: f(std::integral_constant<int, IT_ROUND>()); break;
        default: f(std::integral_constant<int, IT_AMD>()); break;
    }
}

void coop_defer(const uint8_t *rgba, int w, int h, const qt_bc1_params &p, uint8_t *out, bool bc3, int aligned, long n,
                const uint32_t *list, const uint32_t *count, const DeferQueues &d, cudaStream_t s) {
    by_coop_interp(p.interpolator, [&](auto I) {
        constexpr int IT = decltype(I)::value;
        static std::atomic<uint64_t> done{0};
        if (allow_smem(k_bc1_coop_defer<IT>, coop::kFitSmem, done) != cudaSuccess) return;
        const long ctas = (n + tpb::kThreads - 1) / tpb::kThreads;
        const int g = (int)std::min<long>(ctas, (long)num_sms() * kCoopCtas);
        k_bc1_coop_defer<IT><<<g, tpb::kThreads, coop::kFitSmem, s>>>(rgba, w, h, (w + 3) / 4, p, out, bc3, aligned, list, count, d.q, d.c);
    });
}

void coop_defer_rest(const uint8_t *rgba, int w, int h, const qt_bc1_params &p, uint8_t *out, bool bc3, int aligned,
                     const DeferQueues &d, bool cf2, cudaStream_t s) {
    by_coop_interp(p.interpolator, [&](auto I) {
        constexpr int IT = decltype(I)::value;
        static std::atomic<uint64_t> done{0};
        if (allow_smem(k_bc1_coop_cf2<IT>, coop::kFitSmem, done) != cudaSuccess) return;
        const int bw = (w + 3) / 4;
        if (cf2) k_bc1_coop_cf2<IT><<<num_sms() * kCoopCtas, tpb::kThreads, coop::kFitSmem, s>>>(rgba, w, h, bw, p, out, bc3, aligned, d.c, d.q);
        k_bc1_coop_search<IT><<<num_sms() * kCoopSearchCtas, tpb::kThreads, coop::kSearchSmem, s>>>(rgba, w, h, bw, p, out, bc3, aligned, d.q, d.fq);
    });
}

int batch_coop_launch(BatchLaunch *l, int *resident) {
    static std::atomic<uint64_t> done{0};
    const cudaError_t e = allow_smem(k_batch_coop, coop::kFitSmem, done);
    if (e != cudaSuccess) return (int)e;
    l->func = (const void *)k_batch_coop;
    l->smem = coop::kFitSmem;
    *resident = kCoopCtas;
    return 0;
}

cudaError_t upload_coop_tables() { return cudaMemcpyToSymbol(g_tab, &host_tables(), sizeof(DevTables)); }

}  // namespace qtk
