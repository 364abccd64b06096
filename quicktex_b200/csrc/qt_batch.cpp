// qt_batch.cpp — host side of the batched persistent path (qt_batch_* in
// include/quicktex_cuda.h).
//
// A qt_batch owns, per device: the device work queue (texture descriptors,
// tiles, and a control block: head and end of each kernel's range of tiles),
// pinned host staging for it, and a CUDA graph holding the persistent launch. Every qt_batch_run cuts the textures into tiles (tile size per
// format/level from the tuning rules), orders the tiles by estimated cost,
// heaviest first (so the long tiles start early and the cheap ones fill the
// tail), uploads the queue, and replays the graph. BC1/BC3 encodes go to kernels
// of their own beside k_batch, in the same graph: the cooperative encoder
// (levels 16-19) and encoders specialised by interpolator, error mode and
// colour mode. The one graph holds a node for each kernel that a run has needed so far; a run
// switches its own on and the others off.
// It is built again when a run needs a kernel that it lacks, or a queue buffer has to grow.

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include <cuda_runtime.h>

#include "qt_internal.h"

namespace {

constexpr int kLevels = 20;
int fmt_index(int fmt) { return fmt == 1 ? 0 : fmt == 3 ? 1 : fmt == 4 ? 2 : fmt == 5 ? 3 : -1; }
int rule_index(int op, int fmt, int level) {
    const int l = (op == QT_OP_ENCODE && (fmt == 1 || fmt == 3)) ? std::min(std::max(level, 0), kLevels - 1) : 0;
    return (op * 4 + fmt_index(fmt)) * kLevels + l;
}

struct Rule {
    uint32_t tile_blocks;
    float cost;
};

// The preset level whose settings these are (exact match on the fields a
// level sets), else the preset closest in cluster-fit orderings and search
// rounds; used only to pick a tuning rule.
int qtk_level_of(const qt_bc1_params &p) {
    int best = 0;
    long best_d = -1;
    for (int l = 0; l < kLevels; l++) {
        qt_bc1_params q;
        if (qt_bc1_params_for_level((unsigned)l, QT_COLOR_FOUR, 0, &q) != QT_OK) continue;
        if (q.error_mode == p.error_mode && q.endpoint_mode == p.endpoint_mode && q.two_ls_passes == p.two_ls_passes &&
            q.two_ep_passes == p.two_ep_passes && q.two_cf_passes == p.two_cf_passes && q.exhaustive == p.exhaustive &&
            q.search_rounds == p.search_rounds && q.orderings4 == p.orderings4 && q.orderings3 == p.orderings3 &&
            q.power_iterations == p.power_iterations)
            return l;
        const long d = std::labs((long)q.orderings4 * (q.two_cf_passes ? 2 : 1) - (long)p.orderings4 * (p.two_cf_passes ? 2 : 1)) +
                       std::labs((long)q.search_rounds - (long)p.search_rounds) / 4;
        if (best_d < 0 || d < best_d) {
            best_d = d;
            best = l;
        }
    }
    return p.exhaustive ? 19 : best;
}

}  // namespace

struct qt_batch {
    int device = 0;
    std::mutex mu;
    Rule rules[2 * 4 * kLevels];
    int ctas_per_sm = 0;
    int threads = 128;  // per CTA of the persistent kernel
    size_t cap_items = 0, cap_tiles = 0, last_tiles = 0;
    qtk::BatchItemDev *d_items = nullptr, *h_items = nullptr;
    qtk::TileDev *d_tiles = nullptr, *h_tiles = nullptr;
    uint32_t *d_ctl = nullptr, *h_ctl = nullptr;
    cudaEvent_t staged = nullptr;     // the last upload from the pinned staging buffers
    cudaEvent_t done = nullptr;       // the last persistent launch (the queue is in use until then)
    cudaGraph_t graph = nullptr;      // the kernels of `built` (bit k: kind k), side by side
    cudaGraphExec_t exec = nullptr;
    cudaGraphNode_t node[qtk::kBatchKinds] = {};
    uint32_t built = 0, enabled = 0;  // the graph's kernels, and those that the next replay runs
    size_t graphs = 0;                // built so far

    qt_batch() {
        for (int op = 0; op < 2; op++)
            for (int f : {1, 3, 4, 5})
                for (int l = 0; l < kLevels; l++) {
                    Rule &r = rules[rule_index(op, f, l)];
                    // a warp takes one tile; tiles are multiples of its 32 lanes
                    if (op == QT_OP_DECODE) {
                        r = {2048, 0.05f};
                    } else if (f == 4 || f == 5) {
                        r = {2048, 0.1f};
                    } else {  // BC1 / BC3 encode: cost grows steeply with the level's cluster fit and search
                        const float c = l >= 17 ? 25.f : l >= 13 ? 15.f : l >= 9 ? 4.f : l >= 7 ? 2.f : l >= 1 ? 1.5f : 1.f;
                        r = {l >= 13 ? 32u : l >= 7 ? 64u : 256u, c + (f == 3 ? 0.1f : 0.f)};
                    }
                }
    }
};

namespace {

constexpr size_t kMinTiles = 16384;  // the queue's smallest capacity

// Warps that the kernels keep resident, and the most tiles that cutting a run finer than its rules (qt_batch_run) can add
int resident_warps() { return qtk::batch_sms() * 16; }
size_t finer_tiles(size_t items) { return 2 * (size_t)resident_warps() + items; }

constexpr size_t kCtlBytes = 2 * qtk::kBatchKinds * sizeof(uint32_t);

// (nodes stay enabled in a replay that was launched before; the executable goes once that has run)
void drop_graph(qt_batch *b) {
    if (b->exec) {
        cudaEventSynchronize(b->done);
        cudaGraphExecDestroy(b->exec);
    }
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
    b->built = b->enabled = 0;
}

void free_buffers(qt_batch *b) {
    drop_graph(b);
    cudaFree(b->d_items);
    cudaFree(b->d_tiles);
    cudaFreeHost(b->h_items);
    cudaFreeHost(b->h_tiles);
    b->d_items = b->h_items = nullptr;
    b->d_tiles = b->h_tiles = nullptr;
    b->cap_items = b->cap_tiles = 0;
}

int grow(qt_batch *b, size_t items, size_t tiles) {
    if (items <= b->cap_items && tiles <= b->cap_tiles && b->d_items) return QT_OK;
    if (b->staged) cudaEventSynchronize(b->staged);
    cudaDeviceSynchronize();  // the old queue may still be read by a running launch
    const size_t ni = std::max(items, std::max<size_t>(b->cap_items * 2, 64));
    const size_t nt = std::max(tiles, std::max<size_t>(b->cap_tiles * 2, kMinTiles));
    free_buffers(b);
    cudaError_t e;
    if ((e = cudaMalloc(&b->d_items, ni * sizeof(qtk::BatchItemDev))) != cudaSuccess ||
        (e = cudaMalloc(&b->d_tiles, nt * sizeof(qtk::TileDev))) != cudaSuccess ||
        (e = cudaHostAlloc((void **)&b->h_items, ni * sizeof(qtk::BatchItemDev), cudaHostAllocDefault)) != cudaSuccess ||
        (e = cudaHostAlloc((void **)&b->h_tiles, nt * sizeof(qtk::TileDev), cudaHostAllocDefault)) != cudaSuccess) {
        free_buffers(b);
        cudaGetLastError();
        return qtk::cuda_error((int)e, "allocating the batch queue");
    }
    b->cap_items = ni;
    b->cap_tiles = nt;
    return QT_OK;
}

// Builds the graph of the kernels of `kinds` (replays read the queue through fixed pointers): side by side, or one after the
// other where the caller limited the grid, so that the batch holds no more of an SM at any time.
int build_graph(qt_batch *b, uint32_t kinds) {
    drop_graph(b);
    const bool chain = qtk::batch_limited(b->ctas_per_sm, b->threads);
    int before = -1;
    cudaError_t e = cudaGraphCreate(&b->graph, 0);
    for (int k = 0; k < qtk::kBatchKinds && e == cudaSuccess; k++) {
        if (!((kinds >> k) & 1u)) continue;
        qtk::BatchLaunch l;
        if ((e = (cudaError_t)qtk::batch_launch(k, b->ctas_per_sm, b->threads, &l)) != cudaSuccess) break;
        uint32_t *ctl = b->d_ctl + 2 * k;
        void *args[] = {&b->d_items, &b->d_tiles, &ctl};
        cudaKernelNodeParams np = {};
        np.func = const_cast<void *>(l.func);
        np.gridDim = dim3((unsigned)l.grid);
        np.blockDim = dim3((unsigned)l.threads);
        np.sharedMemBytes = (unsigned)l.smem;
        np.kernelParams = args;
        e = cudaGraphAddKernelNode(&b->node[k], b->graph, chain && before >= 0 ? &b->node[before] : nullptr, chain && before >= 0, &np);
        before = k;
        if (e == cudaSuccess && k == 1) {  // its tiles are the long ones: they start first
            cudaLaunchAttributeValue v = {};
            v.priority = -1;
            e = cudaGraphKernelNodeSetAttribute(b->node[k], cudaLaunchAttributePriority, &v);
        }
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&b->exec, b->graph, 0);
    if (e != cudaSuccess) {
        b->exec = nullptr;
        drop_graph(b);
        return qtk::cuda_error((int)e, "building the batch's graph");
    }
    b->built = b->enabled = kinds;
    b->graphs++;
    return QT_OK;
}

// The graph that runs exactly the kernels of `kinds`. One graph with switches, not one per set of kernels: a server's mixes
// form ever new sets, and each would cost an instantiation (~0.2 ms) in a request's path and stay for good. It grows
// by the kernels that runs need, at most kBatchKinds times, and does not start with all of them: 24 switched-off
// kernels cost a run 6-20 us (BC1 level 0 at 64^2 65 -> 79 us, at 2048^2 138 -> 149).
int use_graph(qt_batch *b, uint32_t kinds) {
    if (kinds & ~b->built) {
        if (int rc = build_graph(b, b->built | kinds)) return rc;
    }
    for (uint32_t change = kinds ^ b->enabled; change; change &= change - 1) {
        const int k = __builtin_ctz(change);
        const cudaError_t e = cudaGraphNodeSetEnabled(b->exec, b->node[k], (kinds >> k) & 1u);
        if (e != cudaSuccess) return qtk::cuda_error((int)e, "switching the batch's kernels");
        b->enabled ^= 1u << k;
    }
    return QT_OK;
}

int check_item(const qt_batch_item &it) {
    if (int rc = qtk::check_item_fields(it)) return rc;
    if (!it.src || !it.dst) return qtk::set_error(QT_ERR_ARG, "batch item: NULL buffer");
    const size_t bsz = (it.format == 3 || it.format == 5) ? 16 : 8;
    const size_t a_src = it.op == QT_OP_ENCODE ? 4 : bsz, a_dst = it.op == QT_OP_ENCODE ? bsz : 4;
    if (reinterpret_cast<uintptr_t>(it.src) % a_src || reinterpret_cast<uintptr_t>(it.dst) % a_dst)
        return qtk::set_error(QT_ERR_ARG, "batch item: misaligned buffer");
    return QT_OK;
}

}  // namespace

int qtk::check_item_fields(const qt_batch_item &it) {
    if (it.op != QT_OP_ENCODE && it.op != QT_OP_DECODE) return qtk::set_error(QT_ERR_ARG, "batch item: invalid op");
    if (fmt_index(it.format) < 0) return qtk::set_error(QT_ERR_ARG, "batch item: format must be 1, 3, 4 or 5");
    if (it.width <= 0) return qtk::set_error(QT_ERR_ARG, "Texture width must be greater than 0");
    if (it.height <= 0) return qtk::set_error(QT_ERR_ARG, "Texture height must be greater than 0");
    if (it.chan0 < 0 || it.chan0 > 3 || it.chan1 < 0 || it.chan1 > 3) return qtk::set_error(QT_ERR_ARG, "Channel out of range");
    if (it.op == QT_OP_DECODE && (it.interpolator < 0 || it.interpolator > 3))
        return qtk::set_error(QT_ERR_ARG, "Invalid interpolator type");
    if (it.op == QT_OP_ENCODE && (it.format == 1 || it.format == 3)) return qtk::check_bc1_params(&it.params, it.format == 3);
    return QT_OK;
}

extern "C" size_t qtk_batch_graphs(const qt_batch *b) { return b->graphs; }
extern "C" size_t qtk_batch_kernels(const qt_batch *b, unsigned *ctas, unsigned *threads) {
    size_t n = 0;
    for (uint32_t left = b->enabled; left; left &= left - 1) {
        cudaKernelNodeParams np = {};
        if (cudaGraphKernelNodeGetParams(b->node[__builtin_ctz(left)], &np) != cudaSuccess) return 0;
        ctas[n] = np.gridDim.x;
        threads[n++] = np.blockDim.x;
    }
    return n;
}
extern "C" size_t qtk_batch_edges(const qt_batch *b) {
    size_t n = 0;
    if (b->graph) cudaGraphGetEdges(b->graph, nullptr, nullptr, &n);
    return n;
}

extern "C" {

int qt_batch_create(int device, qt_batch **out) {
    if (!out) return qtk::set_error(QT_ERR_ARG, "out is NULL");
    int prev = 0;
    cudaGetDevice(&prev);
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return qtk::cuda_error((int)e, "cudaSetDevice");
    int rc = qtk::ensure_current_device(nullptr);
    qt_batch *b = nullptr;
    if (rc == QT_OK) {
        b = new qt_batch();
        b->device = device;
        if ((e = cudaEventCreateWithFlags(&b->staged, cudaEventDisableTiming)) != cudaSuccess ||
            (e = cudaEventCreateWithFlags(&b->done, cudaEventDisableTiming)) != cudaSuccess ||
            (e = cudaMalloc(&b->d_ctl, kCtlBytes)) != cudaSuccess ||
            (e = cudaHostAlloc((void **)&b->h_ctl, kCtlBytes, cudaHostAllocDefault)) != cudaSuccess) {
            rc = qtk::cuda_error((int)e, "creating a batch");
            qt_batch_destroy(b);
            b = nullptr;
        }
    }
    cudaSetDevice(prev);
    *out = b;
    return rc;
}

int qt_batch_destroy(qt_batch *b) {
    if (!b) return QT_OK;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(b->device);
    cudaDeviceSynchronize();
    free_buffers(b);
    cudaFree(b->d_ctl);
    cudaFreeHost(b->h_ctl);
    if (b->staged) cudaEventDestroy(b->staged);
    if (b->done) cudaEventDestroy(b->done);
    cudaSetDevice(prev);
    delete b;
    return QT_OK;
}

int qt_batch_set_rules(qt_batch *b, const qt_tile_rule *rules, size_t n) {
    if (!b || (n && !rules)) return qtk::set_error(QT_ERR_ARG, "NULL argument");
    std::lock_guard<std::mutex> lk(b->mu);
    for (size_t i = 0; i < n; i++) {
        const qt_tile_rule &r = rules[i];
        if ((r.op != QT_OP_ENCODE && r.op != QT_OP_DECODE) || fmt_index(r.format) < 0 || r.tile_blocks == 0 ||
            !(r.cost_per_block > 0))
            return qtk::set_error(QT_ERR_ARG, "invalid tile rule");
        const bool leveled = r.op == QT_OP_ENCODE && (r.format == 1 || r.format == 3);
        const int l0 = (leveled && r.level >= 0) ? r.level : 0, l1 = (leveled && r.level >= 0) ? r.level : kLevels - 1;
        for (int l = l0; l <= l1; l++) b->rules[rule_index(r.op, r.format, l)] = {r.tile_blocks, r.cost_per_block};
    }
    return QT_OK;
}

int qt_batch_set_grid(qt_batch *b, int ctas_per_sm) {
    if (!b || ctas_per_sm < 0) return qtk::set_error(QT_ERR_ARG, "invalid grid");
    std::lock_guard<std::mutex> lk(b->mu);
    if (ctas_per_sm != b->ctas_per_sm) drop_graph(b);
    b->ctas_per_sm = ctas_per_sm;
    return QT_OK;
}

int qt_batch_set_threads(qt_batch *b, int threads_per_cta) {
    if (!b || (threads_per_cta != 32 && threads_per_cta != 64 && threads_per_cta != 128))
        return qtk::set_error(QT_ERR_ARG, "threads per CTA must be 32, 64 or 128");
    std::lock_guard<std::mutex> lk(b->mu);
    if (threads_per_cta != b->threads) drop_graph(b);
    b->threads = threads_per_cta;
    return QT_OK;
}

size_t qt_batch_last_tiles(const qt_batch *b) { return b ? b->last_tiles : 0; }

int qt_copy_async(const qt_copy *copies, size_t n, void *stream) {
    if (n && !copies) return qtk::set_error(QT_ERR_ARG, "copies is NULL");
    for (size_t i = 0; i < n; i++) {
        if (!copies[i].bytes) continue;
        if (!copies[i].dst || !copies[i].src) return qtk::set_error(QT_ERR_ARG, "qt_copy_async: NULL buffer");
        const cudaError_t e = cudaMemcpyAsync(copies[i].dst, copies[i].src, copies[i].bytes, cudaMemcpyDefault,
                                              (cudaStream_t)stream);
        if (e != cudaSuccess) return qtk::cuda_error((int)e, "qt_copy_async");
    }
    return QT_OK;
}

int qt_batch_reserve(qt_batch *b, size_t items, size_t tiles) {
    if (!b) return qtk::set_error(QT_ERR_ARG, "NULL argument");
    std::lock_guard<std::mutex> lk(b->mu);
    int cur = 0;
    cudaGetDevice(&cur);
    if (cur != b->device) return qtk::set_error(QT_ERR_STATE, "qt_batch_reserve: the batch belongs to another device");
    return grow(b, std::max<size_t>(items, b->cap_items), std::max<size_t>(tiles + finer_tiles(items), b->cap_tiles));
}

int qt_batch_run(qt_batch *b, const qt_batch_item *items, size_t n, void *stream) {
    if (!b || (n && !items)) return qtk::set_error(QT_ERR_ARG, "NULL argument");
    std::lock_guard<std::mutex> lk(b->mu);
    int cur = 0;
    cudaGetDevice(&cur);
    if (cur != b->device) return qtk::set_error(QT_ERR_STATE, "qt_batch_run: the batch belongs to another device");
    if (int rc = qtk::ensure_current_device(nullptr)) return rc;

    // descriptors, and each item's rule and kernel
    std::vector<qtk::BatchItemDev> dev(n);
    struct Plan {
        Rule rule;
        int kind;
    };
    std::vector<Plan> plan(n);
    double work[2] = {0, 0};  // of the kernels that run a block per lane, of the cooperative one
    for (size_t i = 0; i < n; i++) {
        const qt_batch_item &it = items[i];
        if (int rc = check_item(it)) return rc;
        qtk::BatchItemDev &d = dev[i];
        d.src = it.src;
        d.dst = it.dst;
        d.w = it.width;
        d.h = it.height;
        d.bw = (it.width + 3) / 4;
        d.bh = (it.height + 3) / 4;
        d.op = it.op;
        d.fmt = it.format;
        d.c0 = (it.format == 4 || it.format == 5) ? it.chan0 : 0;
        d.c1 = it.format == 5 ? it.chan1 : d.c0;
        d.interp = it.interpolator;
        d.write_alpha = it.write_alpha != 0;
        d.p = it.params;
        const uint64_t nb = (uint64_t)d.bw * d.bh;
        if (nb > 0xFFFFFFFFull) return qtk::set_error(QT_ERR_ARG, "Texture too large");
        const bool leveled = it.op == QT_OP_ENCODE && (it.format == 1 || it.format == 3);
        Plan &pl = plan[i];
        pl.rule = b->rules[rule_index(it.op, it.format, leveled ? qtk_level_of(it.params) : 0)];
        pl.kind = qtk::batch_kind(it.op, it.format, it.params);
        work[pl.kind == 1] += (double)pl.rule.cost * (double)nb;
    }
    // Tiles of the rules' sizes, or smaller where the resident warps would have fewer than one each (a short batch
    // waits for its longest tile): a cooperative warp works on one block at a time, so its tiles may fall to a few
    // blocks; the others keep 32, a block per lane. The cut depends on this run's work alone. One tile per warp, not more: 1 / 2 / 4 of them take
    // 176 / 214 / 322 us for 300 textures up to 256^2 (uncut 388) and 528 / 576 / 802 for 300 up to 1024^2 (uncut 559), where the
    // host makes the tiles and the copy engine moves them. BC1 level 5 at 256^2 121 -> 41 us, its 64^2 chain 112 -> 30,
    // level 18 at 256^2 285 -> 85, 20 mixed textures up to 256^2 363 -> 157, 200 up to 512^2 at levels 0-10 306 -> 149.
    const double warps = resident_warps();
    struct Tile {
        int kind;
        float cost;
        qtk::TileDev t;
    };
    std::vector<Tile> tiles;
    for (size_t i = 0; i < n; i++) {
        const Plan &pl = plan[i];
        const bool coop = pl.kind == 1;
        const uint64_t nb = (uint64_t)dev[i].bw * dev[i].bh;
        uint64_t tb = pl.rule.tile_blocks;
        const double share = work[coop] / warps / pl.rule.cost;  // this texture's blocks in one warp's share of the run
        if (share < (double)tb) {
            const uint64_t fill = (uint64_t)share + 1;
            tb = std::min(tb, coop ? fill : (fill + 31) / 32 * 32);
        }
        for (uint64_t s0 = 0; s0 < nb; s0 += tb) {
            const uint32_t cnt = (uint32_t)std::min<uint64_t>(tb, nb - s0);
            tiles.push_back({pl.kind, pl.rule.cost * cnt, {(uint32_t)i, (uint32_t)s0, cnt, 0u}});
        }
    }
    // each kernel's tiles together, heaviest first
    std::stable_sort(tiles.begin(), tiles.end(), [](const Tile &a, const Tile &c) { return a.kind != c.kind ? a.kind < c.kind : a.cost > c.cost; });
    b->last_tiles = tiles.size();
    if (tiles.size() > 0xFFFFFFFFull) return qtk::set_error(QT_ERR_ARG, "too many tiles");
    if (tiles.empty()) return QT_OK;

    if (int rc = grow(b, n, tiles.size())) return rc;
    cudaError_t e = cudaEventSynchronize(b->staged);  // the staging buffers are free once the last upload ran
    if (e != cudaSuccess) return qtk::cuda_error((int)e, "batch staging");
    std::memcpy(b->h_items, dev.data(), n * sizeof(qtk::BatchItemDev));
    for (size_t i = 0; i < tiles.size(); i++) b->h_tiles[i] = tiles[i].t;
    uint32_t kinds = 0;
    for (size_t i = 0; i < tiles.size(); i++) {
        const int k = tiles[i].kind;
        if (!((kinds >> k) & 1u)) b->h_ctl[2 * k] = (uint32_t)i;
        b->h_ctl[2 * k + 1] = (uint32_t)i + 1;
        kinds |= 1u << k;
    }
    if (int rc = use_graph(b, kinds)) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    // runs on other streams: do not overwrite the queue before the previous launch finished reading it
    if ((e = cudaStreamWaitEvent(s, b->done, 0)) != cudaSuccess) return qtk::cuda_error((int)e, "batch ordering");
    if ((e = cudaMemcpyAsync(b->d_items, b->h_items, n * sizeof(qtk::BatchItemDev), cudaMemcpyHostToDevice, s)) != cudaSuccess ||
        (e = cudaMemcpyAsync(b->d_tiles, b->h_tiles, tiles.size() * sizeof(qtk::TileDev), cudaMemcpyHostToDevice, s)) != cudaSuccess ||
        (e = cudaMemcpyAsync(b->d_ctl, b->h_ctl, kCtlBytes, cudaMemcpyHostToDevice, s)) != cudaSuccess ||
        (e = cudaEventRecord(b->staged, s)) != cudaSuccess)
        return qtk::cuda_error((int)e, "batch upload");

    if ((e = cudaGraphLaunch(b->exec, s)) != cudaSuccess) return qtk::cuda_error((int)e, "graph launch");
    if ((e = cudaEventRecord(b->done, s)) != cudaSuccess) return qtk::cuda_error((int)e, "graph launch");
    return QT_OK;
}

int qt_batch_run_plain(const qt_batch_item *items, size_t n, void *stream) {
    if (n && !items) return qtk::set_error(QT_ERR_ARG, "items is NULL");
    for (size_t i = 0; i < n; i++) {
        const qt_batch_item &it = items[i];
        if (int rc = check_item(it)) return rc;
        const int w = it.width, h = it.height, f = it.format;
        int rc;
        if (it.op == QT_OP_ENCODE) {
            rc = f == 1   ? qt_bc1_encode_device(it.src, w, h, &it.params, it.dst, stream)
                 : f == 3 ? qt_bc3_encode_device(it.src, w, h, &it.params, it.dst, stream)
                 : f == 4 ? qt_bc4_encode_device(it.src, w, h, it.chan0, it.dst, stream)
                          : qt_bc5_encode_device(it.src, w, h, it.chan0, it.chan1, it.dst, stream);
        } else {
            rc = f == 1   ? qt_bc1_decode_device(it.src, w, h, it.interpolator, it.write_alpha, it.dst, stream)
                 : f == 3 ? qt_bc3_decode_device(it.src, w, h, it.interpolator, it.dst, stream)
                 : f == 4 ? qt_bc4_decode_device(it.src, w, h, it.chan0, it.dst, stream)
                          : qt_bc5_decode_device(it.src, w, h, it.chan0, it.chan1, it.dst, stream);
        }
        if (rc) return rc;
    }
    return QT_OK;
}

}  // extern "C"
