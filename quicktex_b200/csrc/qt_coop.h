// qt_coop.h — the queues of the deferred BC1/BC3 path and the launchers of the warp-cooperative encoder (qt_coop.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "qt_internal.h"

namespace qtk {

struct SearchQueues {
    uint32_t *count;  // [3] entries per queue
    uint32_t *head;   // [3] next entry to take
    uint32_t *b, *lohi, *err, *sel, *mode;  // [3][cap] each
    long cap;
};

// Searches that moved the endpoints, finished by k_bc1_finish: the block, its final endpoints
// and colour mode. The reference keeps the selectors of the last accepted trial, which
// FindSelectors computed from those endpoints (BC1Encoder.cpp:974-990); the search rounds here
// compute errors only, so the selectors are computed once at the end. Done inside the refill loop,
// that would run with one lane of the warp active.
struct FinishQueue {
    uint32_t *count;
    uint32_t *b, *lohi, *mode;  // [cap] each
};

// Blocks whose EncodeBlock continues in k_bc1_cf2 after the first four-colour cluster-fit
// pass (one entry per block: its index, the result after the first pass, the endpoints
// before refinement). Entries that run the second pass fill the arrays from the front,
// entries that only run the 3-colour trials from the back, so warps of k_bc1_cf2 see one
// kind.
struct Cf2Queue {
    uint32_t *count;  // [2]: second-pass entries, 3-colour-only entries
    uint32_t *b, *lohi, *err, *sel, *mode, *orig;  // [cap] each
    long cap;
};

struct DeferQueues {
    SearchQueues q;
    FinishQueue fq;
    Cf2Queue c;
};

int num_sms();
long defer_min_blocks();

bool coop_setting(const qt_bc1_params &p, long n);
cudaError_t upload_coop_tables();
// EncodeBlock of n blocks [b0, b0 + n) or, with list, of the *count <= n listed ones
cudaError_t coop_encode(const uint8_t *rgba, int w, int h, long b0, long n, const qt_bc1_params &p, uint8_t *out, bool bc3, int aligned,
                        const uint32_t *list, const uint32_t *count, cudaStream_t s);
// The deferred path's first pass over a list of at most n blocks, and its passes over the queues up to the searches (the
// caller finishes those that moved). Not with Nvidia's interpolation. A failure is the last CUDA error.
void coop_defer(const uint8_t *rgba, int w, int h, const qt_bc1_params &p, uint8_t *out, bool bc3, int aligned, long n,
                const uint32_t *list, const uint32_t *count, const DeferQueues &d, cudaStream_t s);
void coop_defer_rest(const uint8_t *rgba, int w, int h, const qt_bc1_params &p, uint8_t *out, bool bc3, int aligned,
                     const DeferQueues &d, bool cf2, cudaStream_t s);

}  // namespace qtk
