// C ABI of the B200 expert-FFN path (declared in include/moexb.h): argument checks, launches, resident layers.
#include "moexb.h"
#include "common.cuh"
#include "router.cuh"
#include "experts_simt.cuh"
#include "formats.cuh"
#include "stream.cuh"
#include "tiled.cuh"
#include "grouped.cuh"
#include "decode_stack.cuh"
#include "ep.cuh"
#include "gguf_ingest.h"
#include "st_ingest.h"
#include "gguf_quant.h"

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <algorithm>
#include <atomic>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

using namespace moexb;

namespace {

thread_local char g_err[512] = "";

int fail(int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof g_err, fmt, ap);
    va_end(ap);
    return code;
}

#define REQUIRE(cond, ...) do { if (!(cond)) return fail(MOEXB_ERR_ARG, __VA_ARGS__); } while (0)
#define CUDA_TRY(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) return fail(MOEXB_ERR_CUDA, "%s: %s", #x, cudaGetErrorString(e_)); } while (0)
#define LAUNCHED(name) do { cudaError_t e_ = cudaGetLastError(); if (e_ != cudaSuccess) return fail(MOEXB_ERR_CUDA, "launch of %s: %s", name, cudaGetErrorString(e_)); \
    g_launches.fetch_add(1, std::memory_order_relaxed); } while (0)
std::atomic<long long> g_launches{0};

inline cudaStream_t S(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Launch with programmatic stream serialization: the kernel's blocks may be scheduled before the kernel ahead of it in
// the stream has finished, and wait for it inside (pdl_wait in common.cuh). Only kernels that call pdl_wait before they
// touch their inputs are launched this way. MOEXB_PDL=0 in the environment turns it off (plain launches).
static bool pdl_enabled() {
    static const bool on = [] { const char* e = getenv("MOEXB_PDL"); return !(e && e[0] == '0'); }();
    return on;
}
// The kernels of a prefill-size batch fill every SM for tens of microseconds, and blocks of the next one that wait inside take the
// place of blocks that could run: such a batch is launched the plain way (2048 tokens: 444 us with programmatic launches, 419 without;
// up to a few hundred tokens it is the other way round).
static thread_local bool t_plain_launches = false;
struct PlainLaunches {
    const bool before = t_plain_launches;
    explicit PlainLaunches(bool on) { t_plain_launches = on; }
    ~PlainLaunches() { t_plain_launches = before; }
};
template <typename... P, typename... A>
static cudaError_t launch_dep(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = pdl_enabled() && !t_plain_launches ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
// Function attributes (the opt-in to more than 48 KB of dynamic shared memory, occupancy figures) belong to one device, so
// "once" means once per device: keyed by the device that is current in the calling thread, which is the one the launch
// that follows goes to.
constexpr int MAX_DEVICES = 64;
struct PerDeviceOnce {
    std::mutex mu;
    bool done[MAX_DEVICES] = {};
    cudaError_t err[MAX_DEVICES] = {};
    template <class F>
    cudaError_t run(F&& f) {
        int dev = -1;
        const cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        if (dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
        std::lock_guard<std::mutex> lock(mu);
        if (!done[dev]) { err[dev] = f(); done[dev] = true; }
        return err[dev];
    }
};
// The opt-in of a kernel to `smem` bytes of dynamic shared memory. Its grid is sized for `ctas` CTAs per SM: kernels of which fewer fit
// are counted (moexb_short_residency); they run, but what does not fit waits for a second wave.
std::atomic<int> g_short_residency{0};
template <typename K>
static cudaError_t opt_in(K* kernel, int threads, int smem, int ctas) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    int fit = 0;
    if (e == cudaSuccess && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kernel, threads, smem) == cudaSuccess && fit < ctas) g_short_residency++;
    return e;
}
inline bool fmt_ok(int fmt) { return fmt == FMT_SYM_F32 || fmt == FMT_SYM_F16 || fmt == FMT_ZP; }

// Calls f.template operator()<FMT>() for the run-time format.
template <class F>
int by_fmt(int fmt, F&& f) {
    switch (fmt) {
        case FMT_SYM_F32: return f.template operator()<FMT_SYM_F32>();
        case FMT_SYM_F16: return f.template operator()<FMT_SYM_F16>();
        case FMT_ZP: return f.template operator()<FMT_ZP>();
    }
    return fail(MOEXB_ERR_ARG, "unknown expert format %d", fmt);
}

// ---- half-normal quantile tables of the synthetic generator ---------------------------------------------------------

float half_to_float_host(uint16_t h) { return __half2float(__ushort_as_half(h)); }

// table[i] = fp16 bits of sigma * q, q = the (i + 0.5) / N quantile of |N(0, 1)|, found by bisection on erf.
void build_table(double sigma, uint16_t* table) {
    for (int i = 0; i < SYNTH_TABLE_N; i++) {
        const double p = (i + 0.5) / SYNTH_TABLE_N;
        double lo = 0, hi = 10;
        for (int it = 0; it < 80; it++) {
            const double mid = 0.5 * (lo + hi);
            if (std::erf(mid / std::sqrt(2.0)) < p) lo = mid; else hi = mid;
        }
        table[i] = __half_as_ushort(__float2half_rn((float)(sigma * 0.5 * (lo + hi))));
    }
}
struct Tables { uint16_t s[SYNTH_TABLE_N], d[SYNTH_TABLE_N]; };
const Tables& host_tables() {
    static Tables t;
    static std::once_flag once;
    std::call_once(once, [] { build_table(0.02, t.s); build_table(0.01, t.d); });
    return t;
}

}  // namespace

constexpr int STAGING_BLOBS = 32;

struct moexb_ctx {
    int device = 0, max_tokens = 0, max_experts = 0, top_k = 0;
    uint16_t *table_s = nullptr, *table_d = nullptr;  // device copies of the synthetic tables
    // workspace of the layer-level calls
    float *xf = nullptr, *xn = nullptr, *logits = nullptr, *w = nullptr, *act = nullptr, *ypair = nullptr, *moe = nullptr;
    int *idx = nullptr, *counts = nullptr, *nitems = nullptr;
    moexb_pair_item* items = nullptr;
    moexb_pair* pairs = nullptr;
    const uint8_t** slots = nullptr;  // decode: K+1 blob pointers
    float* wts = nullptr;             // decode: K+1 weights
    // streaming (tensor-core) path
    uint16_t *xs = nullptr, *act_split = nullptr;       // activations / act as 16-bit hi + lo halves, permuted
    moexb_pair_item* subs = nullptr;                    // sub-items of at most 8 pairs
    int *nsub = nullptr, *err = nullptr;
    float *sx = nullptr, *sx_act = nullptr;             // grouped GEMM, zero point: activation sums per 32-input chunk, of the tokens and of act
    int* bcnt = nullptr; moexb_pair* bpairs = nullptr;  // the work list as buckets (null when they would be too large)
    bool buckets_dirty = false;                         // a call failed between its router and its combine: bcnt may not be zero
    bool selftest_fail = false;                         // the next layer call fails there (moexb_ctx_selftest_fail)
    int* route_done = nullptr;                          // per token tile: blocks of the routing kernel that have finished (returns to zero)
    int sms = 0, path = 0;                              // path: 0 = streaming kernels, 1 = fp32 SIMT kernels
    int fused_decode = 1;                               // one-token residual stacks run as one cooperative launch
    int pairs_per_pass = 8;                             // sub-item width of the tiled streaming kernels from 8 tokens on
    int prefill_min_tokens = 256;                       // batches from this size on use the tcgen05 grouped GEMM
    uint8_t* staging = nullptr;                         // reference-layout blobs on their way into a tiled image
    std::vector<void*> owned;
    // optional per-kernel timing of the layer-level calls
    bool profiling = false;
    struct Rec { int tag; cudaEvent_t a, b; };
    std::vector<Rec> recs;
    std::vector<cudaEvent_t> spare;
};

namespace {
// Brackets the launches made inside its scope with two events on the stream when the context is profiling.
struct ProfScope {
    moexb_ctx* c; cudaStream_t st; cudaEvent_t a = nullptr, b = nullptr; int tag;
    ProfScope(moexb_ctx* c_, int tag_, cudaStream_t st_) : c(c_), st(st_), tag(tag_) {
        if (!c || !c->profiling) return;
        auto get = [&] { cudaEvent_t e; if (c->spare.empty()) cudaEventCreate(&e); else { e = c->spare.back(); c->spare.pop_back(); } return e; };
        a = get(); b = get();
        cudaEventRecord(a, st);
    }
    ~ProfScope() { if (a) { cudaEventRecord(b, st); c->recs.push_back({tag, a, b}); } }
};
}  // namespace

#define PROF_CAT2(a, b) a##b
#define PROF_CAT(a, b) PROF_CAT2(a, b)
#define PROF(ctx, tag, stream) ProfScope PROF_CAT(prof_scope_, __LINE__)(ctx, tag, S(stream))

struct moexb_layer {
    moexb_ctx* ctx = nullptr;
    int fmt = 0, n_routed = 0, first_local = 0, n_local = 0, router_dtype = 0, layout = 0;
    uint8_t* image = nullptr;               // n_local + 1 blobs: the held routed experts, then the shared expert
    void* router = nullptr;                 // [n_routed + 1][H]
    const uint8_t** slot_table = nullptr;   // device, n_routed + 1 pointers
    std::vector<const uint8_t*> slot_host;
    GroupedMaps map_gate_up{}, map_down{};  // the image as the grouped GEMM's copies see it (tiled layout)
    // per expert id (index n_routed = the shared expert): weights were put there by an upload, a synthetic fill or a file load.
    // The image starts zeroed, so an expert that was never loaded contributes zeros; the shared expert runs for every token,
    // so the layer-level calls refuse to run it unloaded instead of silently adding nothing.
    std::vector<uint8_t> loaded;
};

extern "C" {

const char* moexb_last_error(void) { return g_err; }
int moexb_version(void) { return 1; }
size_t moexb_expert_bytes(int fmt) { return fmt_ok(fmt) ? expert_bytes(fmt) : 0; }

// ---- router ------------------------------------------------------------------------------------------------------

}  // extern "C"
template <typename WT>
static int gemv_any(const WT* W, const float* x, float* y, int I, int O, void* stream, int rows) {
    REQUIRE(W && x && y, "gemv: null pointer");
    REQUIRE(I > 0 && I % 128 == 0 && O > 0 && rows > 0, "gemv: I=%d must be a positive multiple of 128, O=%d, rows=%d", I, O, rows);
    // A warp per (row, output) re-reads the weights from L2 for every row; the batched kernel's tiles read them once per 8 rows, but of
    // them a small batch has too few to reach every SM. In a chain of calls (f16 / f32 weights, us): 8 rows 3.1 / 3.2 against 6.0 / 5.7,
    // 14 rows 5.2 / 5.2 against 6.0 / 5.7, 16 rows 5.6 / 5.6 against 6.0 / 5.8, 20 rows 6.6 / 6.8 against 6.0 / 5.8; with weights that
    // come from memory the lines cross at 16 (a chunk of 16 tokens over 2 layers: 187 us against 184).
    constexpr int TR = 8, SMEM_MAX = 200 * 1024;
    const int smem = I <= SMEM_MAX / (TR * (int)sizeof(float)) ? TR * I * (int)sizeof(float) : SMEM_MAX + 1;   // of a tile's rows
    if (rows > 24 || (rows >= 16 && smem <= SMEM_MAX)) {   // (up to 24 rows of any length are taken)
        // Tiles of 16 outputs x 8 rows. Up to one tile per SM the warps are what is short: 8 of 2 outputs each (64 rows of 257 outputs
        // 6.2 / 5.9 us, 10.3 / 7.9 with 4 of 4). Beyond, the reads of the rows from shared memory, which a warp's outputs share (65 rows
        // 11.1 / 10.6 us with 8 of 2, 8.8 / 7.2 with 4 of 4; 256 rows 22.6 / 21.5 and 19.5 / 14.8; 2048 rows 163 / 155 and 102 / 89).
        constexpr int TILE = 16;
        REQUIRE(smem <= SMEM_MAX, "gemv: I=%d is too large for the batched kernel", I);
        const dim3 grid((O + TILE - 1) / TILE, (rows + TR - 1) / TR);
        int dev = 0, sms = 0;
        CUDA_TRY(cudaGetDevice(&dev));
        CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        auto tiles = [&]<int WARPS, int U>() -> int {
            constexpr auto kernel = gemm_rows_k<WT, WARPS, TILE / WARPS, TR, U>;
            static PerDeviceOnce once;
            const cudaError_t attr_err = once.run([] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX); });
            if (attr_err != cudaSuccess) return fail(MOEXB_ERR_CUDA, "gemv: shared memory attribute: %s", cudaGetErrorString(attr_err));
            CUDA_TRY(launch_dep(kernel, grid, WARPS * 32, smem, S(stream), W, x, y, I, O, rows));
            return MOEXB_OK;
        };
        const int rc = (size_t)grid.x * grid.y <= (size_t)sms ? tiles.template operator()<8, 8>() : tiles.template operator()<4, sizeof(WT) == 2 ? 2 : 1>();
        if (rc != MOEXB_OK) return rc;
    } else {
        constexpr int WARPS = 8;
        CUDA_TRY(launch_dep(gemv_rows_k<WT, WARPS>, dim3((O + WARPS - 1) / WARPS, rows), WARPS * 32, 0, S(stream), W, x, y, I, O));
    }
    LAUNCHED("gemv");
    return MOEXB_OK;
}
extern "C" {
int moexb_gemv_f16(const void* W, const float* x, float* y, int I, int O, void* stream, int rows) {
    return gemv_any(static_cast<const __half*>(W), x, y, I, O, stream, rows);
}
int moexb_gemv_f32(const float* W, const float* x, float* y, int I, int O, void* stream, int rows) {
    return gemv_any(W, x, y, I, O, stream, rows);
}

static int topk_launch(const float* logits, int E, int K, int norm, int* idx, float* w, void* stream, int T, int ld,
                       const uint8_t* const* slot_table, const uint8_t** slots_out, float* wts_out,
                       moexb_pair_item* dsubs = nullptr, moexb_pair* dpairs = nullptr, int* dnsub = nullptr) {
    REQUIRE(logits && idx && w, "router_topk: null pointer");
    REQUIRE(E > 0 && E % 32 == 0 && E <= 1024, "router_topk: E=%d must be a multiple of 32 up to 1024", E);
    REQUIRE(K > 0 && K < 32 && K <= E, "router_topk: K=%d out of range", K);
    REQUIRE(T > 0 && ld >= E, "router_topk: T=%d, ld=%d", T, ld);
    constexpr int WARPS = 2;
    const TopkOut o{idx, w, slot_table, slots_out, wts_out, dsubs, dpairs, dnsub};
    if (E <= 256) CUDA_TRY(launch_dep(router_topk_k<WARPS, 8>, (T + WARPS - 1) / WARPS, WARPS * 32, 0, S(stream), logits, E, K, norm, ld, T, o));
    else CUDA_TRY(launch_dep(router_topk_k<WARPS, 32>, (T + WARPS - 1) / WARPS, WARPS * 32, 0, S(stream), logits, E, K, norm, ld, T, o));
    LAUNCHED("router_topk");
    return MOEXB_OK;
}
int moexb_router_topk(const float* logits, int E, int K, int norm, int* idx, float* w, void* stream, int T, int ld) {
    return topk_launch(logits, E, K, norm, idx, w, stream, T, ld, nullptr, nullptr, nullptr);
}

// ---- routed experts ------------------------------------------------------------------------------------------------

static int decode_launch(moexb_ctx* prof, int fmt, const uint8_t* const* slots, const float* w, int K, const float* x, float* act,
                         float* out, void* stream, const int* nh) {
    REQUIRE(slots && w && x && act && out, "experts_forward: null pointer");
    REQUIRE(K > 0 && K <= 16, "experts_forward: K=%d out of range 1..16", K);
    return by_fmt(fmt, [&]<int FMT>() {
        constexpr int WARPS = 8;
        {
            PROF(prof, MOEXB_PROF_GATE_UP, stream);
            decode_gate_up_k<FMT, WARPS><<<dim3(EI / WARPS, K), WARPS * 32, 0, S(stream)>>>(slots, K, nh, x, act);
            LAUNCHED("decode_gate_up");
        }
        PROF(prof, MOEXB_PROF_DOWN, stream);
        decode_down_k<FMT, WARPS, 16><<<EH / WARPS, WARPS * 32, K * pad32_size(EI) * sizeof(float), S(stream)>>>(slots, w, K, nh, act, out);
        LAUNCHED("decode_down");
        return (int)MOEXB_OK;
    });
}
}  // extern "C"

// The context whose workspace the pointer-level one-token entry point may use on each device (moexb_set_default_ctx).
static std::mutex g_default_lock;
static moexb_ctx* g_default_ctx[MAX_DEVICES] = {};
static int stream_experts(moexb_ctx* c, int fmt, const moexb_pair* pairs, float* act32, float* ypair, int npairs, void* stream);
static int split_launch(moexb_ctx* c, const float* x, int rows, void* stream, const SidePlan& plan);

extern "C" {

int moexb_set_default_ctx(moexb_ctx* ctx, int device) {
    REQUIRE(device >= 0 && device < MAX_DEVICES, "set_default_ctx: device %d", device);
    REQUIRE(!ctx || ctx->device == device, "set_default_ctx: the context belongs to device %d", ctx ? ctx->device : -1);
    std::lock_guard<std::mutex> lock(g_default_lock);
    g_default_ctx[device] = ctx;
    return MOEXB_OK;
}

int moexb_experts_forward(int fmt, const uint8_t* const* slots, const float* w, int K, const float* x, float* act,
                          float* out, void* stream, const int* nh) {
    moexb_ctx* c = nullptr;
    {
        int dev = -1;
        if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < MAX_DEVICES) { std::lock_guard<std::mutex> lock(g_default_lock); c = g_default_ctx[dev]; }
    }
    if (!c || c->path == 1 || K > c->max_tokens * (c->top_k + 1)) return decode_launch(nullptr, fmt, slots, w, K, x, act, out, stream, nh);
    // With a default context: the streaming tensor-core kernels on the caller's reference-layout blobs. The K experts are K
    // one-pair sub-items of the one token; act receives the fp32 activations as the reference's scratch does.
    REQUIRE(slots && w && x && act && out, "experts_forward: null pointer");
    REQUIRE(K > 0 && K <= 16, "experts_forward: K=%d out of range 1..16", K);
    REQUIRE(fmt_ok(fmt), "experts_forward: unknown expert format %d", fmt);
    cudaStream_t st = S(stream);
    SidePlan plan{};
    plan.slots = slots; plan.w = w; plan.K = K; plan.nh = nh; plan.subs = c->subs; plan.pairs = c->pairs; plan.nsub = c->nsub;
    int rc = split_launch(c, x, 1, stream, plan);
    if (rc != MOEXB_OK) return rc;
    if (nh) CUDA_TRY(cudaMemsetAsync(c->ypair, 0, (size_t)K * EH * sizeof(float), st));   // rows of the experts beyond *nh stay zero
    rc = stream_experts(c, fmt, c->pairs, act, c->ypair, K, stream);
    if (rc != MOEXB_OK) return rc;
    CUDA_TRY(launch_dep(pairs_reduce_k, dim3((EH / 4 + 255) / 256, 1), 256, 0, st, (const float*)c->ypair, (const float*)nullptr, out, K, EH, (const int*)nullptr));
    LAUNCHED("pairs_reduce");
    return MOEXB_OK;
}

static int pairs_launch(moexb_ctx* prof, int fmt, const moexb_pair_item* items, const int* nitems, int grid_items, const moexb_pair* pairs,
                        const float* X, float* act, float* ypair, void* stream) {
    REQUIRE(items && pairs && X && act && ypair, "pairs_forward: null pointer");
    REQUIRE(grid_items > 0 && grid_items <= 65535, "pairs_forward: %d items", grid_items);
    return by_fmt(fmt, [&]<int FMT>() {
        constexpr int WARPS = 8;
        {
            PROF(prof, MOEXB_PROF_GATE_UP, stream);
            pairs_gate_up_k<FMT, WARPS><<<dim3(EI / WARPS, grid_items), WARPS * 32, 0, S(stream)>>>(items, pairs, X, act, nitems);
            LAUNCHED("pairs_gate_up");
        }
        PROF(prof, MOEXB_PROF_DOWN, stream);
        pairs_down_k<FMT, WARPS><<<dim3(EH / WARPS, grid_items), WARPS * 32, 0, S(stream)>>>(items, pairs, act, ypair, nitems);
        LAUNCHED("pairs_down");
        return (int)MOEXB_OK;
    });
}
int moexb_pairs_forward(int fmt, const moexb_pair_item* items, int n_items, const moexb_pair* pairs, const float* X,
                        float* act, float* ypair, void* stream) {
    if (n_items == 0) return fmt_ok(fmt) ? MOEXB_OK : fail(MOEXB_ERR_ARG, "unknown expert format %d", fmt);
    return pairs_launch(nullptr, fmt, items, nullptr, n_items, pairs, X, act, ypair, stream);
}
int moexb_pairs_forward_dev(int fmt, const moexb_pair_item* items, const int* nitems, int max_items,
                            const moexb_pair* pairs, const float* X, float* act, float* ypair, void* stream) {
    REQUIRE(nitems, "pairs_forward_dev: null item count");
    return pairs_launch(nullptr, fmt, items, nitems, max_items, pairs, X, act, ypair, stream);
}

int moexb_pairs_reduce(const float* ypair, const float* ycpu, float* moe, int K, int D, int T, const int* use_cpu, void* stream) {
    REQUIRE(ypair && moe, "pairs_reduce: null pointer");
    REQUIRE(K > 0 && D > 0 && D % 4 == 0 && T > 0 && T <= 65535, "pairs_reduce: K=%d D=%d T=%d", K, D, T);
    CUDA_TRY(launch_dep(pairs_reduce_k, dim3((D / 4 + 255) / 256, T), 256, 0, S(stream), ypair, ycpu, moe, K, D, use_cpu));
    LAUNCHED("pairs_reduce");
    return MOEXB_OK;
}

int moexb_gated_add_rows(float* out, const float* sh, const float* gl, int gl_stride, int D, int T, void* stream) {
    REQUIRE(out && sh && gl, "gated_add_rows: null pointer");
    REQUIRE(D > 0 && T > 0 && T <= 65535 && gl_stride >= 0, "gated_add_rows: D=%d T=%d", D, T);
    gated_add_rows_k<<<dim3((D + 255) / 256, T), 256, 0, S(stream)>>>(out, sh, gl, gl_stride, D);
    LAUNCHED("gated_add_rows");
    return MOEXB_OK;
}

int moexb_group_pairs(const int* idx, const float* w, int T, int K, int E, const uint8_t* const* slot_table,
                      moexb_pair_item* items, moexb_pair* pairs, int* nitems, int* counts, void* stream) {
    REQUIRE(idx && w && slot_table && items && pairs && nitems && counts, "group_pairs: null pointer");
    REQUIRE(T > 0 && K > 0 && E > 0 && E <= 1024, "group_pairs: T=%d K=%d E=%d", T, K, E);
    CUDA_TRY(launch_dep(group_pairs_k, 1, 1024, 0, S(stream), idx, w, T, K, E, slot_table, items, pairs, nitems));
    LAUNCHED("group_pairs");
    return MOEXB_OK;
}

int moexb_shared_expert_add(int fmt, const uint8_t* blob, const float* gl, int gl_stride, const float* X, int T,
                            float* out, float* scratch, void* stream) {
    REQUIRE(blob && gl && X && out && scratch, "shared_expert_add: null pointer");
    REQUIRE(T > 0 && T <= 65535, "shared_expert_add: T=%d", T);
    // scratch: act [T][I]
    return by_fmt(fmt, [&]<int FMT>() {
        constexpr int WARPS = 8;
        const unsigned ty = (unsigned)((T + SH_T - 1) / SH_T);
        CUDA_TRY(launch_dep(shared_gate_up_k<FMT, WARPS>, dim3(EI / WARPS, ty), WARPS * 32, 0, S(stream), blob, X, scratch, T));
        LAUNCHED("shared_gate_up");
        CUDA_TRY(launch_dep(shared_down_k<FMT, WARPS>, dim3(EH / WARPS, ty), WARPS * 32, 0, S(stream), blob, (const float*)scratch, gl, gl_stride, out, T));
        LAUNCHED("shared_down");
        return (int)MOEXB_OK;
    });
}

// ---- formats ---------------------------------------------------------------------------------------------------------

int moexb_dequant(int fmt, const uint8_t* blob, float* out, void* stream) {
    REQUIRE(blob && out, "dequant: null pointer");
    return by_fmt(fmt, [&]<int FMT>() {
        dequant_k<FMT><<<(unsigned)((CHUNKS + 255) / 256), 256, 0, S(stream)>>>(blob, out);
        LAUNCHED("dequant");
        return (int)MOEXB_OK;
    });
}

int moexb_q4k_dequant(const uint8_t* blocks, long long n, float* y, void* stream) {
    REQUIRE(blocks && y, "q4k_dequant: null pointer");
    REQUIRE(n > 0 && n % 256 == 0, "q4k_dequant: n=%lld must be a positive multiple of 256", n);
    const long long threads = n / 256 * 4;
    q4k_dequant_k<<<(unsigned)((threads + 255) / 256), 256, 0, S(stream)>>>(blocks, n / 256, y);
    LAUNCHED("q4k_dequant");
    return MOEXB_OK;
}

int moexb_q4k_to_zp(const uint8_t* gate, const uint8_t* up, const uint8_t* down, uint8_t* blob, void* stream) {
    REQUIRE(gate && up && down && blob, "q4k_to_zp: null pointer");
    q4k_to_zp_k<<<(unsigned)((CHUNKS / 8 + 127) / 128), 128, 0, S(stream)>>>(gate, up, down, blob);
    LAUNCHED("q4k_to_zp");
    return MOEXB_OK;
}

// ---- synthetic experts --------------------------------------------------------------------------------------------------

static int synth_launch(int fmt, unsigned seed, int layer, int e0, int n, uint8_t* dst, const uint16_t* ts, const uint16_t* td, void* stream) {
    REQUIRE(dst && ts && td, "synth_experts: null pointer");
    REQUIRE(n > 0 && n <= 65535 && e0 >= 0 && layer >= 0, "synth_experts: layer=%d e0=%d n=%d", layer, e0, n);
    return by_fmt(fmt, [&]<int FMT>() {
        const size_t work = FMT == FMT_ZP ? CHUNKS / 8 : Q_BYTES / 4;
        synth_experts_k<FMT><<<dim3((unsigned)((work + 255) / 256), n), 256, 0, S(stream)>>>(seed, layer, e0, dst, ts, td);
        LAUNCHED("synth_experts");
        return (int)MOEXB_OK;
    });
}

int moexb_synth_expert_host(int fmt, unsigned seed, int layer, int expert, uint8_t* dst) {
    REQUIRE(dst && fmt_ok(fmt), "synth_expert_host: bad argument");
    const Tables& t = host_tables();
    if (fmt == FMT_ZP) {
        for (size_t sb = 0; sb < CHUNKS / 8; sb++) {
            uint8_t blk[144], *qb, *cs, *sup;
            synth_q4k_block(seed, layer, expert, sb, t.d, blk);
            zp_block_dst(dst, sb, qb, cs, sup);
            q4k_block_to_zp(blk, qb, cs, sup);
        }
        return MOEXB_OK;
    }
    for (size_t i = 0; i < Q_BYTES / 4; i++) {
        const uint32_t w = synth_nibble_word(seed, layer, expert, i);
        memcpy(dst + 4 * i, &w, 4);
    }
    for (size_t g = 0; g < CHUNKS / 2; g++) {
        const uint16_t h = synth_scale_h(seed, layer, expert, g, t.s);
        if (fmt == FMT_SYM_F16) memcpy(dst + Q_BYTES + 2 * g, &h, 2);
        else { const float f = half_to_float_host(h); memcpy(dst + Q_BYTES + 4 * g, &f, 4); }
    }
    return MOEXB_OK;
}

int moexb_synth_q4k_host(unsigned seed, int layer, int expert, uint8_t* gate, uint8_t* up, uint8_t* down) {
    REQUIRE(gate && up && down, "synth_q4k_host: null pointer");
    const Tables& t = host_tables();
    constexpr size_t NB = (size_t)EH * EI / 256;
    for (size_t sb = 0; sb < 3 * NB; sb++) {
        uint8_t* d = sb < NB ? gate + sb * 144 : sb < 2 * NB ? up + (sb - NB) * 144 : down + (sb - 2 * NB) * 144;
        synth_q4k_block(seed, layer, expert, sb, t.d, d);
    }
    return MOEXB_OK;
}

// ---- context and resident layers -----------------------------------------------------------------------------------------

}  // extern "C"
template <class T>
static int dev_alloc(moexb_ctx* ctx, T** p, size_t n) {
    void* v = nullptr;
    cudaError_t e = cudaMalloc(&v, n * sizeof(T));
    if (e != cudaSuccess) return fail(MOEXB_ERR_NOMEM, "cudaMalloc of %zu bytes: %s", n * sizeof(T), cudaGetErrorString(e));
    ctx->owned.push_back(v);
    *p = static_cast<T*>(v);
    return MOEXB_OK;
}

extern "C" {
int moexb_ctx_create(int device, int max_tokens, int max_experts, int top_k, moexb_ctx** out) {
    REQUIRE(out, "ctx_create: null output");
    REQUIRE(max_tokens > 0 && max_tokens <= 65535 && max_experts > 0 && max_experts % 32 == 0 && max_experts <= 1024 && top_k > 0 && top_k <= 15,
            "ctx_create: max_tokens=%d max_experts=%d top_k=%d", max_tokens, max_experts, top_k);
    CUDA_TRY(cudaSetDevice(device));
    moexb_ctx* c = new (std::nothrow) moexb_ctx;
    if (!c) return fail(MOEXB_ERR_NOMEM, "out of host memory");
    c->device = device; c->max_tokens = max_tokens; c->max_experts = max_experts; c->top_k = top_k;
    const size_t T = max_tokens, P = T * (top_k + 1);
    int rc = MOEXB_OK;
    auto A = [&](auto** p, size_t n) { if (rc == MOEXB_OK) rc = dev_alloc(c, p, n); };
    A(&c->table_s, SYNTH_TABLE_N); A(&c->table_d, SYNTH_TABLE_N);
    A(&c->xf, T * EH); A(&c->xn, T * EH); A(&c->logits, T * (max_experts + 1)); A(&c->w, T * top_k); A(&c->idx, T * top_k);
    A(&c->act, P * EI); A(&c->ypair, P * EH); A(&c->moe, T * EH);
    A(&c->counts, (size_t)max_experts); A(&c->nitems, 1); A(&c->items, (size_t)max_experts + 1); A(&c->pairs, P);
    A(&c->slots, (size_t)top_k + 1); A(&c->wts, (size_t)top_k + 1);
    A(&c->xs, T * 2 * EH); A(&c->act_split, P * 2 * EI); A(&c->subs, (size_t)max_experts + 1 + P / ST_MAXP + 1);
    A(&c->nsub, 2); A(&c->err, 1); A(&c->sx, T * (EH / 32)); A(&c->sx_act, P * (EI / 32)); A(&c->route_done, (size_t)max_tokens); A(&c->staging, (size_t)STAGING_BLOBS * expert_bytes(FMT_ZP));
    // buckets of max_tokens places for every expert and the shared one, where that is at most 64 MB (6.3 MB for 2048 tokens, 256 experts)
    if (max_experts <= BK_MAX_E && T * (max_experts + 1) * sizeof(moexb_pair) <= (64u << 20)) {
        A(&c->bcnt, (size_t)max_experts); A(&c->bpairs, T * (max_experts + 1));
        if (rc == MOEXB_OK && cudaMemset(c->bcnt, 0, (size_t)max_experts * sizeof(int)) != cudaSuccess) rc = fail(MOEXB_ERR_CUDA, "ctx_create: memset");
    }
    if (rc == MOEXB_OK && cudaMemset(c->err, 0, sizeof(int)) != cudaSuccess) rc = fail(MOEXB_ERR_CUDA, "ctx_create: memset");
    if (rc == MOEXB_OK && cudaMemset(c->route_done, 0, (size_t)max_tokens * sizeof(int)) != cudaSuccess) rc = fail(MOEXB_ERR_CUDA, "ctx_create: memset");
    if (rc == MOEXB_OK && cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) rc = fail(MOEXB_ERR_CUDA, "ctx_create: device attribute");
    if (rc != MOEXB_OK) { moexb_ctx_destroy(c); return rc; }
    const Tables& t = host_tables();
    cudaError_t e = cudaMemcpy(c->table_s, t.s, sizeof t.s, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(c->table_d, t.d, sizeof t.d, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) { moexb_ctx_destroy(c); return fail(MOEXB_ERR_CUDA, "table upload: %s", cudaGetErrorString(e)); }
    *out = c;
    return MOEXB_OK;
}

int moexb_ctx_destroy(moexb_ctx* ctx) {
    if (!ctx) return MOEXB_OK;
    {
        std::lock_guard<std::mutex> lock(g_default_lock);
        for (moexb_ctx*& d : g_default_ctx) if (d == ctx) d = nullptr;
    }
    for (void* p : ctx->owned) cudaFree(p);
    for (auto& r : ctx->recs) { cudaEventDestroy(r.a); cudaEventDestroy(r.b); }
    for (auto e : ctx->spare) cudaEventDestroy(e);
    delete ctx;
    return MOEXB_OK;
}

int moexb_synth_experts(moexb_ctx* ctx, int fmt, unsigned seed, int layer, int e0, int n, uint8_t* dst, void* stream) {
    REQUIRE(ctx, "synth_experts: null context");
    return synth_launch(fmt, seed, layer, e0, n, dst, ctx->table_s, ctx->table_d, stream);
}

}  // extern "C"
// One tensor map over the image of n_blobs tiled blobs, [slice / 4][K slice][8 bytes]: boxes of `elems` x 8 bytes of 16 slices - the same K
// slice of 16 row tiles (gate/up), or 16 slices in a row (down). The encoder is a driver call, looked up through the runtime.
static int image_map(CUtensorMap* map, const uint8_t* image, int slice_bytes, size_t n_blobs, int elems, bool down) {
    using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void* f = nullptr; cudaDriverEntryPointQueryResult q;
        return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess ? (Encode)f : nullptr;
    }();
    if (!encode) return fail(MOEXB_ERR_CUDA, "layer_create: the driver has no tensor map encoder");
    const cuuint64_t dims[3] = {(cuuint64_t)slice_bytes / 8, 4, (cuuint64_t)n_blobs * (TL_SLICES / 4)}, strides[2] = {(cuuint64_t)slice_bytes, (cuuint64_t)slice_bytes * 4};
    const cuuint32_t box[3] = {(cuuint32_t)elems, down ? 4u : 1u, down ? 4u : 16u}, step[3] = {1, 1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<uint8_t*>(image), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? (int)MOEXB_OK : fail(MOEXB_ERR_CUDA, "layer_create: tensor map: error %d", (int)r);
}
static int layer_maps(moexb_layer* L) {
    return by_fmt(L->fmt, [&]<int FMT>() {
        int rc = MOEXB_OK;
        for (int down = 0; down < 2 && rc == MOEXB_OK; down++) {
            GroupedMaps& m = down ? L->map_down : L->map_gate_up;
            rc = image_map(&m.w, L->image, tl_slice_bytes<FMT>(), L->n_local + 1, GG_CH * tl_group_bytes<FMT>() / 8, down);
            if (rc == MOEXB_OK && FMT == FMT_ZP) rc = image_map(&m.dd, L->image, tl_slice_bytes<FMT>(), L->n_local + 1, 16, down);
        }
        return rc;
    });
}

extern "C" {
int moexb_layer_create(moexb_ctx* ctx, int fmt, int n_routed, int first_local, int n_local, int router_dtype, int layout, moexb_layer** out) {
    REQUIRE(ctx && out, "layer_create: null pointer");
    REQUIRE(fmt_ok(fmt), "layer_create: unknown expert format %d", fmt);
    REQUIRE(n_routed > 0 && n_routed % 32 == 0 && n_routed <= ctx->max_experts, "layer_create: n_routed=%d (context allows %d)", n_routed, ctx->max_experts);
    REQUIRE(first_local >= 0 && n_local >= 0 && first_local + n_local <= n_routed, "layer_create: local experts [%d, %d) outside 0..%d", first_local, first_local + n_local, n_routed);
    REQUIRE(router_dtype == MOEXB_F32 || router_dtype == 2, "layer_create: router dtype %d", router_dtype);
    REQUIRE(layout == MOEXB_LAYOUT_TILED || layout == MOEXB_LAYOUT_REFERENCE, "layer_create: layout %d", layout);
    CUDA_TRY(cudaSetDevice(ctx->device));
    moexb_layer* L = new (std::nothrow) moexb_layer;
    if (!L) return fail(MOEXB_ERR_NOMEM, "out of host memory");
    L->ctx = ctx; L->fmt = fmt; L->n_routed = n_routed; L->first_local = first_local; L->n_local = n_local; L->router_dtype = router_dtype; L->layout = layout;
    const size_t eb = expert_bytes(fmt);
    cudaError_t e = cudaMalloc((void**)&L->image, (size_t)(n_local + 1) * eb);
    if (e == cudaSuccess) e = cudaMemset(L->image, 0, (size_t)(n_local + 1) * eb);
    L->loaded.assign(n_routed + 1, 0);
    if (e == cudaSuccess) e = cudaMalloc(&L->router, (size_t)(n_routed + 1) * EH * (router_dtype == MOEXB_F32 ? 4 : 2));
    if (e == cudaSuccess) e = cudaMalloc((void**)&L->slot_table, (size_t)(n_routed + 1) * sizeof(void*));
    if (e == cudaSuccess) {
        L->slot_host.assign(n_routed + 1, nullptr);
        for (int i = 0; i < n_local; i++) L->slot_host[first_local + i] = L->image + (size_t)i * eb;
        L->slot_host[n_routed] = L->image + (size_t)n_local * eb;
        e = cudaMemcpy(L->slot_table, L->slot_host.data(), L->slot_host.size() * sizeof(void*), cudaMemcpyHostToDevice);
    }
    if (e != cudaSuccess) { moexb_layer_destroy(L); return fail(MOEXB_ERR_NOMEM, "layer_create: %s", cudaGetErrorString(e)); }
    if (layout == MOEXB_LAYOUT_TILED) {
        const int rc = layer_maps(L);
        if (rc != MOEXB_OK) { moexb_layer_destroy(L); return rc; }
    }
    *out = L;
    return MOEXB_OK;
}

int moexb_layer_destroy(moexb_layer* L) {
    if (!L) return MOEXB_OK;
    cudaFree(L->image); cudaFree(L->router); cudaFree((void*)L->slot_table);
    delete L;
    return MOEXB_OK;
}

uint8_t* moexb_layer_blob(moexb_layer* L, int e) {
    if (!L || e < 0 || e > L->n_routed) return nullptr;
    return const_cast<uint8_t*>(L->slot_host[e]);
}
const uint8_t* const* moexb_layer_slot_table(moexb_layer* L) { return L ? L->slot_table : nullptr; }
void* moexb_layer_router(moexb_layer* L) { return L ? L->router : nullptr; }

}  // extern "C"

// Reference-layout blobs at src (device) -> the layer's layout at dst, n experts.
static int to_layer_layout(moexb_layer* L, const uint8_t* src, uint8_t* dst, int n, cudaStream_t st) {
    const size_t eb = expert_bytes(L->fmt);
    if (L->layout == MOEXB_LAYOUT_REFERENCE) {
        CUDA_TRY(cudaMemcpyAsync(dst, src, n * eb, cudaMemcpyDeviceToDevice, st));
        return MOEXB_OK;
    }
    return by_fmt(L->fmt, [&]<int FMT>() {
        tile_expert_k<FMT, true><<<dim3(TL_SLICES, n), 256, 0, st>>>(src, dst);
        LAUNCHED("tile_expert");
        return (int)MOEXB_OK;
    });
}

extern "C" {

int moexb_layer_upload_expert(moexb_layer* L, int e, const uint8_t* blob_host) {
    REQUIRE(L && blob_host, "layer_upload_expert: null pointer");
    REQUIRE(e >= 0 && e <= L->n_routed && L->slot_host[e], "layer_upload_expert: expert %d is not held by this layer", e);
    CUDA_TRY(cudaMemcpy(L->ctx->staging, blob_host, expert_bytes(L->fmt), cudaMemcpyHostToDevice));
    const int rc = to_layer_layout(L, L->ctx->staging, const_cast<uint8_t*>(L->slot_host[e]), 1, nullptr);
    if (rc != MOEXB_OK) return rc;
    CUDA_TRY(cudaStreamSynchronize(nullptr));
    L->loaded[e] = 1;
    return MOEXB_OK;
}

int moexb_layer_export_expert(moexb_layer* L, int e, uint8_t* blob_host) {
    REQUIRE(L && blob_host, "layer_export_expert: null pointer");
    REQUIRE(e >= 0 && e <= L->n_routed && L->slot_host[e], "layer_export_expert: expert %d is not held by this layer", e);
    const uint8_t* src = L->slot_host[e];
    if (L->layout == MOEXB_LAYOUT_TILED) {
        const int rc = by_fmt(L->fmt, [&]<int FMT>() {
            tile_expert_k<FMT, false><<<TL_SLICES, 256>>>(src, L->ctx->staging);
            LAUNCHED("untile_expert");
            return (int)MOEXB_OK;
        });
        if (rc != MOEXB_OK) return rc;
        src = L->ctx->staging;
    }
    CUDA_TRY(cudaMemcpy(blob_host, src, expert_bytes(L->fmt), cudaMemcpyDeviceToHost));
    return MOEXB_OK;
}

int moexb_layer_set_router(moexb_layer* L, const void* W_host) {
    REQUIRE(L && W_host, "layer_set_router: null pointer");
    CUDA_TRY(cudaMemcpy(L->router, W_host, (size_t)(L->n_routed + 1) * EH * (L->router_dtype == MOEXB_F32 ? 4 : 2), cudaMemcpyHostToDevice));
    return MOEXB_OK;
}

int moexb_layer_fill_synth(moexb_layer* L, unsigned seed, int layer_index, void* stream) {
    REQUIRE(L, "layer_fill_synth: null layer");
    const size_t eb = expert_bytes(L->fmt);
    moexb_ctx* c = L->ctx;
    // held routed experts, then the shared expert (id n_routed), through the staging buffer in batches
    for (int i = 0; i < L->n_local + 1; i += STAGING_BLOBS) {
        const int n = min(STAGING_BLOBS, L->n_local + 1 - i);
        const int routed = min(n, max(0, L->n_local - i));
        int rc = MOEXB_OK;
        if (routed) rc = synth_launch(L->fmt, seed, layer_index, L->first_local + i, routed, c->staging, c->table_s, c->table_d, stream);
        if (rc == MOEXB_OK && routed < n) rc = synth_launch(L->fmt, seed, layer_index, L->n_routed, 1, c->staging + routed * eb, c->table_s, c->table_d, stream);
        if (rc == MOEXB_OK) rc = to_layer_layout(L, c->staging, L->image + (size_t)i * eb, n, S(stream));
        if (rc != MOEXB_OK) return rc;
    }
    for (int i = 0; i < L->n_local; i++) L->loaded[L->first_local + i] = 1;
    L->loaded[L->n_routed] = 1;
    return MOEXB_OK;
}

// ---- GGUF ingest ----------------------------------------------------------------------------------------------------------

int moexb_gguf_open(const char* path, moexb_gguf** out) {
    REQUIRE(path && out, "gguf_open: null pointer");
    std::string err;
    moexb_gguf* g = gguf_open(path, err);
    if (!g) return fail(MOEXB_ERR_ARG, "gguf_open: %s", err.c_str());
    *out = g;
    return MOEXB_OK;
}

int moexb_gguf_close(moexb_gguf* g) {
    delete g;
    return MOEXB_OK;
}

int moexb_gguf_tensor_count(const moexb_gguf* g) { return g ? (int)g->tensors.size() : 0; }

const char* moexb_gguf_tensor_name(const moexb_gguf* g, int i) {
    return g && i >= 0 && i < (int)g->tensors.size() ? g->tensors[i].name.c_str() : nullptr;
}

int moexb_gguf_tensor(const moexb_gguf* g, const char* name, int* type, int* n_dims, long long* ne, const void** data, long long* nbytes) {
    REQUIRE(g && name, "gguf_tensor: null pointer");
    const GgufTensor* t = g->find(name);
    if (!t) return fail(MOEXB_ERR_ARG, "tensor %s is missing from the GGUF", name);
    if (type) *type = (int)t->type;
    if (n_dims) *n_dims = t->n_dims;
    if (ne) for (int d = 0; d < 4; d++) ne[d] = t->ne[d];
    if (data) *data = t->data;
    if (nbytes) *nbytes = t->nbytes;
    return MOEXB_OK;
}

}  // extern "C"

// A Q4_K tensor of the block with the shape the path needs, or an error naming what differs.
static int gguf_expect(const moexb_gguf* g, const std::string& name, std::initializer_list<long long> ne, const GgufTensor** out) {
    const GgufTensor* t = g->find(name);
    if (!t) return fail(MOEXB_ERR_ARG, "tensor %s is missing from the GGUF", name.c_str());
    int bn, bb;
    if (!gq_block(t->type, bn, bb) || !t->data)
        return fail(MOEXB_ERR_UNSUPPORTED, "layer_load_gguf: %s has ggml type %u, which this loader cannot re-quantise (Q4_K is carried over bit for bit; "
                    "Q5_K, Q6_K, Q8_0, IQ4_NL, IQ4_XS, Q4_0/1, Q5_0/1, F16, BF16 and F32 are refitted to 4 bits)", name.c_str(), t->type);
    bool same = t->n_dims == (int)ne.size();
    int d = 0;
    for (long long v : ne) same = same && t->ne[d++] == v;
    if (!same) return fail(MOEXB_ERR_ARG, "tensor %s has shape [%lld, %lld, %lld, %lld] (%d dimensions), not the one this layer needs",
                           name.c_str(), t->ne[0], t->ne[1], t->ne[2], t->ne[3], t->n_dims);
    *out = t;
    return MOEXB_OK;
}

// One expert from three GGUF tensors of any readable type (gate, up [I][H]; down [H][I]; row-major, `type[k]` blocks) into a
// zero-point blob in the reference layout, on the host: Q4_K rows are carried over bit for bit, the others refitted
// (gguf_quant.h). What gg_experts does per expert (gguf.h:666-694).
static bool expert_to_zp_host(const uint32_t type[3], const uint8_t* const src[3], uint8_t* blob) {
    std::vector<float> w(EH);
    for (int k = 0; k < 3; k++) {
        const int rows = k < 2 ? EI : EH, cols = k < 2 ? EH : EI;
        int bn, bb;
        if (!gq_block(type[k], bn, bb)) return false;
        const size_t row_bytes = (size_t)cols / bn * bb;
        for (int r = 0; r < rows; r++) {
            const size_t row = (size_t)(k == 0 ? 0 : k == 1 ? EI : 0) + r;   // row inside [gate | up] or inside down
            const size_t qoff = k < 2 ? row * (EH / 2) : DOWN_Q_OFF + row * (EI / 2);
            const size_t c0 = k < 2 ? row * (EH / 32) : DOWN_C_OFF + row * (EI / 32);
            uint8_t* qb = blob + qoff;
            uint8_t* cs = blob + Q_BYTES + c0 * 2;
            uint16_t* sup = reinterpret_cast<uint16_t*>(blob + Q_BYTES + CHUNKS * 2 + (c0 / 8) * 4);
            const uint8_t* p = src[k] + (size_t)r * row_bytes;
            if (type[k] == GQ_Q4_K) {
                for (int b = 0; b < cols / 256; b++) q4k_block_to_zp(p + (size_t)b * 144, qb + b * 128, cs + b * 16, reinterpret_cast<uint8_t*>(sup + 2 * b));
            } else {
                if (!gq_dequant(type[k], p, cols, w.data())) return false;
                zp_row_from_values(w.data(), cols, qb, cs, sup);
            }
        }
    }
    return true;
}

// `n` router values at src (F32, F16 or BF16, by ggml type id) into the layer's router dtype at dst (host).
static bool router_rows_to(uint32_t type, const uint8_t* src, long long n, int router_dtype, void* dst) {
    if (type != GGML_F32 && type != GGML_F16 && type != GGML_BF16) return false;
    for (long long i = 0; i < n; i++) {
        float v;
        if (type == GGML_F32) memcpy(&v, src + 4 * i, 4);
        else {
            uint16_t h; memcpy(&h, src + 2 * i, 2);
            if (type == GGML_F16) { __half hh; memcpy(&hh, &h, 2); v = __half2float(hh); }
            else { const uint32_t u = (uint32_t)h << 16; memcpy(&v, &u, 4); }
        }
        if (router_dtype == MOEXB_F32) static_cast<float*>(dst)[i] = v;
        else static_cast<__half*>(dst)[i] = __float2half_rn(v);
    }
    return true;
}

extern "C" {

int moexb_layer_load_gguf(moexb_layer* L, const moexb_gguf* g, int block, int* loaded) {
    REQUIRE(L && g, "layer_load_gguf: null pointer");
    REQUIRE(block >= 0, "layer_load_gguf: block %d", block);
    if (loaded) *loaded = 0;
    if (L->fmt != FMT_ZP) return fail(MOEXB_ERR_UNSUPPORTED, "layer_load_gguf: GGUF expert tensors load into a MOEXB_FMT_ZP layer (this one has format %d)", L->fmt);
    const std::string p = "blk." + std::to_string(block) + ".";
    const long long E = L->n_routed;
    const GgufTensor* t[3];
    int rc = gguf_expect(g, p + "ffn_gate_exps.weight", {EH, EI, E}, &t[0]);
    if (rc == MOEXB_OK) rc = gguf_expect(g, p + "ffn_up_exps.weight", {EH, EI, E}, &t[1]);
    if (rc == MOEXB_OK) rc = gguf_expect(g, p + "ffn_down_exps.weight", {EI, EH, E}, &t[2]);
    if (rc != MOEXB_OK) return rc;
    moexb_ctx* c = L->ctx;
    CUDA_TRY(cudaSetDevice(c->device));
    constexpr size_t PART = (size_t)EH * EI / 256 * 144;  // raw bytes of one expert's gate, up or down
    const size_t eb = expert_bytes(FMT_ZP);
    static_assert(3 * PART <= (size_t)Q_BYTES + 2 * CHUNKS + CHUNKS / 8 * 4, "raw Q4_K of one expert fits a staging blob");
    constexpr int HALF = STAGING_BLOBS / 2;  // raw tensors in the first half of the staging buffer, blobs in the second
    // src[k] = the three raw tensors of the experts to convert, `n` of them, into the layer from slot `dst0` on
    auto convert = [&](const uint8_t* const* src, int n, uint8_t* dst) -> int {
        for (int i = 0; i < n; i++)
            for (int k = 0; k < 3; k++)
                CUDA_TRY(cudaMemcpyAsync(c->staging + i * eb + k * PART, src[3 * i + k], PART, cudaMemcpyHostToDevice, nullptr));
        for (int i = 0; i < n; i++) {
            const uint8_t* raw = c->staging + i * eb;
            q4k_to_zp_k<<<(unsigned)((CHUNKS / 8 + 127) / 128), 128>>>(raw, raw + PART, raw + 2 * PART, c->staging + (HALF + i) * eb);
            LAUNCHED("q4k_to_zp");
        }
        return to_layer_layout(L, c->staging + HALF * eb, dst, n, nullptr);
    };
    // Any tensor in another type than Q4_K: the experts are re-quantised on the host (gguf_quant.h), a batch of them spread
    // over the host threads, and uploaded as finished blobs. per[k]: bytes of one expert inside tensor k.
    auto convert_host = [&](const GgufTensor* const tt[3], int first, int n, uint8_t* dst) -> int {
        size_t per[3]; uint32_t ty[3];
        for (int k = 0; k < 3; k++) { int bn, bb; gq_block(tt[k]->type, bn, bb); per[k] = (size_t)EH * EI / bn * bb; ty[k] = tt[k]->type; }
        std::vector<uint8_t> blobs((size_t)STAGING_BLOBS * eb);
        for (int i = 0; i < n; i += STAGING_BLOBS) {
            const int m = min(STAGING_BLOBS, n - i);
            std::atomic<int> next{0}, bad{0};
            auto work = [&] {
                for (int j; (j = next.fetch_add(1)) < m;) {
                    const uint8_t* src3[3];
                    for (int k = 0; k < 3; k++) src3[k] = tt[k]->data + (size_t)(first + i + j) * per[k];
                    if (!expert_to_zp_host(ty, src3, blobs.data() + (size_t)j * eb)) bad = 1;
                }
            };
            std::vector<std::thread> th;
            const int nt = (int)std::min<unsigned>(std::max(1u, std::thread::hardware_concurrency()), (unsigned)m);
            for (int q = 1; q < nt; q++) th.emplace_back(work);
            work();
            for (auto& x : th) x.join();
            if (bad) return fail(MOEXB_ERR_UNSUPPORTED, "layer_load_gguf: a block of block %d could not be re-quantised", block);
            CUDA_TRY(cudaMemcpy(c->staging, blobs.data(), (size_t)m * eb, cudaMemcpyHostToDevice));
            const int rc2 = to_layer_layout(L, c->staging, dst + (size_t)i * eb, m, nullptr);
            if (rc2 != MOEXB_OK) return rc2;
            CUDA_TRY(cudaStreamSynchronize(nullptr));
        }
        return MOEXB_OK;
    };
    const uint8_t* src[3 * HALF];
    const bool all_q4k = t[0]->type == GGML_Q4_K && t[1]->type == GGML_Q4_K && t[2]->type == GGML_Q4_K;
    if (!all_q4k) {
        rc = convert_host(t, L->first_local, L->n_local, L->image);
        if (rc != MOEXB_OK) return rc;
    } else
    for (int i = 0; i < L->n_local; i += HALF) {
        const int n = min(HALF, L->n_local - i);
        for (int j = 0; j < n; j++)
            for (int k = 0; k < 3; k++) src[3 * j + k] = t[k]->data + (size_t)(L->first_local + i + j) * PART;
        rc = convert(src, n, L->image + (size_t)i * eb);
        if (rc != MOEXB_OK) return rc;
        CUDA_TRY(cudaStreamSynchronize(nullptr));
    }
    int got = L->n_local ? 1 : 0;
    for (int i = 0; i < L->n_local; i++) L->loaded[L->first_local + i] = 1;
    // the shared expert, when the file holds it as Q4_K too
    const GgufTensor *sg = g->find(p + "ffn_gate_shexp.weight"), *su = g->find(p + "ffn_up_shexp.weight"), *sd = g->find(p + "ffn_down_shexp.weight");
    int sbn, sbb;
    if (sg && su && sd && sg->data && su->data && sd->data && gq_block(sg->type, sbn, sbb) && gq_block(su->type, sbn, sbb) && gq_block(sd->type, sbn, sbb) &&
        sg->n_dims == 2 && su->n_dims == 2 &&
        sd->n_dims == 2 && sg->ne[0] == EH && sg->ne[1] == EI && su->ne[0] == EH && su->ne[1] == EI && sd->ne[0] == EI && sd->ne[1] == EH) {
        if (sg->type == GGML_Q4_K && su->type == GGML_Q4_K && sd->type == GGML_Q4_K) {
            src[0] = sg->data; src[1] = su->data; src[2] = sd->data;
            rc = convert(src, 1, L->image + (size_t)L->n_local * eb);
        } else {
            const GgufTensor* st3[3] = {sg, su, sd};
            rc = convert_host(st3, 0, 1, L->image + (size_t)L->n_local * eb);
        }
        if (rc != MOEXB_OK) return rc;
        CUDA_TRY(cudaStreamSynchronize(nullptr));
        got |= 2;
        L->loaded[L->n_routed] = 1;
    }
    // router rows and the shared expert's gate vector
    const GgufTensor *rt = g->find(p + "ffn_gate_inp.weight"), *rs = g->find(p + "ffn_gate_inp_shexp.weight");
    const size_t esz = L->router_dtype == MOEXB_F32 ? 4 : 2;
    std::vector<uint8_t> rows((size_t)E * EH * esz);
    if (rt && rt->n_dims == 2 && rt->ne[0] == EH && rt->ne[1] == E && rt->data && router_rows_to(rt->type, rt->data, E * EH, L->router_dtype, rows.data())) {
        CUDA_TRY(cudaMemcpy(L->router, rows.data(), rows.size(), cudaMemcpyHostToDevice));
        got |= 4;
    }
    if (rs && rs->ne[0] == EH && rs->nbytes == rs->row_bytes && rs->data && router_rows_to(rs->type, rs->data, EH, L->router_dtype, rows.data())) {
        CUDA_TRY(cudaMemcpy(static_cast<uint8_t*>(L->router) + (size_t)E * EH * esz, rows.data(), EH * esz, cudaMemcpyHostToDevice));
        got |= 8;
    }
    if (loaded) *loaded = got;
    return MOEXB_OK;
}

// gg_dequant (gguf.h:85-255) for the block types this library reads, on the host: n values (a multiple of the block size).
int moexb_gguf_dequant_host(int ggml_type, const uint8_t* src_host, long long n, float* y_host) {
    REQUIRE(src_host && y_host && n > 0, "gguf_dequant_host: bad argument");
    if (!gq_dequant((uint32_t)ggml_type, src_host, n, y_host))
        return fail(MOEXB_ERR_UNSUPPORTED, "gguf_dequant_host: ggml type %d is not readable here, or n=%lld is not a multiple of its block size", ggml_type, n);
    return MOEXB_OK;
}

// gg_zp_row (gguf.h:302-330) on the host: one row of `cols` weights (a multiple of 256) of a GGUF tensor into the zero-point
// form - nibble bytes qb[cols / 2], [sc, mn] cs[cols / 32 * 2], (d, dm) fp16 bits sup[cols / 256 * 2].
int moexb_gguf_row_to_zp(int ggml_type, const uint8_t* src_host, int cols, uint8_t* qb, uint8_t* cs, uint16_t* sup) {
    REQUIRE(src_host && qb && cs && sup, "gguf_row_to_zp: null pointer");
    REQUIRE(cols > 0 && cols % 256 == 0, "gguf_row_to_zp: cols=%d must be a positive multiple of 256", cols);
    if (ggml_type == (int)GQ_Q4_K) {
        for (int b = 0; b < cols / 256; b++) q4k_block_to_zp(src_host + (size_t)b * 144, qb + b * 128, cs + b * 16, reinterpret_cast<uint8_t*>(sup + 2 * b));
        return MOEXB_OK;
    }
    std::vector<float> w(cols);
    if (!gq_dequant((uint32_t)ggml_type, src_host, cols, w.data())) return fail(MOEXB_ERR_UNSUPPORTED, "gguf_row_to_zp: ggml type %d is not readable here", ggml_type);
    zp_row_from_values(w.data(), cols, qb, cs, sup);
    return MOEXB_OK;
}

// ---- safetensors container ingest ----------------------------------------------------------------------------------------

int moexb_st_open(const char* path, moexb_st** out) {
    REQUIRE(path && out, "st_open: null pointer");
    std::string err;
    moexb_st* s = st_open(path, err);
    if (!s) return fail(MOEXB_ERR_ARG, "st_open: %s", err.c_str());
    *out = s;
    return MOEXB_OK;
}

int moexb_st_close(moexb_st* s) {
    delete s;
    return MOEXB_OK;
}

int moexb_st_tensor_count(const moexb_st* s) { return s ? (int)s->tensors.size() : 0; }

const char* moexb_st_tensor_name(const moexb_st* s, int i) {
    return s && i >= 0 && i < (int)s->tensors.size() ? s->tensors[i].name.c_str() : nullptr;
}

int moexb_st_tensor(const moexb_st* s, const char* name, char* dtype, int* n_dims, long long* shape, const void** data, long long* nbytes) {
    REQUIRE(s && name, "st_tensor: null pointer");
    const StTensorInfo* t = s->find(name);
    if (!t) return fail(MOEXB_ERR_ARG, "missing tensor %s", name);
    if (dtype) { strncpy(dtype, t->dtype.c_str(), 7); dtype[7] = 0; }
    if (n_dims) *n_dims = (int)std::min<size_t>(t->shape.size(), 8);
    if (shape) for (size_t d = 0; d < t->shape.size() && d < 8; d++) shape[d] = t->shape[d];
    if (data) *data = t->data;
    if (nbytes) *nbytes = t->nbytes;
    return MOEXB_OK;
}

int moexb_layer_load_st(moexb_layer* L, const moexb_st* s, const char* prefix, int* loaded) {
    REQUIRE(L && s && prefix, "layer_load_st: null pointer");
    if (loaded) *loaded = 0;
    moexb_ctx* c = L->ctx;
    CUDA_TRY(cudaSetDevice(c->device));
    const std::string p(prefix);
    const size_t eb = expert_bytes(L->fmt), sp = eb - Q_BYTES;  // scale part of the layer's format
    // the container's scale part: F32 group scales (symmetric) or the zero-point bytes; an fp16-scale layer takes F32
    // scales only when every one of them is an fp16 value, so that nothing is rounded on the way in
    const size_t sp_file = L->fmt == FMT_ZP ? expert_bytes(FMT_ZP) - Q_BYTES : expert_bytes(FMT_SYM_F32) - Q_BYTES;
    const char* want_dtype = L->fmt == FMT_ZP ? "U8" : "F32";
    std::vector<__half> narrow(L->fmt == FMT_SYM_F16 ? CHUNKS / 2 : 0);
    for (int i = 0; i < L->n_local; i += STAGING_BLOBS) {
        const int n = min(STAGING_BLOBS, L->n_local - i);
        for (int j = 0; j < n; j++) {
            const std::string ep = p + "mlp.experts." + std::to_string(L->first_local + i + j) + ".";
            const StTensorInfo *q = s->find(ep + "merged_weight"), *qs = s->find(ep + "qs");
            if (!q || !qs) return fail(MOEXB_ERR_ARG, "missing tensor %s%s", ep.c_str(), q ? "qs" : "merged_weight");
            if ((size_t)q->nbytes != Q_BYTES) return fail(MOEXB_ERR_ARG, "%smerged_weight has %lld bytes, not the %zu of this expert shape", ep.c_str(), q->nbytes, (size_t)Q_BYTES);
            if ((size_t)qs->nbytes != sp_file || qs->dtype != want_dtype)
                return fail(MOEXB_ERR_UNSUPPORTED, "%sqs (%s, %lld bytes) is not the scale part of this layer's expert format (%s, %zu bytes)",
                            ep.c_str(), qs->dtype.c_str(), qs->nbytes, want_dtype, sp_file);
            uint8_t* dst = c->staging + (size_t)j * eb;
            CUDA_TRY(cudaMemcpyAsync(dst, q->data, Q_BYTES, cudaMemcpyHostToDevice, nullptr));
            if (L->fmt == FMT_SYM_F16) {
                for (size_t k = 0; k < CHUNKS / 2; k++) {
                    float f;
                    memcpy(&f, qs->data + 4 * k, 4);
                    narrow[k] = __float2half_rn(f);
                    if (!(__half2float(narrow[k]) == f))
                        return fail(MOEXB_ERR_UNSUPPORTED, "%sqs: scale %zu (%.9g) is not an fp16 value; load this container into a MOEXB_FMT_SYM_F32 layer", ep.c_str(), k, f);
                }
                CUDA_TRY(cudaMemcpy(dst + Q_BYTES, narrow.data(), sp, cudaMemcpyHostToDevice));  // synchronous: narrow is reused
            } else {
                CUDA_TRY(cudaMemcpyAsync(dst + Q_BYTES, qs->data, sp, cudaMemcpyHostToDevice, nullptr));
            }
        }
        const int rc = to_layer_layout(L, c->staging, L->image + (size_t)i * eb, n, nullptr);
        if (rc != MOEXB_OK) return rc;
        CUDA_TRY(cudaStreamSynchronize(nullptr));
    }
    int got = L->n_local ? 1 : 0;
    for (int i = 0; i < L->n_local; i++) L->loaded[L->first_local + i] = 1;
    // router rows (mlp.gate.weight [E][H]) and the shared expert's gate vector (mlp.shared_expert_gate.weight [1][H])
    const size_t esz = L->router_dtype == MOEXB_F32 ? 4 : 2;
    const long long E = L->n_routed;
    std::vector<uint8_t> rows((size_t)E * EH * esz);
    auto ggml_of = [](const std::string& d) { return d == "F32" ? (int)GGML_F32 : d == "F16" ? (int)GGML_F16 : d == "BF16" ? (int)GGML_BF16 : -1; };
    auto convert = [&](const StTensorInfo* t, long long n) {
        const int ty = t ? ggml_of(t->dtype) : -1;
        if (ty < 0 || t->nbytes != n * (ty == (int)GGML_F32 ? 4 : 2)) return false;
        return router_rows_to((uint32_t)ty, t->data, n, L->router_dtype, rows.data());
    };
    if (convert(s->find(p + "mlp.gate.weight"), E * EH)) {
        CUDA_TRY(cudaMemcpy(L->router, rows.data(), rows.size(), cudaMemcpyHostToDevice));
        got |= 4;
    }
    if (convert(s->find(p + "mlp.shared_expert_gate.weight"), EH)) {
        CUDA_TRY(cudaMemcpy(static_cast<uint8_t*>(L->router) + (size_t)E * EH * esz, rows.data(), EH * esz, cudaMemcpyHostToDevice));
        got |= 8;
    }
    if (loaded) *loaded = got;
    return MOEXB_OK;
}

}  // extern "C"

// ---- streaming (tensor-core) expert path ------------------------------------------------------------------------------------

template <int FMT, bool DOWN, int CPS>
static int stream_launch_cfg(moexb_ctx* c, const StreamArgs& a, void* stream) {
    constexpr int NW = ST_NW, STAGES = (DOWN ? 3 : 2) + (CPS == 2);
    constexpr int SMEM = st_smem_bytes<FMT, DOWN, NW, STAGES>();
    static PerDeviceOnce once;
    const cudaError_t attr_err = once.run([] { return opt_in(stream_k<FMT, DOWN, NW, STAGES>, (NW + ST_NP) * 32, SMEM, CPS); });
    if (attr_err != cudaSuccess) return fail(MOEXB_ERR_CUDA, "stream kernel shared memory: %s", cudaGetErrorString(attr_err));
    PROF(c, DOWN ? MOEXB_PROF_DOWN : MOEXB_PROF_GATE_UP, stream);
    static_assert((SMEM + 1024) * CPS <= 228 * 1024, "shared memory of the resident CTAs");
    CUDA_TRY(launch_dep(stream_k<FMT, DOWN, NW, STAGES>, CPS * c->sms, (NW + ST_NP) * 32, SMEM, S(stream), a));
    LAUNCHED(DOWN ? "stream_down" : "stream_gate_up");
    return MOEXB_OK;
}
// CTAs per SM. Symmetric formats: three - the 12 consumer warps, not the ring's depth, are what the loop is short of with two. The
// zero-point loop is bound by its arithmetic, so that three CTAs do in 3/2 of the time what two do, and two keep a stage more in
// flight: they take it, except where a short list (a few rounds) fills the rounds of three CTAs better. npairs bounds the
// sub-items. 1, 2, 3, 4, 5, 8, 64 tokens, three CTAs against two: 28, 36, 38, 52, 57, 73, 245 us and 24, 28, 43, 46, 58, 73, 239.
template <int FMT, bool DOWN>
static int stream_launch_one(moexb_ctx* c, const StreamArgs& a, int npairs, void* stream) {
    if constexpr (FMT != FMT_ZP) return stream_launch_cfg<FMT, DOWN, 3>(c, a, stream);
    else {
        const long long tiles = (long long)npairs * st_tiles<DOWN>();
        const long long rounds2 = (tiles + 2 * c->sms - 1) / (2 * c->sms), rounds3 = (tiles + 3 * c->sms - 1) / (3 * c->sms);
        return rounds3 <= (DOWN ? 3 : 2) && 3 * rounds3 <= 2 * rounds2 ? stream_launch_cfg<FMT, DOWN, 3>(c, a, stream) : stream_launch_cfg<FMT, DOWN, 2>(c, a, stream);
    }
}

// gate/up then down over the sub-items already planned in the context (subs, nsub);
// xs = the split activations [token][2][H]; act32 optional.
static int stream_experts(moexb_ctx* c, int fmt, const moexb_pair* pairs, float* act32, float* ypair, int npairs, void* stream) {
    StreamArgs a{c->subs, c->nsub, pairs, reinterpret_cast<const __nv_bfloat16*>(c->xs), act32, reinterpret_cast<__nv_bfloat16*>(c->act_split), ypair, c->err};
    return by_fmt(fmt, [&]<int FMT>() {
        int rc = stream_launch_one<FMT, false>(c, a, npairs, stream);
        if (rc != MOEXB_OK) return rc;
        StreamArgs d = a;
        d.xs = reinterpret_cast<const __nv_bfloat16*>(c->act_split);
        return stream_launch_one<FMT, true>(c, d, npairs, stream);
    });
}

template <int FMT, bool DOWN, int NW, int D, int NB, int CPS, int SRC, bool KSP = false>
static int tiled_launch_cfg(moexb_ctx* c, const TiledArgs& a, const PlanArgs& pa, const BucketArgs& ba, void* stream) {
    constexpr int SMEM = tl_smem_bytes<FMT, DOWN, NW, D, NB, SRC, KSP>();
    static_assert(tl_fits<FMT, DOWN, NW, D, NB, CPS, SRC, KSP>(), "shared memory of the resident CTAs");
    static PerDeviceOnce once;
    const cudaError_t attr_err = once.run([] { return opt_in(stream_tiled_k<FMT, DOWN, NW, D, NB, CPS, SRC, KSP>, NW * 32, SMEM, CPS); });
    if (attr_err != cudaSuccess) return fail(MOEXB_ERR_CUDA, "tiled stream kernel shared memory: %s", cudaGetErrorString(attr_err));
    PROF(c, DOWN ? MOEXB_PROF_DOWN : MOEXB_PROF_GATE_UP, stream);
    CUDA_TRY(launch_dep(stream_tiled_k<FMT, DOWN, NW, D, NB, CPS, SRC, KSP>, CPS * c->sms, NW * 32, SMEM, S(stream), a, pa, ba));
    LAUNCHED(DOWN ? "stream_tiled_down" : "stream_tiled_gate_up");
    return MOEXB_OK;
}

// Two shapes of the same kernel, both two CTAs per SM: a few tokens leave only a handful of row tiles per SM, so CTAs of
// 4 warps with 4 slices in flight each spread them over every SM; from 8 tokens on there is work for 16 warps per SM
// (CTAs of 8 warps, 2 slices in flight each - the same bytes in flight, twice the issue slots in use).
// From 8 tokens on the symmetric formats also take sub-items of up to 8 pairs (two column blocks; tiled_maxp below): the
// gate/up columns of 8 pairs are 66 KB, so that kernel runs as one CTA of 16 warps per SM.
template <int FMT, bool DOWN, int SRC>
static int tiled_launch_one(moexb_ctx* c, const TiledArgs& a, int T, int K, void* stream, const PlanArgs& pa, const BucketArgs& ba) {
    static_assert(SRC != TL_PLAN || FMT == FMT_SYM_F16, "the in-kernel work list fits beside the ring of the fp16-scale format only");
    // The K slices of a row tile on four warps: one zero-point token whose K + 1 sub-items give a CTA no more than a third of a whole round
    // (K = 2, 4, 8, 11, 12, 15: 21.8 / 18.9, 24.1 / 19.5, 26.7 / 22.3, 30.1 / 29.5, 30.8 / 30.8, 32.0 / 32.2 us a layer, without and with; symmetric
    // formats 19.2 either way), and 8 to 15 tokens of the symmetric formats, where whole rounds are two or three per CTA and leave many
    // CTAs with one less (8, 9, 11, 14 tokens 47.9, 50.1, 55.8, 58.3 -> 46.7, 49.2, 52.6, 58.0 us; stacks of 10 and 12 43.7, 48.1 -> 41.6, 44.2;
    // 16 and 23 tokens 59.8, 71.5 -> 60.5, 72.1; zero point 9 and 14 tokens 71.4, 92.9 -> 73.1, 90.1). What decides is how many whole rounds the
    // list gives a CTA, which the host does not know: of 312 lists of 2 to 187 sub-items (8 to 15 tokens, 1 to 15 ranks, 32 to 512 experts) those
    // of 0.8 to 1, 1.9 to 2, 2.5 to 3 and more than 3.5 rounds take up to 6.6 % longer, all others up to 27 % less, the mean 4.1 % less. 15 tokens
    // of 256 experts take 57.4 -> 59.3 us when they are independent and 50.0 -> 45.9 when they share experts; a rank's 32 of 256 experts 25.0 -> 21.6
    // (8 tokens) and 29.8 -> 28.0 (15). Asking for the list on the device cost what it gave: both loops in one kernel are compiled worse.
    if constexpr (!DOWN && FMT == FMT_ZP) { if (T == 1 && 12 * (K + 1) <= c->sms) return tiled_launch_cfg<FMT, DOWN, 16, 2, 1, 1, SRC, true>(c, a, pa, ba, stream); }
    else if constexpr (!DOWN) {
        if (T >= 8 && T < 16) return c->pairs_per_pass == 4 ? tiled_launch_cfg<FMT, DOWN, 16, 2, 1, 1, SRC, true>(c, a, pa, ba, stream)
                                                            : tiled_launch_cfg<FMT, DOWN, 16, 2, 2, 1, SRC, true>(c, a, pa, ba, stream);
    }
    if (T < 8) return tiled_launch_cfg<FMT, DOWN, 4, 4, 1, 2, SRC>(c, a, pa, ba, stream);
    if (FMT == FMT_ZP || c->pairs_per_pass == 4) return tiled_launch_cfg<FMT, DOWN, 8, 2, 1, 2, SRC>(c, a, pa, ba, stream);
    if constexpr (FMT == FMT_ZP) return MOEXB_OK;
    else if constexpr (DOWN) return tiled_launch_cfg<FMT, DOWN, 8, 2, 2, 2, SRC>(c, a, pa, ba, stream);
    else return tiled_launch_cfg<FMT, DOWN, 16, 2, 2, 1, SRC>(c, a, pa, ba, stream);
}
// Pairs per sub-item that tiled_launch_one's kernels take.
static int tiled_maxp(const moexb_ctx* c, int fmt, int T) { return (T >= 8 && fmt != FMT_ZP) ? c->pairs_per_pass : 4; }
// Expert parallelism: whether the gate/up kernel makes the work list of this batch itself (tiled.cuh: plan_in_cta) - a planning launch
// would sit behind the wait for the peers. (fp16-scale format: with the wider slices of the others the list does not fit.)
static bool plan_in_kernel(int fmt, int T, int K, int E) {
    static const bool on = [] { const char* e = getenv("MOEXB_PLAN_IN_KERNEL"); return !(e && e[0] == '0'); }();
    return on && fmt == FMT_SYM_F16 && T <= PL_MAX_TOKENS && K <= PL_MAX_K && E <= PL_MAX_E;
}

// The same on blobs in the tiled layout (sub-item slots point into a tiled layer image). The work list: plan = the gate/up kernel
// makes it and leaves it in the context for the down kernel; buckets = the router's; neither = it is in the context.
static int tiled_experts(moexb_ctx* c, int fmt, const moexb_pair* pairs, float* act32, float* ypair, int T, int K, void* stream, const PlanArgs* plan = nullptr,
                         const BucketArgs* buckets = nullptr, bool clear = false) {
    const TiledArgs a{c->subs, c->nsub, buckets ? buckets->pairs : pairs, c->xs, act32, c->act_split, ypair, c->err, nullptr, 0};
    TiledArgs d = a;
    d.xs = c->act_split;
    if (clear && buckets) { d.clear = c->bcnt; d.experts = buckets->E; }
    PlanArgs pa = plan ? *plan : PlanArgs{};
    pa.subs_out = c->subs; pa.nsub_out = c->nsub;
    const BucketArgs ba = buckets ? *buckets : BucketArgs{};
    return by_fmt(fmt, [&]<int FMT>() {
        int rc;
        if (buckets) {
            rc = tiled_launch_one<FMT, false, TL_BUCKETS>(c, a, T, K, stream, pa, ba);
            return rc != MOEXB_OK ? rc : tiled_launch_one<FMT, true, TL_LIST>(c, d, T, K, stream, pa, ba);
        }
        if constexpr (FMT == FMT_SYM_F16) rc = plan ? tiled_launch_one<FMT, false, TL_PLAN>(c, a, T, K, stream, pa, ba) : tiled_launch_one<FMT, false, TL_LIST>(c, a, T, K, stream, pa, ba);
        else rc = tiled_launch_one<FMT, false, TL_LIST>(c, a, T, K, stream, pa, ba);
        return rc != MOEXB_OK ? rc : tiled_launch_one<FMT, true, TL_LIST>(c, d, T, K, stream, pa, ba);
    });
}

// ---- prefill: grouped GEMM on tcgen05 ----------------------------------------------------------------------------------------

template <int FMT, bool DOWN>
static int grouped_launch_one(moexb_ctx* c, const GroupedArgs& a, const GroupedMaps& maps, void* stream) {
    constexpr int SMEM = gg_smem_bytes<FMT>();
    static PerDeviceOnce once;
    const cudaError_t attr_err = once.run([] { return opt_in(grouped_k<FMT, DOWN>, GG_THREADS, SMEM, 1); });
    if (attr_err != cudaSuccess) return fail(MOEXB_ERR_CUDA, "grouped GEMM shared memory: %s", cudaGetErrorString(attr_err));
    PROF(c, DOWN ? MOEXB_PROF_DOWN : MOEXB_PROF_GATE_UP, stream);
    CUDA_TRY(launch_dep(grouped_k<FMT, DOWN>, c->sms, GG_THREADS, SMEM, S(stream), a, maps));
    LAUNCHED(DOWN ? "grouped_down" : "grouped_gate_up");
    return MOEXB_OK;
}

// Batches from this size on run on the grouped GEMM; where the lines cross depends on how many experts the tokens share. Zero-point blobs
// from a third of the symmetric formats' size on: their streaming kernels take twice the MMAs and four pairs a pass. us a layer,
// streaming against grouped, of independent tokens and of a 12-layer stack whose tokens have grown alike:
//   symmetric   192 tokens 157 / 184 and 160 / 174, 256 tokens 188 / 202 and 195 / 186, 288 tokens 207 / 202 and 207 / 188, 336 tokens 230 / 207 and 229 / 194
//   zero point   40 tokens 159 / 169 and 101 / 82, 72 tokens 209 / 213 and 154 / 110, 88 tokens 226 / 217 and 177 / 111, 128 tokens 283 / 219 and 242 / 124
// Independent symmetric tokens cross at about 280, those of a stack at 225: at 256 the ones lose 7 % and the others gain 5 %.
static int grouped_min_tokens(const moexb_ctx* c, int fmt) {
    const int t = c->prefill_min_tokens;
    return fmt == FMT_ZP ? t / 3 + (t % 3 != 0) : t;   // (any threshold up to the largest int)
}

// Pairs per tile of the grouped GEMM.
static int grouped_maxp(int fmt) { return fmt == FMT_ZP ? gg_nmax<FMT_ZP>() : gg_nmax<FMT_SYM_F16>(); }

// Experts of a large batch on the tensor-core grouped GEMM: the tiles are in the context (subs, nsub) or in the buckets, and layer_rows or
// the token owners (expert parallelism) left the activation rows.
static int grouped_experts(moexb_ctx* c, const moexb_layer* L, const moexb_pair* pairs, int parts, float* ypair, void* stream, const BucketArgs* buckets = nullptr) {
    return by_fmt(L->fmt, [&]<int FMT>() {
        GroupedArgs a{L->image, buckets ? nullptr : c->subs, c->nsub, buckets ? *buckets : BucketArgs{}, buckets ? buckets->pairs : pairs, c->xs, c->sx, c->act_split, c->sx_act, ypair, c->err, parts};
        int rc = grouped_launch_one<FMT, false>(c, a, L->map_gate_up, stream);
        if (rc != MOEXB_OK) return rc;
        a.xs = c->act_split; a.sx = c->sx_act; a.parts = 2;
        return grouped_launch_one<FMT, true>(c, a, L->map_down, stream);
    });
}

// The bf16 split of f32 rows into the context; plan: made on the side by one more block.
static int split_launch(moexb_ctx* c, const float* x, int rows, void* stream, const SidePlan& plan) {
    PROF(c, MOEXB_PROF_OTHER, stream);
    CUDA_TRY(launch_dep(split_rows_k, rows + 1, 256, 0, S(stream), x, c->xs, rows, plan));
    LAUNCHED("split_rows");
    return MOEXB_OK;
}

// What a layer makes of its input rows (layer_rows_k): xf = bf16 rows widened, xn = their rmsnorm (norm), xs = the split of either.
static int layer_rows(moexb_ctx* c, const void* X, int x_dtype, int rows, float* xf, bool norm, float* xn, int mode, uint16_t* xs, int parts, void* stream) {
    PROF(c, MOEXB_PROF_OTHER, stream);
    auto run = [&]<typename XT, bool NORM, int MODE>() -> int {
        CUDA_TRY(launch_dep(layer_rows_k<XT, NORM, MODE>, rows, 256, 0, S(stream), static_cast<const XT*>(X), xf, xn, xs, c->sx, parts, 1e-6f));
        LAUNCHED("layer_rows");
        return MOEXB_OK;
    };
    auto by_mode = [&]<typename XT, bool NORM>() -> int {
        switch (mode) {
            case ROWS_F16: return run.template operator()<XT, NORM, ROWS_F16>();
            case ROWS_BF16: return run.template operator()<XT, NORM, ROWS_BF16>();
            case ROWS_GEMM: return run.template operator()<XT, NORM, ROWS_GEMM>();
            case ROWS_GEMM_Z: return run.template operator()<XT, NORM, ROWS_GEMM_Z>();
        }
        if constexpr (NORM || sizeof(XT) == 2) return run.template operator()<XT, NORM, ROWS_NONE>();
        else return (int)MOEXB_OK;   // f32 rows as they are
    };
    if (x_dtype == MOEXB_BF16) return norm ? by_mode.template operator()<__nv_bfloat16, true>() : by_mode.template operator()<__nv_bfloat16, false>();
    return norm ? by_mode.template operator()<float, true>() : by_mode.template operator()<float, false>();
}

extern "C" int moexb_pairs_forward_tc(moexb_ctx* c, int fmt, const moexb_pair_item* items, int n_items, const moexb_pair* pairs,
                                      const float* X, int T, int npairs, float* act, float* ypair, void* stream) {
    REQUIRE(c && items && pairs && X && ypair, "pairs_forward_tc: null pointer");
    REQUIRE(fmt_ok(fmt), "pairs_forward_tc: unknown expert format %d", fmt);
    REQUIRE(T > 0 && T <= c->max_tokens, "pairs_forward_tc: T=%d exceeds the context's max_tokens=%d", T, c->max_tokens);
    REQUIRE(npairs > 0 && npairs <= c->max_tokens * (c->top_k + 1), "pairs_forward_tc: npairs=%d exceeds the context's capacity %d", npairs, c->max_tokens * (c->top_k + 1));
    REQUIRE(n_items >= 0 && n_items <= c->max_experts + 1, "pairs_forward_tc: n_items=%d exceeds the context's capacity %d", n_items, c->max_experts + 1);
    if (n_items == 0) return MOEXB_OK;
    SidePlan plan{};
    plan.items = items; plan.n_items = n_items; plan.maxp = ST_MAXP; plan.subs = c->subs; plan.nsub = c->nsub;
    int rc = split_launch(c, X, T, stream, plan);
    if (rc != MOEXB_OK) return rc;
    return stream_experts(c, fmt, pairs, act, ypair, npairs, stream);
}

extern "C" int moexb_ctx_set_fused_decode(moexb_ctx* c, int on) {
    REQUIRE(c, "ctx_set_fused_decode: null context");
    c->fused_decode = on != 0;
    return MOEXB_OK;
}

extern "C" int moexb_ctx_set_pairs_per_pass(moexb_ctx* c, int pairs) {
    REQUIRE(c && (pairs == 4 || pairs == 8), "ctx_set_pairs_per_pass: 4 or 8");
    c->pairs_per_pass = pairs;
    return MOEXB_OK;
}

extern "C" int moexb_ctx_set_prefill_min_tokens(moexb_ctx* c, int tokens) {
    REQUIRE(c && tokens >= 1, "ctx_set_prefill_min_tokens: bad argument");
    c->prefill_min_tokens = tokens;
    return MOEXB_OK;
}

extern "C" int moexb_ctx_selftest_fail(moexb_ctx* c) {
    REQUIRE(c, "ctx_selftest_fail: null pointer");
    c->selftest_fail = true;
    return MOEXB_OK;
}

extern "C" int moexb_ctx_set_path(moexb_ctx* c, int path) {
    REQUIRE(c && (path == 0 || path == 1), "ctx_set_path: path must be 0 (streaming) or 1 (fp32 SIMT)");
    c->path = path;
    return MOEXB_OK;
}

// Waits for the device and returns the error word of the streaming kernels (0 = none; 1 / 2 = a consumer / the producer
// gave up waiting on a pipeline barrier), clearing it.
extern "C" int moexb_ctx_status(moexb_ctx* c, int* status) {
    REQUIRE(c && status, "ctx_status: null pointer");
    CUDA_TRY(cudaDeviceSynchronize());
    CUDA_TRY(cudaMemcpy(status, c->err, sizeof(int), cudaMemcpyDeviceToHost));
    if (*status) CUDA_TRY(cudaMemset(c->err, 0, sizeof(int)));
    return MOEXB_OK;
}

// Makes one bounded device-side wait run out on purpose and reports what the kernels' error word then holds.
// which = 0: the mbarrier wait of the streaming / grouped-GEMM pipelines (a barrier that expects bytes nobody sends);
// which = 1: the grid barrier of the one-token stack kernel (one CTA, two arrivals expected); which = 2: the wait of the
// expert-parallel kernels for a flag that another GPU raises (nobody raises it). All with `polls` polls instead of the
// production limits. Nothing faults or hangs: the kernel returns, the context stays usable.
extern "C" int moexb_ctx_selftest_timeout(moexb_ctx* c, int which, int polls, int* status) {
    REQUIRE(c && status, "ctx_selftest_timeout: null pointer");
    REQUIRE(which >= 0 && which <= 2 && polls > 0 && polls <= (1 << 20), "ctx_selftest_timeout: which=%d polls=%d", which, polls);
    CUDA_TRY(cudaSetDevice(c->device));
    CUDA_TRY(cudaMemset(c->nsub, 0, 2 * sizeof(int)));   // scratch of the self-test: [0] result of the wait
    unsigned* sync = reinterpret_cast<unsigned*>(c->counts);       // scratch: barrier counter and abort flag
    CUDA_TRY(cudaMemset(sync, 0, 2 * sizeof(unsigned)));
    if (which == 0) selftest_mbar_timeout_k<<<1, 32>>>(c->err, ST_ERR_FULL_WAIT, polls, c->nsub);
    else if (which == 1) selftest_grid_barrier_timeout_k<<<1, 32>>>(sync, c->err, polls, c->nsub);
    else selftest_ep_wait_timeout_k<<<1, 32>>>(sync, c->err, polls, c->nsub);
    LAUNCHED("selftest_timeout");
    return moexb_ctx_status(c, status);
}

extern "C" int moexb_ctx_selftest_swiglu(moexb_ctx* c, unsigned long long out[3]) {
    REQUIRE(c && out, "ctx_selftest_swiglu: null pointer");
    CUDA_TRY(cudaSetDevice(c->device));
    unsigned long long* d = nullptr;
    CUDA_TRY(cudaMalloc((void**)&d, 3 * sizeof(*d)));
    cudaError_t e = cudaMemset(d, 0, 3 * sizeof(*d));
    if (e == cudaSuccess) { selftest_swiglu_k<<<c->sms * 8, 256>>>(d); e = cudaGetLastError(); }
    if (e == cudaSuccess) e = cudaMemcpy(out, d, 3 * sizeof(*d), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? MOEXB_OK : fail(MOEXB_ERR_CUDA, "ctx_selftest_swiglu: %s", cudaGetErrorString(e));
}

extern "C" {

// Router logits (column n_routed = the shared expert's gate logit) and top-K for T tokens, into the context workspace.
// decode: also emit the K+1 one-pair sub-items of a single token (slots, weights, sub-items, pairs).
}  // extern "C"
// Router logits (into the context, [T][E + 1]) and the top-K selection in one launch; decode: also the K + 1 one-pair
// sub-items of a single token.
struct RouteEp { const EpDevice* dev; int row_bytes; unsigned phase; const unsigned* step; };
// pairs into the buckets (with the shared expert's); the caller's copies of ids and weights; split: the rows of x (x_dtype) are split by
// the routing kernel (ROWS_F16, ROWS_BF16; only where route_splits)
struct RouteOut { bool buckets = false, shared = false; int* idx = nullptr; float* w = nullptr; int x_dtype = MOEXB_F32, split = ROWS_NONE; };
// A layer whose router also makes its input rows and, split, leaves them in the context (combine_route_k): in a stack the end of the layer
// before (ranks rows of ypair a token; residual rows x; out; a dozen tokens at most), or the norm of the rows x of x_dtype (ranks = 0)
struct RouteCombine { const void* x; int x_dtype, ranks; float* out; bool f16; };
// A block per eight outputs of a token, which also splits its rows: up to 7 tokens, and 8 where the blocks are no more than two per SM (288
// experts); beyond, tiles of 8 tokens x 16 outputs. us a layer, tiles against blocks per token: 8 tokens of 32, 128, 256, 512 and 1024 experts
// 35.0 / 29.7, 42.4 / 36.6, 45.6 / 42.0, 59.3 / 60.1 and 67.0 / 75.7, of bf16 rows 35.0 / 31.1, 42.2 / 39.4, 45.5 / 45.6, 59.0 / 66.1 and
// 67.1 / 86.0; 256 experts 9 bf16 tokens 49.5 / 50.7, 12 and 16 tokens 54.3 / 54.7 and 59.4 / 59.5, 24 tokens 70.7 / 76.2.
static int route_blocks(int T, int E) { return T * ((E + 8) / 8); }
static bool route_splits(const moexb_ctx* c, int T, int E) { return T < 8 || (T == 8 && route_blocks(T, E) <= 2 * c->sms); }
template <typename WT>
static int route_launch(moexb_ctx* c, moexb_layer* L, const void* x, int T, int K, void* stream, bool decode, const RouteOut& ro, int tok0 = 0, const RouteEp* rep = nullptr,
                        const RouteCombine* rc = nullptr) {
    const float* xf = static_cast<const float*>(x);
    // tok0: the T rows at xf are tokens tok0.. of the batch - their logits, ids and weights go to those rows of the workspace
    const int E = L->n_routed;
    const WT* W = static_cast<const WT*>(L->router);
    float* logits = c->logits + (size_t)tok0 * (E + 1);
    TopkOut o{c->idx + (size_t)tok0 * K, c->w + (size_t)tok0 * K, L->slot_table, decode ? c->slots : nullptr, decode ? c->wts : nullptr,
              decode ? c->subs : nullptr, decode ? c->pairs : nullptr, decode ? c->nsub : nullptr};
    if (ro.buckets) {
        o.bcnt = c->bcnt; o.bpairs = c->bpairs; o.bstride = c->max_tokens; o.e_lo = L->first_local; o.e_hi = L->first_local + L->n_local; o.npairs = T * K;
        o.bshared = ro.shared; o.err = c->err;
    }
    o.idx2 = ro.idx; o.w2 = ro.w;
    if (rep) { o.ep = rep->dev; o.ep_row_bytes = rep->row_bytes; o.ep_phase = rep->phase; o.ep_step = rep->step; }
    auto run = [&]<int NJ>() -> int {
        if (rc) {
            auto combine = [&]<bool F16, typename XT>() -> int {
                constexpr auto kernel = combine_route_k<WT, NJ, F16, XT>;
                constexpr int SMEM = 8 * EH * (int)sizeof(WT);
                static PerDeviceOnce once;
                const cudaError_t attr_err = once.run([] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM); });
                if (attr_err != cudaSuccess) return fail(MOEXB_ERR_CUDA, "router kernel shared memory: %s", cudaGetErrorString(attr_err));
                const float *ypair = c->ypair, *extra = rc->ranks ? c->ypair + (size_t)T * K * EH : nullptr;
                CUDA_TRY(launch_dep(kernel, dim3((E + 1 + 7) / 8 + 1, T), 256, SMEM, S(stream), W, logits, E, K, 1, c->route_done, o, ypair, extra, static_cast<const XT*>(rc->x), rc->ranks,
                                    rc->out, c->xs, 1e-6f));
                LAUNCHED("combine_route");
                return MOEXB_OK;
            };
            if (rc->x_dtype == MOEXB_BF16) return rc->f16 ? combine.template operator()<true, __nv_bfloat16>() : combine.template operator()<false, __nv_bfloat16>();
            return rc->f16 ? combine.template operator()<true, float>() : combine.template operator()<false, float>();
        }
        // expert parallelism with few own tokens: one token per block row, so that each token's selection and dispatch stores are
        // done by a block of their own instead of one block sending a whole tile of 8
        if (route_splits(c, T, E) || (rep && T <= 16)) {
            constexpr int WARPS = 8;
            const dim3 grid((E + 1 + WARPS - 1) / WARPS + (ro.split ? 1 : 0), T);
            uint16_t* xs = ro.split ? c->xs : nullptr;
            if (ro.x_dtype == MOEXB_BF16)
                CUDA_TRY(launch_dep(route_gemv_k<WT, __nv_bfloat16, WARPS, NJ>, grid, WARPS * 32, 0, S(stream), W, static_cast<const __nv_bfloat16*>(x), logits, EH, E, K, 1, c->route_done, o, xs, ro.split));
            else CUDA_TRY(launch_dep(route_gemv_k<WT, float, WARPS, NJ>, grid, WARPS * 32, 0, S(stream), W, xf, logits, EH, E, K, 1, c->route_done, o, xs, ro.split));
        } else {
            // a small batch: 16 outputs x 8 tokens per block, to reach every SM; a prefill chunk goes to the register-tiled
            // kernel (64 tokens x 16 outputs per block, FMA-bound)
            auto gemm = [&]() -> int {
                constexpr int WARPS = 8, TO = 2, TR = 8, SMEM = TR * EH * (int)sizeof(float);
                static PerDeviceOnce once;
                const cudaError_t attr_err = once.run([] { return cudaFuncSetAttribute(route_gemm_k<WT, WARPS, TO, TR, NJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM); });
                if (attr_err != cudaSuccess) return fail(MOEXB_ERR_CUDA, "router kernel shared memory: %s", cudaGetErrorString(attr_err));
                CUDA_TRY(launch_dep(route_gemm_k<WT, WARPS, TO, TR, NJ>, dim3((E + 1 + WARPS * TO - 1) / (WARPS * TO), (T + TR - 1) / TR), WARPS * 32, SMEM, S(stream),
                                    W, xf, logits, EH, E, K, 1, T, c->route_done, o));
                return MOEXB_OK;
            };
            auto gemm2 = [&]() -> int {
                constexpr int SMEM = RG2_ST * rg2_stage_bytes<WT>();
                static PerDeviceOnce once;
                const cudaError_t attr_err = once.run([] { return cudaFuncSetAttribute(route_gemm2_k<WT, NJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM); });
                if (attr_err != cudaSuccess) return fail(MOEXB_ERR_CUDA, "router kernel shared memory: %s", cudaGetErrorString(attr_err));
                CUDA_TRY(launch_dep(route_gemm2_k<WT, NJ>, dim3((E + 1 + RG2_TN - 1) / RG2_TN, (T + RG2_TM - 1) / RG2_TM), 256, SMEM, S(stream),
                                    W, xf, logits, E, K, 1, T, c->route_done, o, rep ? 1 : 0));
                if (!rep) {
                    LAUNCHED("route");
                    CUDA_TRY(launch_dep(router_topk_k<8, NJ>, (T + 7) / 8, 256, 0, S(stream), (const float*)logits, E, K, 1, E + 1, T, o));
                }
                return MOEXB_OK;
            };
            const int rc = T >= 256 ? gemm2() : gemm();
            if (rc != MOEXB_OK) return rc;
        }
        LAUNCHED("route");
        return MOEXB_OK;
    };
    return E <= 256 ? run.template operator()<8>() : run.template operator()<32>();
}

extern "C" {
static int layer_route(moexb_ctx* c, moexb_layer* L, const void* xf, int T, int K, void* stream, bool decode, const RouteOut& ro, int tok0 = 0, const RouteEp* rep = nullptr, const RouteCombine* rc = nullptr) {
    PROF(c, MOEXB_PROF_ROUTER, stream);
    return L->router_dtype == MOEXB_F32 ? route_launch<float>(c, L, xf, T, K, stream, decode, ro, tok0, rep, rc) : route_launch<__half>(c, L, xf, T, K, stream, decode, ro, tok0, rep, rc);
}

// Zeroes the bucket counts on `st`. Under capture the graph does it when it runs, so what is in memory now stays marked.
static int clear_buckets(moexb_ctx* c, cudaStream_t st) {
    c->buckets_dirty = true;
    CUDA_TRY(cudaMemsetAsync(c->bcnt, 0, (size_t)c->max_experts * sizeof(int), st));
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CUDA_TRY(cudaStreamIsCapturing(st, &cap));
    c->buckets_dirty = cap != cudaStreamCaptureStatusNone;
    return MOEXB_OK;
}
// The router adds to the bucket counts; the combine kernel clears them, or the down kernel where there is none (a layer of a small stack that
// leaves its end to the next one). A call that returns between the two clears them itself, so that neither the next call nor the replay of a graph finds its pairs there. Where that fails too, the next call does it.
struct BucketCounts {
    moexb_ctx* c; cudaStream_t st; bool open = false;
    ~BucketCounts() {
        if (!open) return;
        char why[sizeof(g_err)];
        memcpy(why, g_err, sizeof(g_err));
        cudaGetLastError();
        clear_buckets(c, st);
        memcpy(g_err, why, sizeof(g_err));   // what the caller is told stays the first failure
    }
};

// One layer. X: the layer input [T][H] of x_dtype. flags as moexb_layer_forward. pre_normed: the context already holds
// rmsnorm(X) and its split (left there by the previous layer of a stack); next_norm: leave rmsnorm(out) and its
// split in the context for the next layer. chain_x (a stack of 2 to 12 tokens): the layer before left its end to this one's router, whose
// kernel makes X from chain_x, the residual rows of that layer; chain_next: this one leaves its end to the next one.
static int layer_impl(moexb_ctx* c, moexb_layer* L, const void* X, int x_dtype, int T, int K, float* out, int* idx_out, float* w_out, int flags,
                      void* stream, bool pre_normed, bool next_norm, int sh0 = 0, int sh1 = -1, const float* chain_x = nullptr, bool chain_next = false) {
    if (sh1 < 0) sh1 = T;
    const bool shared = !(flags & 1) && sh1 > sh0, block = flags & 2, partial = flags & 4, bf16 = x_dtype == MOEXB_BF16;
    const bool all_local = L->n_local == L->n_routed;
    const int E = L->n_routed, ld = E + 1;
    cudaStream_t st = S(stream);
    const bool tiled = L->layout == MOEXB_LAYOUT_TILED;
    const bool streaming = tiled || c->path == 0;
    // large batches go to the tcgen05 grouped GEMM; the rest to the streaming kernels
    const bool prefill = tiled && T >= grouped_min_tokens(c, L->fmt);
    const PlainLaunches plain(prefill);
    const bool f16 = tiled && L->fmt != FMT_ZP && !prefill;  // element type of the split activations the streaming kernels read
    const int parts = prefill && bf16 && !block ? 1 : 2;
    const int mode = !streaming ? ROWS_NONE : prefill ? (L->fmt == FMT_ZP ? ROWS_GEMM_Z : ROWS_GEMM) : f16 ? ROWS_F16 : ROWS_BF16;
    // xin: the input as f32 (for the residual and the fp32 kernels); xr: what the router sees, of xr_dtype
    const float* xin = bf16 ? c->xf : static_cast<const float*>(X);
    const void* xr = xin;
    RouteOut ro;
    int rc = MOEXB_OK;
    // A few tokens: the routing kernel normalises and splits the rows itself, up to 16 tokens and as many blocks as read their outputs' weights
    // in about the time of that launch (f16 weights are half as long). us a layer, by a launch before it against that: 256 experts 9, 12, 16,
    // 20 tokens 50.0 / 47.6, 55.5 / 53.9, 60.2 / 59.4, 68.1 / 70.4; zero point 9 and 12 tokens 72.9 / 70.5, 89.7 / 88.8; 512 experts 12 and 16
    // tokens 69.0 / 66.1 and 79.7 / 80.6, 1024 experts 8, 10, 12, 16 tokens 67.8 / 66.5, 72.8 / 73.1, 76.9 / 82.2, 88.4 / 99.5; f16 weights 512
    // experts 16 tokens 82.0 / 77.8, 1024 experts 10, 12, 16 tokens 74.2 / 69.1, 78.4 / 77.7, 90.6 / 94.6.
    const bool norm_in_route = block && !pre_normed && streaming && !prefill && T <= 16 && route_blocks(T, E) <= (L->router_dtype == MOEXB_F32 ? 7 : 11) * c->sms;
    if (block) {
        xr = c->xn;
        if (chain_x || norm_in_route) {}
        else if (!pre_normed || prefill) {   // (the previous layer leaves no rows for the grouped GEMM)
            rc = layer_rows(c, X, x_dtype, T, c->xf, true, c->xn, mode, c->xs, parts, stream);
        } else if (bf16) rc = layer_rows(c, X, x_dtype, T, c->xf, false, nullptr, ROWS_NONE, nullptr, 2, stream);
    } else if (streaming && !prefill && route_splits(c, T, E)) {
        xr = X; ro.x_dtype = x_dtype; ro.split = mode;
    } else if (mode != ROWS_NONE || bf16) rc = layer_rows(c, X, x_dtype, T, c->xf, false, nullptr, mode, c->xs, parts, stream);
    if (rc != MOEXB_OK) return rc;
    const float* xf = block ? c->xn : xin;   // what the router and the experts see, as f32
    const bool decode = T == 1 && all_local && shared && !partial && !prefill;
    const bool buckets = tiled && !decode && c->bpairs;
    ro.buckets = buckets; ro.shared = buckets && shared; ro.idx = idx_out; ro.w = w_out;
    if (buckets && c->buckets_dirty) { rc = clear_buckets(c, st); if (rc != MOEXB_OK) return rc; }
    BucketCounts counts{c, st, buckets};
    const RouteCombine rows = chain_x ? RouteCombine{chain_x, MOEXB_F32, K, const_cast<float*>(xin), f16} : RouteCombine{X, x_dtype, 0, bf16 ? c->xf : nullptr, f16};
    rc = layer_route(c, L, xr, T, K, stream, decode, ro, 0, nullptr, chain_x || norm_in_route ? &rows : nullptr);
    if (rc != MOEXB_OK) return rc;
    if (c->selftest_fail) { c->selftest_fail = false; return fail(MOEXB_ERR_CUDA, "layer: the failure that a self-test asked for"); }
    int ranks = K;                  // rows of ypair per token that the final reduction adds
    const float* extra = nullptr;   // + the shared expert's rows
    if (partial && !streaming) return fail(MOEXB_ERR_UNSUPPORTED, "layer_forward: partial outputs need the streaming kernels");
    if (decode && !streaming) {
        // one token on the fp32 SIMT kernels: the K routed experts and the shared expert as K+1 decode experts
        rc = decode_launch(c, L->fmt, c->slots, c->wts, K + 1, xf, c->act, block ? c->moe : out, stream, nullptr);
        if (rc != MOEXB_OK) return rc;
        if (block) {
            PROF(c, MOEXB_PROF_COMBINE, stream);
            residual_add_k<<<(unsigned)((EH / 4 + 255) / 256), 256, 0, st>>>(xin, c->moe, out, EH);
            LAUNCHED("residual_add");
            if (next_norm) { rc = layer_rows(c, out, MOEXB_F32, 1, nullptr, true, c->xn, ROWS_BF16, c->xs, 2, stream); if (rc != MOEXB_OK) return rc; }
        }
        ranks = 0;
    } else if (decode) {
        rc = tiled ? tiled_experts(c, L->fmt, c->pairs, nullptr, c->ypair, T, K, stream) : stream_experts(c, L->fmt, c->pairs, nullptr, c->ypair, K + 1, stream);
        if (rc != MOEXB_OK) return rc;
        ranks = K + 1;
    } else {
        const int maxp = prefill ? grouped_maxp(L->fmt) : (tiled ? tiled_maxp(c, L->fmt, T) : ST_MAXP);
        const BucketArgs bk{c->bcnt, c->bpairs, c->max_tokens, E, shared ? sh0 : 0, shared ? sh1 : 0, maxp, L->image - L->first_local * expert_bytes(L->fmt), L->slot_host[E]};
        if (!buckets) {
            PROF(c, MOEXB_PROF_GROUP, stream);
            // room in shared memory for the routed pairs (12 bytes each), so that the list is written out in full lines
            constexpr int PLAN_STAGE_MAX = 196608;
            static PerDeviceOnce plan_once;
            const cudaError_t plan_attr = plan_once.run([] { return cudaFuncSetAttribute(group_plan1_k<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, PLAN_STAGE_MAX); });
            const int stage_pairs = plan_attr == cudaSuccess && (size_t)T * K * 12 <= PLAN_STAGE_MAX ? T * K : 0;
            CUDA_TRY(launch_dep(group_plan1_k<false>, 1, 1024, (size_t)stage_pairs * 12, st, c->idx, c->w, T, K, E, L->slot_table, c->items, c->pairs, c->nitems, c->subs, c->nsub, maxp,
                                shared ? c->logits + E : nullptr, ld, sh0, sh1, stage_pairs,
                                (const unsigned*)nullptr, (const unsigned*)nullptr, 0u, 0, 0, (int*)nullptr));
            LAUNCHED("group_plan");
            // pairs of experts that are not held here are never written: the SIMT reduction path needs zeros there, the fused
            // reduction skips them by expert id
            if (!all_local && !streaming) CUDA_TRY(cudaMemsetAsync(c->ypair, 0, (size_t)T * K * EH * sizeof(float), st));
        }
        rc = prefill ? grouped_experts(c, L, c->pairs, parts, c->ypair, stream, buckets ? &bk : nullptr)
           : tiled ? tiled_experts(c, L->fmt, c->pairs, nullptr, c->ypair, T, K, stream, nullptr, buckets ? &bk : nullptr, chain_next)
           : streaming ? stream_experts(c, L->fmt, c->pairs, nullptr, c->ypair, T * (K + 1), stream)
                       : pairs_launch(c, L->fmt, c->items, c->nitems, min(E, T * K) + 1, c->pairs, xf, c->act, c->ypair, stream);
        if (rc != MOEXB_OK) return rc;
        if (shared) extra = c->ypair + (size_t)T * K * EH;
    }
    if (chain_next) { counts.open = false; return MOEXB_OK; }
    if (ranks) {
        PROF(c, MOEXB_PROF_COMBINE, stream);
        const float* xres = (block && !partial) ? xin : nullptr;
        float* xn_next = next_norm ? c->xn : nullptr;
        const int* held = (!all_local && ranks == K) ? c->idx : nullptr;
        if (f16) CUDA_TRY(launch_dep(reduce_residual_norm_k<true>, T, 256, 0, st, c->ypair, extra, xres, out, ranks, xn_next, c->xs, 1e-6f, sh0, sh1, held, L->first_local, L->first_local + L->n_local, buckets ? c->bcnt : (int*)nullptr, E));
        else CUDA_TRY(launch_dep(reduce_residual_norm_k<false>, T, 256, 0, st, c->ypair, extra, xres, out, ranks, xn_next, prefill ? (uint16_t*)nullptr : c->xs, 1e-6f, sh0, sh1, held, L->first_local, L->first_local + L->n_local, buckets ? c->bcnt : (int*)nullptr, E));
        LAUNCHED("reduce_residual_norm");
        counts.open = false;
    }
    return MOEXB_OK;
}

int moexb_layer_forward(moexb_ctx* c, moexb_layer* L, const void* X, int x_dtype, int T, int K, float* out, int* idx_out,
                        float* w_out, int flags, void* stream) {
    REQUIRE(c && L && X && out, "layer_forward: null pointer");
    REQUIRE(L->ctx == c, "layer_forward: layer belongs to another context");
    REQUIRE(T > 0 && T <= c->max_tokens, "layer_forward: T=%d exceeds the context's max_tokens=%d", T, c->max_tokens);
    REQUIRE(K > 0 && K <= c->top_k, "layer_forward: K=%d exceeds the context's top_k=%d", K, c->top_k);
    REQUIRE(x_dtype == MOEXB_F32 || x_dtype == MOEXB_BF16, "layer_forward: x_dtype=%d", x_dtype);
    REQUIRE((flags & 1) || L->loaded[L->n_routed], "layer_forward: the shared expert of this layer was never loaded (upload it, or pass flags bit 0 to leave it out)");
    return layer_impl(c, L, X, x_dtype, T, K, out, idx_out, w_out, flags, stream, false, false);
}

int moexb_layer_forward_ep(moexb_ctx* c, moexb_layer* L, const void* X, int x_dtype, int T, int K, float* out, int* idx_out,
                           float* w_out, int shared_t0, int shared_t1, int pre_normed, void* stream) {
    REQUIRE(c && L && X && out, "layer_forward_ep: null pointer");
    REQUIRE(L->ctx == c, "layer_forward_ep: layer belongs to another context");
    REQUIRE(T > 0 && T <= c->max_tokens, "layer_forward_ep: T=%d exceeds the context's max_tokens=%d", T, c->max_tokens);
    REQUIRE(K > 0 && K <= c->top_k, "layer_forward_ep: K=%d exceeds the context's top_k=%d", K, c->top_k);
    REQUIRE(x_dtype == MOEXB_F32 || x_dtype == MOEXB_BF16, "layer_forward_ep: x_dtype=%d", x_dtype);
    REQUIRE(shared_t0 >= 0 && shared_t0 <= shared_t1 && shared_t1 <= T, "layer_forward_ep: shared token range [%d, %d) outside 0..%d", shared_t0, shared_t1, T);
    REQUIRE(shared_t0 == shared_t1 || L->loaded[L->n_routed], "layer_forward_ep: the shared expert of this layer was never loaded");
    return layer_impl(c, L, X, x_dtype, T, K, out, idx_out, w_out, 2 | 4, stream, pre_normed != 0, false, shared_t0, shared_t1);
}

int moexb_ep_residual_norm(moexb_ctx* c, moexb_layer* next, const float* x, const float* total, float* out, int T, void* stream) {
    REQUIRE(c && x && total && out, "ep_residual_norm: null pointer");
    REQUIRE(T > 0 && T <= c->max_tokens, "ep_residual_norm: T=%d exceeds the context's max_tokens=%d", T, c->max_tokens);
    const bool f16 = next && next->layout == MOEXB_LAYOUT_TILED && next->fmt != FMT_ZP;
    float* xn = next ? c->xn : nullptr;
    PROF(c, MOEXB_PROF_COMBINE, stream);
    const float* no_extra = nullptr; const int* no_idx = nullptr;
    if (f16) CUDA_TRY(launch_dep(reduce_residual_norm_k<true>, T, 256, 0, S(stream), total, no_extra, x, out, 1, xn, c->xs, 1e-6f, 0, 0, no_idx, 0, 0, (int*)nullptr, 0));
    else CUDA_TRY(launch_dep(reduce_residual_norm_k<false>, T, 256, 0, S(stream), total, no_extra, x, out, 1, xn, c->xs, 1e-6f, 0, 0, no_idx, 0, 0, (int*)nullptr, 0));
    LAUNCHED("ep_residual_norm");
    return MOEXB_OK;
}

// ---- stack of layers as one CUDA graph ----------------------------------------------------------------------------------

struct moexb_stack {
    moexb_ctx* ctx = nullptr;
    int T = 0, K = 0, x_dtype = 0, n_layers = 0, kernels = 0;
    int out_rows = 0;            // rows of the result: T, or the own tokens of an expert-parallel rank
    void* x_in = nullptr;        // [T][H] of x_dtype
    float* buf[2] = {nullptr, nullptr};
    float* result = nullptr;     // = buf[(n_layers - 1) & 1]
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaStream_t cap = nullptr;
    // one-token residual stacks: a single cooperative launch instead of a graph
    bool fused = false;
    DecodeLayer* dlayers = nullptr;   // device
    unsigned* dsync = nullptr;        // device: barrier counter, abort flag
    int fmt = 0, router_dtype = 0, n_routed = 0;
};

int moexb_stack_destroy(moexb_stack* s) {
    if (!s) return MOEXB_OK;
    if (s->exec) cudaGraphExecDestroy(s->exec);
    if (s->graph) cudaGraphDestroy(s->graph);
    if (s->cap) cudaStreamDestroy(s->cap);
    cudaFree(s->x_in); cudaFree(s->buf[0]); cudaFree(s->buf[1]); cudaFree(s->dlayers); cudaFree(s->dsync);
    delete s;
    return MOEXB_OK;
}

}  // extern "C"
template <int FMT, typename WT, bool XBF>
static int decode_stack_launch(moexb_stack* s, const void* X, float* out, void* stream) {
    moexb_ctx* c = s->ctx;
    constexpr int SMEM = ds_smem_bytes<FMT>();
    static PerDeviceOnce once;
    const cudaError_t attr_err = once.run([] {
        cudaError_t e = cudaFuncSetAttribute(decode_stack_k<FMT, WT, XBF>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        int per_sm = 0;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, decode_stack_k<FMT, WT, XBF>, DS_THREADS, SMEM);
        if (e == cudaSuccess && per_sm < 1) e = cudaErrorLaunchOutOfResources;   // the persistent CTA does not fit an SM of this device
        return e;
    });
    if (attr_err != cudaSuccess) return fail(MOEXB_ERR_CUDA, "decode stack kernel: %s", cudaGetErrorString(attr_err));
    DecodeStackArgs a{s->dlayers, s->n_layers, s->n_routed, s->K, X, out, c->logits, c->act_split, c->ypair, c->wts, nullptr, nullptr, s->dsync, c->err};
    void* args[] = {&a};
    // cooperative: every CTA is resident, which the grid barrier inside relies on
    CUDA_TRY(cudaLaunchCooperativeKernel((void*)decode_stack_k<FMT, WT, XBF>, dim3(c->sms), dim3(DS_THREADS), args, SMEM, S(stream)));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return MOEXB_OK;
}
static int decode_stack_run(moexb_stack* s, const void* X, float* out, void* stream) {
    auto by_x = [&]<int FMT, typename WT>() {
        return s->x_dtype == MOEXB_BF16 ? decode_stack_launch<FMT, WT, true>(s, X, out, stream) : decode_stack_launch<FMT, WT, false>(s, X, out, stream);
    };
    auto by_w = [&]<int FMT>() {
        return s->router_dtype == MOEXB_F32 ? by_x.template operator()<FMT, float>() : by_x.template operator()<FMT, __half>();
    };
    return s->fmt == FMT_SYM_F16 ? by_w.template operator()<FMT_SYM_F16>() : s->fmt == FMT_ZP ? by_w.template operator()<FMT_ZP>() : by_w.template operator()<FMT_SYM_F32>();
}
extern "C" {

int moexb_stack_create(moexb_ctx* c, moexb_layer* const* layers, int n_layers, int T, int K, int x_dtype, int residual, moexb_stack** out) {
    REQUIRE(c && layers && out, "stack_create: null pointer");
    REQUIRE(n_layers > 0 && T > 0 && T <= c->max_tokens && K > 0 && K <= c->top_k, "stack_create: n_layers=%d T=%d K=%d", n_layers, T, K);
    REQUIRE(x_dtype == MOEXB_F32 || x_dtype == MOEXB_BF16, "stack_create: x_dtype=%d", x_dtype);
    REQUIRE(!c->profiling, "stack_create: switch profiling off before capturing a graph");
    for (int l = 0; l < n_layers; l++) {
        REQUIRE(layers[l] && layers[l]->ctx == c, "stack_create: layer %d is null or belongs to another context", l);
        REQUIRE(layers[l]->fmt == layers[0]->fmt && layers[l]->layout == layers[0]->layout, "stack_create: layer %d differs from layer 0 in format or layout", l);
        REQUIRE(layers[l]->loaded[layers[l]->n_routed], "stack_create: the shared expert of layer %d was never loaded", l);
    }
    CUDA_TRY(cudaSetDevice(c->device));
    moexb_stack* s = new (std::nothrow) moexb_stack;
    if (!s) return fail(MOEXB_ERR_NOMEM, "out of host memory");
    s->ctx = c; s->T = T; s->K = K; s->x_dtype = x_dtype; s->n_layers = n_layers; s->out_rows = T;
    const size_t n = (size_t)T * EH;
    cudaError_t e = cudaMalloc(&s->x_in, n * (x_dtype == MOEXB_BF16 ? 2 : 4));
    if (e == cudaSuccess) e = cudaMalloc((void**)&s->buf[0], n * 4);
    if (e == cudaSuccess) e = cudaMalloc((void**)&s->buf[1], n * 4);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s->cap, cudaStreamNonBlocking);
    if (e != cudaSuccess) { moexb_stack_destroy(s); return fail(MOEXB_ERR_NOMEM, "stack_create: %s", cudaGetErrorString(e)); }
    // one token through residual blocks of resident symmetric-format experts: one cooperative launch for the whole stack
    // (a CTA of the cooperative kernel owns at most two router rows, so E + 1 <= 2 x SMs)
    bool fused = c->fused_decode && T == 1 && residual && K <= DS_MAXK && n_layers <= DS_MAXLAYERS && layers[0]->n_routed + 1 <= 2 * c->sms && layers[0]->layout == MOEXB_LAYOUT_TILED;
    for (int l = 0; l < n_layers && fused; l++)
        fused = layers[l]->n_local == layers[l]->n_routed && layers[l]->n_routed == layers[0]->n_routed && layers[l]->n_routed <= 256 &&
                layers[l]->n_routed % 32 == 0 && layers[l]->router_dtype == layers[0]->router_dtype;
    if (fused) {
        std::vector<DecodeLayer> h(n_layers);
        for (int l = 0; l < n_layers; l++) h[l] = {layers[l]->router, layers[l]->slot_table};
        e = cudaMalloc((void**)&s->dlayers, n_layers * sizeof(DecodeLayer));
        if (e == cudaSuccess) e = cudaMalloc((void**)&s->dsync, 3 * sizeof(unsigned));
        if (e == cudaSuccess) e = cudaMemset(s->dsync, 0, 3 * sizeof(unsigned));
        if (e == cudaSuccess) e = cudaMemcpy(s->dlayers, h.data(), n_layers * sizeof(DecodeLayer), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) { moexb_stack_destroy(s); return fail(MOEXB_ERR_NOMEM, "stack_create: %s", cudaGetErrorString(e)); }
        s->fused = true; s->fmt = layers[0]->fmt; s->router_dtype = layers[0]->router_dtype; s->n_routed = layers[0]->n_routed;
        s->kernels = 1; s->result = s->buf[0];
        *out = s;
        return MOEXB_OK;
    }
    const long long before = g_launches.load();
    e = cudaStreamBeginCapture(s->cap, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) { moexb_stack_destroy(s); return fail(MOEXB_ERR_CUDA, "stack_create: begin capture: %s", cudaGetErrorString(e)); }
    // 2 to 12 tokens (zero point 8): a layer's end and the next one's routing are one kernel, where every layer has its buckets and all its experts here
    // (us a layer, two kernels against one: 9, 10, 12, 16, 20 tokens 40.0 / 37.8, 41.2 / 40.4, 44.5 / 44.1, 50.3 / 50.0, 54.8 / 58.0;
    // zero point 8 and 12 tokens 45.9 / 41.8 and 58.2 / 61.2; 4 to 15 ranks and 32 to 256 experts, from 15 % less to 0.4 % more)
    bool chain = residual && T > 1 && T <= (layers[0]->fmt == FMT_ZP ? 8 : 12) && layers[0]->layout == MOEXB_LAYOUT_TILED && c->bpairs && T < grouped_min_tokens(c, layers[0]->fmt);
    for (int l = 0; l < n_layers && chain; l++) chain = layers[l]->n_local == layers[l]->n_routed;
    const void* xin = s->x_in;
    const float* res = x_dtype == MOEXB_BF16 ? c->xf : static_cast<const float*>(s->x_in);   // the residual rows of the layer before
    int rc = MOEXB_OK;
    for (int l = 0; l < n_layers && rc == MOEXB_OK; l++) {
        // layer l leaves rmsnorm(x_{l+1}) and its split in the context, so layer l+1 starts at its router
        const int dt = l ? MOEXB_F32 : x_dtype;
        if (residual) rc = layer_impl(c, layers[l], xin, dt, T, K, s->buf[l & 1], nullptr, nullptr, 2, s->cap, l > 0, l + 1 < n_layers, 0, -1,
                                      chain && l ? res : nullptr, chain && l + 1 < n_layers);
        else rc = layer_impl(c, layers[l], xin, dt, T, K, s->buf[l & 1], nullptr, nullptr, 0, s->cap, false, false);
        if (l) res = static_cast<const float*>(xin);
        xin = s->buf[l & 1];
    }
    e = cudaStreamEndCapture(s->cap, &s->graph);
    s->kernels = (int)(g_launches.load() - before);
    g_launches.store(before);  // captured, not yet run
    if (rc != MOEXB_OK) { moexb_stack_destroy(s); return rc; }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&s->exec, s->graph, 0);
    if (e != cudaSuccess) { moexb_stack_destroy(s); return fail(MOEXB_ERR_CUDA, "stack_create: graph: %s", cudaGetErrorString(e)); }
    s->result = s->buf[(n_layers - 1) & 1];
    *out = s;
    return MOEXB_OK;
}

int moexb_stack_kernel_count(moexb_stack* s) { return s ? s->kernels : 0; }

int moexb_stack_run(moexb_stack* s, const void* X, float* out, void* stream) {
    REQUIRE(s && X && out, "stack_run: null pointer");
    const size_t n = (size_t)s->T * EH;
    // the one-token kernel reads and writes the caller's buffers itself where they allow 16-byte accesses
    if (s->fused && !((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(out)) & 15)) return decode_stack_run(s, X, out, stream);
    if (s->ctx->buckets_dirty) { const int rc = clear_buckets(s->ctx, S(stream)); if (rc != MOEXB_OK) return rc; }
    CUDA_TRY(cudaMemcpyAsync(s->x_in, X, n * (s->x_dtype == MOEXB_BF16 ? 2 : 4), cudaMemcpyDeviceToDevice, S(stream)));
    if (s->fused) { const int rc = decode_stack_run(s, s->x_in, s->buf[0], stream); if (rc != MOEXB_OK) return rc; }
    else {
        CUDA_TRY(cudaGraphLaunch(s->exec, S(stream)));
        g_launches.fetch_add(s->kernels, std::memory_order_relaxed);
    }
    CUDA_TRY(cudaMemcpyAsync(out, s->result, (size_t)s->out_rows * EH * 4, cudaMemcpyDeviceToDevice, S(stream)));
    return MOEXB_OK;
}

int moexb_stack_run_host(moexb_stack* s, const void* X_host, float* out_host, void* stream) {
    REQUIRE(s && X_host && out_host, "stack_run_host: null pointer");
    const size_t n = (size_t)s->T * EH;
    if (s->ctx->buckets_dirty) { const int rc = clear_buckets(s->ctx, S(stream)); if (rc != MOEXB_OK) return rc; }
    CUDA_TRY(cudaMemcpyAsync(s->x_in, X_host, n * (s->x_dtype == MOEXB_BF16 ? 2 : 4), cudaMemcpyHostToDevice, S(stream)));
    if (s->fused) { const int rc = decode_stack_run(s, s->x_in, s->buf[0], stream); if (rc != MOEXB_OK) return rc; }
    else {
        CUDA_TRY(cudaGraphLaunch(s->exec, S(stream)));
        g_launches.fetch_add(s->kernels, std::memory_order_relaxed);
    }
    CUDA_TRY(cudaMemcpyAsync(out_host, s->result, (size_t)s->out_rows * EH * 4, cudaMemcpyDeviceToHost, S(stream)));
    CUDA_TRY(cudaStreamSynchronize(S(stream)));
    return MOEXB_OK;
}

// ---- expert parallelism: token all-to-all over peer memory (ep.cuh) -----------------------------------------------------------

struct moexb_ep {
    moexb_ctx* ctx = nullptr;
    EpGeom g{};
    EpPeers peers{};
    EpLayout lay{};
    int n_routed = 0;
    float* x = nullptr;         // [n_own_max][H] residual rows of the own tokens
    unsigned* step = nullptr;   // device: steps begun so far
    EpDevice* dev = nullptr;    // device copy of geometry, peer pointers and layout (what the routing kernel's push reads)
    // what the context pointed at before its activations, ids and weights moved into the exchange buffer
    uint16_t* saved_xs = nullptr; int* saved_idx = nullptr; float* saved_w = nullptr;
    // host-side state of the layer in progress (set by dispatch, used by experts)
    bool prefill = false; int parts = 2;
};

size_t moexb_ep_buffer_bytes(int max_tokens, int top_k, int world) {
    if (max_tokens <= 0 || top_k <= 0 || world <= 0 || world > EP_MAX_RANKS) return 0;
    return ep_layout(max_tokens, top_k, world).bytes;
}

int moexb_ep_buffer_alloc(size_t bytes, void** ptr, unsigned char* handle) {
    REQUIRE(ptr && bytes > 0, "ep_buffer_alloc: bad argument");
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, bytes);
    if (e != cudaSuccess) return fail(MOEXB_ERR_NOMEM, "ep_buffer_alloc: cudaMalloc of %zu bytes: %s", bytes, cudaGetErrorString(e));
    e = cudaMemset(p, 0, bytes);
    if (e == cudaSuccess && handle) {
        static_assert(sizeof(cudaIpcMemHandle_t) == 64, "an IPC handle is 64 bytes");
        cudaIpcMemHandle_t h;
        e = cudaIpcGetMemHandle(&h, p);
        if (e == cudaSuccess) memcpy(handle, &h, 64);
    }
    if (e != cudaSuccess) { cudaFree(p); return fail(MOEXB_ERR_CUDA, "ep_buffer_alloc: %s", cudaGetErrorString(e)); }
    *ptr = p;
    return MOEXB_OK;
}

int moexb_ep_buffer_open(const unsigned char* handle, void** ptr) {
    REQUIRE(handle && ptr, "ep_buffer_open: null pointer");
    cudaIpcMemHandle_t h;
    memcpy(&h, handle, 64);
    CUDA_TRY(cudaIpcOpenMemHandle(ptr, h, cudaIpcMemLazyEnablePeerAccess));
    return MOEXB_OK;
}

int moexb_ep_buffer_close(void* ptr) {
    if (ptr) CUDA_TRY(cudaIpcCloseMemHandle(ptr));
    return MOEXB_OK;
}

int moexb_ep_buffer_free(void* ptr) {
    if (ptr) CUDA_TRY(cudaFree(ptr));
    return MOEXB_OK;
}

int moexb_ep_create(moexb_ctx* c, int rank, int world, int T, int K, int n_routed, void* const* bufs, moexb_ep** out) {
    REQUIRE(c && bufs && out, "ep_create: null pointer");
    REQUIRE(world >= 1 && world <= EP_MAX_RANKS && rank >= 0 && rank < world, "ep_create: rank %d of %d (at most %d ranks)", rank, world, EP_MAX_RANKS);
    REQUIRE(T >= world && T <= c->max_tokens, "ep_create: T=%d must be at least the number of ranks (%d) and at most the context's max_tokens=%d", T, world, c->max_tokens);
    REQUIRE(K > 0 && K <= c->top_k, "ep_create: K=%d exceeds the context's top_k=%d", K, c->top_k);
    REQUIRE(n_routed >= world && n_routed <= c->max_experts, "ep_create: n_routed=%d", n_routed);
    for (int r = 0; r < world; r++) REQUIRE(bufs[r], "ep_create: the exchange buffer of rank %d is null", r);
    CUDA_TRY(cudaSetDevice(c->device));
    moexb_ep* e = new (std::nothrow) moexb_ep;
    if (!e) return fail(MOEXB_ERR_NOMEM, "out of host memory");
    e->ctx = c; e->n_routed = n_routed;
    e->g.rank = rank; e->g.world = world; e->g.T = T; e->g.K = K; e->g.n_own_max = (T + world - 1) / world;
    for (int r = 0; r <= EP_MAX_RANKS; r++) {
        const int rr = min(r, world);
        e->g.tok0[r] = rr * (T / world) + min(rr, T % world);
        e->g.exp0[r] = rr * (n_routed / world) + min(rr, n_routed % world);
    }
    for (int r = 0; r < EP_MAX_RANKS; r++) e->peers.base[r] = r < world ? static_cast<uint8_t*>(bufs[r]) : nullptr;
    e->lay = ep_layout(T, K, world);
    cudaError_t err = cudaMalloc((void**)&e->x, (size_t)e->g.n_own_max * EH * sizeof(float));
    if (err == cudaSuccess) err = cudaMalloc((void**)&e->step, sizeof(unsigned));
    if (err == cudaSuccess) err = cudaMalloc((void**)&e->dev, sizeof(EpDevice));
    if (err == cudaSuccess) err = cudaMemset(e->step, 0, sizeof(unsigned));
    if (err == cudaSuccess) { const EpDevice h{e->g, e->peers, e->lay}; err = cudaMemcpy(e->dev, &h, sizeof h, cudaMemcpyHostToDevice); }
    if (err != cudaSuccess) { cudaFree(e->x); cudaFree(e->step); cudaFree(e->dev); delete e; return fail(MOEXB_ERR_NOMEM, "ep_create: %s", cudaGetErrorString(err)); }
    // the context's activation columns, ids and weights now live in this rank's exchange buffer, where the peers write them
    uint8_t* local = e->peers.base[rank];
    e->saved_xs = c->xs; e->saved_idx = c->idx; e->saved_w = c->w;
    c->xs = reinterpret_cast<uint16_t*>(local + e->lay.xs);
    c->idx = reinterpret_cast<int*>(local + e->lay.idx);
    c->w = reinterpret_cast<float*>(local + e->lay.w);
    *out = e;
    return MOEXB_OK;
}

int moexb_ep_destroy(moexb_ep* e) {
    if (!e) return MOEXB_OK;
    e->ctx->xs = e->saved_xs; e->ctx->idx = e->saved_idx; e->ctx->w = e->saved_w;
    cudaFree(e->x); cudaFree(e->step); cudaFree(e->dev);
    delete e;
    return MOEXB_OK;
}

int moexb_ep_own_tokens(const moexb_ep* e, int* first, int* count) {
    REQUIRE(e, "ep_own_tokens: null pointer");
    if (first) *first = e->g.tok0[e->g.rank];
    if (count) *count = e->g.tok0[e->g.rank + 1] - e->g.tok0[e->g.rank];
    return MOEXB_OK;
}

int moexb_ep_read_routing(moexb_ep* e, int* idx_out, float* w_out, void* stream) {
    REQUIRE(e, "ep_read_routing: null pointer");
    const size_t n = (size_t)e->g.T * e->g.K;
    if (idx_out) CUDA_TRY(cudaMemcpyAsync(idx_out, e->ctx->idx, n * sizeof(int), cudaMemcpyDeviceToDevice, S(stream)));
    if (w_out) CUDA_TRY(cudaMemcpyAsync(w_out, e->ctx->w, n * sizeof(float), cudaMemcpyDeviceToDevice, S(stream)));
    return MOEXB_OK;
}

int moexb_ep_begin_step(moexb_ep* e, void* stream) {
    REQUIRE(e, "ep_begin_step: null pointer");
    ep_step_k<<<1, 1, 0, S(stream)>>>(e->step);
    LAUNCHED("ep_step");
    return MOEXB_OK;
}

}  // extern "C"

static int ep_check_layer(const moexb_ep* e, const moexb_layer* L, int l, const char* who) {
    REQUIRE(e && L, "%s: null pointer", who);
    REQUIRE(L->ctx == e->ctx, "%s: layer belongs to another context", who);
    REQUIRE(l >= 0 && l + 1 < (int)EP_PHASES, "%s: layer index %d", who, l);
    REQUIRE(L->n_routed == e->n_routed && L->first_local == e->g.exp0[e->g.rank] && L->n_local == e->g.exp0[e->g.rank + 1] - e->g.exp0[e->g.rank],
            "%s: the layer holds experts [%d, %d) of %d, this rank's share is [%d, %d) of %d", who, L->first_local, L->first_local + L->n_local,
            L->n_routed, e->g.exp0[e->g.rank], e->g.exp0[e->g.rank + 1], e->n_routed);
    REQUIRE(L->loaded[L->n_routed], "%s: the shared expert of this layer was never loaded", who);
    return MOEXB_OK;
}

// The owner's side of the combine of layer `l - 1` (l >= 1), leaving the next layer's input (or, with `out`, the result).
static int ep_combine(moexb_ep* e, bool f16, bool residual, unsigned phase, float* out, bool next, bool split, void* stream) {
    moexb_ctx* c = e->ctx;
    const int n_own = e->g.tok0[e->g.rank + 1] - e->g.tok0[e->g.rank];
    const float* extra = c->ypair + (size_t)e->g.T * e->g.K * EH;   // the shared expert's rows, by absolute token
    float* x = residual ? e->x : nullptr;
    float* xn = next ? c->xn : nullptr;
    uint16_t* xs = next && split ? c->xs : nullptr;
    PROF(c, MOEXB_PROF_COMBINE, stream);
    if (f16) CUDA_TRY(launch_dep(ep_combine_norm_k<true>, n_own, 256, 0, S(stream), e->g, (const uint8_t*)e->peers.base[e->g.rank], e->lay, extra, x, out, xn, xs, residual ? 1 : 0, 1e-6f, (const unsigned*)e->step, phase, c->err));
    else CUDA_TRY(launch_dep(ep_combine_norm_k<false>, n_own, 256, 0, S(stream), e->g, (const uint8_t*)e->peers.base[e->g.rank], e->lay, extra, x, out, xn, xs, residual ? 1 : 0, 1e-6f, (const unsigned*)e->step, phase, c->err));
    LAUNCHED("ep_combine_norm");
    return MOEXB_OK;
}

extern "C" {

int moexb_ep_dispatch(moexb_ep* e, moexb_layer* L, int l, const void* X, int x_dtype, int residual, void* stream) {
    int rc = ep_check_layer(e, L, l, "ep_dispatch");
    if (rc != MOEXB_OK) return rc;
    REQUIRE(l > 0 || X, "ep_dispatch: layer 0 needs the input");
    REQUIRE(x_dtype == MOEXB_F32 || x_dtype == MOEXB_BF16, "ep_dispatch: x_dtype=%d", x_dtype);
    moexb_ctx* c = e->ctx;
    cudaStream_t st = S(stream);
    const int T = e->g.T, K = e->g.K, t0 = e->g.tok0[e->g.rank], n_own = e->g.tok0[e->g.rank + 1] - t0;
    const bool tiled = L->layout == MOEXB_LAYOUT_TILED;
    REQUIRE(tiled || c->path == 0, "ep_dispatch: expert parallelism runs on the streaming kernels");
    // (zero point stays on the streaming kernels: the grouped GEMM's chunk sums are not among what the owners send)
    const bool prefill = tiled && L->fmt != FMT_ZP && T >= grouped_min_tokens(c, L->fmt);
    const bool f16 = tiled && L->fmt != FMT_ZP && !prefill;
    // activation columns per token: the grouped GEMM takes one when the layer input is exactly bf16, else hi + lo
    const int parts = prefill && x_dtype == MOEXB_BF16 && !residual && l == 0 ? 1 : 2;
    e->prefill = prefill; e->parts = parts;
    const int mode = prefill ? ROWS_GEMM : f16 ? ROWS_F16 : ROWS_BF16;
    float* xn_own = c->xn + (size_t)t0 * EH;
    if (l == 0) {
        // the own rows of the input as fp32 into the residual rows (blocks) or straight into the layer input (plain layers), with the
        // norm and the split in the same pass
        float* dst = residual ? e->x : xn_own;
        const size_t n = (size_t)n_own * EH;
        const uint8_t* own = static_cast<const uint8_t*>(X) + (size_t)t0 * EH * (x_dtype == MOEXB_BF16 ? 2 : 4);
        const bool f32 = x_dtype == MOEXB_F32;
        if (f32) CUDA_TRY(cudaMemcpyAsync(dst, own, n * sizeof(float), cudaMemcpyDeviceToDevice, st));
        // f32 rows are read from the copy: the caller's may begin at any float
        rc = layer_rows(c, f32 ? static_cast<const void*>(dst) : own, x_dtype, n_own, dst, residual != 0, xn_own, mode, c->xs + (size_t)t0 * parts * EH, parts, stream);
        if (rc != MOEXB_OK) return rc;
    } else {
        rc = ep_combine(e, f16, residual != 0, (unsigned)l, nullptr, true, !prefill, stream);
        if (rc != MOEXB_OK) return rc;
        if (prefill) {
            rc = layer_rows(c, xn_own, MOEXB_F32, n_own, nullptr, false, nullptr, mode, c->xs + (size_t)t0 * parts * EH, parts, stream);
            if (rc != MOEXB_OK) return rc;
        }
    }
    // the routing kernel sends each token to the peers as soon as its experts are selected and raises the tokens' flags
    const RouteEp rep{e->dev, parts * EH * 2, (unsigned)(l + 1), e->step};
    return layer_route(c, L, xn_own, n_own, K, stream, false, RouteOut{}, t0, &rep);
}

int moexb_ep_experts(moexb_ep* e, moexb_layer* L, int l, void* stream) {
    int rc = ep_check_layer(e, L, l, "ep_experts");
    if (rc != MOEXB_OK) return rc;
    moexb_ctx* c = e->ctx;
    cudaStream_t st = S(stream);
    const int T = e->g.T, K = e->g.K, E = L->n_routed, t0 = e->g.tok0[e->g.rank], t1 = e->g.tok0[e->g.rank + 1];
    const bool tiled = L->layout == MOEXB_LAYOUT_TILED, prefill = e->prefill;
    const int maxp = prefill ? grouped_maxp(L->fmt) : (tiled ? tiled_maxp(c, L->fmt, T) : ST_MAXP);
    const unsigned* flags = reinterpret_cast<const unsigned*>(e->peers.base[e->g.rank] + e->lay.flag_a);
    const bool in_kernel = tiled && !prefill && plan_in_kernel(L->fmt, T, K, E);
    // the dispatch flags of all tokens are waited for by whoever makes the work list: the gate/up CTAs, or the planning kernel
    const PlanArgs plan{c->idx, c->w, T, K, E, L->slot_table, L->first_local, L->first_local + L->n_local, c->logits + E, E + 1, t0, t1, maxp, c->subs, c->pairs, c->nsub, flags, e->step, (unsigned)(l + 1)};
    if (!in_kernel) {
        PROF(c, MOEXB_PROF_GROUP, stream);
        constexpr int PLAN_STAGE_MAX = 196608;
        static PerDeviceOnce plan_once;
        const cudaError_t plan_attr = plan_once.run([] { return cudaFuncSetAttribute(group_plan1_k<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, PLAN_STAGE_MAX); });
        const int stage_pairs = plan_attr == cudaSuccess && (size_t)T * K * 12 <= PLAN_STAGE_MAX ? T * K : 0;
        CUDA_TRY(launch_dep(group_plan1_k<true>, 1, 1024, (size_t)stage_pairs * 12, st, (const int*)c->idx, (const float*)c->w, T, K, E, L->slot_table, c->items, c->pairs, c->nitems,
                            c->subs, c->nsub, maxp, (const float*)(c->logits + E), E + 1, t0, t1, stage_pairs,
                            flags, (const unsigned*)e->step, (unsigned)(l + 1), e->g.world, e->g.rank, c->err));
        LAUNCHED("group_plan");
    }
    rc = prefill ? grouped_experts(c, L, c->pairs, e->parts, c->ypair, stream)
       : tiled ? tiled_experts(c, L->fmt, c->pairs, nullptr, c->ypair, T, K, stream, in_kernel ? &plan : nullptr)
               : stream_experts(c, L->fmt, c->pairs, nullptr, c->ypair, T * (K + 1), stream);
    if (rc != MOEXB_OK) return rc;
    PROF(c, MOEXB_PROF_COMBINE, stream);
    CUDA_TRY(launch_dep(ep_partial_push_k, T, 256, 0, st, e->g, e->peers, e->lay, (const float*)c->ypair, (const unsigned*)e->step, (unsigned)(l + 1)));
    LAUNCHED("ep_partial_push");
    return MOEXB_OK;
}

int moexb_ep_finish(moexb_ep* e, int n_layers, int residual, float* out_own, void* stream) {
    REQUIRE(e && out_own, "ep_finish: null pointer");
    REQUIRE(n_layers >= 1 && n_layers < (int)EP_PHASES, "ep_finish: %d layers", n_layers);
    return ep_combine(e, true, residual != 0, (unsigned)n_layers, out_own, false, false, stream);
}

// One whole step on `stream`: begin, per layer dispatch + experts, finish. X [T][H] of x_dtype (every rank passes the whole
// batch and uses its own rows), out_own [own tokens][H].
int moexb_ep_step(moexb_ep* e, moexb_layer* const* layers, int n_layers, const void* X, int x_dtype, int residual, float* out_own, void* stream) {
    REQUIRE(e && layers && X && out_own, "ep_step: null pointer");
    int rc = moexb_ep_begin_step(e, stream);
    for (int l = 0; l < n_layers && rc == MOEXB_OK; l++) {
        rc = moexb_ep_dispatch(e, layers[l], l, X, x_dtype, residual, stream);
        if (rc == MOEXB_OK) rc = moexb_ep_experts(e, layers[l], l, stream);
    }
    if (rc == MOEXB_OK) rc = moexb_ep_finish(e, n_layers, residual, out_own, stream);
    return rc;
}

int moexb_ep_stack_create(moexb_ep* e, moexb_layer* const* layers, int n_layers, int x_dtype, int residual, moexb_stack** out) {
    REQUIRE(e && layers && out, "ep_stack_create: null pointer");
    REQUIRE(n_layers >= 1 && n_layers < (int)EP_PHASES, "ep_stack_create: %d layers", n_layers);
    REQUIRE(residual || n_layers == 1, "ep_stack_create: plain (non-residual) layers are chained one at a time");
    moexb_ctx* c = e->ctx;
    REQUIRE(!c->profiling, "ep_stack_create: switch profiling off before capturing a graph");
    CUDA_TRY(cudaSetDevice(c->device));
    moexb_stack* s = new (std::nothrow) moexb_stack;
    if (!s) return fail(MOEXB_ERR_NOMEM, "out of host memory");
    const int T = e->g.T;
    s->ctx = c; s->T = T; s->K = e->g.K; s->x_dtype = x_dtype; s->n_layers = n_layers;
    s->out_rows = e->g.tok0[e->g.rank + 1] - e->g.tok0[e->g.rank];
    const size_t n = (size_t)T * EH;
    cudaError_t err = cudaMalloc(&s->x_in, n * (x_dtype == MOEXB_BF16 ? 2 : 4));
    if (err == cudaSuccess) err = cudaMalloc((void**)&s->buf[0], (size_t)e->g.n_own_max * EH * 4);
    if (err == cudaSuccess) err = cudaStreamCreateWithFlags(&s->cap, cudaStreamNonBlocking);
    if (err != cudaSuccess) { moexb_stack_destroy(s); return fail(MOEXB_ERR_NOMEM, "ep_stack_create: %s", cudaGetErrorString(err)); }
    const long long before = g_launches.load();
    err = cudaStreamBeginCapture(s->cap, cudaStreamCaptureModeThreadLocal);
    if (err != cudaSuccess) { moexb_stack_destroy(s); return fail(MOEXB_ERR_CUDA, "ep_stack_create: begin capture: %s", cudaGetErrorString(err)); }
    const int rc = moexb_ep_step(e, layers, n_layers, s->x_in, x_dtype, residual, s->buf[0], s->cap);
    err = cudaStreamEndCapture(s->cap, &s->graph);
    s->kernels = (int)(g_launches.load() - before);
    g_launches.store(before);
    if (rc != MOEXB_OK) { moexb_stack_destroy(s); return rc; }
    if (err == cudaSuccess) err = cudaGraphInstantiate(&s->exec, s->graph, 0);
    if (err != cudaSuccess) { moexb_stack_destroy(s); return fail(MOEXB_ERR_CUDA, "ep_stack_create: graph: %s", cudaGetErrorString(err)); }
    s->result = s->buf[0];
    *out = s;
    return MOEXB_OK;
}

// ---- instrumentation ------------------------------------------------------------------------------------------------------

long long moexb_launch_count(void) { return g_launches.load(); }
int moexb_short_residency(void) { return g_short_residency.load(); }

int moexb_ctx_profile(moexb_ctx* c, int on) {
    REQUIRE(c, "ctx_profile: null context");
    c->profiling = on != 0;
    return MOEXB_OK;
}

int moexb_ctx_profile_read(moexb_ctx* c, float* ms, int* launches) {
    REQUIRE(c && ms && launches, "ctx_profile_read: null pointer");
    CUDA_TRY(cudaDeviceSynchronize());
    for (int i = 0; i < MOEXB_PROF_TAGS; i++) { ms[i] = 0.f; launches[i] = 0; }
    for (auto& r : c->recs) {
        float t = 0.f;
        CUDA_TRY(cudaEventElapsedTime(&t, r.a, r.b));
        ms[r.tag] += t; launches[r.tag]++;
        c->spare.push_back(r.a); c->spare.push_back(r.b);
    }
    c->recs.clear();
    return MOEXB_OK;
}

}  // extern "C"

// ---- one-token experts with built-in scratch ------------------------------------------------------------------------------
//
// moexb_experts_forward_static is for callers that cannot allocate device memory: an engine that sizes its expert cache
// from whatever memory is free at load time has no bytes left to ask for afterwards, and code on a latency-critical
// decode thread must not call cudaMalloc at all, because an allocation can block on the whole device.
// moexb_experts_forward asks such a caller for an `act` buffer; this variant brings its own.

namespace {
constexpr int STATIC_MAX_K = 16;  // experts per call: the scratch holds STATIC_MAX_K x I floats = 32 KB
constexpr int STATIC_MAX_DEVICES = 64;
// act[k][I] of the call in flight. Every GPU that loads the library holds these 32 KB until the process exits.
// In host code this name is only a handle for cudaGetSymbolAddress, never a device address to hand to a kernel.
static __device__ __align__(256) float g_static_act[STATIC_MAX_K * EI];
std::mutex g_static_lock;
float* g_static_ptr[STATIC_MAX_DEVICES];  // device address of g_static_act per device, resolved on first use
}  // namespace

extern "C" int moexb_experts_forward_static(int fmt, const uint8_t* const* slots, const float* w, int K, const float* x, float* out,
                                            void* stream, const int* nh) {
    REQUIRE(slots && w && x && out, "experts_forward_static: null pointer");
    REQUIRE(K >= 1 && K <= STATIC_MAX_K, "experts_forward_static: K=%d exceeds the built-in scratch (at most %d experts per call)", K, STATIC_MAX_K);
    REQUIRE(fmt_ok(fmt), "experts_forward_static: unknown expert format %d", fmt);
    int dev = -1;
    CUDA_TRY(cudaGetDevice(&dev));
    REQUIRE(dev >= 0 && dev < STATIC_MAX_DEVICES, "experts_forward_static: device %d out of range", dev);
    float* act;
    {
        // Set-up, once per device and with that device current: ask the runtime where the array lives on this GPU.
        std::lock_guard<std::mutex> lock(g_static_lock);
        if (!g_static_ptr[dev]) {
            void* p = nullptr;
            CUDA_TRY(cudaGetSymbolAddress(&p, g_static_act));
            REQUIRE(p, "experts_forward_static: the scratch array has no address on device %d", dev);
            g_static_ptr[dev] = static_cast<float*>(p);
        }
        act = g_static_ptr[dev];
    }
    // Nothing in the array has to start at zero: the first kernel writes rows k < K (or < *nh), the second reads only those.
    return by_fmt(fmt, [&]<int FMT>() {
        constexpr int WARPS = 8;
        decode_gate_up_k<FMT, WARPS><<<dim3(EI / WARPS, K), WARPS * 32, 0, S(stream)>>>(slots, K, nh, x, act);
        LAUNCHED("decode_gate_up (static scratch)");
        decode_down_k<FMT, WARPS, STATIC_MAX_K><<<EH / WARPS, WARPS * 32, K * pad32_size(EI) * sizeof(float), S(stream)>>>(slots, w, K, nh, act, out);
        LAUNCHED("decode_down (static scratch)");
        return (int)MOEXB_OK;
    });
}
