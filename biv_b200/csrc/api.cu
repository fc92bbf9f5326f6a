// The C ABI of include/bivmoe.h: layer objects, weight upload and repack,
// workspace, the forward sequence and the parity taps.
#include <cuda.h>
#include <cuda_fp16.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <new>
#include <string>
#include <vector>

#include "common.cuh"
#include "host_buffers.h"
#include "launch.cuh"

namespace bivmoe {

static std::atomic<uint64_t> g_launches{0};
void count_launch(int n) { g_launches.fetch_add((uint64_t)n, std::memory_order_relaxed); }

static thread_local std::string g_error;
static thread_local uint64_t g_oom_bytes = 0;   // size of the device allocation that failed last

// cudaMalloc that remembers the size of a failed request (Error::OutOfMemory{bytes})
static cudaError_t dev_alloc(void** p, size_t bytes) {
    const cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) {
        g_oom_bytes = bytes;
        cudaGetLastError();   // reported by the caller: a later call must not find it
    }
    return e;
}

static int set_err(std::string* dst, int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    (dst ? *dst : g_error) = buf;
    return code;
}

struct Arena {   // carves 256-byte aligned pieces out of one allocation
    size_t off = 0;
    uint8_t* base = nullptr;
    template <class T> T* take(size_t count) {
        size_t bytes = (count * sizeof(T) + 255) & ~(size_t)255;
        T* p = base && count ? (T*)(base + off) : nullptr;
        off += bytes;
        return p;
    }
};

}  // namespace bivmoe

using namespace bivmoe;

// bivmoe_forward_host: the most sections of one call, by the rule and by request
constexpr int kHostSectionsDefault = 6, kHostSectionsMax = 8;
// up to this many bytes of rows the kernels read and write page-locked host memory themselves
constexpr size_t kHostDirectBytes = 8 << 20;
// rows of more than this many bytes (that no cache holds) share their place in a workspace
constexpr size_t kShareBytes = 128 << 20;
// shapes of bivmoe_forward calls a layer keeps a graph for (an engine's batch size moves
// between a few values from step to step)
constexpr int kForwardGraphs = 8;

struct bivmoe_layer {
    int device = 0, sm_count = 0;
    bool all_bf16 = false;   // every matrix is BF16: three-term activations, the products on the tensor cores
    bool dense = false;   // made by bivmoe_dense_create: one expert behind a router of zeros
    int e = 0, n_expert = 0, k = 0, ff = 0, ff_sh = 0, max_tokens = 0;
    bool has_shared = false;
    DevTiles gate_up, down, sh_gate_up, sh_down;
    float* router = nullptr;      // [n_expert + 1][e]; the last row is the shared-gate vector
    float* post_norm = nullptr;   // [e]
    float norm_eps = 0.0f;
    uint64_t state_id = 0;        // new_state_id() of what a stack's graph holds of the layer by value
    uint8_t* ws_mem = nullptr;
    size_t ws_bytes = 0, weight_bytes = 0;
    Workspace ws{};
    cudaStream_t own_stream = nullptr;   // bivmoe_forward_host
    // a host-buffer call over many rows runs in sections: the copy-in of the next section
    // and the copy-out of the last one (streams of their own) overlap the section at work
    cudaStream_t in_stream = nullptr, out_stream = nullptr;
    cudaEvent_t host_ev[2 * (kHostSectionsMax + 1) + 2] = {};
    float* host_in = nullptr;            // device staging of forward_host
    float* host_out = nullptr;
    int last_n = 0;              // rows of the last call, which the taps describe
    bool last_wide = false;      // that call's quantised rows are f16 records
    bool last_few = false;       // that call's rows were quantised by experts_few_kernel: token t's at position t
    bool in_sections = false;    // that call was a host call in sections: the workspace holds the last one's rows
    int host_sections_forced = 0;    // BIVMOE_HOST_SECTIONS when the layer was made
    bool host_in_sections = false;   // ... of the host call enqueued or captured last
    // the launch sequences of recent forward calls as CUDA graphs, one per (n, accumulate)
    struct ForwardGraph {
        cudaGraphExec_t exec = nullptr;
        int n = -1, accumulate = -1;
        int seen = 0;            // calls of this shape seen; the graph is built on the second
        int launches = 0;
        uint64_t used = 0;       // for the choice of the entry a new shape replaces
        const float* h = nullptr;
        float* out = nullptr;
        // the nodes that hold the caller's buffers, for calls that bring others
        struct Io { cudaGraphNode_t node; cudaKernelNodeParams params; std::vector<void*> args; std::vector<int> h_at, out_at; };
        std::vector<Io> io;
        cudaGraph_t graph = nullptr;   // owns what `io` points into
    } graphs[kForwardGraphs];
    uint64_t graph_clock = 0;
    // bivmoe_forward_host with page-locked buffers: both copies, the launches and the
    // status read are one graph, replayed while the call's arguments, and what the device's
    // page tables say of them, stay the same
    struct {
        cudaGraphExec_t exec = nullptr;
        HostBuffers buf;
        int seen = 0, launches = 0;
    } host_graph;
    // bivmoe_forward_stack, kept by the stack's first layer: the launches of all layers as
    // one graph, replayed while the same layers in the same state, rows and stream come back
    struct {
        cudaGraphExec_t exec = nullptr;
        std::vector<uint64_t> layers;   // their state_id: an address may come back with another layer
        float* x = nullptr;
        int n = -1, seen = 0, launches = 0;
        cudaStream_t stream = nullptr;
    } stack_graph;
    int32_t* status_host = nullptr;   // page-locked copy of the device status words
    void* status_view = nullptr;      // its address on the device
    int prefill_min = 0;   // set at create when the tcgen05 kernels support the layer's types
    BigGroups big;         // the rule for its groups
    BigGroups big_alone;   // and for the shared expert's where it runs by itself (expert parallelism)
    int prefill_tile = kPrefillTile;
    int tile_rows = kFloatTile;
    bool quant = false;        // every matrix is quantised
    int wide_min = 0;          // rows a group on average from which a pass goes to experts_tc.cu, on f16 records
    bool wide_tiles = false;   // every matrix has a kernel for 16-row tiles
    // expert parallelism (bivmoe_ep_create): this rank's experts are global ids
    // ep_rank * n_local .. +n_local; `ws` serves the rank's own tokens (routing over all
    // experts, the shared expert), `ws_owner` the rows received for the local experts
    int ep_rank = 0, ep_world = 1, n_local = 0, max_recv = 0, ep_n = 0;
    Workspace ws_owner{};
    int32_t* ep_slot = nullptr;       // [max_tokens][world] a token's slot among a rank's rows, or -1
    int32_t* ep_counts = nullptr;     // [world] rows for each rank
    int32_t* ep_rank_ids = nullptr;   // [max_tokens][world] the rank, or -1: the home combine's "ids"
    int32_t* ep_rank_pos = nullptr;   // [max_tokens][world] the row's index among the sent rows
    float* ep_ones = nullptr;         // [max_tokens][world] the home combine's weights
    // the peer-store exchange (bivmoe_ep_peer_*): this rank's block, the ranks' blocks as
    // mapped into this process
    uint8_t* peer_block = nullptr;
    PeerLayout peer_lay{};
    PeerTable peers{};
    bool peers_attached = false;
    unsigned long long barrier_limit_ns = 2000000000ull;   // how long bivmoe_ep_peer_wait waits
    std::vector<void*> ipc_opened;
    bool use_graph = true;
    std::string error, device_name;
    std::vector<void*> allocs;
};

// A number no layer of this process has had: a layer gets one when it is made and another one
// whenever something changes that a captured launch holds by value (the norm's eps).
static uint64_t new_state_id() {
    static std::atomic<uint64_t> last{0};
    return last.fetch_add(1, std::memory_order_relaxed) + 1;
}

// whether the kernels take a product in parts: all but the float kernel
static bool in_parts(const bivmoe_layer* L) {
    return L->all_bf16 || (!type_uses_f32_act(L->gate_up.ty) && !type_uses_f32_act(L->down.ty));
}
// In how many parts a dense layer's product runs along K.  `items`: its tiles times its
// chunks.  The warp-MMA kernel has up to four groups per SM and each works on an item of its
// own: one token of 4096 / 12288 gives gate+up 192 items and down 32, 16 and 48 K-slices
// long (20 and 40 us; in 3 and 16 parts 9 and 8).  The tensor-core kernel has one item per SM at a time.
// Parts of at least two (four) K-slices, so that the copies of a part overlap its products.
static int quant_parts(const bivmoe_layer* L, int items, int nslices) {
    return std::max(1, std::min({4 * L->sm_count / std::max(items, 1), nslices / 2, 16}));
}
// (A BF16 item is two chunks, a slice of it a quarter as long.)
static int prefill_parts(const bivmoe_layer* L, int tiles) {
    const int items = tiles * (L->all_bf16 ? (L->down.chunks + 1) / 2 : L->down.chunks);
    return std::max(1, std::min({2 * L->sm_count / std::max(items, 1), L->down.nslices / (L->all_bf16 ? 8 : 4), 16}));
}
// room for what these rules allow: a part of an item is 128 rows x a tile's tokens, and there
// are at most 16 parts of the rows there may be
static size_t dense_parts_floats(const bivmoe_layer* L) {
    if (!in_parts(L)) return 0;
    const size_t rows = (size_t)16 * L->max_tokens * std::max(2 * L->ff, L->e);
    const size_t quant = (size_t)4 * L->sm_count * kChunkRows * kQuantTile;
    const size_t prefill = (size_t)2 * L->sm_count * kChunkRows * kPrefillTile * (L->all_bf16 ? 2 : 1);
    return std::min(rows, L->prefill_min > 0 || L->wide_min > 0 ? std::max(quant, prefill) : quant);
}

// Whether a pass of n rows goes to experts_tc.cu: from 36 rows a group on (a pass of 2048 / 512, Q4_K / Q6_K,
// us, by the small groups' kernels / by that one: 256 experts, 16 rows a group 271 / 329, 20 rows 335 / 350,
// 32 rows 450 / 397; 64 experts, 19 rows 112 / 113, 28 rows unevenly 129 / 128, 47 rows 190 / 142; 128
// experts, 37 rows unevenly 274 / 253), the one group of a dense layer, whose products have few work items,
// from 128 on (Q4_K, 64 rows of 4096 / 12288 109 / 98, 100 rows of 2048 / 6144 60 / 62, 150 rows of 1024 /
// 3072 35 / 33).  Both lines lie on the safe side of where the two meet, about 24 rows and 64 to 100.
// BIVMOE_WIDE_MIN, as it is when the layer is made, overrides both.
static bool wide_pass(const bivmoe_layer* L, int n) {
    return L->wide_min > 0 && n > 8 && (size_t)n * L->k >= (size_t)L->wide_min * L->n_expert;
}

// One workspace: `N` rows of `k` pairs over `ne` experts.  `routed_rows` false: only
// the shared group's positions get activation buffers (the home side of expert
// parallelism, whose routed rows are computed elsewhere).
static void layout_one(bivmoe_layer* L, Arena& a, Workspace& w, size_t N, size_t k, size_t ne,
                       bool routed_rows) {
    const size_t P = N * k, e = L->e;
    const size_t mid = std::max(L->ff, L->ff_sh);
    w.logits = a.take<float>(N * (ne + 1));
    w.ids = a.take<int32_t>(P);
    w.weights = a.take<float>(P);
    w.counts = a.take<int32_t>(ne);
    w.offsets = a.take<int32_t>(ne + 1);
    w.order = a.take<int32_t>(((N + 7) / 8) * 8 + P + 8 * ne + 8 + kPrefillPad);
    w.pos_of = a.take<int32_t>(P);
    w.blk_counts = a.take<int32_t>(((N + 255) / 256) * ne);
    w.grp_expert = a.take<int32_t>(ne + 1);
    w.grp_start = a.take<int32_t>(ne + 1);
    w.grp_count = a.take<int32_t>(ne + 1);
    w.n_groups = a.take<int32_t>(1);
    const size_t tiles = P / 8 + N / 8 + ne + 2;
    w.tile_desc = a.take<int4>(tiles);
    w.n_tiles = a.take<int32_t>(2);
    const size_t ptiles = (P + N) / kPrefillTile + ne + 2;
    w.ptile_group = a.take<int32_t>(ptiles);
    w.ptile_t0 = a.take<int32_t>(ptiles);
    w.big_min = a.take<int32_t>(1);
    w.n_ptiles = a.take<int32_t>(2);
    w.status = a.take<int32_t>(4);
    // positions: the tokens (shared group), then the routed groups, each padded to 8
    // (+kPrefillPad: a tile of the tcgen05 kernels copies up to that many positions from its first one)
    const size_t R = ((N + 7) / 8) * 8 + (routed_rows ? P + 8 * ne : 0) + 8 + kPrefillPad;
    w.act_rows = (int)R;
    const bool qact = !type_uses_f32_act(L->gate_up.ty) || (L->has_shared && !type_uses_f32_act(L->sh_gate_up.ty));
    const bool fact = type_uses_f32_act(L->gate_up.ty) || (L->has_shared && type_uses_f32_act(L->sh_gate_up.ty));
    const bool qmid = !type_uses_f32_act(L->down.ty) || (L->has_shared && !type_uses_f32_act(L->sh_down.ty));
    const size_t rec = L->wide_min > 0 ? kHalfRec : kActTileBytes;   // room for either form
    w.act_t = a.take<uint8_t>(qact ? (e / 256) * (R / 8) * rec : 0);
    const bool qrows = qact && N >= 256;   // the by-token rows of passes of many tokens
    w.tok_q = a.take<int8_t>(qrows ? N * e : 0);
    w.tok_s = a.take<float2>(qrows ? N * (e / 32) : 0);
    w.act_f = a.take<float>(fact && !L->all_bf16 ? R * e : 0);
    const bool brec = L->prefill_min > 0 && L->gate_up.ty == BIVMOE_BF16;   // bf16 hi/lo records
    w.tok_b = a.take<uint8_t>(brec ? N * (e / 64) * kTokBRec : 0);
    w.mid = a.take<float>(R * mid);
    w.mid_t = a.take<uint8_t>(qmid ? (mid / 256) * (R / 8) * rec : 0);
    if (L->all_bf16) {
        // One place each for what is not alive at the same time: the three-term rows are last
        // read by the small groups' gate+up, before any product's rows are written to pair_out;
        // the three-term SwiGLU rows by their down product, before the tcgen05 kernels begin.
        // (Small workspaces keep two places for the first: 33 tokens 199.0 us a pass so, 200.6 in one.)
        const size_t rows_3 = (e / 64) * (R / 8) * kAct3Rec, rows_out = R * e * 4;
        const bool one_place = rows_out > kShareBytes;
        w.act_3 = a.take<uint8_t>(one_place ? std::max(rows_3, rows_out) : rows_3);
        w.pair_out = one_place ? (float*)w.act_3 : a.take<float>(R * e);
        w.mid_3 = a.take<uint8_t>((mid / 64) * (R / 8) * kAct3Rec);
        w.mid_b = brec ? w.mid_3 : nullptr;
        static_assert(kActBRec <= kAct3Rec, "the two-term records fit where the three-term ones lie");
    } else {
        w.act_3 = w.mid_3 = nullptr;
        w.mid_b = a.take<uint8_t>(brec ? (mid / 64) * (R / 8) * kActBRec : 0);
        w.pair_out = a.take<float>(R * e);
    }
    w.h_norm = a.take<float>(N * e);
    w.row_scale = a.take<float>(N);
    w.parts = a.take<float>(L->dense ? dense_parts_floats(L) : 0);
}

static void layout_workspace(bivmoe_layer* L, Arena& a) {
    if (L->ep_world <= 1) {
        layout_one(L, a, L->ws, (size_t)L->max_tokens, (size_t)L->k, (size_t)L->n_expert, true);
        return;
    }
    layout_one(L, a, L->ws, (size_t)L->max_tokens, (size_t)L->k, (size_t)L->n_expert, false);
    layout_one(L, a, L->ws_owner, (size_t)L->max_recv, (size_t)L->k, (size_t)L->n_local, true);
    const size_t nw = (size_t)L->max_tokens * L->ep_world;
    L->ep_slot = a.take<int32_t>(nw);
    L->ep_counts = a.take<int32_t>((size_t)L->ep_world);
    L->ep_rank_ids = a.take<int32_t>(nw);
    L->ep_rank_pos = a.take<int32_t>(nw);
    L->ep_ones = a.take<float>(nw);
}

#define CU(call)                                                                          \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess) {                                                          \
            cudaGetLastError();   /* reported here: a later call must not find it */       \
            return set_err(errp, e_ == cudaErrorMemoryAllocation ? BIVMOE_ERR_OOM         \
                                                                 : BIVMOE_ERR_CUDA,       \
                           "%s: %s", #call, cudaGetErrorString(e_));                      \
        }                                                                                 \
    } while (0)

static int check_stack(std::string* errp, const char* name, const bivmoe_experts& s, int64_t cols,
                       int64_t rows, int64_t n, bool is_down) {
    if (!s.data) return set_err(errp, BIVMOE_ERR_ARGUMENT, "%s: null data", name);
    if (s.cols != cols || s.rows != rows || s.n != n)
        return set_err(errp, BIVMOE_ERR_ARGUMENT,
                       "%s: shape [%lld x %lld] x %lld, expected [%lld x %lld] x %lld", name,
                       (long long)s.rows, (long long)s.cols, (long long)s.n, (long long)rows,
                       (long long)cols, (long long)n);
    if (!experts_supported(s.ggml_type, (int)cols, (int)rows, is_down))
        return set_err(errp, BIVMOE_ERR_UNSUPPORTED,
                       "%s: no kernel for ggml type %d with %lld columns, %lld rows", name,
                       s.ggml_type, (long long)cols, (long long)rows);
    return BIVMOE_OK;
}

// Copies one product's stacks (gate and up, or down alone) to the device and
// repacks them into the tiled layout.
static int upload_tiles(bivmoe_layer* L, std::string* errp, const bivmoe_experts* a,
                        const bivmoe_experts* b, int chunk_rows, DevTiles* out) {
    const SliceGeom g = slice_geom(a->ggml_type);
    out->ty = a->ggml_type;
    out->cols = (int)a->cols; out->rows = (int)a->rows; out->n = (int)a->n;
    out->chunk_rows = chunk_rows;
    out->chunks = (int)(a->rows / chunk_rows);
    out->slice_bytes = g.sl;
    out->nslices = (int)(a->cols / g.elems);
    out->stage_bytes = slice_stage_bytes(a->ggml_type);
    out->expert_bytes = (int64_t)out->chunks * out->nslices * out->stage_bytes;
    const size_t dev_bytes = (size_t)(a->n * out->expert_bytes);
    void* p = nullptr;
    CU(dev_alloc(&p, dev_bytes));
    L->allocs.push_back(p);
    L->weight_bytes += dev_bytes;
    out->data = (uint8_t*)p;
    const bivmoe_experts* srcs[2] = {a, b};
    for (int i = 0; i < 2; i++) {
        const bivmoe_experts* s = srcs[i];
        if (!s) continue;
        const int64_t mat = s->rows * gguf_row_bytes(s->ggml_type, s->cols);
        const int64_t stride = s->stride_bytes ? s->stride_bytes : mat;
        void* staging = nullptr;
        CU(dev_alloc(&staging, (size_t)(s->n * mat)));
        cudaError_t e1 = cudaMemcpy2D(staging, (size_t)mat, (const uint8_t*)s->data + s->offset_bytes,
                                      (size_t)stride, (size_t)mat, (size_t)s->n, cudaMemcpyHostToDevice);
        if (e1 == cudaSuccess) e1 = launch_repack(*out, (const uint8_t*)staging, 2 * i, 0);
        if (e1 == cudaSuccess) e1 = cudaDeviceSynchronize();
        cudaFree(staging);
        CU(e1);
    }
    return BIVMOE_OK;
}

namespace bivmoe {
// A read-only view of the routing tensors for entry points kept in other files;
// with `error_or_null` it instead records that text as the layer's last error.
int layer_route_view(bivmoe_layer* L, RouteView* out, const char* error_or_null) {
    if (!L) return BIVMOE_ERR_ARGUMENT;
    if (error_or_null) {
        L->error = error_or_null;
        return BIVMOE_OK;
    }
    *out = RouteView{L->device, L->sm_count, L->e, L->n_expert, L->k, L->has_shared ? 1 : 0,
                     L->router, L->ws.status};
    return BIVMOE_OK;
}
}  // namespace bivmoe

extern "C" {

const char* bivmoe_global_error(void) { return g_error.c_str(); }
const char* bivmoe_last_error(const bivmoe_layer* layer) {
    return layer ? layer->error.c_str() : g_error.c_str();
}
uint64_t bivmoe_launch_count(void) { return g_launches.load(); }
uint64_t bivmoe_last_oom_bytes(void) { return g_oom_bytes; }

void bivmoe_destroy(bivmoe_layer* L) {
    if (!L) return;
    DeviceScope on_device(L->device);
    for (auto& g : L->graphs) {
        if (g.exec) cudaGraphExecDestroy(g.exec);
        if (g.graph) cudaGraphDestroy(g.graph);
    }
    if (L->host_graph.exec) cudaGraphExecDestroy(L->host_graph.exec);
    if (L->stack_graph.exec) cudaGraphExecDestroy(L->stack_graph.exec);
    if (L->status_host) cudaFreeHost(L->status_host);
    for (void* p : L->ipc_opened) cudaIpcCloseMemHandle(p);
    for (void* p : L->allocs) cudaFree(p);
    if (L->own_stream) cudaStreamDestroy(L->own_stream);
    if (L->in_stream) cudaStreamDestroy(L->in_stream);
    if (L->out_stream) cudaStreamDestroy(L->out_stream);
    for (cudaEvent_t ev : L->host_ev)
        if (ev) cudaEventDestroy(ev);
    delete L;
}

static int create_impl(const bivmoe_desc* d, int ep_rank, int ep_world, int max_recv,
                       bivmoe_layer** out, bool dense = false) {
    std::string* errp = nullptr;
    if (out) *out = nullptr;
    if (!d || !out) return set_err(errp, BIVMOE_ERR_ARGUMENT, "null descriptor or output");
    if (ep_world < 1 || ep_rank < 0 || ep_rank >= ep_world)
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "rank %d outside 0..%d", ep_rank, ep_world);
    if (ep_world > 1 && (d->n_expert % ep_world || max_recv <= 0 || ep_world > 32))
        return set_err(errp, BIVMOE_ERR_ARGUMENT,
                       "%d experts do not split over %d ranks (at most 32), or max_recv_rows %d is not positive",
                       d->n_expert, ep_world, max_recv);
    const int n_local = d->n_expert / ep_world;
    if (d->n_embd <= 0 || d->n_expert <= 0 || d->n_ff_exp <= 0 || d->max_tokens <= 0 || !d->router)
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "non-positive dimension or null router");
    // model.rs:108-112: 1 <= n_expert_used <= n_expert
    if (d->n_expert_used < 1 || d->n_expert_used > d->n_expert || d->n_expert_used > 32)
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "n_expert_used %d outside 1..min(%d, 32)",
                       d->n_expert_used, d->n_expert);
    if (d->n_expert > 1024)
        return set_err(errp, BIVMOE_ERR_UNSUPPORTED, "more than 1024 experts");
    if (d->n_embd % 256)
        return set_err(errp, BIVMOE_ERR_UNSUPPORTED, "n_embd %d is not a multiple of 256", d->n_embd);
    int rc;
    if ((rc = check_stack(errp, "ffn_gate_exps", d->gate, d->n_embd, d->n_ff_exp, n_local, false)) ||
        (rc = check_stack(errp, "ffn_up_exps", d->up, d->n_embd, d->n_ff_exp, n_local, false)) ||
        (rc = check_stack(errp, "ffn_down_exps", d->down, d->n_ff_exp, d->n_embd, n_local, true)))
        return rc;
    if (d->gate.ggml_type != d->up.ggml_type)
        return set_err(errp, BIVMOE_ERR_UNSUPPORTED, "gate and up of different types");
    const bool shared = d->n_ff_shexp > 0;
    if (shared) {
        if (!d->sh_gate_inp) return set_err(errp, BIVMOE_ERR_ARGUMENT, "null ffn_gate_inp_shexp");
        if ((rc = check_stack(errp, "ffn_gate_shexp", d->sh_gate, d->n_embd, d->n_ff_shexp, 1, false)) ||
            (rc = check_stack(errp, "ffn_up_shexp", d->sh_up, d->n_embd, d->n_ff_shexp, 1, false)) ||
            (rc = check_stack(errp, "ffn_down_shexp", d->sh_down, d->n_ff_shexp, d->n_embd, 1, true)))
            return rc;
        if (d->sh_gate.ggml_type != d->sh_up.ggml_type)
            return set_err(errp, BIVMOE_ERR_UNSUPPORTED, "shared gate and up of different types");
    }
    DeviceScope on_device(d->device);   // the caller's device is current again on return
    {
        int cur = -1;
        CU(cudaGetDevice(&cur));
        if (cur != d->device) CU(cudaSetDevice(d->device));   // reports an invalid ordinal
    }
    cudaDeviceProp prop;
    CU(cudaGetDeviceProperties(&prop, d->device));
    if (prop.major != 10)
        return set_err(errp, BIVMOE_ERR_UNSUPPORTED,
                       "device %d is sm_%d%d; this library is built for sm_100a only", d->device,
                       prop.major, prop.minor);
    bivmoe_layer* L = new (std::nothrow) bivmoe_layer();
    if (!L) return set_err(errp, BIVMOE_ERR_OOM, "host allocation failed");
    L->device = d->device;
    L->state_id = new_state_id();
    if (const char* v = getenv("BIVMOE_HOST_SECTIONS")) L->host_sections_forced = atoi(v);
    L->dense = dense;
    L->sm_count = prop.multiProcessorCount;
    L->device_name = prop.name;
    L->e = d->n_embd; L->n_expert = d->n_expert; L->k = d->n_expert_used;
    L->ff = d->n_ff_exp; L->ff_sh = d->n_ff_shexp; L->max_tokens = d->max_tokens;
    L->has_shared = shared;
    L->ep_rank = ep_rank; L->ep_world = ep_world; L->n_local = n_local; L->max_recv = max_recv;
    auto fail = [&](int code) { g_error = g_error.empty() ? L->error : g_error; bivmoe_destroy(L); return code; };
    if ((rc = upload_tiles(L, errp, &d->gate, &d->up, 64, &L->gate_up)) ||
        (rc = upload_tiles(L, errp, &d->down, nullptr, 128, &L->down)))
        return fail(rc);
    if (shared && ((rc = upload_tiles(L, errp, &d->sh_gate, &d->sh_up, 64, &L->sh_gate_up)) ||
                   (rc = upload_tiles(L, errp, &d->sh_down, nullptr, 128, &L->sh_down))))
        return fail(rc);
    auto cu_fail = [&](cudaError_t e, const char* what) {
        set_err(errp, e == cudaErrorMemoryAllocation ? BIVMOE_ERR_OOM : BIVMOE_ERR_CUDA, "%s: %s",
                what, cudaGetErrorString(e));
        return fail(e == cudaErrorMemoryAllocation ? BIVMOE_ERR_OOM : BIVMOE_ERR_CUDA);
    };
    cudaError_t ce;
    const size_t rbytes = (size_t)(L->n_expert + 1) * L->e * sizeof(float);
    if ((ce = dev_alloc((void**)&L->router, rbytes)) != cudaSuccess) return cu_fail(ce, "router");
    L->allocs.push_back(L->router);
    L->weight_bytes += rbytes;
    if ((ce = cudaMemset(L->router, 0, rbytes)) != cudaSuccess) return cu_fail(ce, "router");
    if ((ce = cudaMemcpy(L->router, d->router, (size_t)L->n_expert * L->e * 4,
                         cudaMemcpyHostToDevice)) != cudaSuccess)
        return cu_fail(ce, "router upload");
    if (shared && (ce = cudaMemcpy(L->router + (size_t)L->n_expert * L->e, d->sh_gate_inp,
                                   (size_t)L->e * 4, cudaMemcpyHostToDevice)) != cudaSuccess)
        return cu_fail(ce, "shared gate upload");
    // groups of at least this many tokens run on the tcgen05 kernels, where they exist
    // for the layer's types (shared expert of the same types, or none).  Q8_0: a group of
    // more than two 8-row tiles.  With groups of 32 rows on average (256 experts, 2048 / 512)
    // a pass takes 0.64 ms from 96 rows on, 0.55 from 33, 0.46 from 17 or 9; with 16 on
    // average 0.40, 0.39, 0.36 and 0.37: two tiles of the warp-MMA kernel cost what one
    // tensor-core tile costs.  BF16: the tcgen05 kernel sizes its MMA to the tile's rows and
    // reads the weights once per group, the warp-MMA kernel once per 8 rows: a group that needs
    // more than one 8-row tile is read again there (balanced groups of 12 rows, 384 tokens: 371
    // us a pass by the tcgen05 kernels, 422 without).
    L->all_bf16 = L->gate_up.ty == BIVMOE_BF16 && L->down.ty == BIVMOE_BF16 &&
                  (!shared || (L->sh_gate_up.ty == BIVMOE_BF16 && L->sh_down.ty == BIVMOE_BF16));
    if (prefill_supported(L->gate_up.ty, L->down.ty) &&
        (!shared || (L->sh_gate_up.ty == L->gate_up.ty && L->sh_down.ty == L->down.ty))) {
        const char* env = getenv("BIVMOE_PREFILL_MIN");
        L->prefill_min = env ? atoi(env) : L->gate_up.ty == BIVMOE_BF16 ? 9 : 17;
        L->prefill_tile = L->gate_up.ty == BIVMOE_BF16 ? kPrefillTileBf16 : kPrefillTile;
        // a pass whose large groups are few or small leaves them to the small groups' kernels
        // (big_groups.h); with a threshold from the environment every group of that size counts
        L->big.min = L->prefill_min;
        L->big.tile_bytes = L->gate_up.expert_bytes + L->down.expert_bytes;
        L->big.worth = env ? 0 : big_worth(L->all_bf16, L->e, L->ff, L->big.tile_bytes);
        L->big.sh_tile_bytes = L->sh_gate_up.expert_bytes + L->sh_down.expert_bytes;
        L->big_alone = BigGroups{L->prefill_min, env ? 0 : big_worth_alone(L->e, L->ff_sh), 0, L->big.sh_tile_bytes};
    }
    // the tile list serves both products of the routed and of the shared experts
    if (!type_uses_f32_act(L->gate_up.ty) && !type_uses_f32_act(L->down.ty) &&
        (!shared || (!type_uses_f32_act(L->sh_gate_up.ty) && !type_uses_f32_act(L->sh_down.ty))))
        L->tile_rows = kQuantTile, L->quant = true;
    auto k_quant = [](int ty) { return ty == BIVMOE_Q4_K || ty == BIVMOE_Q5_K || ty == BIVMOE_Q6_K; };
    L->wide_tiles = k_quant(L->gate_up.ty) && k_quant(L->down.ty) &&
                    (!shared || (k_quant(L->sh_gate_up.ty) && k_quant(L->sh_down.ty)));
    if (L->wide_tiles && ep_world == 1) {
        const char* env = getenv("BIVMOE_WIDE_MIN");
        L->wide_min = env ? atoi(env) : dense ? 128 : 36;
        if (!wide_pass(L, L->max_tokens)) L->wide_min = 0;   // no pass of this layer: no room for it
    }
    Arena probe;
    layout_workspace(L, probe);
    L->ws_bytes = probe.off;
    if ((ce = dev_alloc((void**)&L->ws_mem, L->ws_bytes)) != cudaSuccess) {
        set_err(errp, BIVMOE_ERR_OOM, "workspace of %zu bytes: %s", L->ws_bytes, cudaGetErrorString(ce));
        return fail(BIVMOE_ERR_OOM);
    }
    L->allocs.push_back(L->ws_mem);
    Arena real;
    real.base = L->ws_mem;
    layout_workspace(L, real);
    if ((ce = cudaMemset(L->ws.status, 0, 16)) != cudaSuccess) return cu_fail(ce, "status");
    if (ep_world > 1) {
        if ((ce = cudaMemset(L->ws_owner.status, 0, 16)) != cudaSuccess) return cu_fail(ce, "status");
        std::vector<float> ones((size_t)L->max_tokens * ep_world, 1.0f);
        if ((ce = cudaMemcpy(L->ep_ones, ones.data(), ones.size() * 4, cudaMemcpyHostToDevice)) != cudaSuccess)
            return cu_fail(ce, "weights of one");
    }
    if ((ce = cudaStreamCreateWithFlags(&L->own_stream, cudaStreamNonBlocking)) != cudaSuccess)
        return cu_fail(ce, "stream");
    if ((ce = cudaDeviceSynchronize()) != cudaSuccess) return cu_fail(ce, "upload");
    *out = L;
    return BIVMOE_OK;
}

int bivmoe_create(const bivmoe_desc* d, bivmoe_layer** out) { return create_impl(d, 0, 1, 0, out); }

int bivmoe_dense_create(int32_t device, int32_t n_embd, int32_t n_ff, int32_t max_tokens,
                        const bivmoe_experts* gate, const bivmoe_experts* up,
                        const bivmoe_experts* down, bivmoe_layer** out) {
    if (out) *out = nullptr;
    if (!gate || !up || !down || !out || n_embd <= 0)
        return set_err(nullptr, BIVMOE_ERR_ARGUMENT, "null pointer or non-positive n_embd");
    // one expert behind a router of zeros: softmax of one logit is 1, so is the
    // renormalised weight, and the combine's w * y is y
    std::vector<float> router((size_t)n_embd, 0.0f);
    bivmoe_desc d{};
    d.n_embd = n_embd; d.n_expert = 1; d.n_expert_used = 1;
    d.n_ff_exp = n_ff; d.n_ff_shexp = 0;
    d.max_tokens = max_tokens; d.device = device;
    d.router = router.data();
    d.gate = *gate; d.up = *up; d.down = *down;
    return create_impl(&d, 0, 1, 0, out, true);
}

int bivmoe_ep_create(const bivmoe_desc* d, int32_t ep_rank, int32_t ep_world, int32_t max_recv_rows,
                     bivmoe_layer** out) {
    if (ep_world == 1) return create_impl(d, 0, 1, 0, out);
    return create_impl(d, ep_rank, ep_world, max_recv_rows, out);
}

int bivmoe_set_post_norm(bivmoe_layer* L, const float* w, float eps) {
    if (!L || !w) return set_err(nullptr, BIVMOE_ERR_ARGUMENT, "null layer or weights");
    std::string* errp = &L->error;
    DeviceScope on_device(L->device);
    if (!L->post_norm) {
        CU(dev_alloc((void**)&L->post_norm, (size_t)L->e * 4));
        L->allocs.push_back(L->post_norm);
        L->weight_bytes += (size_t)L->e * 4;
    }
    CU(cudaMemcpy(L->post_norm, w, (size_t)L->e * 4, cudaMemcpyHostToDevice));
    L->norm_eps = eps;
    L->state_id = new_state_id();
    return BIVMOE_OK;
}

// Whether a pass of n rows takes the kernel that routes a few tokens by itself: quantised types, gate
// and up of one with the shared expert's, no group for the tcgen05 kernels, and not a dense layer by
// itself (which has no routing; in a stack, where the norm is fused, it is a layer like any other).
static bool few_pass(const bivmoe_layer* L, int n, bool norm) {
    return L->quant && (!L->dense || norm) && (L->big.min == 0 || n < L->big.min) && L->ep_world == 1 &&
           few_supported(n, L->k, L->e, L->n_expert, L->gate_up.ty) && (!L->has_shared || L->sh_gate_up.ty == L->gate_up.ty);
}

// What the taps have to know about the last pass: `n` rows, a section of a call of `call` rows or all of
// them.  Decided here alone, for the call that enqueues the launches, which goes by it, as for those
// that replay them.
static void note_pass(bivmoe_layer* L, int n, int call, bool norm) {
    L->last_n = n;
    L->in_sections = false;
    L->last_wide = wide_pass(L, call);
    L->last_few = !L->last_wide && few_pass(L, n, norm);
}

// `norm`: `h` holds the residual rows and the router and dispatch kernels apply the
// layer's rms_norm themselves (bivmoe_forward_stack).  `of`: the rows are a section of a call of that
// many.  The choice of the k-quants' kernels, and all of a dense layer's (the kernels, and into how
// many parts K is cut), go by the call's rows, so that a section rounds as the call in one piece
// would.  The groups of a BF16 mixture go by the section's: those that are large ones only in the
// whole call round as small ones do.  `next`: the pass may leave the rows normed for the layer after
// this one in a stack, and says whether it did.
struct NextLayer {
    bivmoe_layer* layer;   // none: the last of the stack
    bool normed = false;   // its ws.h_norm holds this pass's rows
};
static int forward_impl(bivmoe_layer* L, const float* h, float* out, int n, int accumulate,
                        cudaStream_t stream, cudaEvent_t* ev = nullptr, const RowNorm* norm = nullptr, int of = 0,
                        NextLayer* next = nullptr) {
    std::string* errp = &L->error;
    if (n < 0 || n > L->max_tokens)
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "n = %d outside 0..max_tokens = %d", n, L->max_tokens);
    if (n > 0 && (!h || !out)) return set_err(errp, BIVMOE_ERR_ARGUMENT, "null activation pointer");
    if (L->ep_world > 1)
        return set_err(errp, BIVMOE_ERR_ARGUMENT,
                       "the layer holds 1/%d of the experts: use the bivmoe_ep_* steps", L->ep_world);
    const int call = std::max(n, of);   // rows of the call
    note_pass(L, n, call, norm != nullptr);
    if (n == 0) return BIVMOE_OK;
    LaunchCfg c{stream, n, L->k, L->e, L->n_expert, L->ff, L->ff_sh, L->has_shared ? 1 : 0, L->sm_count};
    c.ev = ev;
    c.big = L->dense && !norm ? L->big : big_for(L->big, n, c.k, c.has_shared);
    c.prefill_tile = L->prefill_tile;
    c.tile_rows = L->tile_rows;
    mark(c, EV_START);
    // 16-row tiles from 8 rows a group on, where more than one tile in two has both its records
    // (256 experts, 8 a token: 200 tokens 154 -> 164 us, 300 tokens 200 -> 194, 1024 tokens 473 ->
    // 418; dense: 16 rows 62 -> 65, 40 rows 57 -> 53)
    if (L->wide_tiles && n * c.k >= 8 * c.n_expert && n >= 32) c.tile_rows = 2 * kQuantTile;
    if (L->dense && !norm && c.big.worth > 0) {
        // the same question for a dense layer's one group, whose products fill the chip either
        // way: the small groups' kernels read the weights again for every 8 rows, which costs as
        // much as the tensor-core kernels' longer start when they read some 200 MB more (BF16),
        // 85 MB (Q8_0, whose products also cost more).  1024 / 3072, 64 rows: 45 against 50 us and
        // 43 against 47; 4096 / 12288, 32 rows: 181 against 109 and 123 against 92
        const long long again = (call - 1) / kQuantTile * c.big.tile_bytes;
        if (again < (L->all_bf16 ? 200 : 85) * 1000000ll) c.big.min = 0;
        else if (call >= c.big.min) c.big.min = std::min(c.big.min, n);   // a section, however short, as its call
    }
    // of a mixture's pass, whichever kernels came before
    auto combine = [&]() -> cudaError_t {
        bivmoe_layer* after = next ? next->layer : nullptr;
        if (!after || after->device != L->device || after->e != L->e || !combine_norms(n, L->e))
            return launch_combine(c, combine_src(L->ws), out, accumulate);
        const RowNorm ahead{after->post_norm, after->norm_eps, nullptr};
        next->normed = true;
        return launch_combine(c, combine_src(L->ws), out, accumulate, &ahead, after->ws.h_norm);
    };
    const bool to_prefill = c.big.min > 0 && n >= c.big.min;   // a token selects an expert once: no group is larger than n
    c.wide = L->last_wide;
    if (c.wide) c.tile_rows = kWideTile;
    if (L->dense && !norm) {
        c.dense = 1;
        if (in_parts(L)) {
            const int tiles = (call + kQuantTile - 1) / kQuantTile, ptiles = (call + c.prefill_tile - 1) / c.prefill_tile;
            if (to_prefill) {
                c.down_parts = prefill_parts(L, ptiles);
            } else if (c.wide) {
                c.down_parts = prefill_parts(L, (call + c.tile_rows - 1) / c.tile_rows);
            } else {
                // (long rows only: a part's own rounding may move a re-quantised value of a
                // SwiGLU row by one step, which has to stay small against the whole row)
                if (L->ff >= 2048) c.gateup_parts = quant_parts(L, tiles * L->gate_up.chunks, L->gate_up.nslices);
                c.down_parts = quant_parts(L, tiles * L->down.chunks, L->down.nslices);
            }
        }
        CU(launch_route_dense(c, h, L->ws));   // lays the quantised rows out, too
        mark(c, EV_ROUTER);
        mark(c, EV_TOPK);
    } else {
        CU(launch_router(c, L->router, h, L->ws, norm));
        mark(c, EV_ROUTER);
        if (L->last_few) {   // the rest of the routing and the rows' quantiser are the gate+up kernel's
            mark(c, EV_TOPK);
            mark(c, EV_SORT);
            mark(c, EV_QUANT);
            CU(launch_experts_few(c, h, L->gate_up, L->sh_gate_up, L->ws, norm));
            CU(launch_experts(c, L->gate_up, L->down, L->sh_gate_up, L->sh_down, L->ws, true));
            mark(c, EV_DOWN);
            CU(combine());
            mark(c, EV_COMBINE);
            return BIVMOE_OK;
        }
        if (topk_and_sort_fuse(n, L->n_expert)) {
            mark(c, EV_TOPK);
            CU(launch_topk_sort(c, L->ws));
        } else {
            if (!norm) c.rows_ready = rows_with_topk(c, L->ws, L->ws.act_t != nullptr, L->ws.act_f || L->ws.act_3);
            CU(launch_route_topk(c, L->ws, h, c.rows_ready));
            mark(c, EV_TOPK);
            CU(launch_sort(c, L->ws));
        }
    }
    mark(c, EV_SORT);
    CU(launch_dispatch(c, h, L->ws, L->ws.act_t != nullptr && !c.dense, L->ws.act_f || L->ws.act_3, norm));
    mark(c, EV_QUANT);
    if (c.dense && to_prefill) mark(c, EV_GATEUP);   // the one group is the tensor-core kernels'
    else CU(launch_experts(c, L->gate_up, L->down, L->sh_gate_up, L->sh_down, L->ws));
    if (to_prefill) CU(launch_experts_prefill(c, L->gate_up, L->down, L->sh_gate_up, L->sh_down, L->ws));
    mark(c, EV_DOWN);
    if (c.dense) CU(launch_combine_dense(c, L->ws, out, accumulate));
    else CU(combine());
    mark(c, EV_COMBINE);
    return BIVMOE_OK;
}

// The nodes of a captured pass that hold the caller's rows or the caller's output, with their
// argument lists: one for every launch that was given one of them while it was captured.
static cudaError_t find_io_nodes(bivmoe_layer::ForwardGraph& G, const LaunchWatch& watch) {
    size_t count = 0;
    cudaError_t e = cudaGraphGetNodes(G.graph, nullptr, &count);
    if (e != cudaSuccess) return e;
    std::vector<cudaGraphNode_t> nodes(count);
    if ((e = cudaGraphGetNodes(G.graph, nodes.data(), &count)) != cudaSuccess) return e;
    std::vector<bool> found(watch.seen.size(), false);
    for (cudaGraphNode_t node : nodes) {
        cudaGraphNodeType type;
        if ((e = cudaGraphNodeGetType(node, &type)) != cudaSuccess) return e;
        if (type != cudaGraphNodeTypeKernel) continue;
        bivmoe_layer::ForwardGraph::Io io{};
        io.node = node;
        if ((e = cudaGraphKernelNodeGetParams(node, &io.params)) != cudaSuccess) return e;
        for (size_t i = 0; i < watch.seen.size(); i++) {
            const LaunchWatch::Seen& s = watch.seen[i];
            if (found[i] || !is_kernel(io.params.func, s.kernel)) continue;
            // the same kernel may be launched several times: this node's arguments decide
            const auto holds = [&](const std::vector<int>& at, const void* p) {
                return std::all_of(at.begin(), at.end(), [&](int k) { return *(const void**)io.params.kernelParams[k] == p; });
            };
            if (!holds(s.h_at, watch.h) || !holds(s.out_at, watch.out)) continue;
            found[i] = true;
            io.h_at = s.h_at;
            io.out_at = s.out_at;
            io.args.assign(io.params.kernelParams, io.params.kernelParams + s.args);
            G.io.push_back(std::move(io));
            break;
        }
    }
    for (auto& io : G.io) io.params.kernelParams = io.args.data();   // the vectors have their places now
    return std::all_of(found.begin(), found.end(), [](bool f) { return f; }) ? cudaSuccess : cudaErrorInvalidValue;
}

// forward_impl, replayed from a CUDA graph when a call of the same shape repeats: the
// launches then cost one graph launch and run back to back on the device (0.3 us apart
// instead of the 2.3 us of separate launches on the default stream).  The capture happens
// on the layer's own stream, so the graph serves every stream of the caller, the legacy
// default stream - which cannot be captured - included; a call that brings other buffers
// rewrites the pointers in the graph's nodes (at most four nodes hold them).
static int forward_graphed(bivmoe_layer* L, const float* h, float* out, int n, int accumulate,
                           cudaStream_t stream) {
    std::string* errp = &L->error;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (!L->use_graph || n <= 0 ||
        (stream != nullptr && stream != cudaStreamLegacy &&
         (cudaStreamIsCapturing(stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone)))
        return forward_impl(L, h, out, n, accumulate, stream);   // also when the caller captures us
    bivmoe_layer::ForwardGraph* G = nullptr;
    for (auto& g : L->graphs)
        if (g.n == n && g.accumulate == accumulate) { G = &g; break; }
    if (!G) {   // the shape that was used longest ago makes room
        G = &L->graphs[0];
        for (auto& g : L->graphs)
            if (g.used < G->used) G = &g;
        if (G->exec) cudaGraphExecDestroy(G->exec);
        if (G->graph) cudaGraphDestroy(G->graph);
        *G = bivmoe_layer::ForwardGraph{};
        G->n = n;
        G->accumulate = accumulate;
    }
    G->used = ++L->graph_clock;
    if (!G->exec) {
        if (++G->seen < 2)   // the first call runs plainly (it also sets the kernels' attributes)
            return forward_impl(L, h, out, n, accumulate, stream);
        const uint64_t before = bivmoe_launch_count();
        CU(cudaStreamBeginCapture(L->own_stream, cudaStreamCaptureModeThreadLocal));
        LaunchWatch watch;
        watch.h = h;
        watch.out = out;
        launch_watch() = &watch;
        const int rc = forward_impl(L, h, out, n, accumulate, L->own_stream);
        launch_watch() = nullptr;
        cudaError_t ce = cudaStreamEndCapture(L->own_stream, &G->graph);
        G->launches = (int)(bivmoe_launch_count() - before);
        count_launch(-G->launches);   // captured, not launched yet
        if (!rc && ce == cudaSuccess && G->graph) ce = find_io_nodes(*G, watch);
        if (!rc && ce == cudaSuccess && G->graph) ce = cudaGraphInstantiate(&G->exec, G->graph, 0);
        if (rc || ce != cudaSuccess || !G->exec) {
            G->exec = nullptr;
            L->use_graph = false;   // plain launches from here on
            cudaGetLastError();
            return rc ? rc : forward_impl(L, h, out, n, accumulate, stream);
        }
        G->h = h;
        G->out = out;
    }
    if (G->h != h || G->out != out) {
        for (auto& io : G->io) {
            for (int at : io.h_at) io.args[at] = &h;
            for (int at : io.out_at) io.args[at] = &out;
            if ((!io.h_at.empty() && G->h != h) || (!io.out_at.empty() && G->out != out))
                CU(cudaGraphExecKernelNodeSetParams(G->exec, io.node, &io.params));
        }
        G->h = h;
        G->out = out;
    }
    note_pass(L, n, n, false);
    CU(cudaGraphLaunch(G->exec, stream));
    count_launch(G->launches);
    return BIVMOE_OK;
}

int bivmoe_forward(bivmoe_layer* L, const float* h_dev, float* out_dev, int32_t n,
                   int32_t accumulate, void* stream) {
    if (!L) return set_err(nullptr, BIVMOE_ERR_ARGUMENT, "null layer");
    DeviceScope on_device(L->device);
    if (n < 0 || n > L->max_tokens)
        return set_err(&L->error, BIVMOE_ERR_ARGUMENT, "n = %d outside 0..max_tokens = %d", n,
                       L->max_tokens);
    if (n == 0) {   // no rows (their pointers may be null): nothing to do
        note_pass(L, 0, 0, false);
        return BIVMOE_OK;
    }
    if (!h_dev || !out_dev) return set_err(&L->error, BIVMOE_ERR_ARGUMENT, "null activation pointer");
    return forward_graphed(L, h_dev, out_dev, n, accumulate, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// expert parallelism: the device steps between the caller's two exchanges

static int ep_check(bivmoe_layer* L, const char* what) {
    if (!L) return set_err(nullptr, BIVMOE_ERR_ARGUMENT, "null layer");
    if (L->ep_world <= 1)
        return set_err(&L->error, BIVMOE_ERR_ARGUMENT, "%s: the layer was not made by bivmoe_ep_create "
                       "with more than one rank", what);
    return BIVMOE_OK;
}

int bivmoe_ep_route(bivmoe_layer* L, const float* h_dev, int32_t n, float* send_rows_dev,
                    int32_t* send_tags_dev, int32_t* send_counts_dev, void* stream) {
    if (int rc = ep_check(L, "bivmoe_ep_route")) return rc;
    DeviceScope on_device(L->device);
    std::string* errp = &L->error;
    if (!h_dev || !send_rows_dev || !send_tags_dev || !send_counts_dev)
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "null pointer");
    if (n < 0 || n > L->max_tokens)
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "n = %d outside 0..max_tokens = %d", n, L->max_tokens);
    cudaStream_t s = (cudaStream_t)stream;
    L->ep_n = n;
    L->last_n = n;
    if (n == 0) {
        CU(cudaMemsetAsync(send_counts_dev, 0, (size_t)L->ep_world * 4, s));
        return BIVMOE_OK;
    }
    LaunchCfg c{s, n, L->k, L->e, L->n_expert, L->ff, L->ff_sh, L->has_shared ? 1 : 0, L->sm_count};
    // the lists of the shared expert's group, which is computed here; its size decides
    // its kernel (the routed pairs are sorted by the ranks that own their experts)
    c.big = big_for(L->big_alone, n, 0, 1);
    c.prefill_tile = L->prefill_tile;
    c.tile_rows = L->tile_rows;
    CU(launch_router(c, L->router, h_dev, L->ws));
    CU(launch_route_topk(c, L->ws));
    if (L->has_shared) CU(launch_shared_lists(c, L->ws));
    CU(launch_ep_gather(c, h_dev, L->ws, L->ep_world, L->n_local, L->ep_slot, L->ep_counts,
                        L->ep_rank_ids, L->ep_rank_pos, send_rows_dev, send_tags_dev, send_counts_dev));
    return BIVMOE_OK;
}

int bivmoe_ep_shared(bivmoe_layer* L, const float* h_dev, void* stream) {
    if (int rc = ep_check(L, "bivmoe_ep_shared")) return rc;
    DeviceScope on_device(L->device);
    std::string* errp = &L->error;
    const int n = L->ep_n;
    if (!L->has_shared || n == 0) return BIVMOE_OK;
    if (!h_dev) return set_err(errp, BIVMOE_ERR_ARGUMENT, "null pointer");
    cudaStream_t s = (cudaStream_t)stream;
    LaunchCfg c{s, n, 0, L->e, L->n_expert, L->ff, L->ff_sh, 1, L->sm_count};   // k = 0: no pair rows
    c.big = big_for(L->big_alone, n, 0, 1);
    c.prefill_tile = L->prefill_tile;
    c.tile_rows = L->tile_rows;
    c.only_shared = 1;
    CU(launch_dispatch(c, h_dev, L->ws, L->ws.act_t != nullptr && !type_uses_f32_act(L->sh_gate_up.ty),
                       (L->ws.act_f || L->ws.act_3) && type_uses_f32_act(L->sh_gate_up.ty)));
    c.k = L->k;
    CU(launch_experts(c, L->gate_up, L->down, L->sh_gate_up, L->sh_down, L->ws));
    if (c.big.min > 0)
        CU(launch_experts_prefill(c, L->gate_up, L->down, L->sh_gate_up, L->sh_down, L->ws));
    return BIVMOE_OK;
}

int bivmoe_ep_experts(bivmoe_layer* L, const float* recv_rows_dev, const int32_t* recv_tags_dev,
                      int32_t m, float* out_rows_dev, void* stream) {
    if (int rc = ep_check(L, "bivmoe_ep_experts")) return rc;
    DeviceScope on_device(L->device);
    std::string* errp = &L->error;
    if (m < 0 || m > L->max_recv)
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "m = %d outside 0..max_recv_rows = %d", m, L->max_recv);
    if (m == 0) return BIVMOE_OK;
    if (!recv_rows_dev || !recv_tags_dev || !out_rows_dev)
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "null pointer");
    cudaStream_t s = (cudaStream_t)stream;
    // the received rows with their tags are a routing result over the local experts with
    // empty slots for the experts other ranks own; no shared expert here
    LaunchCfg c{s, m, L->k, L->e, L->n_local, L->ff, 0, 0, L->sm_count};
    c.big = big_for(L->big, m, L->k, 0);
    c.prefill_tile = L->prefill_tile;
    c.tile_rows = L->tile_rows;
    const Workspace& w = L->ws_owner;
    const DevTiles none{};
    CU(launch_ep_localize(c, recv_tags_dev, L->ep_rank * L->n_local, w));
    CU(launch_sort(c, w));
    CU(launch_dispatch(c, recv_rows_dev, w, w.act_t != nullptr && !type_uses_f32_act(L->gate_up.ty),
                       (w.act_f || w.act_3) && type_uses_f32_act(L->gate_up.ty)));
    CU(launch_experts(c, L->gate_up, L->down, none, none, w));
    if (c.big.min > 0) CU(launch_experts_prefill(c, L->gate_up, L->down, none, none, w));
    CU(launch_combine(c, combine_src(w), out_rows_dev, 0));   // the weighted sum over the local experts
    return BIVMOE_OK;
}

int bivmoe_ep_combine(bivmoe_layer* L, const float* returned_rows_dev, float* out_dev, int32_t n,
                      int32_t accumulate, void* stream) {
    if (int rc = ep_check(L, "bivmoe_ep_combine")) return rc;
    DeviceScope on_device(L->device);
    std::string* errp = &L->error;
    if (n != L->ep_n)
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "n = %d, but bivmoe_ep_route ran on %d rows", n, L->ep_n);
    if (n == 0) return BIVMOE_OK;
    if (!returned_rows_dev || !out_dev) return set_err(errp, BIVMOE_ERR_ARGUMENT, "null pointer");
    // the ranks take the experts' place: weight one, ascending rank = ascending expert id
    LaunchCfg c{(cudaStream_t)stream, n, L->ep_world, L->e, L->n_expert, L->ff, L->ff_sh,
                L->has_shared ? 1 : 0, L->sm_count};
    const CombineSrc src{L->ep_rank_ids, L->ep_ones, returned_rows_dev, L->ep_rank_pos, L->ws.pair_out,
                         L->ws.logits};
    CU(launch_combine(c, src, out_dev, accumulate));
    return BIVMOE_OK;
}

// ---- the peer-store exchange ------------------------------------------------------

static int peer_check(bivmoe_layer* L, const char* what, bool attached) {
    if (int rc = ep_check(L, what)) return rc;
    if (attached && !L->peers_attached)
        return set_err(&L->error, BIVMOE_ERR_ARGUMENT, "%s before bivmoe_ep_peer_attach", what);
    return BIVMOE_OK;
}

int bivmoe_ep_peer_info(bivmoe_layer* L, bivmoe_peer_info* info) {
    if (int rc = peer_check(L, "bivmoe_ep_peer_info", false)) return rc;
    std::string* errp = &L->error;
    if (!info) return set_err(errp, BIVMOE_ERR_ARGUMENT, "null pointer");
    DeviceScope on_device(L->device);
    if (!L->peer_block) {
        const size_t W = (size_t)L->ep_world, cap = (size_t)L->max_tokens, e = (size_t)L->e;
        if ((size_t)L->max_recv < W * cap)
            return set_err(errp, BIVMOE_ERR_ARGUMENT,
                           "max_recv_rows %d is below world * max_tokens = %zu, the rows of the regions",
                           L->max_recv, W * cap);
        PeerLayout lay{};
        lay.cap = (int)cap;
        lay.rows = 0;
        lay.returned = W * cap * e * 4;
        lay.tags = 2 * lay.returned;
        lay.counts = lay.tags + ((W * cap * 2 * (size_t)L->k * 4 + 255) & ~(size_t)255);
        lay.flags = lay.counts + 256;
        lay.bytes = lay.flags + 1024;
        void* p = nullptr;
        CU(dev_alloc(&p, lay.bytes));
        L->allocs.push_back(p);
        CU(cudaMemset(p, 0, lay.bytes));
        L->peer_block = (uint8_t*)p;
        L->peer_lay = lay;
        L->ws_bytes += lay.bytes;
    }
    memset(info, 0, sizeof(*info));
    cudaIpcMemHandle_t hnd;
    CU(cudaIpcGetMemHandle(&hnd, L->peer_block));
    static_assert(sizeof(hnd) == sizeof(info->ipc_handle), "cudaIpcMemHandle_t is 64 bytes");
    memcpy(info->ipc_handle, &hnd, sizeof(hnd));
    info->base = L->peer_block;
    info->pid = (int64_t)getpid();
    info->device = L->device;
    info->bytes = (int64_t)L->peer_lay.bytes;
    return BIVMOE_OK;
}

int bivmoe_ep_peer_attach(bivmoe_layer* L, const bivmoe_peer_info* all) {
    if (int rc = peer_check(L, "bivmoe_ep_peer_attach", false)) return rc;
    std::string* errp = &L->error;
    if (!all) return set_err(errp, BIVMOE_ERR_ARGUMENT, "null pointer");
    if (!L->peer_block) return set_err(errp, BIVMOE_ERR_ARGUMENT, "bivmoe_ep_peer_info comes first");
    if (L->peers_attached) return set_err(errp, BIVMOE_ERR_ARGUMENT, "already attached");
    DeviceScope on_device(L->device);
    for (int r = 0; r < L->ep_world; r++) {
        const bivmoe_peer_info& pi = all[r];
        if (pi.bytes != (int64_t)L->peer_lay.bytes)
            return set_err(errp, BIVMOE_ERR_ARGUMENT,
                           "rank %d's block has %lld bytes, this rank's %zu: the ranks' shapes differ", r,
                           (long long)pi.bytes, L->peer_lay.bytes);
        if (r == L->ep_rank) {
            L->peers.base[r] = L->peer_block;
        } else if (pi.pid == (int64_t)getpid()) {   // a rank of this process: its pointer as it is
            if (pi.device != L->device) {
                int can = 0;
                CU(cudaDeviceCanAccessPeer(&can, L->device, pi.device));
                if (!can)
                    return set_err(errp, BIVMOE_ERR_UNSUPPORTED, "device %d cannot map device %d's memory",
                                   L->device, pi.device);
                const cudaError_t pe = cudaDeviceEnablePeerAccess(pi.device, 0);
                if (pe != cudaSuccess && pe != cudaErrorPeerAccessAlreadyEnabled) CU(pe);
                cudaGetLastError();
            }
            L->peers.base[r] = (uint8_t*)pi.base;
        } else {
            cudaIpcMemHandle_t hnd;
            memcpy(&hnd, pi.ipc_handle, sizeof(hnd));
            void* p = nullptr;
            CU(cudaIpcOpenMemHandle(&p, hnd, cudaIpcMemLazyEnablePeerAccess));
            L->ipc_opened.push_back(p);
            L->peers.base[r] = (uint8_t*)p;
        }
    }
    L->peers_attached = true;
    return BIVMOE_OK;
}

int bivmoe_ep_peer_dispatch(bivmoe_layer* L, const float* h_dev, int32_t n, void* stream) {
    if (int rc = peer_check(L, "bivmoe_ep_peer_dispatch", true)) return rc;
    DeviceScope on_device(L->device);
    std::string* errp = &L->error;
    if (n < 0 || n > L->max_tokens)
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "n = %d outside 0..max_tokens = %d", n, L->max_tokens);
    if (n > 0 && !h_dev) return set_err(errp, BIVMOE_ERR_ARGUMENT, "null pointer");
    cudaStream_t s = (cudaStream_t)stream;
    L->ep_n = n;
    LaunchCfg c{s, n, L->k, L->e, L->n_expert, L->ff, L->ff_sh, L->has_shared ? 1 : 0, L->sm_count};
    c.big = big_for(L->big_alone, n, 0, 1);
    c.prefill_tile = L->prefill_tile;
    c.tile_rows = L->tile_rows;
    if (n > 0) {
        CU(launch_router(c, L->router, h_dev, L->ws));
        CU(launch_route_topk(c, L->ws));
        if (L->has_shared) CU(launch_shared_lists(c, L->ws));
    }
    CU(launch_ep_peer_scatter(c, h_dev, L->ws, L->ep_world, L->ep_rank, L->n_local, L->ep_slot, L->ep_counts,
                              L->ep_rank_ids, L->ep_rank_pos, L->peers, L->peer_lay));
    return BIVMOE_OK;
}

int bivmoe_ep_peer_experts(bivmoe_layer* L, void* stream) {
    if (int rc = peer_check(L, "bivmoe_ep_peer_experts", true)) return rc;
    DeviceScope on_device(L->device);
    std::string* errp = &L->error;
    cudaStream_t s = (cudaStream_t)stream;
    const int m = L->ep_world * L->peer_lay.cap;
    LaunchCfg c{s, m, L->k, L->e, L->n_local, L->ff, 0, 0, L->sm_count};
    c.big = big_for(L->big, m, L->k, 0);
    c.prefill_tile = L->prefill_tile;
    c.tile_rows = L->tile_rows;
    const Workspace& w = L->ws_owner;
    const DevTiles none{};
    const float* rows = (const float*)(L->peer_block + L->peer_lay.rows);
    CU(launch_ep_peer_localize(c, L->peer_block, L->peer_lay, L->ep_rank * L->n_local, w));
    CU(launch_sort(c, w));
    CU(launch_dispatch(c, rows, w, w.act_t != nullptr && !type_uses_f32_act(L->gate_up.ty),
                       (w.act_f || w.act_3) && type_uses_f32_act(L->gate_up.ty)));
    CU(launch_experts(c, L->gate_up, L->down, none, none, w));
    if (c.big.min > 0) CU(launch_experts_prefill(c, L->gate_up, L->down, none, none, w));
    // the weighted sum over the local experts, stored where its home rank reads it
    CU(launch_combine_to_peers(c, combine_src(w), L->peer_block, L->ep_rank, L->peers, L->peer_lay));
    return BIVMOE_OK;
}

int bivmoe_ep_peer_combine(bivmoe_layer* L, float* out_dev, int32_t n, int32_t accumulate, void* stream) {
    if (int rc = peer_check(L, "bivmoe_ep_peer_combine", true)) return rc;
    return bivmoe_ep_combine(L, (const float*)(L->peer_block + L->peer_lay.returned), out_dev, n, accumulate,
                             stream);
}

int bivmoe_ep_peer_signal(bivmoe_layer* L, void* stream) {
    if (int rc = peer_check(L, "bivmoe_ep_peer_signal", true)) return rc;
    DeviceScope on_device(L->device);
    std::string* errp = &L->error;
    CU(launch_ep_peer_signal((cudaStream_t)stream, L->peer_block, L->ep_rank, L->ep_world, L->peers,
                             L->peer_lay));
    return BIVMOE_OK;
}

int bivmoe_ep_peer_wait(bivmoe_layer* L, void* stream) {
    if (int rc = peer_check(L, "bivmoe_ep_peer_wait", true)) return rc;
    DeviceScope on_device(L->device);
    std::string* errp = &L->error;
    CU(launch_ep_peer_wait((cudaStream_t)stream, L->peer_block, L->ep_world, L->peer_lay,
                           L->barrier_limit_ns, L->ws.status));
    return BIVMOE_OK;
}

int bivmoe_ep_peer_barrier(bivmoe_layer* L, void* stream) {
    if (int rc = bivmoe_ep_peer_signal(L, stream)) return rc;
    return bivmoe_ep_peer_wait(L, stream);
}

int bivmoe_ep_peer_wait_limit(bivmoe_layer* L, uint64_t microseconds) {
    if (int rc = ep_check(L, "bivmoe_ep_peer_wait_limit")) return rc;
    if (microseconds == 0 || microseconds > 60000000ull)
        return set_err(&L->error, BIVMOE_ERR_ARGUMENT, "a wait limit of %llu us is outside 1 us .. 60 s",
                       (unsigned long long)microseconds);
    L->barrier_limit_ns = microseconds * 1000ull;
    return BIVMOE_OK;
}

int bivmoe_status(bivmoe_layer* L, void* stream) {
    if (!L) return set_err(nullptr, BIVMOE_ERR_ARGUMENT, "null layer");
    DeviceScope on_device(L->device);
    std::string* errp = &L->error;
    cudaStream_t s = (cudaStream_t)stream;
    const bool ep = L->ep_world > 1;
    int32_t st[2][4] = {};
    CU(cudaMemcpyAsync(st[0], L->ws.status, 16, cudaMemcpyDeviceToHost, s));
    if (ep) CU(cudaMemcpyAsync(st[1], L->ws_owner.status, 16, cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
    if (st[0][0] || st[1][0]) {
        cudaMemsetAsync(L->ws.status, 0, 16, s);
        if (ep) cudaMemsetAsync(L->ws_owner.status, 0, 16, s);
        const int which = st[0][0] ? 0 : 1;
        return set_err(errp, st[which][0], "a device-side bounded wait gave up (status %d, wait site %d)",
                       st[which][0], st[which][2]);
    }
    return BIVMOE_OK;
}

int bivmoe_ep_status(bivmoe_layer* L, void* stream) {
    if (int rc = ep_check(L, "bivmoe_ep_status")) return rc;
    return bivmoe_status(L, stream);
}

int bivmoe_forward_profile(bivmoe_layer* L, const float* h_dev, float* out_dev, int32_t n,
                           void* stream, float* ms) {
    if (!L || !ms) return set_err(nullptr, BIVMOE_ERR_ARGUMENT, "null layer or buffer");
    DeviceScope on_device(L->device);
    std::string* errp = &L->error;
    cudaEvent_t ev[EV_COUNT];
    for (int i = 0; i < EV_COUNT; i++) CU(cudaEventCreate(&ev[i]));
    int rc = forward_impl(L, h_dev, out_dev, n, 0, (cudaStream_t)stream, ev);
    cudaError_t ce = cudaEventSynchronize(ev[EV_COMBINE]);
    for (int i = 1; i < EV_COUNT && ce == cudaSuccess && !rc; i++)
        ce = cudaEventElapsedTime(&ms[i - 1], ev[i - 1], ev[i]);
    for (int i = 0; i < EV_COUNT; i++) cudaEventDestroy(ev[i]);
    if (rc) return rc;
    CU(ce);
    return BIVMOE_OK;
}

// The page-locked range that `p` lies in (0.1 us; from the driver, as the runtime tells only
// whether one address is page-locked).
static LockedRange look_up(const void* p) {
    using Get = CUresult (*)(unsigned, CUpointer_attribute*, void**, CUdeviceptr);
    static const Get get = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found;
        const cudaError_t e = cudaGetDriverEntryPoint("cuPointerGetAttributes", &f, cudaEnableDefault, &found);
        return e == cudaSuccess && found == cudaDriverEntryPointSuccess ? (Get)f : nullptr;
    }();
    unsigned type = 0, access = 0;
    CUdeviceptr dev = 0, start = 0;
    size_t bytes = 0;
    CUpointer_attribute what[5] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_DEVICE_POINTER,
                                   CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE,
                                   CU_POINTER_ATTRIBUTE_ACCESS_FLAGS};
    void* into[5] = {&type, &dev, &start, &bytes, &access};
    if (!get || get(5, what, into, (CUdeviceptr)p) != CUDA_SUCCESS || type != CU_MEMORYTYPE_HOST) return {};
    return {(uintptr_t)dev, (uintptr_t)start, bytes, (access & CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READWRITE) ==
                                                         CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READWRITE};
}

// How many sections a host-buffer call of n rows runs in.  The layer is row-wise, so a
// section's result does not depend on the rows of the others.  More sections hide more of the
// copies (54 GB/s each way: with one nothing, with two half of them, with three or more, whose
// first and last are half as long, all but 1 / S), and each costs another 60 us of launches and
// short kernels and one more reading of the weights, 0.19 us per MB with what that delays.
// Measured in 1 / 2 / 3 sections, ms: 3000 BF16 rows (1.6 GB of weights) 1.48 / 1.39 / 1.80, 6000
// rows 2.80 / 2.06 / 2.16, 8192 rows - / 2.78 / 2.47 (four: 2.73); 2048 rows Q8_0 (0.9 GB) 1.28 /
// 1.20 / 1.46; 3000 BF16 rows of 1024, 64 experts (0.2 GB) 0.69 / 0.55 / 0.56.  Long calls gain
// by more sections than that explains, one per 455 us of copy-in: 12000 BF16 rows in 3 / 4 / 5
// take 3.40 / 3.18 / 3.48, 16384 rows 4.60 / 4.24 / 3.94.
// BIVMOE_HOST_SECTIONS, as it is when the layer is made, overrides the rule (1 = no overlap).
static int host_sections(const bivmoe_layer* L, int n) {
    const int forced = L->host_sections_forced;
    int c = forced > 0 ? forced : 1;
    if (forced <= 0) {
        const double copy = (double)n * L->e * 4 / 54e3, section = 60.0 + 0.19e-6 * (double)L->weight_bytes;
        double best = 2.0 * copy;
        for (int k = 2; k <= kHostSectionsDefault; k++) {
            const double cost = k == 2 ? copy + section : copy / k + k * section;   // from 3 on there is one more
            if (cost < best) { best = cost; c = k; }
        }
        c = std::min(std::max(c, (int)(copy / 455.0 + 0.5)), kHostSectionsDefault);
    }
    c = std::min(c, kHostSectionsMax);
    c = std::min(c, n / 8);
    return std::max(c, 1);
}

// copy in, the layer, copy out, status out - enqueued on the layer's own stream; with
// more than one section the copies run on two more streams, forked from and joined to it
// by events (so that the whole can be captured from the layer's stream)
static int forward_host_enqueue(bivmoe_layer* L, const HostBuffers& buf) {
    std::string* errp = &L->error;
    const float* h_host = buf.h;
    float* out_host = buf.out;
    const int n = buf.n;
    const size_t bytes = (size_t)n * L->e * 4;
    cudaStream_t s = L->own_stream;
    const int sections = host_sections(L, n);
    if (sections > 1) {
        cudaStream_t si = L->in_stream, so = L->out_stream;
        cudaEvent_t* ev = L->host_ev;
        cudaEvent_t fork = ev[2 * (kHostSectionsMax + 1)], join = ev[2 * (kHostSectionsMax + 1) + 1];
        // Section boundaries.  With three sections or more the first and the last are half
        // as long as the others (one more section in all): what cannot overlap anything is
        // the first section's copy-in and the last one's copy-out.
        int bound[kHostSectionsMax + 2];
        int nsec = 0;
        {
            const int per = ((n + sections - 1) / sections + 7) / 8 * 8;
            const int edge = sections >= 3 ? (per / 2 + 7) / 8 * 8 : per;
            bound[0] = 0;
            for (int t0 = edge; t0 < n; t0 += (n - t0 > per + edge / 2 ? per : n - t0)) bound[++nsec] = t0;
            bound[++nsec] = n;
            if (sections >= 3 && nsec >= 3 && bound[nsec] - bound[nsec - 1] > edge) {
                // the tail came out long: cut it so that the last section is an edge
                const int cut = (bound[nsec] - edge) / 8 * 8;
                if (cut > bound[nsec - 1] && nsec < kHostSectionsMax + 1) {
                    bound[nsec + 1] = bound[nsec];
                    bound[nsec] = cut;
                    nsec++;
                }
            }
        }
        CU(cudaEventRecord(fork, s));
        CU(cudaStreamWaitEvent(si, fork, 0));
        CU(cudaStreamWaitEvent(so, fork, 0));
        for (int c = 0; c < nsec; c++) {
            const size_t off = (size_t)bound[c] * L->e, nb = (size_t)(bound[c + 1] - bound[c]) * L->e * 4;
            CU(cudaMemcpyAsync(L->host_in + off, h_host + off, nb, cudaMemcpyHostToDevice, si));
            CU(cudaEventRecord(ev[2 * c], si));
        }
        for (int c = 0; c < nsec; c++) {
            const size_t off = (size_t)bound[c] * L->e;
            const int rows = bound[c + 1] - bound[c];
            CU(cudaStreamWaitEvent(s, ev[2 * c], 0));
            if (int rc = forward_impl(L, L->host_in + off, L->host_out + off, rows, 0, s, nullptr, nullptr, n)) return rc;
            CU(cudaEventRecord(ev[2 * c + 1], s));
            CU(cudaStreamWaitEvent(so, ev[2 * c + 1], 0));
            CU(cudaMemcpyAsync(out_host + off, L->host_out + off, (size_t)rows * L->e * 4,
                               cudaMemcpyDeviceToHost, so));
        }
        CU(cudaEventRecord(join, so));
        CU(cudaStreamWaitEvent(s, join, 0));
        CU(cudaMemcpyAsync(L->status_host, L->ws.status, 16, cudaMemcpyDeviceToHost, s));
        L->host_in_sections = true;
        return BIVMOE_OK;
    }
    L->host_in_sections = false;
    // Few rows: between a copy node and a kernel of a graph lie 5 us, as long as the copy of 16
    // rows itself.  A kernel brings the rows in, the combine stores the result where it belongs
    // and a last kernel the status: 122 -> 107 us for 16 rows of 2048, 528 -> 518 for 512.
    if (bytes <= kHostDirectBytes && buf.direct()) {
        LaunchCfg c{s, n, L->k, L->e, L->n_expert, L->ff, L->ff_sh, L->has_shared ? 1 : 0, L->sm_count};
        CU(launch_copy_words(c, (const void*)buf.h_dev, L->host_in, bytes));
        if (int rc = forward_graphed(L, L->host_in, (float*)buf.out_dev, n, 0, s)) return rc;
        CU(launch_copy_words(c, L->ws.status, L->status_view, 16));
        return BIVMOE_OK;
    }
    CU(cudaMemcpyAsync(L->host_in, h_host, bytes, cudaMemcpyHostToDevice, s));
    int rc = forward_graphed(L, L->host_in, L->host_out, n, 0, s);   // plain launches under a capture
    if (rc) return rc;
    CU(cudaMemcpyAsync(out_host, L->host_out, bytes, cudaMemcpyDeviceToHost, s));
    CU(cudaMemcpyAsync(L->status_host, L->ws.status, 16, cudaMemcpyDeviceToHost, s));
    return BIVMOE_OK;
}

// What the host-buffer calls keep, made on the first one.  A step that fails leaves the ones
// before it to the next call, which goes on from there: nothing runs until all are done.
static int host_set_up(bivmoe_layer* L) {
    std::string* errp = &L->error;
    const size_t bytes = (size_t)L->max_tokens * L->e * 4;
    for (float** buf : {&L->host_in, &L->host_out}) {
        if (*buf) continue;
        void* p = nullptr;
        CU(dev_alloc(&p, bytes));
        L->allocs.push_back(p);
        L->ws_bytes += bytes;
        *buf = (float*)p;
    }
    if (!L->status_host) {
        CU(cudaHostAlloc((void**)&L->status_host, 16, cudaHostAllocDefault));
        memset(L->status_host, 0, 16);
    }
    if (!L->status_view) CU(cudaHostGetDevicePointer(&L->status_view, L->status_host, 0));
    for (cudaStream_t* st : {&L->in_stream, &L->out_stream})
        if (!*st) CU(cudaStreamCreateWithFlags(st, cudaStreamNonBlocking));
    for (cudaEvent_t& ev : L->host_ev)
        if (!ev) CU(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    return BIVMOE_OK;
}

int bivmoe_forward_host_async(bivmoe_layer* L, const float* h_host, float* out_host, int32_t n) {
    if (!L) return set_err(nullptr, BIVMOE_ERR_ARGUMENT, "null layer");
    std::string* errp = &L->error;
    if (n < 0 || n > L->max_tokens)
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "n = %d outside 0..max_tokens = %d", n, L->max_tokens);
    if (n == 0) {
        note_pass(L, 0, 0, false);
        return BIVMOE_OK;
    }
    if (!h_host || !out_host) return set_err(errp, BIVMOE_ERR_ARGUMENT, "null host pointer");
    DeviceScope on_device(L->device);
    if (int rc = host_set_up(L)) return rc;
    cudaStream_t s = L->own_stream;
    auto& G = L->host_graph;
    const HostBuffers buf = host_buffers(h_host, out_host, n, (size_t)L->e * 4, look_up);
    if (!(G.buf == buf)) {
        if (G.exec) { cudaGraphExecDestroy(G.exec); G.exec = nullptr; }
        G.buf = buf;
        G.seen = 0;
    }
    bool launched = false;
    if (G.exec) {
        CU(cudaGraphLaunch(G.exec, s));
        count_launch(G.launches);
        launched = true;
    } else if (L->use_graph && ++G.seen >= 2 && buf.locked()) {
        // the second identical call with page-locked buffers: capture the whole sequence
        cudaGraph_t graph = nullptr;
        const uint64_t before = bivmoe_launch_count();
        CU(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        const int rc = forward_host_enqueue(L, buf);
        cudaError_t ce = cudaStreamEndCapture(s, &graph);
        G.launches = (int)(bivmoe_launch_count() - before);
        if (!rc && ce == cudaSuccess && graph) ce = cudaGraphInstantiate(&G.exec, graph, 0);
        if (graph) cudaGraphDestroy(graph);
        if (rc || ce != cudaSuccess) {
            G.exec = nullptr;
            L->use_graph = false;   // plain launches from here on
            cudaGetLastError();
            if (rc) return rc;
        } else {
            CU(cudaGraphLaunch(G.exec, s));
            launched = true;
        }
    }
    if (!launched) {
        int rc = forward_host_enqueue(L, buf);
        if (rc) return rc;
    }
    note_pass(L, n, n, false);
    L->in_sections = L->host_in_sections;
    return BIVMOE_OK;
}

int bivmoe_host_wait(bivmoe_layer* L) {
    if (!L) return set_err(nullptr, BIVMOE_ERR_ARGUMENT, "null layer");
    std::string* errp = &L->error;
    if (!L->status_view) return BIVMOE_OK;   // no host-buffer call was ever made
    DeviceScope on_device(L->device);
    cudaStream_t s = L->own_stream;
    CU(cudaStreamSynchronize(s));
    if (L->status_host[0]) {
        const int code = L->status_host[0];
        cudaMemsetAsync(L->ws.status, 0, 16, s);
        return set_err(errp, code, "a device-side bounded wait gave up (status %d)", code);
    }
    return BIVMOE_OK;
}

int bivmoe_forward_host(bivmoe_layer* L, const float* h_host, float* out_host, int32_t n) {
    if (int rc = bivmoe_forward_host_async(L, h_host, out_host, n)) return rc;
    return n > 0 ? bivmoe_host_wait(L) : BIVMOE_OK;
}

// the launches of every layer of the stack, in order, on `stream`
static int stack_enqueue(bivmoe_layer* const* layers, int n_layers, float* x_dev, int n, cudaStream_t stream) {
    bool normed = false;   // by the layer before
    for (int l = 0; l < n_layers; l++) {
        bivmoe_layer* L = layers[l];
        std::string* errp = &L->error;
        DeviceScope on_device(L->device);
        LaunchCfg c{stream, n, L->k, L->e, L->n_expert, L->ff, L->ff_sh, L->has_shared ? 1 : 0, L->sm_count};
        int rc;
        if (router_fuses_norm(n, L->e)) {
            // the router kernel normalises the rows it stages and publishes the scales; the
            // dispatch kernel applies them on the fly: the normed rows never reach HBM
            const RowNorm norm{L->post_norm, L->norm_eps, L->ws.row_scale};
            rc = forward_impl(L, x_dev, x_dev, n, 1, stream, nullptr, &norm);
            normed = false;
        } else {
            if (!normed) CU(launch_rms_norm(c, x_dev, L->post_norm, L->norm_eps, L->ws.h_norm));
            NextLayer next{l + 1 < n_layers ? layers[l + 1] : nullptr};
            rc = forward_impl(L, L->ws.h_norm, x_dev, n, 1, stream, nullptr, nullptr, 0, &next);
            normed = next.normed;
        }
        if (rc) return rc;
    }
    return BIVMOE_OK;
}

int bivmoe_forward_stack(bivmoe_layer* const* layers, int32_t n_layers, float* x_dev, int32_t n,
                         void* stream) {
    if (!layers || n_layers <= 0 || !layers[0])
        return set_err(nullptr, BIVMOE_ERR_ARGUMENT, "no layers");
    bool one_device = true;
    for (int l = 0; l < n_layers; l++) {
        bivmoe_layer* L = layers[l];
        std::string* errp = L ? &L->error : nullptr;
        if (!L || !L->post_norm)
            return set_err(errp, BIVMOE_ERR_ARGUMENT, "layer %d has no post_norm weights", l);
        if (n < 0 || n > L->max_tokens)
            return set_err(errp, BIVMOE_ERR_ARGUMENT, "n = %d outside 0..max_tokens", n);
        one_device = one_device && L->device == layers[0]->device;
    }
    if (n == 0) return BIVMOE_OK;
    // The same stack over the same rows again (an engine's decode loop): the launches of all
    // layers - 4 each up to eight rows of a quantised layer, else 7 or more - are replayed as one graph from the second
    // identical call on.
    bivmoe_layer* L0 = layers[0];
    std::string* errp = &L0->error;
    cudaStream_t s = (cudaStream_t)stream;
    auto& G = L0->stack_graph;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    const bool can_graph = L0->use_graph && one_device && s != nullptr && s != cudaStreamLegacy &&
                           cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone;
    if (!can_graph) return stack_enqueue(layers, n_layers, x_dev, n, s);
    DeviceScope on_device(L0->device);
    const bool same = G.x == x_dev && G.n == n && G.stream == s && (int)G.layers.size() == n_layers &&
                      std::equal(G.layers.begin(), G.layers.end(), layers,
                                 [](uint64_t id, const bivmoe_layer* l) { return id == l->state_id; });
    if (same && G.exec) {
        CU(cudaGraphLaunch(G.exec, s));
        count_launch(G.launches);
        for (int l = 0; l < n_layers; l++) note_pass(layers[l], n, n, router_fuses_norm(n, layers[l]->e));
        return BIVMOE_OK;
    }
    if (!same) {
        if (G.exec) { cudaGraphExecDestroy(G.exec); G.exec = nullptr; }
        G.layers.clear();
        for (int l = 0; l < n_layers; l++) G.layers.push_back(layers[l]->state_id);
        G.x = x_dev; G.n = n; G.stream = s; G.seen = 0;
    }
    if (++G.seen < 2) return stack_enqueue(layers, n_layers, x_dev, n, s);   // the first call also sets kernel attributes
    cudaGraph_t graph = nullptr;
    const uint64_t before = bivmoe_launch_count();
    CU(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    const int rc = stack_enqueue(layers, n_layers, x_dev, n, s);
    cudaError_t ce = cudaStreamEndCapture(s, &graph);
    G.launches = (int)(bivmoe_launch_count() - before);
    if (!rc && ce == cudaSuccess && graph) ce = cudaGraphInstantiate(&G.exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    if (rc || ce != cudaSuccess) {
        G.exec = nullptr;
        L0->use_graph = false;   // plain launches from here on
        cudaGetLastError();
        return rc ? rc : stack_enqueue(layers, n_layers, x_dev, n, s);
    }
    CU(cudaGraphLaunch(G.exec, s));
    return BIVMOE_OK;
}

// ---------------------------------------------------------------------------
// taps

static int copy_out(bivmoe_layer* L, void* dst, const void* src, size_t want, size_t have) {
    std::string* errp = &L->error;
    if (want != have)
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "tap buffer of %zu bytes, expected %zu", want, have);
    CU(cudaMemcpy(dst, src, have, cudaMemcpyDeviceToHost));
    return BIVMOE_OK;
}

// Waits for the device, and has the workspace describe all rows of the last call: a host call
// that ran in sections is run once more in one piece, from the rows in its staging buffer.
static int tap_begin(bivmoe_layer* L) {
    std::string* errp = &L->error;
    CU(cudaSetDevice(L->device));
    CU(cudaDeviceSynchronize());
    if (!L->in_sections) return BIVMOE_OK;
    if (int rc = forward_impl(L, L->host_in, L->host_out, L->last_n, 0, L->own_stream)) return rc;
    CU(cudaStreamSynchronize(L->own_stream));
    return BIVMOE_OK;
}

int bivmoe_tap(bivmoe_layer* L, int32_t which, void* dst, size_t bytes) {
    if (!L || !dst) return set_err(nullptr, BIVMOE_ERR_ARGUMENT, "null layer or buffer");
    std::string* errp = &L->error;
    if (L->ep_world > 1)
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "taps read a whole layer's workspace; this layer is sharded");
    if (int rc = tap_begin(L)) return rc;
    const size_t n = (size_t)L->last_n, k = L->k, ne = L->n_expert, e = L->e, P = n * k;
    const size_t mid = std::max(L->ff, L->ff_sh);
    const Workspace& w = L->ws;
    switch (which) {
        case BIVMOE_TAP_LOGITS:
        case BIVMOE_TAP_SHARED_GATE: {
            std::vector<float> tmp(n * (ne + 1));
            CU(cudaMemcpy(tmp.data(), w.logits, tmp.size() * 4, cudaMemcpyDeviceToHost));
            const bool lg = which == BIVMOE_TAP_LOGITS;
            if (bytes != (lg ? n * ne : n) * 4)
                return set_err(errp, BIVMOE_ERR_ARGUMENT, "tap buffer size mismatch");
            float* o = (float*)dst;
            for (size_t t = 0; t < n; t++) {
                if (lg) memcpy(o + t * ne, tmp.data() + t * (ne + 1), ne * 4);
                else o[t] = tmp[t * (ne + 1) + ne];
            }
            return BIVMOE_OK;
        }
        case BIVMOE_TAP_IDS: return copy_out(L, dst, w.ids, bytes, P * 4);
        case BIVMOE_TAP_WEIGHTS: return copy_out(L, dst, w.weights, bytes, P * 4);
        case BIVMOE_TAP_COUNTS: return copy_out(L, dst, w.counts, bytes, ne * 4);
        case BIVMOE_TAP_ORDER: {   // the padded position space, compacted expert by expert
            if (bytes != P * 4) return set_err(errp, BIVMOE_ERR_ARGUMENT, "tap buffer size mismatch");
            std::vector<int32_t> cnt(ne), off(ne + 1), ord(w.act_rows);
            CU(cudaMemcpy(cnt.data(), w.counts, ne * 4, cudaMemcpyDeviceToHost));
            CU(cudaMemcpy(off.data(), w.offsets, (ne + 1) * 4, cudaMemcpyDeviceToHost));
            CU(cudaMemcpy(ord.data(), w.order, ord.size() * 4, cudaMemcpyDeviceToHost));
            size_t o = 0;
            for (size_t x = 0; x < ne; x++)
                for (int j = 0; j < cnt[x]; j++) ((int32_t*)dst)[o++] = ord[off[x] + j];
            return BIVMOE_OK;
        }
        case BIVMOE_TAP_ACT_Q:
        case BIVMOE_TAP_ACT_D:
        case BIVMOE_TAP_ACT_S: {
            // the tokens' rows are positions 0..n of the slice-major arrays
            if (!w.act_t) return set_err(errp, BIVMOE_ERR_ARGUMENT, "no quantised activations");
            const size_t R = w.act_rows, nsl = e / 256;
            const bool q = which == BIVMOE_TAP_ACT_Q;
            if (bytes != (q ? n * e : n * e / 32 * 4))
                return set_err(errp, BIVMOE_ERR_ARGUMENT, "tap buffer size mismatch");
            // a token's row: its position in the shared group, else its first pair's position
            std::vector<int32_t> tpos(n);
            for (size_t t = 0; t < n; t++) tpos[t] = (int32_t)t;
            if (!L->has_shared && !L->last_few)
                CU(cudaMemcpy2D(tpos.data(), 4, w.pos_of, (size_t)k * 4, 4, n, cudaMemcpyDeviceToHost));
            const bool half = L->last_wide;
            const size_t rb = half ? kHalfRec : kActTileBytes;
            std::vector<uint8_t> rec(nsl * (R / 8) * rb);
            CU(cudaMemcpy(rec.data(), w.act_t, rec.size(), cudaMemcpyDeviceToHost));
            for (size_t t = 0; t < n; t++)
                for (size_t sl = 0; sl < nsl; sl++) {
                    const uint8_t* r0 = rec.data() + (sl * (R / 8) + tpos[t] / 8) * rb;
                    const int tk = tpos[t] % 8;
                    if (q)
                        for (int i = 0; i < 256; i++) {
                            __half_raw v{};
                            if (half) memcpy(&v.x, r0 + half_q_off(tk, i), 2);
                            ((int8_t*)dst)[t * e + sl * 256 + i] = half ? (int8_t)__half2float(__half(v)) : (int8_t)r0[act_q_off(tk, i)];
                        }
                    else
                        for (int b = 0; b < 8; b++) {
                            const int sc = which == BIVMOE_TAP_ACT_S ? 3 : 0;
                            ((float*)dst)[t * (e / 32) + sl * 8 + b] =
                                *(const float*)(r0 + (half ? half_scale_off(sc, b, tk) : act_scale_off(sc, b, tk)));
                        }
                }
            return BIVMOE_OK;
        }
        case BIVMOE_TAP_MID: {
            const size_t R = w.act_rows, ffw = L->ff;
            if (bytes != P * ffw * 4) return set_err(errp, BIVMOE_ERR_ARGUMENT, "tap buffer size mismatch");
            std::vector<float> tmp(R * mid);
            std::vector<int32_t> pos(P);
            CU(cudaMemcpy(tmp.data(), w.mid, tmp.size() * 4, cudaMemcpyDeviceToHost));
            CU(cudaMemcpy(pos.data(), w.pos_of, P * 4, cudaMemcpyDeviceToHost));
            // pairs of groups the BF16 tensor-core kernels took have no f32 mid row: theirs is
            // the sum of the two bf16 terms the down product reads (mid to 2^-17)
            std::vector<uint8_t> terms;
            std::vector<int32_t> ids, cnt;
            int32_t big_min = 0;   // as the pass set it
            const bool has_terms = w.mid_b && L->prefill_min > 0;
            if (has_terms) {
                terms.resize((mid / 64) * (R / 8) * (size_t)kActBRec);
                ids.resize(P);
                cnt.resize(ne);
                CU(cudaMemcpy(terms.data(), w.mid_b, terms.size(), cudaMemcpyDeviceToHost));
                CU(cudaMemcpy(ids.data(), w.ids, P * 4, cudaMemcpyDeviceToHost));
                CU(cudaMemcpy(cnt.data(), w.counts, ne * 4, cudaMemcpyDeviceToHost));
                CU(cudaMemcpy(&big_min, w.big_min, 4, cudaMemcpyDeviceToHost));
            }
            auto bf = [](uint16_t v) { uint32_t u = (uint32_t)v << 16; float f; memcpy(&f, &u, 4); return f; };
            for (size_t p = 0; p < P; p++) {
                float* o = (float*)dst + p * ffw;
                if (pos[p] < 0) { memset(o, 0, ffw * 4); continue; }
                const bool big = has_terms && big_min > 0 && ids[p] >= 0 && cnt[ids[p]] >= big_min;
                for (size_t sl = 0; sl < ffw / 64; sl++) {
                    if (!big) {
                        memcpy(o + sl * 64, tmp.data() + (sl * R + pos[p]) * 64, 256);
                        continue;
                    }
                    const uint8_t* rec = terms.data() + (sl * (R / 8) + pos[p] / 8) * (size_t)kActBRec;
                    for (int i = 0; i < 64; i++) {
                        uint16_t hi, lo;
                        memcpy(&hi, rec + act_b_off(pos[p] % 8, i), 2);
                        memcpy(&lo, rec + kActBLo + act_b_off(pos[p] % 8, i), 2);
                        o[sl * 64 + i] = bf(hi) + bf(lo);
                    }
                }
            }
            return BIVMOE_OK;
        }
        case BIVMOE_TAP_PAIR_OUT: {
            if (bytes != P * e * 4) return set_err(errp, BIVMOE_ERR_ARGUMENT, "tap buffer size mismatch");
            std::vector<float> tmp((size_t)w.act_rows * e);
            std::vector<int32_t> pos(P);
            CU(cudaMemcpy(tmp.data(), w.pair_out, tmp.size() * 4, cudaMemcpyDeviceToHost));
            CU(cudaMemcpy(pos.data(), w.pos_of, P * 4, cudaMemcpyDeviceToHost));
            for (size_t p = 0; p < P; p++)
                memcpy((float*)dst + p * e, tmp.data() + (size_t)pos[p] * e, e * 4);
            return BIVMOE_OK;
        }
        case BIVMOE_TAP_SHARED_OUT:
            if (!L->has_shared) return set_err(errp, BIVMOE_ERR_ARGUMENT, "no shared expert");
            return copy_out(L, dst, w.pair_out, bytes, n * e * 4);
        case BIVMOE_TAP_BIG_MIN: return copy_out(L, dst, w.big_min, bytes, 4);
        default: return set_err(errp, BIVMOE_ERR_ARGUMENT, "unknown tap %d", which);
    }
}

int bivmoe_tap_block_dots(bivmoe_layer* L, int32_t matrix, int32_t expert, int32_t row,
                          int32_t act_row, int32_t* out) {
    if (!L || !out) return set_err(nullptr, BIVMOE_ERR_ARGUMENT, "null layer or buffer");
    std::string* errp = &L->error;
    if (L->ep_world > 1)
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "taps read a whole layer's workspace; this layer is sharded");
    if (int rc = tap_begin(L)) return rc;
    if (matrix < 0 || matrix > 5 || (matrix >= 3 && !L->has_shared))
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "matrix %d", matrix);
    const bool shared = matrix >= 3, is_down = matrix % 3 == 2;
    const DevTiles& m = is_down ? (shared ? L->sh_down : L->down) : (shared ? L->sh_gate_up : L->gate_up);
    const int tile_base = matrix % 3 == 1 ? 2 : 0;   // up rows are tiles 2, 3 of a gate+up chunk
    const int n = L->last_n, P = n * L->k;
    if (expert < 0 || expert >= m.n || row < 0 || row >= m.rows || act_row < 0 ||
        act_row >= (is_down && !shared ? P : n))
        return set_err(errp, BIVMOE_ERR_ARGUMENT, "index out of range");
    if (type_uses_f32_act(m.ty))
        return set_err(errp, BIVMOE_ERR_UNSUPPORTED, "type %d has no integer block dots", m.ty);
    const int nb = m.cols / 32;
    int32_t* dots = nullptr;
    CU(cudaMalloc((void**)&dots, (size_t)nb * 4));
    cudaError_t ce = cudaSuccess;
    // gate/up rows meet the token's Q8 row of h (position = token); down rows the
    // Q8 row of the pair's mid vector at the pair's position
    int32_t pos = act_row;
    if (is_down && !shared) ce = cudaMemcpy(&pos, L->ws.pos_of + act_row, 4, cudaMemcpyDeviceToHost);
    if (!is_down && !L->has_shared && !L->last_few)
        ce = cudaMemcpy(&pos, L->ws.pos_of + (size_t)act_row * L->k, 4, cudaMemcpyDeviceToHost);
    if (ce == cudaSuccess)
        ce = launch_block_dots(m, tile_base, expert, row, is_down ? L->ws.mid_t : L->ws.act_t,
                               L->ws.act_rows, pos, L->last_wide, dots, 0);
    if (ce == cudaSuccess) ce = cudaMemcpy(out, dots, (size_t)nb * 4, cudaMemcpyDeviceToHost);
    cudaFree(dots);
    CU(ce);
    return BIVMOE_OK;
}

int bivmoe_int8_peak(bivmoe_layer* L, double* tops) {
    if (!L || !tops) return set_err(nullptr, BIVMOE_ERR_ARGUMENT, "null layer or result");
    std::string* errp = &L->error;
    DeviceScope on_device(L->device);
    CU(measure_int8_peak(L->sm_count, L->ws.status + 1, L->own_stream, tops));
    int32_t st = 0;
    CU(cudaMemcpy(&st, L->ws.status + 1, 4, cudaMemcpyDeviceToHost));
    if (st) {
        cudaMemset(L->ws.status + 1, 0, 4);
        return set_err(errp, st, "the probe's bounded wait gave up");
    }
    return BIVMOE_OK;
}

int bivmoe_numerics(const bivmoe_layer* L, char* buf, size_t len) {
    if (!L || !buf || !len) return set_err(nullptr, BIVMOE_ERR_ARGUMENT, "null layer or buffer");
    // which expert kernels this layer's types get: groups that are few or small (and every group
    // of types without a tcgen05 kernel) take the warp-level kernels
    const bool f32act = type_uses_f32_act(L->gate_up.ty);
    const char* small = L->all_bf16 ? "mma.sync-three-bf16-terms" : f32act ? "f32-fma" : "mma.sync-s8-block-dots";
    char big[96] = "";
    if (L->prefill_min > 0)
        snprintf(big, sizeof big, "+tcgen05-%s-from-%d-rows", L->gate_up.ty == BIVMOE_BF16 ? "f16-two-bf16-terms" : "i8-block-dots",
                 L->prefill_min);
    if (L->wide_min > 0) snprintf(big, sizeof big, "+tcgen05-f16-scaled-integers-from-%d-rows-a-group", L->wide_min);
    snprintf(buf, len,
             "kind=cuda device=%s sms=%d repack=v%d experts=%s/bulk-copy-ring/tiled-weights%s "
             "router=f32-avx2-order combine=ordered-fma types=%d/%d/%d",
             L->device_name.c_str(), L->sm_count, kRepackVersion, small, big, L->gate_up.ty, L->gate_up.ty,
             L->down.ty);
    return BIVMOE_OK;
}

int bivmoe_memory(const bivmoe_layer* L, uint64_t* weight_bytes, uint64_t* workspace_bytes) {
    if (!L) return set_err(nullptr, BIVMOE_ERR_ARGUMENT, "null layer");
    if (weight_bytes) *weight_bytes = L->weight_bytes;
    if (workspace_bytes) *workspace_bytes = L->ws_bytes;
    return BIVMOE_OK;
}

}  // extern "C"
