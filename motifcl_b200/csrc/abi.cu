// C-ABI layer of libmotifcl_cuda.so: contexts, argument checks, dispatch to the kernels.
// The declarations and the reference interfaces they replace are in include/motifcl_cuda.h.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <set>
#include <string>
#include <vector>

#include "kernels.h"
#include "motifcl_cuda.h"

// Decode GEMVs of a recording: launches that take a list of matrices each.
struct GemvList {
    mcl_cuda_ctx* ctx;                     // the recording context or a lane of it
    bool tc;                               // two nodes of gemv_tc.cu, or one of gemv_mma.cu
    cudaGraphNode_t node[2];               // what is recorded behind the launch depends on the last of them
    int M;
    std::vector<mcl::GemvItem> items;
    void* ws;                              // tc: of the digits and sums
    size_t ws_bytes;
};
struct GemvRecord {
    std::vector<GemvList> lists;
    size_t open = 0;                       // from here on: with nothing else between and behind them, open to further matrices
    cudaGraphNode_t tail = nullptr;        // last node of the last one, and the capture it belongs to: a handle alone may come back for a
    unsigned long long capture = 0;        // node of a later one
    void close() { open = lists.size(); tail = nullptr; }
};

struct mcl_cuda_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int sm_count = 0;
    size_t max_smem = 0;
    size_t device_mem = 0;
    std::string name;
    std::string error;
    uint64_t launches = 0;
    // grow-only workspace used by entry points that need scratch (row tiles of grad_w, ...)
    void* ws = nullptr;
    size_t ws_bytes = 0;
    bool ws_recorded = false;    // the recording holds addresses inside it
    bool ws_held = false;        // and so may a graph that live_batches does not count: a capture of the caller, a batch this context was a lane of
    std::vector<void*> ws_kept;  // earlier ones that a graph may hold
    size_t ws_kept_bytes = 0;
    // how the contractions run (mcl_cuda_set_gemm_mode)
    int gemm_mode = MCL_CUDA_GEMM_AUTO;
    int* err_word = nullptr;     // device word the tensor-core kernels set when a bounded wait gives up
    const uint32_t* seed_offset = nullptr;   // device word added to every update seed (mcl_cuda_set_seed_offset)
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    uint64_t lane_mark = 0;      // launches at the last lane_fork (when this context is a lane)
    bool recording = false;      // between mcl_cuda_batch_begin and mcl_cuda_batch_end, on a lane between fork and join
    bool is_lane = false;        // of the recording
    uint64_t recorded_launches = 0;
    GemvRecord gemvs;            // of the recording
    int live_batches = 0;        // recorded batches not yet destroyed: they hold addresses inside the workspace
};

struct mcl_cuda_batch {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    uint64_t kernels = 0;        // kernel launches one replay stands for
    mcl_cuda_ctx* ctx = nullptr; // the context it was recorded on (looked up among the live contexts before use)
};

namespace {

thread_local std::string g_error;   // errors raised before a context exists

// live contexts, so that a batch destroyed after its context does not touch freed memory
std::mutex g_ctx_mutex;
std::set<mcl_cuda_ctx*> g_live_ctx;

int fail(mcl_cuda_ctx* ctx, int code, const std::string& msg) {
    if (ctx) ctx->error = msg; else g_error = msg;
    return code;
}
int fail_cuda(mcl_cuda_ctx* ctx, const char* what, cudaError_t e) {
    return fail(ctx, MCL_CUDA_ECUDA, std::string(what) + ": " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")");
}

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        cudaGetDevice(&prev);
        if (prev != dev) cudaSetDevice(dev);
        else prev = -1;
    }
    ~DeviceGuard() { if (prev >= 0) cudaSetDevice(prev); }
};

// Shared checks, worded after the reference's wrappers (src/runtime/vulkan_backend.cpp:8497-8521).
int check_counter_dims(mcl_cuda_ctx* ctx, const char* op, size_t C, size_t in_features,
                       size_t out_features) {
    const std::string o(op);
    if (C == 0 || in_features == 0 || out_features == 0)
        return fail(ctx, MCL_CUDA_EINVAL, o + " requires non-zero dimensions");
    if (in_features % 4 != 0) return fail(ctx, MCL_CUDA_EINVAL, o + " requires in_features % 4 == 0");
    if (C > 32 || 3 * (2 * C - 1) > 64)
        return fail(ctx, MCL_CUDA_EINVAL, o + ": C too large for 6-bit packed state encoding");
    if (in_features > 0x7fffffffull || out_features > 0x7fffffffull ||
        in_features * out_features > 0x7fffffffull)
        return fail(ctx, MCL_CUDA_EINVAL, o + ": out_features * in_features exceeds 32-bit element indexing");
    return MCL_CUDA_OK;
}
int check_ptr(mcl_cuda_ctx* ctx, const char* op, const char* name, const void* p, size_t align) {
    if (p == nullptr) return fail(ctx, MCL_CUDA_EINVAL, std::string(op) + ": " + name + " is NULL");
    if (reinterpret_cast<uintptr_t>(p) % align != 0)
        return fail(ctx, MCL_CUDA_EINVAL, std::string(op) + ": " + name + " must be " + std::to_string(align) + "-byte aligned");
    return MCL_CUDA_OK;
}
int check_hypers(mcl_cuda_ctx* ctx, const char* op, float lr, float lr_scale, float rms_beta, float rms_eps) {
    const std::string o(op);
    if (!std::isfinite(lr)) return fail(ctx, MCL_CUDA_EINVAL, o + " requires finite lr");
    if (!std::isfinite(lr_scale)) return fail(ctx, MCL_CUDA_EINVAL, o + " requires finite lr_scale");
    if (!std::isfinite(rms_beta)) return fail(ctx, MCL_CUDA_EINVAL, o + " requires finite rms_beta");
    if (!std::isfinite(rms_eps) || rms_eps < 0.0f)
        return fail(ctx, MCL_CUDA_EINVAL, o + " requires non-negative finite rms_eps");
    return MCL_CUDA_OK;
}

// A larger workspace.  The old one is freed, or kept as long as the context where a graph may hold addresses inside it; the new one is then
// half as large again at least where it can be, so that all kept ones together stay below twice the one in use.
int ws_grow(mcl_cuda_ctx* ctx, size_t bytes) {
    const bool keep = ctx->ws && (ctx->ws_held || ctx->ws_recorded || ctx->live_batches > 0);
    void* fresh = nullptr;
    size_t take = keep ? std::max(bytes, ctx->ws_bytes / 2 * 3) : bytes;
    cudaError_t e = cudaMalloc(&fresh, take);
    if (e != cudaSuccess && take > bytes) { cudaGetLastError(); e = cudaMalloc(&fresh, take = bytes); }
    if (!keep && ctx->ws) {
        const cudaError_t busy = cudaStreamSynchronize(ctx->stream);
        if (busy != cudaSuccess) { if (e == cudaSuccess) cudaFree(fresh); return fail_cuda(ctx, "workspace sync", busy); }
        cudaFree(ctx->ws);
        ctx->ws = nullptr;
        if (e != cudaSuccess) {            // both do not fit side by side
            cudaGetLastError();
            e = cudaMalloc(&fresh, bytes);
            if (e != cudaSuccess && cudaMalloc(&ctx->ws, ctx->ws_bytes) != cudaSuccess) { ctx->ws = nullptr; ctx->ws_bytes = 0; }
        }
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(ctx, MCL_CUDA_ENOMEM, "workspace allocation of " + std::to_string(bytes) + " bytes failed");
    }
    if (keep) { ctx->ws_kept.push_back(ctx->ws); ctx->ws_kept_bytes += ctx->ws_bytes; }
    ctx->ws = fresh;
    ctx->ws_bytes = take;
    ctx->ws_held = ctx->ws_recorded = false;
    return MCL_CUDA_OK;
}
// whether the caller captures the context's stream
bool foreign_capture(const mcl_cuda_ctx* ctx) {
    if (ctx->recording) return false;
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &st) != cudaSuccess) cudaGetLastError();
    return st != cudaStreamCaptureStatusNone;
}
int ws_reserve(mcl_cuda_ctx* ctx, size_t bytes, void** out) {
    const bool foreign = foreign_capture(ctx);
    if (bytes > ctx->ws_bytes) {
        if (ctx->recording)
            return fail(ctx, MCL_CUDA_EINVAL, "workspace would grow while recording a batch: run the same calls once unrecorded first");
        if (ctx->live_batches > 0)
            return fail(ctx, MCL_CUDA_EINVAL, "workspace would grow (to " + std::to_string(bytes) + " bytes) while " +
                                                  std::to_string(ctx->live_batches) + " recorded batch(es) hold addresses inside it: "
                                                  "run the largest call once before recording, or destroy the batches first");
        // a capture that the caller runs on the stream would be broken by the wait and the allocation
        if (foreign)
            return fail(ctx, MCL_CUDA_EINVAL, "workspace would grow while the stream is being captured: run the same calls once uncaptured first");
        const int rc = ws_grow(ctx, bytes);
        if (rc != MCL_CUDA_OK) return rc;
    }
    if (foreign || ctx->is_lane) ctx->ws_held = true;
    else if (ctx->recording) ctx->ws_recorded = true;
    *out = ctx->ws;
    return MCL_CUDA_OK;
}

#define MCL_TRY(expr) do { int _rc = (expr); if (_rc != MCL_CUDA_OK) return _rc; } while (0)
#define MCL_NEED_CTX(ctx) do { if (!(ctx)) return fail(nullptr, MCL_CUDA_EINVAL, "context is NULL"); } while (0)
#define MCL_NOT_RECORDING(ctx, what) do { if ((ctx)->recording) return fail(ctx, MCL_CUDA_EINVAL, what " is not allowed while recording a batch"); } while (0)
#define MCL_LAUNCH(ctx, what, call) do { cudaError_t _e = (call); if (_e != cudaSuccess) return fail_cuda(ctx, what, _e); ++(ctx)->launches; } while (0)

int create_impl(int device, cudaStream_t stream, bool own, mcl_cuda_ctx** out_ctx) {
    if (!out_ctx) return fail(nullptr, MCL_CUDA_EINVAL, "out_ctx is NULL");
    *out_ctx = nullptr;
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n <= 0) {
        cudaGetLastError();
        return fail(nullptr, MCL_CUDA_ENODEVICE, "no CUDA device available");
    }
    if (device < 0 || device >= n) return fail(nullptr, MCL_CUDA_EINVAL, "device index out of range");
    cudaDeviceProp prop;
    e = cudaGetDeviceProperties(&prop, device);
    if (e != cudaSuccess) return fail_cuda(nullptr, "cudaGetDeviceProperties", e);
    if (prop.major != 10)
        return fail(nullptr, MCL_CUDA_EUNSUPPORTED,
                    std::string("this library is built for sm_100a only; device is ") + prop.name +
                        " (sm_" + std::to_string(prop.major) + std::to_string(prop.minor) + ")");
    mcl_cuda_ctx* ctx = new (std::nothrow) mcl_cuda_ctx();
    if (!ctx) return fail(nullptr, MCL_CUDA_ENOMEM, "out of host memory");
    ctx->device = device;
    ctx->sm_count = prop.multiProcessorCount;
    ctx->max_smem = prop.sharedMemPerBlockOptin;
    ctx->device_mem = prop.totalGlobalMem;
    ctx->name = prop.name;
    DeviceGuard guard(device);
    if (own) {
        e = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking);
        if (e != cudaSuccess) { delete ctx; return fail_cuda(nullptr, "cudaStreamCreate", e); }
        ctx->own_stream = true;
    } else {
        ctx->stream = stream;
    }
    {   // keep freed blocks in the default pool instead of returning them to the driver at every synchronisation
        cudaMemPool_t pool = nullptr;
        unsigned long long keep = ~0ull;
        if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess)
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        cudaGetLastError();
    }
    // [0] error word, [8] work items drawn and [9] CTAs done of the running contraction (tc_gemm.cu leaves both at zero)
    e = cudaMalloc(reinterpret_cast<void**>(&ctx->err_word), 16 * sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(ctx->err_word, 0, 16 * sizeof(int));
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ctx->ev_fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ctx->ev_join, cudaEventDisableTiming);
    if (e != cudaSuccess) {
        if (ctx->own_stream) cudaStreamDestroy(ctx->stream);
        delete ctx;
        return fail_cuda(nullptr, "context setup", e);
    }
    {
        std::lock_guard<std::mutex> lock(g_ctx_mutex);
        g_live_ctx.insert(ctx);
    }
    *out_ctx = ctx;
    return MCL_CUDA_OK;
}

// Reads (after the stream has drained) whether a tensor-core kernel abandoned a wait.
int check_device_error(mcl_cuda_ctx* ctx) {
    int w = 0;
    cudaError_t e = cudaMemcpy(&w, ctx->err_word, sizeof(int), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return fail_cuda(ctx, "error-word read", e);
    if (w != 0) {
        cudaMemset(ctx->err_word, 0, sizeof(int));
        const char* who;
        switch (w) {
            case 1: case 11: who = "copy lane (ring slot never released)"; break;
            case 2: case 12: who = "MMA lane (operand tile never arrived)"; break;
            case 13: case 15: who = "epilogue / converter warps (accumulator or tile never completed)"; break;
            case 14: who = "MMA lane (accumulator never drained)"; break;
            case 16: case 17: who = "work items (the drawing warp and its readers lost step)"; break;
            case 21: who = "wide-row counter update (a row slot was never marked ready or released)"; break;
            case 41: who = "single-layer kernel (a k-tile's MMAs never completed)"; break;
            case 31: who = "peer all-reduce (a rank never announced its partial result)"; break;
            default: who = "epilogue (accumulator never completed)"; break;
        }
        return fail(ctx, MCL_CUDA_ECUDA, std::string("a kernel gave up a bounded wait: ") + who + " [code " +
                                             std::to_string(w) + "]; results of that call are invalid");
    }
    return MCL_CUDA_OK;
}

struct Carver {
    char* base = nullptr;
    size_t off = 0;
    size_t reserve(size_t bytes) { off = (off + 1023) & ~size_t(1023); const size_t at = off; off += bytes; return at; }
};

inline int up8(size_t x) { return (int)((x + 7) & ~size_t(7)); }

// out, col_scale: where the output goes and what its columns are scaled by (null: not checked)
bool tc_wanted(const mcl_cuda_ctx* ctx, size_t M, size_t N, size_t K, const void* out = nullptr, const void* col_scale = nullptr) {
    if (ctx->gemm_mode == MCL_CUDA_GEMM_EXACT) return false;
    if (N % 4 != 0) return false;                       // rows of the output are written in 16-byte units
    if ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(col_scale)) & 15) return false;
    if (M > 0x7fffffffull / 2 || N > 0x7fffffffull / 2 || K > 0x7fffffffull / 2) return false;
    if (ctx->gemm_mode == MCL_CUDA_GEMM_TENSOR) return true;
    return (double)M * (double)N * (double)K >= (double)(1u << 22);
}

// one-launch kernels of narrow layers (layer_kernels.cu)
bool layer_wanted(const mcl_cuda_ctx* ctx, size_t tokens, size_t I, size_t O) {
    if (ctx->gemm_mode == MCL_CUDA_GEMM_EXACT || !mcl::layer_kernels_fit(tokens, I, O)) return false;
    return ctx->gemm_mode == MCL_CUDA_GEMM_TENSOR || (double)tokens * (double)I * (double)O >= (double)(1u << 22);
}

#define MCL_CU(ctx, what, call) do { cudaError_t _e = (call); if (_e != cudaSuccess) return fail_cuda(ctx, what, _e); } while (0)

// Tensor-core products on fp16 terms (tc_gemm.cu).  A call carves the terms of its tensors from the workspace, fills them, and
// runs its products.
enum Scaling { kByRow, kByPartner };     // planes: a scale per row, or one that completes those of the partner's rows (kernels.h, SplitDesc)
struct TermBuf { size_t planes, scaled, words, inv, inv_s; size_t rows; int cols, ld; Scaling how; };
size_t term_bytes(size_t rows, size_t cols) { return 2 * rows * (size_t)up8(cols) * 2 + mcl::kTermPad; }
size_t digit_bytes(size_t O, size_t I) { return O * (size_t)up8(I) * 2 + mcl::kTermPad; }
TermBuf carve_terms(Carver* cv, size_t rows, size_t cols, bool plain, bool scaled, Scaling how) {
    TermBuf t = {0, 0, 0, 0, 0, rows, (int)cols, up8(cols), how};
    if (plain) t.planes = cv->reserve(term_bytes(rows, cols));
    if (plain && how == kByRow) t.inv = cv->reserve(rows * sizeof(float));
    if (plain && how == kByPartner) t.words = cv->reserve(2 * sizeof(uint32_t));
    if (scaled) { t.scaled = cv->reserve(term_bytes(rows, cols)); t.inv_s = cv->reserve(rows * sizeof(float)); }
    return t;
}
// col_scale != null: the scaled terms are made too; partner: whose row scales the plain planes complete (null: none)
mcl::SplitDesc split_of(char* w, const TermBuf& t, const float* src, const float* col_scale, bool plain, const TermBuf* partner) {
    mcl::SplitDesc d = {src, (int)t.rows, t.cols, t.ld, col_scale, plain ? w + t.planes : nullptr, col_scale ? w + t.scaled : nullptr,
                        plain && t.how == kByRow ? reinterpret_cast<float*>(w + t.inv) : nullptr,
                        col_scale ? reinterpret_cast<float*>(w + t.inv_s) : nullptr,
                        plain && partner ? reinterpret_cast<const float*>(w + partner->inv) : nullptr,
                        plain && t.how == kByPartner ? reinterpret_cast<uint32_t*>(w + t.words) : nullptr};
    return d;
}
mcl::TcOperand terms_of(char* w, const TermBuf& t, bool scaled, bool mn_major) {
    mcl::TcOperand o = {w + (scaled ? t.scaled : t.planes), (int)t.rows, t.cols, t.ld, 2, mn_major ? 1 : 0, nullptr, nullptr};
    if (scaled) o.inv = reinterpret_cast<const float*>(w + t.inv_s);
    else if (t.how == kByPartner) o.words = reinterpret_cast<const uint32_t*>(w + t.words);
    else if (!mn_major) o.inv = reinterpret_cast<const float*>(w + t.inv);
    return o;
}
mcl::TcOperand digits_of(const char* T, size_t O, size_t I, bool mn_major) {
    mcl::TcOperand o = {T, (int)O, (int)I, up8(I), 1, mn_major ? 1 : 0, nullptr, nullptr};
    return o;
}
#define MCL_TC(ctx, op, call) do { int _n = 0; cudaError_t _e = (call); (ctx)->launches += _n; if (_e != cudaSuccess) return fail_cuda(ctx, op, _e); } while (0)

// plan of a product with ternary digits (depth unbounded: exact digits) or of two split tensors
mcl::TcPlan digit_plan(const mcl_cuda_ctx* ctx, size_t M, size_t N, size_t K) { return mcl::tc_plan((int)M, (int)N, (int)K, 2, ctx->sm_count, 0); }
mcl::TcPlan dense_plan(const mcl_cuda_ctx* ctx, size_t M, size_t N, size_t K) {
    return mcl::tc_plan((int)M, (int)N, (int)K, 3, ctx->sm_count, mcl::kGradDepthLimit);
}
mcl::TcProblem tc_problem(const mcl::TcOperand& a, const mcl::TcOperand& b, float* c, size_t M, size_t N, size_t K, const mcl::TcPlan& plan,
                          const float* col_scale, void* splitk_ws) {
    mcl::TcProblem q = {a, b, c, (int)M, (int)N, (int)K, plan, col_scale, static_cast<float*>(splitk_ws), 0};
    return q;
}
cudaError_t reduce_of(const mcl::TcProblem& q, cudaStream_t stream) {
    const int rows = q.turned ? q.N : q.M, cols = q.turned ? q.M : q.N;
    return mcl::launch_splitk_reduce(q.splitk_ws, q.c, q.col_scale, rows, cols, cols, q.plan.splits, stream);
}
int tc_product(mcl_cuda_ctx* ctx, const char* op, const mcl::TcProblem& q) {
    MCL_TC(ctx, op, mcl::launch_tc_products(&q, 1, ctx->err_word, ctx->max_smem, ctx->sm_count, ctx->stream, &_n));
    if (q.plan.splits > 1)
        MCL_LAUNCH(ctx, op, reduce_of(q, ctx->stream));
    return MCL_CUDA_OK;
}
int split_tensors(mcl_cuda_ctx* ctx, const char* op, const mcl::SplitDesc* d, int n) {
    MCL_TC(ctx, op, mcl::launch_split_terms(d, n, ctx->sm_count, ctx->stream, &_n));
    return MCL_CUDA_OK;
}

// Y, dX and dW of several layers; the ternary digits come from the packed 6-bit state or, when state == NULL, from the 2-bit
// words.  y, grad_x, grad_w may be NULL.
struct ProductLayer {
    const float* x;
    const float* grad_out;
    const uint8_t* state;
    const uint32_t* packed2;
    const float* scale;
    float* y;
    float* grad_x;
    float* grad_w;
    size_t I, O, Nt;
};
size_t layer_term_bytes(const ProductLayer& L) {
    return (L.y || L.grad_w ? term_bytes(L.Nt, L.I) : 0) + (L.grad_w ? term_bytes(L.Nt, L.O) : 0) + (L.grad_x ? term_bytes(L.Nt, L.O) : 0) +
           (L.y || L.grad_x ? digit_bytes(L.O, L.I) : 0);
}
// One chunk of layers.  w == null: returns in *bytes the workspace it needs; else runs it.
int products_chunk(mcl_cuda_ctx* ctx, const char* op, const ProductLayer* L, size_t n, size_t C, char* w, size_t* bytes) {
    std::vector<TermBuf> xb(n), gb(n);
    std::vector<size_t> t_off(n, 0);
    std::vector<mcl::TcProblem> pr;
    std::vector<size_t> k_off;
    Carver cv;
    // dW of many layers: a CTA or a pair per tile, whichever takes less in sum
    int dw_cg = 1;
    // Where the operands of all dW are more than L2 holds (126 MB), a plane is read once; measured over 42 layers of dim 288: -1.5 %
    // at 131 MB, +2 % at 262 MB, +6 % at 1.1 GB.
    size_t dw_bytes = 0;
    for (size_t i = 0; i < n; ++i) dw_bytes += L[i].grad_w ? 4 * L[i].Nt * (L[i].I + L[i].O) : 0;
    const bool together = n > 1 && dw_bytes > (size_t)192 << 20;
    const int min_items = (int)((3 * (size_t)ctx->sm_count + n - 1) / n);
    if (n > 1) {
        double cost[2] = {0, 0};
        for (size_t i = 0; i < n; ++i)
            for (int cg = 1; cg <= 2 && L[i].grad_w; ++cg)
                cost[cg - 1] += mcl::tc_plan_shared((int)L[i].O, (int)L[i].I, (int)L[i].Nt, 3, cg, mcl::kGradDepthLimit, min_items, together).cost;
        dw_cg = cost[1] < cost[0] ? 2 : 1;
    }
    // A product with digits alone in its launch runs as C^T = T X^T where that wastes less of the last tile of tokens: tokens are then its
    // columns, in tiles of 64 to 256, not its rows, in tiles of 128 or 256 (777 tokens: 800 columns for 1024 rows).  Forwards one after the other on a
    // stream, us: 777 x 4096 -> 14336 205 -> 180, 300 x 4096 -> 4096 62 -> 53.  Not where an accumulator would take a longer
    // slice of K: its error grows with it (40 x 4096 -> 14336, 5 slices: 86 us and 1.1e-7, turned in one 89 and 3.1e-7).
    auto row_plan = [&](size_t M, size_t N, size_t K, bool* turned) {
        if (n > 1) return mcl::tc_plan_shared((int)M, (int)N, (int)K, 2, M > 128 ? 2 : 1, 0, 0);
        const mcl::TcPlan straight = digit_plan(ctx, M, N, K), other = digit_plan(ctx, N, M, K);
        *turned = other.cost < 0.98 * straight.cost && other.ktiles_per_split <= straight.ktiles_per_split;
        return *turned ? other : straight;
    };
    for (size_t i = 0; i < n; ++i) {
        const ProductLayer& l = L[i];
        xb[i] = carve_terms(&cv, l.Nt, l.I, l.y || l.grad_w, false, kByRow);
        gb[i] = carve_terms(&cv, l.Nt, l.O, l.grad_w != nullptr, l.grad_x != nullptr, kByPartner);
        if (l.y || l.grad_x) t_off[i] = cv.reserve(digit_bytes(l.O, l.I));
    }
    for (size_t i = 0; i < n; ++i) {
        const ProductLayer& l = L[i];
        auto add = [&](const mcl::TcOperand& a, const mcl::TcOperand& b, float* c, size_t M, size_t N, size_t K, const mcl::TcPlan& plan, const float* cs) {
            k_off.push_back(plan.splits > 1 ? cv.reserve(plan.workspace_bytes) : 0);
            pr.push_back(tc_problem(a, b, c, M, N, K, plan, cs, w + k_off.back()));
        };
        auto add_rows = [&](const mcl::TcOperand& terms, const mcl::TcOperand& digits, float* c, size_t N, size_t K, const float* cs) {
            bool turned = false;
            const mcl::TcPlan plan = row_plan(l.Nt, N, K, &turned);
            if (turned) add(digits, terms, c, N, l.Nt, K, plan, cs);
            else add(terms, digits, c, l.Nt, N, K, plan, cs);
            pr.back().turned = turned;
        };
        if (l.y) add_rows(terms_of(w, xb[i], false, false), digits_of(w + t_off[i], l.O, l.I, false), l.y, l.O, l.I, l.scale);
        if (l.grad_x) add_rows(terms_of(w, gb[i], true, false), digits_of(w + t_off[i], l.O, l.I, true), l.grad_x, l.I, l.O, nullptr);
        if (l.grad_w)
            add(terms_of(w, gb[i], false, true), terms_of(w, xb[i], false, true), l.grad_w, l.O, l.I, l.Nt,
                n == 1 ? dense_plan(ctx, l.O, l.I, l.Nt)
                       : mcl::tc_plan_shared((int)l.O, (int)l.I, (int)l.Nt, 3, dw_cg, mcl::kGradDepthLimit, min_items, together), nullptr);
    }
    if (!w) { *bytes = cv.off; return MCL_CUDA_OK; }
    std::vector<mcl::SplitDesc> sd;
    std::vector<mcl::ExpandDesc> ed;
    for (size_t i = 0; i < n; ++i) {
        const ProductLayer& l = L[i];
        if (l.y || l.grad_w) sd.push_back(split_of(w, xb[i], l.x, nullptr, true, nullptr));
        if (l.grad_x || l.grad_w) sd.push_back(split_of(w, gb[i], l.grad_out, l.grad_x ? l.scale : nullptr, l.grad_w != nullptr, &xb[i]));
        if (l.y || l.grad_x) {
            const mcl::ExpandDesc d = {l.state, l.packed2, (int)l.O, (int)l.I, up8(l.I), w + t_off[i]};
            ed.push_back(d);
        }
    }
    MCL_TRY(split_tensors(ctx, op, sd.data(), (int)sd.size()));
    if (!ed.empty()) MCL_TC(ctx, op, mcl::launch_expand_ternary(ed.data(), (int)ed.size(), (int)C, ctx->sm_count, ctx->stream, &_n));
    // products of one kind together, the longest items first (they are drawn in this order)
    std::stable_sort(pr.begin(), pr.end(), [](const mcl::TcProblem& a, const mcl::TcProblem& b) {
        const int ta = a.turned ? 2 : a.b.planes + 1, tb = b.turned ? 2 : b.b.planes + 1;
        if (ta != tb) return ta > tb;
        if (a.plan.pair != b.plan.pair) return a.plan.pair > b.plan.pair;
        return (long long)ta * a.plan.ktiles_per_split * a.plan.bn > (long long)tb * b.plan.ktiles_per_split * b.plan.bn;
    });
    MCL_TC(ctx, op, mcl::launch_tc_products(pr.data(), (int)pr.size(), ctx->err_word, ctx->max_smem, ctx->sm_count, ctx->stream, &_n));
    std::vector<const float*> part;
    std::vector<float*> out;
    std::vector<long long> elems;
    std::vector<int> splits;
    for (const mcl::TcProblem& q : pr) {
        if (q.plan.splits <= 1) continue;
        if (q.col_scale) {
            MCL_LAUNCH(ctx, op, reduce_of(q, ctx->stream));
            continue;
        }
        part.push_back(q.splitk_ws); out.push_back(q.c); elems.push_back((long long)q.M * q.N); splits.push_back(q.plan.splits);
    }
    if (!part.empty())
        MCL_TC(ctx, op, mcl::launch_splitk_reduce_group(part.data(), out.data(), elems.data(), splits.data(), (int)part.size(), ctx->sm_count, ctx->stream, &_n));
    return MCL_CUDA_OK;
}
// One product of a layer that the one-launch kernels can take: by them, unless the terms split once are faster and their workspace
// can be had (it cannot grow in a recording or under live batches, and these kernels need none)
bool layer_route(mcl_cuda_ctx* ctx, const char* op, const ProductLayer& l, size_t N, size_t K, size_t C) {
    if (!layer_wanted(ctx, l.Nt, l.I, l.O)) return false;
    if (!tc_wanted(ctx, l.Nt, N, K, l.y ? l.y : l.grad_x, l.y ? l.scale : nullptr) || mcl::layer_rows_pay(l.Nt, N, K, ctx->sm_count)) return true;
    size_t bytes = 0;
    void* wsp = nullptr;
    return products_chunk(ctx, op, &l, 1, C, nullptr, &bytes) != MCL_CUDA_OK || ws_reserve(ctx, bytes, &wsp) != MCL_CUDA_OK;
}
// Layers go together while their terms fit kChunkBytes.
constexpr size_t kChunkBytes = (size_t)6 << 30;
int products_group(mcl_cuda_ctx* ctx, const char* op, const ProductLayer* L, size_t n, size_t C) {
    std::vector<size_t> ends;
    size_t need = 0;
    for (size_t i = 0; i < n;) {
        size_t k = i, sum = 0;
        while (k < n && (k == i || sum + layer_term_bytes(L[k]) <= kChunkBytes)) sum += layer_term_bytes(L[k++]);
        size_t b = 0;
        MCL_TRY(products_chunk(ctx, op, L + i, k - i, C, nullptr, &b));
        if (b > need) need = b;
        ends.push_back(k);
        i = k;
    }
    void* wsp = nullptr;
    MCL_TRY(ws_reserve(ctx, need, &wsp));
    size_t i = 0;
    for (size_t e : ends) {
        MCL_TRY(products_chunk(ctx, op, L + i, e - i, C, static_cast<char*>(wsp), nullptr));
        i = e;
    }
    return MCL_CUDA_OK;
}

// The one node that the next launch of a recording will depend on, or null; *capture: id of the recording.
cudaGraphNode_t recorded_tail(mcl_cuda_ctx* ctx, unsigned long long* capture) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    cudaGraph_t graph = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    size_t n = 0;
    if (!ctx->recording || cudaStreamGetCaptureInfo_v2(ctx->stream, &st, capture, &graph, &deps, &n) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    return st == cudaStreamCaptureStatusActive && n == 1 ? deps[0] : nullptr;
}

// Puts `item` into the earliest open list with room, behind which nothing reads or writes what the item writes, or writes what it reads.
// False: there is none.  The list's nodes take it when the recording is complete.
bool join_gemvs(mcl_cuda_ctx* ctx, const mcl::GemvItem& item, int M, bool mma, bool tc) {
    GemvRecord& rec = ctx->gemvs;
    struct Range { uintptr_t begin, end; };
    const auto range = [](const void* p, size_t bytes) { const uintptr_t b = reinterpret_cast<uintptr_t>(p); return Range{b, b + bytes}; };
    const auto meet = [](Range a, Range b) { return a.begin < b.end && b.begin < a.end; };
    const auto out = [&](const mcl::GemvItem& i, int m) { return range(i.y, (size_t)m * i.out_features * 4); };
    const auto takes = [&](const mcl::GemvItem& i, int m, Range r) {
        return meet(range(i.x, (size_t)m * i.in_features * 4), r) || meet(range(i.packed2, (size_t)i.in_features / 4 * i.out_features), r) ||
               meet(range(i.scale, (size_t)i.out_features * 4), r);
    };
    const auto room = [&](GemvList& at) {
        if (at.M != M || at.items.size() >= mcl::kGemvListCap || !(at.tc ? tc : mma)) return false;
        at.items.push_back(item);
        const int n = (int)at.items.size();
        const bool fits = at.tc ? mcl::gemv_tc_workspace_bytes(at.items.data(), n, M, ctx->sm_count) <= at.ws_bytes
                                : mcl::gemv_mma_takes(at.items.data(), n, M, ctx->max_smem);
        at.items.pop_back();
        return fits;
    };
    GemvList* found = nullptr;
    size_t l = rec.lists.size();
    for (bool met = false; l-- > rec.open && !met;) {
        GemvList& at = rec.lists[l];
        for (const mcl::GemvItem& i : at.items)
            met = met || meet(out(i, at.M), out(item, M)) || takes(i, at.M, out(item, M)) || takes(item, M, out(i, at.M));
        if (!met && room(at)) found = &at;
    }
    if (found) found->items.push_back(item);
    return found != nullptr;
}

// The recording is complete: the nodes take their lists.  A list of gemv_mma.cu that has become long enough for gemv_tc.cu goes there,
// where its context's workspace is large enough or can grow (the capture has ended; what the graph already holds of the old one is
// kept).  Its node, on which whatever was recorded behind it depends, becomes the contraction; the digits get a node in front of it.
cudaError_t lay_out_gemvs(mcl_cuda_ctx* ctx, cudaGraph_t graph) {
    std::vector<GemvList> lists;
    lists.swap(ctx->gemvs.lists);
    ctx->gemvs = GemvRecord();
    std::vector<size_t> need(lists.size(), 0);         // 0: stays where it is
    std::map<mcl_cuda_ctx*, size_t> most;
    for (size_t l = 0; l < lists.size(); ++l) {
        const GemvList& at = lists[l];
        const mcl::GemvItem* items = at.items.data();
        const int n = (int)at.items.size();
        if (at.ctx != ctx) {
            std::lock_guard<std::mutex> lock(g_ctx_mutex);
            if (!g_live_ctx.count(at.ctx)) continue;
        }
        bool go = !at.tc && mcl::gemv_tc_pays(items, n, at.M, ctx->sm_count);
        for (const mcl::GemvItem& i : at.items) go = go && mcl::gemv_tc_supported(at.M, i.in_features, i.packed2);
        const size_t bytes = go ? mcl::gemv_tc_workspace_bytes(items, n, at.M, ctx->sm_count) : ~size_t(0);
        if (bytes == ~size_t(0)) continue;
        need[l] = bytes;
        most[at.ctx] = std::max(most[at.ctx], bytes);
    }
    for (const auto& m : most) {
        const std::string error = m.first->error;
        if (m.second > m.first->ws_bytes && ws_grow(m.first, m.second) != MCL_CUDA_OK) m.first->error = error;
        if (m.first != ctx) m.first->ws_held = true;
    }
    for (size_t l = 0; l < lists.size(); ++l) {
        const GemvList& at = lists[l];
        const mcl::GemvItem* items = at.items.data();
        const int n = (int)at.items.size();
        const bool go = need[l] > 0 && need[l] <= at.ctx->ws_bytes;
        if (!go && n == 1) continue;
        const cudaGraphNode_t front[2] = {nullptr, at.node[0]};
        const cudaError_t e = go || at.tc ? mcl::launch_ternary_gemv_tc(items, n, at.M, go ? at.ctx->ws : at.ws, 3, false, go ? front : at.node, graph, ctx->err_word,
                                                                        ctx->sm_count, ctx->max_smem, ctx->stream)
                                          : mcl::launch_ternary_gemv_mma(items, n, at.M, false, at.node, ctx->sm_count, ctx->max_smem, ctx->stream);
        if (e != cudaSuccess) return e;
        if (go) ++ctx->launches;
    }
    return cudaSuccess;
}

}  // namespace

extern "C" {

int mcl_cuda_device_count(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) { cudaGetLastError(); return 0; }
    return n;
}
int mcl_cuda_create(int device, mcl_cuda_ctx** out_ctx) { return create_impl(device, nullptr, true, out_ctx); }
int mcl_cuda_create_on_stream(int device, void* cuda_stream, mcl_cuda_ctx** out_ctx) {
    return create_impl(device, static_cast<cudaStream_t>(cuda_stream), false, out_ctx);
}
void mcl_cuda_destroy(mcl_cuda_ctx* ctx) {
    if (!ctx) return;
    {
        std::lock_guard<std::mutex> lock(g_ctx_mutex);
        g_live_ctx.erase(ctx);
    }
    DeviceGuard guard(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    if (ctx->ws) cudaFree(ctx->ws);
    for (void* w : ctx->ws_kept) cudaFree(w);
    if (ctx->err_word) cudaFree(ctx->err_word);
    if (ctx->ev_fork) cudaEventDestroy(ctx->ev_fork);
    if (ctx->ev_join) cudaEventDestroy(ctx->ev_join);
    if (ctx->own_stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
}
const char* mcl_cuda_last_error(mcl_cuda_ctx* ctx) { return ctx ? ctx->error.c_str() : g_error.c_str(); }
const char* mcl_cuda_device_name(mcl_cuda_ctx* ctx) { return ctx ? ctx->name.c_str() : ""; }
int mcl_cuda_sm_count(mcl_cuda_ctx* ctx) { return ctx ? ctx->sm_count : 0; }
size_t mcl_cuda_device_memory_bytes(mcl_cuda_ctx* ctx) { return ctx ? ctx->device_mem : 0; }
uint64_t mcl_cuda_launch_count(mcl_cuda_ctx* ctx) { return ctx ? ctx->launches : 0; }
size_t mcl_cuda_workspace_bytes(mcl_cuda_ctx* ctx) { return ctx ? ctx->ws_bytes + ctx->ws_kept_bytes : 0; }

int mcl_cuda_batch_begin(mcl_cuda_ctx* ctx) {
    MCL_NEED_CTX(ctx);
    if (ctx->recording) return fail(ctx, MCL_CUDA_EINVAL, "batch_begin: already recording");
    if (ctx->stream == nullptr || ctx->stream == cudaStreamLegacy || ctx->stream == cudaStreamPerThread)
        return fail(ctx, MCL_CUDA_EUNSUPPORTED, "batch_begin: the context runs on a default stream, which cannot be recorded; "
                                              "create the context with its own stream");
    DeviceGuard guard(ctx->device);
    cudaError_t e = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return fail_cuda(ctx, "batch_begin", e);
    ctx->recording = true;
    ctx->gemvs = GemvRecord();
    ctx->recorded_launches = ctx->launches;
    return MCL_CUDA_OK;
}
int mcl_cuda_batch_end(mcl_cuda_ctx* ctx, mcl_cuda_batch** out_batch) {
    MCL_NEED_CTX(ctx);
    if (!out_batch) return fail(ctx, MCL_CUDA_EINVAL, "batch_end: out_batch is NULL");
    *out_batch = nullptr;
    if (!ctx->recording) return fail(ctx, MCL_CUDA_EINVAL, "batch_end without batch_begin");
    DeviceGuard guard(ctx->device);
    ctx->recording = false;
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamEndCapture(ctx->stream, &graph);
    if (e != cudaSuccess || graph == nullptr) { cudaGetLastError(); ctx->ws_recorded = false; return fail_cuda(ctx, "batch_end", e); }
    e = lay_out_gemvs(ctx, graph);
    ctx->ws_recorded = false;                   // from here on the batch counts
    if (e != cudaSuccess) { cudaGraphDestroy(graph); return fail_cuda(ctx, "batch_end (decode lists)", e); }
    mcl_cuda_batch* b = new (std::nothrow) mcl_cuda_batch();
    if (!b) { cudaGraphDestroy(graph); return fail(ctx, MCL_CUDA_ENOMEM, "out of host memory"); }
    b->graph = graph;
    b->kernels = ctx->launches - ctx->recorded_launches;
    ctx->launches = ctx->recorded_launches;     // recorded, not run
    e = cudaGraphInstantiate(&b->exec, graph, 0);
    if (e != cudaSuccess) { cudaGraphDestroy(graph); delete b; return fail_cuda(ctx, "batch_end (instantiate)", e); }
    b->ctx = ctx;
    ++ctx->live_batches;
    *out_batch = b;
    return MCL_CUDA_OK;
}
int mcl_cuda_batch_launch(mcl_cuda_ctx* ctx, mcl_cuda_batch* batch) {
    MCL_NEED_CTX(ctx);
    if (!batch || !batch->exec) return fail(ctx, MCL_CUDA_EINVAL, "batch_launch: batch is NULL");
    MCL_NOT_RECORDING(ctx, "batch_launch");
    DeviceGuard guard(ctx->device);
    cudaError_t e = cudaGraphLaunch(batch->exec, ctx->stream);
    if (e != cudaSuccess) return fail_cuda(ctx, "batch_launch", e);
    ctx->launches += batch->kernels;
    return MCL_CUDA_OK;
}
void mcl_cuda_batch_destroy(mcl_cuda_batch* batch) {
    if (!batch) return;
    {
        std::lock_guard<std::mutex> lock(g_ctx_mutex);
        if (batch->ctx && g_live_ctx.count(batch->ctx) && batch->ctx->live_batches > 0) --batch->ctx->live_batches;
    }
    if (batch->exec) cudaGraphExecDestroy(batch->exec);
    if (batch->graph) cudaGraphDestroy(batch->graph);
    delete batch;
}

int mcl_cuda_lane_fork(mcl_cuda_ctx* ctx, mcl_cuda_ctx* lane) {
    MCL_NEED_CTX(ctx);
    if (!lane || lane == ctx) return fail(ctx, MCL_CUDA_EINVAL, "lane_fork: lane must be another context");
    if (lane->device != ctx->device) return fail(ctx, MCL_CUDA_EINVAL, "lane_fork: lane is on another device");
    DeviceGuard guard(ctx->device);
    cudaError_t e = cudaEventRecord(lane->ev_fork, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(lane->stream, lane->ev_fork, 0);
    if (e != cudaSuccess) return fail_cuda(ctx, "lane_fork", e);
    ctx->gemvs.close();                        // what the lane does from here on stands behind what was recorded
    lane->gemvs = GemvRecord();
    lane->recording = lane->is_lane = ctx->recording;
    lane->lane_mark = lane->launches;
    return MCL_CUDA_OK;
}
int mcl_cuda_lane_join(mcl_cuda_ctx* ctx, mcl_cuda_ctx* lane) {
    MCL_NEED_CTX(ctx);
    if (!lane || lane == ctx) return fail(ctx, MCL_CUDA_EINVAL, "lane_join: lane must be another context");
    DeviceGuard guard(ctx->device);
    cudaError_t e = cudaEventRecord(lane->ev_join, lane->stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(ctx->stream, lane->ev_join, 0);
    if (e != cudaSuccess) return fail_cuda(ctx, "lane_join", e);
    ctx->gemvs.lists.insert(ctx->gemvs.lists.end(), lane->gemvs.lists.begin(), lane->gemvs.lists.end());
    ctx->gemvs.close();
    lane->gemvs = GemvRecord();
    lane->recording = lane->is_lane = false;
    ctx->launches += lane->launches - lane->lane_mark;    // account the lane's kernels to the owner
    lane->launches = lane->lane_mark;
    return MCL_CUDA_OK;
}

int mcl_cuda_finish(mcl_cuda_ctx* ctx) {
    MCL_NEED_CTX(ctx);
    MCL_NOT_RECORDING(ctx, "finish");
    DeviceGuard guard(ctx->device);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return fail_cuda(ctx, "finish", e);
    return check_device_error(ctx);
}

int mcl_cuda_set_seed_offset(mcl_cuda_ctx* ctx, const uint32_t* device_word) {
    MCL_NEED_CTX(ctx);
    if (device_word && reinterpret_cast<uintptr_t>(device_word) % 4 != 0)
        return fail(ctx, MCL_CUDA_EINVAL, "set_seed_offset: pointer must be 4-byte aligned");
    ctx->seed_offset = device_word;
    return MCL_CUDA_OK;
}

int mcl_cuda_set_gemm_mode(mcl_cuda_ctx* ctx, int mode, int act_terms, int grad_terms) {
    MCL_NEED_CTX(ctx);
    if (mode != MCL_CUDA_GEMM_AUTO && mode != MCL_CUDA_GEMM_EXACT && mode != MCL_CUDA_GEMM_TENSOR)
        return fail(ctx, MCL_CUDA_EINVAL, "set_gemm_mode: unknown mode");
    if (act_terms != 2 && act_terms != 3) return fail(ctx, MCL_CUDA_EINVAL, "set_gemm_mode: act_terms must be 2 or 3");
    if (grad_terms != 3 && grad_terms != 6) return fail(ctx, MCL_CUDA_EINVAL, "set_gemm_mode: grad_terms must be 3 or 6");
    ctx->gemm_mode = mode;                 // every setting runs the same two fp16 terms
    return MCL_CUDA_OK;
}
int mcl_cuda_alloc(mcl_cuda_ctx* ctx, size_t bytes, void** out_dptr) {
    MCL_NEED_CTX(ctx);
    MCL_NOT_RECORDING(ctx, "alloc");
    if (!out_dptr) return fail(ctx, MCL_CUDA_EINVAL, "alloc: out_dptr is NULL");
    *out_dptr = nullptr;
    if (bytes == 0) return fail(ctx, MCL_CUDA_EINVAL, "alloc: zero-size buffer");
    DeviceGuard guard(ctx->device);
    // Stream-ordered allocation from the device's default pool: a training step allocates and drops
    // hundreds of intermediate tensors, and the pool serves them without a device synchronisation.
    cudaError_t e = cudaMallocAsync(out_dptr, bytes, ctx->stream);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(ctx, MCL_CUDA_ENOMEM, "alloc of " + std::to_string(bytes) + " bytes failed: " + cudaGetErrorString(e));
    }
    return MCL_CUDA_OK;
}
int mcl_cuda_free(mcl_cuda_ctx* ctx, void* dptr) {
    MCL_NEED_CTX(ctx);
    MCL_NOT_RECORDING(ctx, "free");
    if (!dptr) return MCL_CUDA_OK;
    DeviceGuard guard(ctx->device);
    // Work that still uses the buffer may be queued: the free is ordered after it on the context's
    // stream, which keeps the reference's "free while pending is safe" behaviour without a wait.
    cudaError_t e = cudaFreeAsync(dptr, ctx->stream);
    if (e != cudaSuccess) return fail_cuda(ctx, "free", e);
    return MCL_CUDA_OK;
}
int mcl_cuda_upload(mcl_cuda_ctx* ctx, void* dst, const void* src_host, size_t bytes) {
    MCL_NEED_CTX(ctx);
    MCL_NOT_RECORDING(ctx, "upload");
    if (bytes == 0) return MCL_CUDA_OK;
    if (!dst || !src_host) return fail(ctx, MCL_CUDA_EINVAL, "upload: NULL pointer");
    DeviceGuard guard(ctx->device);
    cudaError_t e = cudaMemcpyAsync(dst, src_host, bytes, cudaMemcpyHostToDevice, ctx->stream);
    if (e != cudaSuccess) return fail_cuda(ctx, "upload", e);
    // pageable sources are staged before the call returns; pinned ones are read later, so
    // wait to give upload the reference's synchronous semantics (src/tensor/tensor.cpp:311-348)
    e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return fail_cuda(ctx, "upload", e);
    return MCL_CUDA_OK;
}
int mcl_cuda_download(mcl_cuda_ctx* ctx, void* dst_host, const void* src, size_t bytes) {
    MCL_NEED_CTX(ctx);
    MCL_NOT_RECORDING(ctx, "download");
    if (bytes == 0) return MCL_CUDA_OK;
    if (!dst_host || !src) return fail(ctx, MCL_CUDA_EINVAL, "download: NULL pointer");
    DeviceGuard guard(ctx->device);
    cudaError_t e = cudaMemcpyAsync(dst_host, src, bytes, cudaMemcpyDeviceToHost, ctx->stream);
    if (e != cudaSuccess) return fail_cuda(ctx, "download", e);
    e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return fail_cuda(ctx, "download", e);
    return MCL_CUDA_OK;
}

int mcl_cuda_counter_decode_weight(mcl_cuda_ctx* ctx, const uint8_t* state, const float* scale,
                                   float* weight, size_t in_features, size_t out_features, size_t C) {
    MCL_NEED_CTX(ctx);
    const char* op = "counter decode_weight";
    MCL_TRY(check_counter_dims(ctx, op, C, in_features, out_features));
    MCL_TRY(check_ptr(ctx, op, "state", state, 1));
    MCL_TRY(check_ptr(ctx, op, "scale", scale, 4));
    MCL_TRY(check_ptr(ctx, op, "weight", weight, 16));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_decode_weight(state, scale, weight, (int)C, (int)in_features,
                                                  (int)out_features, ctx->sm_count, ctx->stream));
    return MCL_CUDA_OK;
}

int mcl_cuda_counter_pack2(mcl_cuda_ctx* ctx, const uint8_t* state, uint32_t* packed2,
                           size_t in_features, size_t out_features, size_t C) {
    MCL_NEED_CTX(ctx);
    const char* op = "counter pack2";
    MCL_TRY(check_counter_dims(ctx, op, C, in_features, out_features));
    if (in_features % 16 != 0) return fail(ctx, MCL_CUDA_EINVAL, "counter pack2 requires in_features % 16 == 0");
    MCL_TRY(check_ptr(ctx, op, "state", state, 4));
    MCL_TRY(check_ptr(ctx, op, "packed2", packed2, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_pack2(state, packed2, (int)C, (int)in_features, (int)out_features,
                                          ctx->sm_count, ctx->stream));
    return MCL_CUDA_OK;
}

int mcl_cuda_counter_forward(mcl_cuda_ctx* ctx, const float* x, const uint8_t* state,
                             const float* scale, float* y, size_t batch, size_t in_features,
                             size_t out_features, size_t C) {
    MCL_NEED_CTX(ctx);
    const char* op = "counter forward";
    MCL_TRY(check_counter_dims(ctx, op, C, in_features, out_features));
    if (batch == 0 || batch > 0x7fffffffull) return fail(ctx, MCL_CUDA_EINVAL, "counter forward requires 0 < batch < 2^31");
    MCL_TRY(check_ptr(ctx, op, "x", x, 4));
    MCL_TRY(check_ptr(ctx, op, "state", state, 1));
    MCL_TRY(check_ptr(ctx, op, "scale", scale, 4));
    MCL_TRY(check_ptr(ctx, op, "y", y, 4));
    DeviceGuard guard(ctx->device);
    const ProductLayer l = {x, nullptr, state, nullptr, scale, y, nullptr, nullptr, in_features, out_features, batch};
    if (layer_route(ctx, op, l, out_features, in_features, C)) {
        MCL_LAUNCH(ctx, op, mcl::launch_layer_rows(0, x, state, scale, y, (int)batch, (int)in_features, (int)out_features, (int)C,
                                                   ctx->err_word, ctx->max_smem, ctx->sm_count, ctx->stream));
        return MCL_CUDA_OK;
    }
    if (tc_wanted(ctx, batch, out_features, in_features, y, scale)) return products_group(ctx, op, &l, 1, C);
    MCL_LAUNCH(ctx, op, mcl::launch_simt_counter_forward(x, state, scale, y, (int)batch, (int)in_features,
                                                         (int)out_features, (int)C, ctx->stream));
    return MCL_CUDA_OK;
}

int mcl_cuda_counter_backward_input(mcl_cuda_ctx* ctx, const uint8_t* state, const float* scale,
                                    const float* grad_out, float* grad_x, size_t batch,
                                    size_t in_features, size_t out_features, size_t C) {
    MCL_NEED_CTX(ctx);
    const char* op = "counter backward_input";
    MCL_TRY(check_counter_dims(ctx, op, C, in_features, out_features));
    if (batch == 0 || batch > 0x7fffffffull) return fail(ctx, MCL_CUDA_EINVAL, "counter backward_input requires 0 < batch < 2^31");
    MCL_TRY(check_ptr(ctx, op, "state", state, 1));
    MCL_TRY(check_ptr(ctx, op, "scale", scale, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_out", grad_out, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_x", grad_x, 4));
    DeviceGuard guard(ctx->device);
    const ProductLayer l = {nullptr, grad_out, state, nullptr, scale, nullptr, grad_x, nullptr, in_features, out_features, batch};
    if (layer_route(ctx, op, l, in_features, out_features, C)) {
        MCL_LAUNCH(ctx, op, mcl::launch_layer_rows(1, grad_out, state, scale, grad_x, (int)batch, (int)in_features, (int)out_features, (int)C,
                                                   ctx->err_word, ctx->max_smem, ctx->sm_count, ctx->stream));
        return MCL_CUDA_OK;
    }
    if (tc_wanted(ctx, batch, in_features, out_features, grad_x)) return products_group(ctx, op, &l, 1, C);
    MCL_LAUNCH(ctx, op, mcl::launch_simt_counter_backward_input(state, scale, grad_out, grad_x, (int)batch,
                                                                (int)in_features, (int)out_features,
                                                                (int)C, ctx->stream));
    return MCL_CUDA_OK;
}

int mcl_cuda_counter_update_dense(mcl_cuda_ctx* ctx, uint8_t* state, float* scale, float* v,
                                  const float* grad_w, uint32_t* packed2_out, size_t C,
                                  size_t in_features, size_t rows, size_t row_offset, float lr,
                                  float lr_scale, float rms_beta, float rms_eps, uint32_t seed) {
    MCL_NEED_CTX(ctx);
    const char* op = "counter update";
    MCL_TRY(check_counter_dims(ctx, op, C, in_features, rows));
    MCL_TRY(check_hypers(ctx, op, lr, lr_scale, rms_beta, rms_eps));
    if ((row_offset + rows) * in_features > 0xffffffffull)
        return fail(ctx, MCL_CUDA_EINVAL, "counter update: (row_offset + rows) * in_features exceeds 32-bit element indexing");
    MCL_TRY(check_ptr(ctx, op, "state", state, 1));
    MCL_TRY(check_ptr(ctx, op, "scale", scale, 4));
    MCL_TRY(check_ptr(ctx, op, "v", v, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_w", grad_w, 16));
    if (packed2_out) {
        if (in_features % 16 != 0) return fail(ctx, MCL_CUDA_EINVAL, "counter update: packed2 output requires in_features % 16 == 0");
        MCL_TRY(check_ptr(ctx, op, "packed2_out", packed2_out, 4));
    }
    DeviceGuard guard(ctx->device);
    cudaError_t e = mcl::launch_counter_update_dense(state, scale, v, grad_w, packed2_out, (int)C,
                                                     (int)in_features, (int)rows, (int)row_offset, lr,
                                                     lr_scale, rms_beta, rms_eps, seed, ctx->seed_offset, ctx->err_word,
                                                     ctx->sm_count, ctx->max_smem, ctx->stream);
    if (e == cudaErrorInvalidConfiguration)
        return fail(ctx, MCL_CUDA_EUNSUPPORTED, "counter update: in_features too large for one row in shared memory");
    if (e != cudaSuccess) return fail_cuda(ctx, op, e);
    ++ctx->launches;
    return MCL_CUDA_OK;
}

int mcl_cuda_counter_update_fused(mcl_cuda_ctx* ctx, uint8_t* state, float* scale, float* v,
                                  const float* grad_out, const float* x, float* scale_new_scratch,
                                  float* denom_scratch, uint32_t* packed2_out, size_t C,
                                  size_t in_features, size_t out_features, size_t batch, float lr,
                                  float lr_scale, float rms_beta, float rms_eps, uint32_t seed) {
    (void)scale_new_scratch; (void)denom_scratch;
    MCL_NEED_CTX(ctx);
    const char* op = "counter update";
    MCL_TRY(check_counter_dims(ctx, op, C, in_features, out_features));
    if (batch == 0 || batch > 0x7fffffffull) return fail(ctx, MCL_CUDA_EINVAL, "counter update requires 0 < batch < 2^31");
    MCL_TRY(check_hypers(ctx, op, lr, lr_scale, rms_beta, rms_eps));
    MCL_TRY(check_ptr(ctx, op, "grad_out", grad_out, 4));
    MCL_TRY(check_ptr(ctx, op, "x", x, 4));
    MCL_TRY(check_ptr(ctx, op, "state", state, 1));
    if (packed2_out && in_features % 16 != 0)
        return fail(ctx, MCL_CUDA_EINVAL, "counter update: packed2 output requires in_features % 16 == 0");
    // Row tile of grad_w: 1/8 of the dense [out,in] gradient, raised to 4 MiB where that is still under 1/5 of the
    // dense gradient (fewer launches for mid-sized layers) and capped at 32 MiB; at least one row; rounded to a multiple
    // of 128 rows when that fits.  The dense gradient is never materialised: the reference's memory-truth gate
    // (tests/test_memory_truth_gate.cpp:30-126) allows the update less than a quarter of a dense weight, and that
    // holds for every layer of more than four rows here.
    const size_t row_b = in_features * sizeof(float);
    const size_t dense = out_features * row_b;
    size_t budget = dense / 8;
    if (budget < (4u << 20)) budget = (4u << 20) < dense / 5 ? (4u << 20) : dense / 5;
    if (budget > (32u << 20)) budget = 32u << 20;
    size_t tile_rows = budget / row_b;
    if (tile_rows < 1) tile_rows = 1;
    if (tile_rows > 128) tile_rows &= ~size_t(127);
    if (tile_rows > out_features) tile_rows = out_features;
    DeviceGuard guard(ctx->device);
    const size_t state_row = in_features / 4 * 3;
    const bool tc = tc_wanted(ctx, tile_rows, in_features, batch) && tile_rows >= 64;
    if (tc) tile_rows &= ~size_t(7);      // a tile starts at a 16-byte aligned column of the terms of grad_out
    mcl::TcPlan plan = {};
    Carver cv;
    const size_t o_gw = cv.reserve(tile_rows * row_b);
    size_t o_k = 0;
    TermBuf gb, xb;
    if (tc) {
        plan = dense_plan(ctx, tile_rows, in_features, batch);
        gb = carve_terms(&cv, batch, out_features, true, false, kByPartner);      // activation-sized, not weight-sized
        xb = carve_terms(&cv, batch, in_features, true, false, kByRow);
        o_k = cv.reserve(plan.workspace_bytes);
    }
    void* wsp = nullptr;
    const bool fused = mcl::layer_kernels_fit(batch, in_features, out_features) && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    // few multiply-adds without tensor cores: one launch, the same sums
    const bool small = fused && !layer_wanted(ctx, batch, in_features, out_features) && (double)batch * (double)in_features * (double)out_features < (double)(1u << 22);
    if (small || (fused && layer_wanted(ctx, batch, in_features, out_features) &&
        (!tc || mcl::layer_update_pays(batch, in_features, out_features, (out_features + tile_rows - 1) / tile_rows, ctx->sm_count) ||
         ws_reserve(ctx, cv.off, &wsp) != MCL_CUDA_OK))) {
        MCL_TRY(check_ptr(ctx, op, "scale", scale, 4));
        MCL_TRY(check_ptr(ctx, op, "v", v, 4));
        if (packed2_out) MCL_TRY(check_ptr(ctx, op, "packed2_out", packed2_out, 4));
        mcl::UpdateDesc d;
        d.state = state; d.scale = scale; d.v = v; d.grad_w = nullptr; d.packed2 = packed2_out;
        d.in_features = (int)in_features; d.rows = (int)out_features; d.row_offset = 0;
        if (small) {
            MCL_LAUNCH(ctx, op, mcl::launch_exact_update(d, grad_out, x, (int)batch, (int)C, lr, lr_scale, rms_beta, rms_eps, seed, ctx->seed_offset,
                                                         ctx->sm_count, ctx->max_smem, ctx->stream));
            return MCL_CUDA_OK;
        }
        MCL_LAUNCH(ctx, op, mcl::launch_layer_update(d, grad_out, x, (int)batch, (int)C, lr, lr_scale, rms_beta, rms_eps, seed, ctx->seed_offset,
                                                     ctx->err_word, ctx->sm_count, ctx->max_smem, ctx->stream));
        return MCL_CUDA_OK;
    }
    MCL_TRY(ws_reserve(ctx, cv.off, &wsp));
    char* w = static_cast<char*>(wsp);
    float* gw = reinterpret_cast<float*>(w + o_gw);
    if (tc) {
        const mcl::SplitDesc sd[2] = {split_of(w, xb, x, nullptr, true, nullptr), split_of(w, gb, grad_out, nullptr, true, &xb)};
        MCL_TRY(split_tensors(ctx, op, sd, 2));
    }
    for (size_t r0 = 0; r0 < out_features; r0 += tile_rows) {
        const size_t nr = (out_features - r0 < tile_rows) ? out_features - r0 : tile_rows;
        if (tc) {
            mcl::TcOperand a = terms_of(w, gb, false, true);
            a.ptr = static_cast<const char*>(a.ptr) + r0 * 2;
            a.cols = (int)nr;
            MCL_TRY(tc_product(ctx, op, tc_problem(a, terms_of(w, xb, false, true), gw, nr, in_features, batch, plan, nullptr, w + o_k)));
        } else {
            MCL_LAUNCH(ctx, "counter update (grad_w tile)",
                       mcl::launch_simt_grad_w(grad_out, x, gw, (int)batch, (int)in_features,
                                               (int)out_features, (int)r0, (int)nr, ctx->stream));
        }
        int rc = mcl_cuda_counter_update_dense(ctx, state + r0 * state_row, scale + r0, v + r0, gw,
                                               packed2_out ? packed2_out + r0 * (in_features / 16) : nullptr,
                                               C, in_features, nr, r0, lr, lr_scale, rms_beta, rms_eps, seed);
        if (rc != MCL_CUDA_OK) return rc;
    }
    return MCL_CUDA_OK;
}

static int linear_products(mcl_cuda_ctx* ctx, const char* op, const float* x, const float* grad_out,
                           const uint8_t* state, const uint32_t* packed2, const float* scale, float* y,
                           float* grad_x, float* grad_w, size_t C, size_t I, size_t O, size_t Nt) {
    const bool tc = tc_wanted(ctx, Nt, O, I, y, scale) && tc_wanted(ctx, Nt, I, O, grad_x) && tc_wanted(ctx, O, I, Nt, grad_w);
    if (!tc) {
        if (state) {
            if (y) MCL_TRY(mcl_cuda_counter_forward(ctx, x, state, scale, y, Nt, I, O, C));
            if (grad_x) MCL_TRY(mcl_cuda_counter_backward_input(ctx, state, scale, grad_out, grad_x, Nt, I, O, C));
        } else {
            if (y) MCL_LAUNCH(ctx, op, mcl::launch_simt_ternary_forward(x, packed2, scale, y, (int)Nt, (int)I, (int)O, ctx->stream));
            if (grad_x) MCL_LAUNCH(ctx, op, mcl::launch_simt_ternary_backward_input(packed2, scale, grad_out, grad_x, (int)Nt,
                                                                                 (int)I, (int)O, ctx->stream));
        }
        if (grad_w) MCL_TRY(mcl_cuda_matmul_f32(ctx, grad_out, x, grad_w, O, Nt, I, 1, 0));
        return MCL_CUDA_OK;
    }
    const ProductLayer l = {x, grad_out, state, packed2, scale, y, grad_x, grad_w, I, O, Nt};
    return products_group(ctx, op, &l, 1, C);
}

int mcl_cuda_counter_linear_step(mcl_cuda_ctx* ctx, const float* x, const float* grad_out,
                                 uint8_t* state, float* scale, float* v, float* y, float* grad_x,
                                 float* grad_w, uint32_t* packed2_out, size_t C, size_t in_features,
                                 size_t out_features, size_t batch, size_t update_rows,
                                 size_t row_offset, float lr, float lr_scale, float rms_beta,
                                 float rms_eps, uint32_t seed) {
    MCL_NEED_CTX(ctx);
    const char* op = "counter linear step";
    MCL_TRY(check_counter_dims(ctx, op, C, in_features, out_features));
    if (batch == 0 || batch > 0x7fffffffull) return fail(ctx, MCL_CUDA_EINVAL, "counter linear step requires 0 < batch < 2^31");
    MCL_TRY(check_hypers(ctx, op, lr, lr_scale, rms_beta, rms_eps));
    MCL_TRY(check_ptr(ctx, op, "x", x, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_out", grad_out, 4));
    MCL_TRY(check_ptr(ctx, op, "state", state, 1));
    MCL_TRY(check_ptr(ctx, op, "scale", scale, 4));
    MCL_TRY(check_ptr(ctx, op, "v", v, 4));
    if (grad_w) MCL_TRY(check_ptr(ctx, op, "grad_w", grad_w, 16));
    else if (update_rows != 0) return fail(ctx, MCL_CUDA_EINVAL, "counter linear step: an update needs grad_w");
    if (row_offset + update_rows > out_features)
        return fail(ctx, MCL_CUDA_EINVAL, "counter linear step: update rows exceed out_features");
    const size_t state_row = in_features / 4 * 3;
    const size_t I = in_features;
    DeviceGuard guard(ctx->device);
    MCL_TRY(linear_products(ctx, op, x, grad_out, state, nullptr, scale, y, grad_x, grad_w, C, in_features,
                            out_features, batch));
    if (update_rows > 0)
        return mcl_cuda_counter_update_dense(ctx, state + row_offset * state_row, scale + row_offset, v + row_offset,
                                             grad_w + row_offset * I,
                                             packed2_out ? packed2_out + row_offset * (I / 16) : nullptr, C, I,
                                             update_rows, row_offset, lr, lr_scale, rms_beta, rms_eps, seed);
    return MCL_CUDA_OK;
}

int mcl_cuda_counter_linear_step_many(mcl_cuda_ctx* ctx, const mcl_cuda_linear_desc* layers, size_t n_layers,
                                      size_t C, float lr, float lr_scale, float rms_beta, float rms_eps,
                                      uint32_t seed) {
    MCL_NEED_CTX(ctx);
    const char* op = "counter linear step (many)";
    if (!layers || n_layers == 0) return fail(ctx, MCL_CUDA_EINVAL, "counter linear step (many): no layers");
    MCL_TRY(check_hypers(ctx, op, lr, lr_scale, rms_beta, rms_eps));
    std::vector<size_t> grouped, single;
    for (size_t i = 0; i < n_layers; ++i) {
        const mcl_cuda_linear_desc& L = layers[i];
        MCL_TRY(check_counter_dims(ctx, op, C, L.in_features, L.out_features));
        if (L.batch == 0 || L.batch > 0x7fffffffull) return fail(ctx, MCL_CUDA_EINVAL, "counter linear step (many) requires 0 < batch < 2^31");
        MCL_TRY(check_ptr(ctx, op, "x", L.x, 4));
        MCL_TRY(check_ptr(ctx, op, "grad_out", L.grad_out, 4));
        MCL_TRY(check_ptr(ctx, op, "scale", L.scale, 4));
        if (L.grad_w) MCL_TRY(check_ptr(ctx, op, "grad_w", L.grad_w, 16));
        else if (L.update_rows != 0) return fail(ctx, MCL_CUDA_EINVAL, "counter linear step (many): an update needs grad_w");
        if (!L.grad_w && !L.y && !L.grad_x) return fail(ctx, MCL_CUDA_EINVAL, "counter linear step (many): a layer asks for no product");
        if (L.state != nullptr) {
            MCL_TRY(check_ptr(ctx, op, "v", L.v, 4));
        } else {
            MCL_TRY(check_ptr(ctx, op, "packed2_in", L.packed2_in, 4));
            if (L.update_rows != 0)
                return fail(ctx, MCL_CUDA_EINVAL, "counter linear step (many): a layer given by its 2-bit words cannot be updated");
            if (L.in_features % 16 != 0)
                return fail(ctx, MCL_CUDA_EINVAL, "counter linear step (many): 2-bit words require in_features % 16 == 0");
        }
        if (L.row_offset + L.update_rows > L.out_features)
            return fail(ctx, MCL_CUDA_EINVAL, "counter linear step (many): update rows exceed out_features");
        if (tc_wanted(ctx, L.batch, L.out_features, L.in_features, L.y, L.scale) && tc_wanted(ctx, L.batch, L.in_features, L.out_features, L.grad_x) &&
            tc_wanted(ctx, L.out_features, L.in_features, L.batch, L.grad_w))
            grouped.push_back(i);
        else
            single.push_back(i);
    }
    DeviceGuard guard(ctx->device);
    for (size_t i : single) {
        const mcl_cuda_linear_desc& L = layers[i];
        if (L.state == nullptr) {
            MCL_TRY(mcl_cuda_ternary_linear_products(ctx, L.x, L.grad_out, L.packed2_in, L.scale, L.y, L.grad_x, L.grad_w,
                                                     L.in_features, L.out_features, L.batch));
            continue;
        }
        MCL_TRY(mcl_cuda_counter_linear_step(ctx, L.x, L.grad_out, L.state, L.scale, L.v, L.y, L.grad_x, L.grad_w, L.packed2_out,
                                             C, L.in_features, L.out_features, L.batch, L.update_rows, L.row_offset, lr,
                                             lr_scale, rms_beta, rms_eps, seed));
    }
    if (grouped.empty()) return MCL_CUDA_OK;
    const size_t ng = grouped.size();
    std::vector<ProductLayer> pl;
    for (size_t gi : grouped) {
        const mcl_cuda_linear_desc& L = layers[gi];
        const ProductLayer l = {L.x, L.grad_out, L.state, L.packed2_in, L.scale, L.y, L.grad_x, L.grad_w, L.in_features, L.out_features, L.batch};
        pl.push_back(l);
    }
    MCL_TRY(products_group(ctx, op, pl.data(), ng, C));
    // the updates of all layers
    {
        std::vector<mcl::UpdateDesc> ud;
        for (size_t gi = 0; gi < ng; ++gi) {
            const mcl_cuda_linear_desc& L = layers[grouped[gi]];
            if (L.update_rows == 0) continue;
            if ((L.row_offset + L.update_rows) * L.in_features > 0xffffffffull)
                return fail(ctx, MCL_CUDA_EINVAL, "counter update: (row_offset + rows) * in_features exceeds 32-bit element indexing");
            const size_t I = L.in_features, rb = I / 4 * 3;
            mcl::UpdateDesc u;
            u.state = L.state + L.row_offset * rb; u.scale = L.scale + L.row_offset; u.v = L.v + L.row_offset;
            u.grad_w = L.grad_w + L.row_offset * I;
            u.packed2 = L.packed2_out ? L.packed2_out + L.row_offset * (I / 16) : nullptr;
            u.in_features = (int)I; u.rows = (int)L.update_rows; u.row_offset = (int)L.row_offset;
            ud.push_back(u);
        }
        if (!ud.empty()) {
            int launches = 0;
            cudaError_t e = mcl::launch_counter_update_group(ud.data(), (int)ud.size(), (int)C, lr, lr_scale, rms_beta, rms_eps, seed,
                                                             ctx->seed_offset, ctx->err_word, ctx->sm_count, ctx->max_smem, ctx->stream, &launches);
            ctx->launches += launches;
            if (e == cudaErrorNotSupported) {
                for (const mcl::UpdateDesc& u : ud)
                    MCL_TRY(mcl_cuda_counter_update_dense(ctx, u.state, u.scale, u.v, u.grad_w, u.packed2, C, (size_t)u.in_features,
                                                          (size_t)u.rows, (size_t)u.row_offset, lr, lr_scale, rms_beta, rms_eps, seed));
            } else if (e != cudaSuccess) {
                return fail_cuda(ctx, op, e);
            }
        }
    }
    return MCL_CUDA_OK;
}

int mcl_cuda_counter_update_dense_many(mcl_cuda_ctx* ctx, const mcl_cuda_update_desc* layers, size_t n_layers,
                                       size_t C, float lr, float lr_scale, float rms_beta, float rms_eps,
                                       uint32_t seed) {
    MCL_NEED_CTX(ctx);
    const char* op = "counter update (many)";
    if (!layers || n_layers == 0) return fail(ctx, MCL_CUDA_EINVAL, "counter update (many): no layers");
    MCL_TRY(check_hypers(ctx, op, lr, lr_scale, rms_beta, rms_eps));
    std::vector<mcl::UpdateDesc> ud;
    for (size_t i = 0; i < n_layers; ++i) {
        const mcl_cuda_update_desc& L = layers[i];
        if (L.rows == 0) continue;
        MCL_TRY(check_counter_dims(ctx, op, C, L.in_features, L.rows));
        if ((L.row_offset + L.rows) * L.in_features > 0xffffffffull)
            return fail(ctx, MCL_CUDA_EINVAL, "counter update: (row_offset + rows) * in_features exceeds 32-bit element indexing");
        MCL_TRY(check_ptr(ctx, op, "state", L.state, 1));
        MCL_TRY(check_ptr(ctx, op, "scale", L.scale, 4));
        MCL_TRY(check_ptr(ctx, op, "v", L.v, 4));
        MCL_TRY(check_ptr(ctx, op, "grad_w", L.grad_w, 16));
        mcl::UpdateDesc u;
        u.state = L.state; u.scale = L.scale; u.v = L.v; u.grad_w = L.grad_w; u.packed2 = L.packed2_out;
        u.in_features = (int)L.in_features; u.rows = (int)L.rows; u.row_offset = (int)L.row_offset;
        ud.push_back(u);
    }
    if (ud.empty()) return MCL_CUDA_OK;
    DeviceGuard guard(ctx->device);
    int launches = 0;
    cudaError_t e = mcl::launch_counter_update_group(ud.data(), (int)ud.size(), (int)C, lr, lr_scale, rms_beta, rms_eps, seed,
                                                     ctx->seed_offset, ctx->err_word, ctx->sm_count, ctx->max_smem, ctx->stream, &launches);
    ctx->launches += launches;
    if (e == cudaErrorNotSupported) {
        for (const mcl::UpdateDesc& u : ud)
            MCL_TRY(mcl_cuda_counter_update_dense(ctx, u.state, u.scale, u.v, u.grad_w, u.packed2, C, (size_t)u.in_features,
                                                  (size_t)u.rows, (size_t)u.row_offset, lr, lr_scale, rms_beta, rms_eps, seed));
        return MCL_CUDA_OK;
    }
    if (e != cudaSuccess) return fail_cuda(ctx, op, e);
    return MCL_CUDA_OK;
}

int mcl_cuda_ternary_linear_products(mcl_cuda_ctx* ctx, const float* x, const float* grad_out,
                                     const uint32_t* packed2, const float* scale, float* y, float* grad_x,
                                     float* grad_w, size_t in_features, size_t out_features, size_t batch) {
    MCL_NEED_CTX(ctx);
    const char* op = "ternary linear products";
    if (in_features == 0 || out_features == 0 || batch == 0)
        return fail(ctx, MCL_CUDA_EINVAL, "ternary linear products requires non-zero dimensions");
    if (in_features % 16 != 0) return fail(ctx, MCL_CUDA_EINVAL, "ternary linear products requires in_features % 16 == 0");
    if (in_features > 0x7fffffffull || out_features > 0x7fffffffull || batch > 0x7fffffffull ||
        in_features * out_features > 0x7fffffffull)
        return fail(ctx, MCL_CUDA_EINVAL, "ternary linear products: dimension exceeds 32-bit indexing");
    MCL_TRY(check_ptr(ctx, op, "x", x, 4));
    MCL_TRY(check_ptr(ctx, op, "packed2", packed2, 4));
    MCL_TRY(check_ptr(ctx, op, "scale", scale, 4));
    if (grad_x || grad_w) MCL_TRY(check_ptr(ctx, op, "grad_out", grad_out, 4));
    if (grad_w) MCL_TRY(check_ptr(ctx, op, "grad_w", grad_w, 16));
    DeviceGuard guard(ctx->device);
    return linear_products(ctx, op, x, grad_out, nullptr, packed2, scale, y, grad_x, grad_w, 11, in_features,
                           out_features, batch);
}

int mcl_cuda_matmul_f32(mcl_cuda_ctx* ctx, const float* a, const float* b, float* c, size_t M,
                        size_t K, size_t N, int trans_a, int trans_b) {
    MCL_NEED_CTX(ctx);
    const char* op = "matmul_f32";
    if (M == 0 || N == 0 || K == 0) return fail(ctx, MCL_CUDA_EINVAL, "matmul_f32 requires non-zero dimensions");
    if (M > 0x7fffffffull || N > 0x7fffffffull || K > 0x7fffffffull)
        return fail(ctx, MCL_CUDA_EINVAL, "matmul_f32 dimension exceeds 2^31");
    MCL_TRY(check_ptr(ctx, op, "a", a, 4));
    MCL_TRY(check_ptr(ctx, op, "b", b, 4));
    MCL_TRY(check_ptr(ctx, op, "c", c, 4));
    DeviceGuard guard(ctx->device);
    if (tc_wanted(ctx, M, N, K, c)) {
        const mcl::TcPlan plan = dense_plan(ctx, M, N, K);
        Carver cv;
        // a stored [M,K] or (trans_a) [K,M], b stored [K,N] or (trans_b) [N,K]: split as stored, read in the needed orientation.  Rows
        // that are rows or columns of c are scaled by row; of two that are both contracted over, the larger is, and the
        // smaller completes it.
        const bool both = trans_a && !trans_b, a_rows = !trans_a || (both && M >= N), b_rows = trans_b || (both && M < N);
        const TermBuf ab = carve_terms(&cv, trans_a ? K : M, trans_a ? M : K, true, false, a_rows ? kByRow : kByPartner);
        const TermBuf bb = carve_terms(&cv, trans_b ? N : K, trans_b ? K : N, true, false, b_rows ? kByRow : kByPartner);
        const size_t o_k = cv.reserve(plan.workspace_bytes);
        void* wsp = nullptr;
        MCL_TRY(ws_reserve(ctx, cv.off, &wsp));
        char* w = static_cast<char*>(wsp);
        const mcl::SplitDesc sd[2] = {split_of(w, ab, a, nullptr, true, both && !a_rows ? &bb : nullptr), split_of(w, bb, b, nullptr, true, both && !b_rows ? &ab : nullptr)};
        MCL_TRY(split_tensors(ctx, op, sd, 2));
        return tc_product(ctx, op, tc_problem(terms_of(w, ab, false, trans_a != 0), terms_of(w, bb, false, trans_b == 0), c, M, N, K, plan, nullptr, w + o_k));
    }
    MCL_LAUNCH(ctx, op, mcl::launch_simt_matmul_f32(a, b, c, (int)M, (int)K, (int)N, trans_a, trans_b, ctx->stream));
    return MCL_CUDA_OK;
}

int mcl_cuda_eltwise_f32(mcl_cuda_ctx* ctx, int op, const float* a, const float* b, float* out, size_t elements,
                         float alpha) {
    MCL_NEED_CTX(ctx);
    const char* name = "eltwise_f32";
    if (op < 0 || op > MCL_CUDA_ELT_SGD) return fail(ctx, MCL_CUDA_EINVAL, "eltwise_f32: unknown op");
    if (elements == 0) return fail(ctx, MCL_CUDA_EINVAL, "eltwise_f32 requires non-zero elements");
    MCL_TRY(check_ptr(ctx, name, "out", out, 4));
    if (op != MCL_CUDA_ELT_ZERO) MCL_TRY(check_ptr(ctx, name, "a", a, 4));
    if (op <= MCL_CUDA_ELT_MUL || op == MCL_CUDA_ELT_SGD) MCL_TRY(check_ptr(ctx, name, "b", b, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, name, mcl::launch_eltwise_f32(op, a, b, out, elements, alpha, ctx->sm_count, ctx->stream));
    return MCL_CUDA_OK;
}

// ---- fp32 row ops of the block stack around the counter layers ----------------------------------------
namespace {
int check_rows(mcl_cuda_ctx* ctx, const char* op, size_t rows, size_t cols) {
    if (rows == 0 || cols == 0) return fail(ctx, MCL_CUDA_EINVAL, std::string(op) + " requires non-zero dimensions");
    if (cols > 0x7fffffffull || rows > 0xffffffffull) return fail(ctx, MCL_CUDA_EINVAL, std::string(op) + " dimension is too large");
    return MCL_CUDA_OK;
}
}  // namespace

int mcl_cuda_rmsnorm(mcl_cuda_ctx* ctx, const float* x, const float* weight, float* out, size_t rows, size_t cols,
                     float eps) {
    MCL_NEED_CTX(ctx);
    const char* op = "rmsnorm";
    MCL_TRY(check_rows(ctx, op, rows, cols));
    MCL_TRY(check_ptr(ctx, op, "x", x, 4));
    MCL_TRY(check_ptr(ctx, op, "weight", weight, 4));
    MCL_TRY(check_ptr(ctx, op, "out", out, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_rmsnorm(x, weight, out, rows, (int)cols, eps, ctx->sm_count, ctx->stream));
    return MCL_CUDA_OK;
}
int mcl_cuda_rmsnorm_backward_x(mcl_cuda_ctx* ctx, const float* x, const float* weight, const float* grad_out,
                                float* grad_x, size_t rows, size_t cols, float eps) {
    MCL_NEED_CTX(ctx);
    const char* op = "rmsnorm backward_x";
    MCL_TRY(check_rows(ctx, op, rows, cols));
    MCL_TRY(check_ptr(ctx, op, "x", x, 4));
    MCL_TRY(check_ptr(ctx, op, "weight", weight, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_out", grad_out, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_x", grad_x, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_rmsnorm_backward_x(x, weight, grad_out, grad_x, rows, (int)cols, eps, ctx->sm_count, ctx->stream));
    return MCL_CUDA_OK;
}
int mcl_cuda_rmsnorm_backward_weight(mcl_cuda_ctx* ctx, const float* x, const float* grad_out, float* row_inv_scratch,
                                     float* grad_weight, size_t rows, size_t cols, float eps) {
    MCL_NEED_CTX(ctx);
    const char* op = "rmsnorm backward_weight";
    MCL_TRY(check_rows(ctx, op, rows, cols));
    MCL_TRY(check_ptr(ctx, op, "x", x, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_out", grad_out, 4));
    MCL_TRY(check_ptr(ctx, op, "row_inv_scratch", row_inv_scratch, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_weight", grad_weight, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_rmsnorm_backward_weight(x, grad_out, row_inv_scratch, grad_weight, rows, (int)cols, eps, ctx->sm_count, ctx->stream));
    if (cols > 1024) ctx->launches += 1;     // a row pass and a column pass
    return MCL_CUDA_OK;
}
int mcl_cuda_mse_loss_partial(mcl_cuda_ctx* ctx, const float* pred, const float* target, float* partial, size_t n) {
    MCL_NEED_CTX(ctx);
    const char* op = "mse_loss_partial";
    if (n == 0 || n > 0x7fffffffull) return fail(ctx, MCL_CUDA_EINVAL, "mse_loss_partial needs 0 < n < 2^31");
    MCL_TRY(check_ptr(ctx, op, "pred", pred, 4));
    MCL_TRY(check_ptr(ctx, op, "target", target, 4));
    MCL_TRY(check_ptr(ctx, op, "partial", partial, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_mse_loss_partial(pred, target, partial, n, ctx->stream));
    return MCL_CUDA_OK;
}
int mcl_cuda_mean_reduce(mcl_cuda_ctx* ctx, const float* partial, float* out, size_t count, size_t denominator) {
    MCL_NEED_CTX(ctx);
    const char* op = "mean_reduce";
    if (count > 0x7fffffffull || denominator > 0x7fffffffull) return fail(ctx, MCL_CUDA_EINVAL, "mean_reduce counts exceed 2^31");
    MCL_TRY(check_ptr(ctx, op, "partial", partial, 4));
    MCL_TRY(check_ptr(ctx, op, "out", out, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_mean_reduce(partial, out, (int)count, (int)denominator, ctx->stream));
    return MCL_CUDA_OK;
}
int mcl_cuda_mse_backward(mcl_cuda_ctx* ctx, const float* pred, const float* target, const float* grad_out,
                          float* grad_pred, size_t n) {
    MCL_NEED_CTX(ctx);
    const char* op = "mse_backward";
    if (n == 0 || n > 0x7fffffffull) return fail(ctx, MCL_CUDA_EINVAL, "mse_backward needs 0 < n < 2^31");
    MCL_TRY(check_ptr(ctx, op, "pred", pred, 4));
    MCL_TRY(check_ptr(ctx, op, "target", target, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_out", grad_out, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_pred", grad_pred, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_mse_backward(pred, target, grad_out, grad_pred, n, ctx->stream));
    return MCL_CUDA_OK;
}
int mcl_cuda_swiglu(mcl_cuda_ctx* ctx, const float* packed, float* out, size_t rows, size_t hidden) {
    MCL_NEED_CTX(ctx);
    const char* op = "swiglu";
    MCL_TRY(check_rows(ctx, op, rows, hidden));
    MCL_TRY(check_ptr(ctx, op, "packed", packed, 4));
    MCL_TRY(check_ptr(ctx, op, "out", out, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_swiglu(packed, out, rows, (int)hidden, ctx->sm_count, ctx->stream));
    return MCL_CUDA_OK;
}
int mcl_cuda_swiglu_backward(mcl_cuda_ctx* ctx, const float* packed, const float* grad_out, float* grad_packed,
                             size_t rows, size_t hidden) {
    MCL_NEED_CTX(ctx);
    const char* op = "swiglu backward";
    MCL_TRY(check_rows(ctx, op, rows, hidden));
    MCL_TRY(check_ptr(ctx, op, "packed", packed, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_out", grad_out, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_packed", grad_packed, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_swiglu_backward(packed, grad_out, grad_packed, rows, (int)hidden, ctx->sm_count, ctx->stream));
    return MCL_CUDA_OK;
}
int mcl_cuda_softmax_cross_entropy(mcl_cuda_ctx* ctx, const float* logits, const int32_t* targets, float* partial,
                                   float* out, size_t rows, size_t cols) {
    MCL_NEED_CTX(ctx);
    const char* op = "softmax_cross_entropy";
    MCL_TRY(check_rows(ctx, op, rows, cols));
    MCL_TRY(check_ptr(ctx, op, "logits", logits, 4));
    MCL_TRY(check_ptr(ctx, op, "targets", targets, 4));
    MCL_TRY(check_ptr(ctx, op, "partial", partial, 4));
    MCL_TRY(check_ptr(ctx, op, "out", out, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_softmax_cross_entropy(logits, targets, partial, out, rows, (int)cols, ctx->sm_count, ctx->stream));
    ctx->launches += 1;     // row losses, then their mean
    return MCL_CUDA_OK;
}
int mcl_cuda_softmax_cross_entropy_backward(mcl_cuda_ctx* ctx, const float* logits, const int32_t* targets,
                                            const float* grad_out, float* grad_logits, size_t rows, size_t cols) {
    MCL_NEED_CTX(ctx);
    const char* op = "softmax_cross_entropy backward";
    MCL_TRY(check_rows(ctx, op, rows, cols));
    MCL_TRY(check_ptr(ctx, op, "logits", logits, 4));
    MCL_TRY(check_ptr(ctx, op, "targets", targets, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_out", grad_out, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_logits", grad_logits, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_softmax_cross_entropy_backward(logits, targets, grad_out, grad_logits, rows, (int)cols, ctx->sm_count, ctx->stream));
    return MCL_CUDA_OK;
}

namespace {
int check_gqa(mcl_cuda_ctx* ctx, const char* op, size_t batch, size_t tq, size_t tk, size_t key_stride, size_t n_head,
              size_t n_kv, size_t hd, size_t vhd, size_t q_off, size_t window, bool backward) {
    if (batch == 0 || tq == 0 || tk == 0 || n_head == 0 || n_kv == 0 || hd == 0 || vhd == 0)
        return fail(ctx, MCL_CUDA_EINVAL, std::string(op) + " requires non-zero dimensions");
    if (n_head % n_kv != 0) return fail(ctx, MCL_CUDA_EINVAL, std::string(op) + " requires n_head % n_kv_head == 0");
    if (key_stride < tk) return fail(ctx, MCL_CUDA_EINVAL, std::string(op) + " requires key_stride >= key_tokens");
    if (batch * n_head > 65535 || tq > 0x7fffffffull || tk > 0x7fffffffull || q_off > 0x3fffffffull ||
        window > 0x3fffffffull || hd > 65536 || vhd > 65536)
        return fail(ctx, MCL_CUDA_EINVAL, std::string(op) + " dimension is too large");
    (void)backward;
    return MCL_CUDA_OK;
}
}  // namespace

int mcl_cuda_gqa_forward(mcl_cuda_ctx* ctx, const float* q, const float* k, const float* v, float* out, size_t batch,
                         size_t query_tokens, size_t key_tokens, size_t key_stride, size_t n_head, size_t n_kv_head,
                         size_t head_dim, size_t v_head_dim, int causal, size_t query_offset, size_t sliding_window,
                         float scale) {
    MCL_NEED_CTX(ctx);
    const char* op = "grouped_query_attention";
    MCL_TRY(check_gqa(ctx, op, batch, query_tokens, key_tokens, key_stride, n_head, n_kv_head, head_dim, v_head_dim,
                      query_offset, sliding_window, false));
    MCL_TRY(check_ptr(ctx, op, "q", q, 4));
    MCL_TRY(check_ptr(ctx, op, "k", k, 4));
    MCL_TRY(check_ptr(ctx, op, "v", v, 4));
    MCL_TRY(check_ptr(ctx, op, "out", out, 4));
    DeviceGuard guard(ctx->device);
    // scores of every (batch, head, query) row live in the workspace between the two products; the batch is
    // served in slices that keep it under 4 GiB (one batch element at least)
    // (the tiled kernels need none)
    const size_t per_batch = mcl::gqa_forward_scratch_floats((int)batch, (int)query_tokens, (int)key_tokens, (int)n_head, (int)head_dim,
                                                             (int)v_head_dim) / batch * sizeof(float);
    size_t slice = per_batch ? ((size_t)4 << 30) / per_batch : batch;
    if (slice < 1) slice = 1;
    if (slice > batch) slice = batch;
    void* ws = nullptr;
    if (per_batch) MCL_TRY(ws_reserve(ctx, slice * per_batch, &ws));
    int launches = 0;
    cudaError_t e = cudaSuccess;
    for (size_t b0 = 0; b0 < batch && e == cudaSuccess; b0 += slice) {
        const size_t nb = batch - b0 < slice ? batch - b0 : slice;
        e = mcl::launch_gqa_forward(q + b0 * query_tokens * n_head * head_dim, k + b0 * key_stride * n_kv_head * head_dim,
                                    v + b0 * key_stride * n_kv_head * v_head_dim, out + b0 * query_tokens * n_head * v_head_dim,
                                    (int)nb, (int)query_tokens, (int)key_tokens, (int)key_stride, (int)n_head, (int)n_kv_head,
                                    (int)head_dim, (int)v_head_dim, causal ? 1 : 0, (int)query_offset, (int)sliding_window,
                                    scale, static_cast<float*>(ws), ctx->stream, &launches);
    }
    if (e != cudaSuccess) return fail_cuda(ctx, op, e);
    ctx->launches += launches;
    return MCL_CUDA_OK;
}
int mcl_cuda_gqa_backward(mcl_cuda_ctx* ctx, const float* q, const float* k, const float* v, const float* grad_out,
                          float* probs_scratch, float* ds_scratch, float* grad_q, float* grad_k, float* grad_v,
                          size_t batch, size_t query_tokens, size_t key_tokens, size_t n_head, size_t n_kv_head,
                          size_t head_dim, int causal, size_t query_offset, float scale) {
    MCL_NEED_CTX(ctx);
    const char* op = "grouped_query_attention backward";
    MCL_TRY(check_gqa(ctx, op, batch, query_tokens, key_tokens, key_tokens, n_head, n_kv_head, head_dim, head_dim,
                      query_offset, 0, true));
    MCL_TRY(check_ptr(ctx, op, "q", q, 4));
    MCL_TRY(check_ptr(ctx, op, "k", k, 4));
    MCL_TRY(check_ptr(ctx, op, "v", v, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_out", grad_out, 4));
    MCL_TRY(check_ptr(ctx, op, "probs_scratch", probs_scratch, 4));
    MCL_TRY(check_ptr(ctx, op, "ds_scratch", ds_scratch, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_q", grad_q, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_k", grad_k, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_v", grad_v, 4));
    DeviceGuard guard(ctx->device);
    int launches = 0;
    cudaError_t e = mcl::launch_gqa_backward(q, k, v, grad_out, probs_scratch, ds_scratch, grad_q, grad_k, grad_v,
                                             (int)batch, (int)query_tokens, (int)key_tokens, (int)n_head, (int)n_kv_head,
                                             (int)head_dim, causal ? 1 : 0, (int)query_offset, scale, ctx->stream, &launches);
    if (e != cudaSuccess) return fail_cuda(ctx, op, e);
    ctx->launches += launches;
    return MCL_CUDA_OK;
}

int mcl_cuda_token_position_embedding(mcl_cuda_ctx* ctx, const float* token_weight, const float* pos_weight,
                                      const int32_t* token_ids, float* out, size_t token_count, size_t vocab_size,
                                      size_t seq_len, size_t embed_dim) {
    MCL_NEED_CTX(ctx);
    const char* op = "token_position_embedding";
    if (token_count == 0 || vocab_size == 0 || embed_dim == 0 || (pos_weight && seq_len == 0))
        return fail(ctx, MCL_CUDA_EINVAL, "token_position_embedding requires non-zero shapes");
    if (vocab_size > 0x7fffffffull || embed_dim > 0x7fffffffull || seq_len > 0x7fffffffull)
        return fail(ctx, MCL_CUDA_EINVAL, "token_position_embedding dimension is too large");
    MCL_TRY(check_ptr(ctx, op, "token_weight", token_weight, 4));
    MCL_TRY(check_ptr(ctx, op, "token_ids", token_ids, 4));
    MCL_TRY(check_ptr(ctx, op, "out", out, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_embedding(token_weight, pos_weight, token_ids, out, token_count, (int)vocab_size,
                                              (int)(seq_len ? seq_len : 1), (int)embed_dim, ctx->sm_count, ctx->stream));
    return MCL_CUDA_OK;
}
int mcl_cuda_embedding_weight_backward(mcl_cuda_ctx* ctx, const int32_t* indices, const float* grad_out, float* grad_weight,
                                       size_t vocab_size, size_t embed_dim, size_t token_count, int zero_first) {
    MCL_NEED_CTX(ctx);
    const char* op = "embedding weight backward";
    if (vocab_size == 0 || embed_dim == 0) return fail(ctx, MCL_CUDA_EINVAL, "embedding weight backward requires non-zero shapes");
    if (vocab_size > 0x7fffffffull || embed_dim > 0x7fffffffull)
        return fail(ctx, MCL_CUDA_EINVAL, "embedding weight backward dimension is too large");
    MCL_TRY(check_ptr(ctx, op, "grad_weight", grad_weight, 4));
    DeviceGuard guard(ctx->device);
    if (zero_first) {
        cudaError_t e = cudaMemsetAsync(grad_weight, 0, vocab_size * embed_dim * sizeof(float), ctx->stream);
        if (e != cudaSuccess) return fail_cuda(ctx, op, e);
    }
    if (token_count == 0) return MCL_CUDA_OK;
    MCL_TRY(check_ptr(ctx, op, "indices", indices, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_out", grad_out, 4));
    MCL_LAUNCH(ctx, op, mcl::launch_embedding_scatter(indices, grad_out, grad_weight, token_count, (int)vocab_size, (int)embed_dim,
                                                      ctx->sm_count, ctx->stream));
    return MCL_CUDA_OK;
}
int mcl_cuda_position_embedding_backward(mcl_cuda_ctx* ctx, const float* grad_out, float* grad_position, size_t batch,
                                         size_t seq_len, size_t embed_dim) {
    MCL_NEED_CTX(ctx);
    const char* op = "position embedding backward";
    if (batch == 0 || seq_len == 0 || embed_dim == 0 || batch > 0x7fffffffull || seq_len > 0x7fffffffull || embed_dim > 0x7fffffffull)
        return fail(ctx, MCL_CUDA_EINVAL, "position embedding backward requires non-zero shapes below 2^31");
    MCL_TRY(check_ptr(ctx, op, "grad_out", grad_out, 4));
    MCL_TRY(check_ptr(ctx, op, "grad_position", grad_position, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_position_backward(grad_out, grad_position, (int)batch, (int)seq_len, (int)embed_dim,
                                                      ctx->sm_count, ctx->stream));
    return MCL_CUDA_OK;
}
int mcl_cuda_rope(mcl_cuda_ctx* ctx, const float* x, float* out, size_t batch, size_t tokens, size_t channels, size_t n_head,
                  size_t head_dim, size_t rotary_dim, size_t token_offset, float theta, int inverse, int split_half) {
    MCL_NEED_CTX(ctx);
    const char* op = "rope";
    if (batch == 0 || tokens == 0 || channels == 0 || n_head == 0 || head_dim == 0)
        return fail(ctx, MCL_CUDA_EINVAL, "rope requires non-zero shapes");
    if (tokens > 0x7fffffffull || channels > 0x7fffffffull || token_offset > 0x3fffffffull || rotary_dim > head_dim)
        return fail(ctx, MCL_CUDA_EINVAL, "rope dimension is out of range");
    if (n_head * head_dim > channels) return fail(ctx, MCL_CUDA_EINVAL, "rope requires n_head * head_dim <= channels");
    MCL_TRY(check_ptr(ctx, op, "x", x, 4));
    MCL_TRY(check_ptr(ctx, op, "out", out, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_rope(x, out, batch * tokens, (int)tokens, (int)channels, (int)n_head, (int)head_dim,
                                         (int)rotary_dim, (int)token_offset, theta, inverse ? 1 : 0, split_half ? 1 : 0,
                                         ctx->sm_count, ctx->stream));
    return MCL_CUDA_OK;
}
int mcl_cuda_adam_update(mcl_cuda_ctx* ctx, float* param, const float* grad, float* m, float* v, size_t elements, float lr,
                         float beta1, float beta2, float eps, float weight_decay, float c1, float c2) {
    MCL_NEED_CTX(ctx);
    const char* op = "adam_update";
    if (elements == 0) return fail(ctx, MCL_CUDA_EINVAL, "adam_update requires non-zero elements");
    MCL_TRY(check_ptr(ctx, op, "param", param, 4));
    MCL_TRY(check_ptr(ctx, op, "grad", grad, 4));
    MCL_TRY(check_ptr(ctx, op, "m", m, 4));
    MCL_TRY(check_ptr(ctx, op, "v", v, 4));
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_adam(param, grad, m, v, elements, lr, beta1, beta2, eps, weight_decay, c1, c2, ctx->sm_count,
                                         ctx->stream));
    return MCL_CUDA_OK;
}

int mcl_cuda_peer_buffer_create(mcl_cuda_ctx* ctx, size_t bytes, void** out_dptr, unsigned char* handle64) {
    MCL_NEED_CTX(ctx);
    MCL_NOT_RECORDING(ctx, "peer_buffer_create");
    if (!out_dptr || !handle64 || bytes == 0) return fail(ctx, MCL_CUDA_EINVAL, "peer_buffer_create: null argument or zero size");
    static_assert(sizeof(cudaIpcMemHandle_t) == MCL_CUDA_IPC_HANDLE_BYTES, "IPC handle size");
    DeviceGuard guard(ctx->device);
    void* d = nullptr;
    // plain cudaMalloc: memory of the stream-ordered pool cannot be exported to other processes
    cudaError_t e = cudaMalloc(&d, bytes);
    if (e != cudaSuccess) return fail_cuda(ctx, "peer_buffer_create (cudaMalloc)", e);
    e = cudaMemset(d, 0, bytes);
    cudaIpcMemHandle_t h;
    if (e == cudaSuccess) e = cudaIpcGetMemHandle(&h, d);
    if (e != cudaSuccess) { cudaFree(d); return fail_cuda(ctx, "peer_buffer_create (export)", e); }
    std::memcpy(handle64, &h, sizeof(h));
    *out_dptr = d;
    return MCL_CUDA_OK;
}
int mcl_cuda_peer_buffer_open(mcl_cuda_ctx* ctx, const unsigned char* handle64, void** out_dptr) {
    MCL_NEED_CTX(ctx);
    MCL_NOT_RECORDING(ctx, "peer_buffer_open");
    if (!out_dptr || !handle64) return fail(ctx, MCL_CUDA_EINVAL, "peer_buffer_open: null argument");
    DeviceGuard guard(ctx->device);
    cudaIpcMemHandle_t h;
    std::memcpy(&h, handle64, sizeof(h));
    void* d = nullptr;
    cudaError_t e = cudaIpcOpenMemHandle(&d, h, cudaIpcMemLazyEnablePeerAccess);
    if (e != cudaSuccess) return fail_cuda(ctx, "peer_buffer_open", e);
    *out_dptr = d;
    return MCL_CUDA_OK;
}
int mcl_cuda_peer_buffer_close(mcl_cuda_ctx* ctx, void* dptr) {
    MCL_NEED_CTX(ctx);
    if (!dptr) return MCL_CUDA_OK;
    DeviceGuard guard(ctx->device);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e == cudaSuccess) e = cudaIpcCloseMemHandle(dptr);
    if (e != cudaSuccess) return fail_cuda(ctx, "peer_buffer_close", e);
    return MCL_CUDA_OK;
}
int mcl_cuda_peer_buffer_destroy(mcl_cuda_ctx* ctx, void* dptr) {
    MCL_NEED_CTX(ctx);
    if (!dptr) return MCL_CUDA_OK;
    DeviceGuard guard(ctx->device);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e == cudaSuccess) e = cudaFree(dptr);
    if (e != cudaSuccess) return fail_cuda(ctx, "peer_buffer_destroy", e);
    return MCL_CUDA_OK;
}
int mcl_cuda_peer_allreduce_f32(mcl_cuda_ctx* ctx, const void* const* peer_data, void* const* peer_flags, int rank,
                                int world, size_t n, size_t parity_stride, int parity, float* out) {
    MCL_NEED_CTX(ctx);
    const char* op = "peer allreduce";
    if (world < 1 || world > mcl::kPeerMaxWorld || rank < 0 || rank >= world)
        return fail(ctx, MCL_CUDA_EINVAL, "peer allreduce serves 1 to 8 ranks of one node");
    if (parity != 0 && parity != 1) return fail(ctx, MCL_CUDA_EINVAL, "peer allreduce: parity is 0 or 1");
    if (n == 0 || n % 4 != 0 || parity_stride % 4 != 0 || n > parity_stride || n > 0x7fffffffull)
        return fail(ctx, MCL_CUDA_EINVAL, "peer allreduce needs n and parity_stride in multiples of 4 floats, n <= parity_stride");
    if (!peer_data || !peer_flags) return fail(ctx, MCL_CUDA_EINVAL, "peer allreduce: null pointer tables");
    MCL_TRY(check_ptr(ctx, op, "out", out, 16));
    mcl::PeerTable tab{};
    for (int r = 0; r < world; ++r) {
        if (!peer_data[r] || !peer_flags[r] || reinterpret_cast<uintptr_t>(peer_data[r]) % 16 != 0 ||
            reinterpret_cast<uintptr_t>(peer_flags[r]) % 4 != 0)
            return fail(ctx, MCL_CUDA_EINVAL, "peer allreduce: every rank's data must be 16-byte and its flags 4-byte aligned");
        tab.data[r] = static_cast<const float*>(peer_data[r]);
        tab.flags[r] = static_cast<uint32_t*>(peer_flags[r]);
    }
    tab.parity_stride4 = parity_stride / 4;
    tab.rank = rank; tab.world = world;
    DeviceGuard guard(ctx->device);
    MCL_LAUNCH(ctx, op, mcl::launch_peer_allreduce(tab, n, parity, out, ctx->err_word, ctx->stream));
    return MCL_CUDA_OK;
}

int mcl_cuda_ternary_gemv(mcl_cuda_ctx* ctx, const float* x, const uint32_t* packed2,
                          const float* scale, float* y, size_t M, size_t in_features,
                          size_t out_features) {
    MCL_NEED_CTX(ctx);
    const char* op = "ternary gemv";
    if (M == 0 || in_features == 0 || out_features == 0) return fail(ctx, MCL_CUDA_EINVAL, "ternary gemv requires non-zero dimensions");
    if (M > 16) return fail(ctx, MCL_CUDA_EINVAL, "ternary gemv serves M <= 16; use counter forward for larger batches");
    if (in_features % 16 != 0) return fail(ctx, MCL_CUDA_EINVAL, "ternary gemv requires in_features % 16 == 0");
    if (in_features > 0x7fffffffull || out_features > 0x7fffffffull) return fail(ctx, MCL_CUDA_EINVAL, "ternary gemv dimension exceeds 2^31");
    MCL_TRY(check_ptr(ctx, op, "x", x, 16));
    MCL_TRY(check_ptr(ctx, op, "packed2", packed2, 4));
    MCL_TRY(check_ptr(ctx, op, "scale", scale, 4));
    MCL_TRY(check_ptr(ctx, op, "y", y, 4));
    DeviceGuard guard(ctx->device);
    const mcl::GemvItem item = {x, packed2, scale, y, (int)in_features, (int)out_features};
    const bool exact = ctx->gemm_mode == MCL_CUDA_GEMM_EXACT;
    const bool mma = !exact && mcl::gemv_mma_supported((int)M, (int)in_features, packed2, ctx->max_smem);
    const bool tc = !exact && mcl::gemv_tc_supported((int)M, (int)in_features, packed2) && (mma || out_features >= 128) && (mma || M > 1);
    if (mma || tc) {
        // Only in a recording is it known what runs before and after: a matrix joins a launch there where nothing that was recorded since
        // has to do with it.
        GemvRecord& rec = ctx->gemvs;
        unsigned long long capture = 0;
        const cudaGraphNode_t tail = recorded_tail(ctx, &capture);
        const bool follows = tail != nullptr && tail == rec.tail && capture == rec.capture;
        if (!follows) rec.close();
        if (join_gemvs(ctx, item, (int)M, mma, tc)) return MCL_CUDA_OK;
        // up to 8 rows the workspace is taken outside captures only: what a recording makes of its lists is settled when it is complete
        GemvList at = {ctx, !mma || (tc && !ctx->recording && mcl::gemv_tc_pays(&item, 1, (int)M, ctx->sm_count) && !foreign_capture(ctx)), {}, (int)M, {item}, nullptr, 0};
        void* wsp = nullptr;
        if (at.tc) {
            // more rows than gemv_mma.cu takes: with room for the digits of further xs, which the launches of a recording may take together
            const size_t need = mcl::gemv_tc_workspace_bytes(&item, 1, (int)M, ctx->sm_count);
            const std::string error = ctx->error;
            const int rc = ws_reserve(ctx, mma || need <= ctx->ws_bytes ? need : need + (size_t(16) << 20), &wsp);
            if (rc != MCL_CUDA_OK && !mma) return rc;
            if (rc != MCL_CUDA_OK) { ctx->error = error; at.tc = false; }
            at.ws = ctx->ws;
            at.ws_bytes = ctx->ws_bytes;
        }
        if (at.tc) {
            for (int part = 0; part < 2; ++part) {
                MCL_LAUNCH(ctx, op, mcl::launch_ternary_gemv_tc(&item, 1, (int)M, wsp, 1 << part, follows, nullptr, nullptr, ctx->err_word, ctx->sm_count, ctx->max_smem, ctx->stream));
                at.node[part] = recorded_tail(ctx, &rec.capture);
            }
        } else {
            MCL_LAUNCH(ctx, op, mcl::launch_ternary_gemv_mma(&item, 1, (int)M, follows, nullptr, ctx->sm_count, ctx->max_smem, ctx->stream));
            at.node[0] = recorded_tail(ctx, &rec.capture);
        }
        rec.tail = at.node[at.tc ? 1 : 0];
        if (rec.tail) rec.lists.push_back(at);
        return MCL_CUDA_OK;
    }
    if (!exact && M == 1) {
        // a single activation row whose shape the integer MMAs do not take: streaming the words through the CUDA
        // cores in one launch still beats the launches of the tensor-core route
        MCL_LAUNCH(ctx, op, mcl::launch_ternary_gemv_stream(x, packed2, scale, y, (int)M, (int)in_features, (int)out_features,
                                                            ctx->sm_count, ctx->stream));
        return MCL_CUDA_OK;
    }
    MCL_LAUNCH(ctx, op, mcl::launch_ternary_gemv(x, packed2, scale, y, (int)M, (int)in_features,
                                                 (int)out_features, ctx->sm_count, ctx->stream));
    return MCL_CUDA_OK;
}

}  // extern "C"
