// Internal launch interface between the C-ABI layer (abi.cu) and the kernel files.
// Every launcher enqueues on `stream` and returns the launch status; none synchronises.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace mcl {

// Launches that follow one another on a stream overlap at their seams (programmatic dependent launch): a kernel launched with
// launch_chained may start when all CTAs of the one before it run, sets itself up, and in grid_wait() waits until that one has completed
// and its results can be read.  Rules: nothing of global memory that another launch may write is touched before grid_wait() nor, behind it, read
// otherwise than by ordinary loads (load_behind), every CTA gets there, and grid_release() comes after a CTA has its tensor memory, so that no CTA waits for memory that a later launch holds.
// What it saves is a few microseconds a launch: one layer of 288 x 288 at 256 rows (three launches) 38 -> 30 us, of 288 x 1536 at 4096 123 ->
// 115, the fp32 ops of a block (13 launches) 219 -> 206, the update of 8192 x 4096 98 -> 95.  Not for the launches of tc_gemm.cu: long
// kernels that fill the GPU gain nothing, and split_terms_kernel's waiting CTAs keep other streams' work off (a stack of 42 layers beside two
// others 1591 -> 1623 us).
template <class... P, class... A>
cudaError_t launch_chained(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}
#ifdef __CUDACC__
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// What an earlier launch may have written, behind grid_wait(): an ordinary load that keeps its place.  The read-only path (__ldg, const
// __restrict__) is for data that nobody writes while the kernel runs, and a kernel that overlaps runs while the one before it writes.
template <class T>
__device__ __forceinline__ T load_behind(const T* p) {
    static_assert(sizeof(T) == 1 || sizeof(T) == 4 || sizeof(T) == 16, "8, 32 or 128 bits");
    union { T v; uint32_t w[sizeof(T) == 16 ? 4 : 1]; } u;
    if constexpr (sizeof(T) == 16) {
        asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(u.w[0]), "=r"(u.w[1]), "=r"(u.w[2]), "=r"(u.w[3]) : "l"(p));
        return u.v;
    } else if constexpr (sizeof(T) == 4) {
        asm volatile("ld.global.u32 %0, [%1];" : "=r"(u.w[0]) : "l"(p));
        return u.v;
    } else {
        uint32_t w;
        asm volatile("ld.global.u8 %0, [%1];" : "=r"(w) : "l"(p));
        return static_cast<T>(w);
    }
}
#endif

// counter_update.cu
cudaError_t ensure_dynamic_smem(const void* kern, int slot, size_t max_smem);
// err_word (may be null): device word that the wide-row kernel sets when a bounded wait gives up
cudaError_t launch_counter_update_dense(uint8_t* state, float* scale, float* v, const float* grad_w,
                                        uint32_t* packed2, int C, int in_features, int rows,
                                        int row_offset, float lr, float lr_scale, float rms_beta,
                                        float rms_eps, uint32_t seed, const uint32_t* seed_offset, int* err_word,
                                        int sm_count, size_t max_smem, cudaStream_t stream);
struct UpdateDesc {            // rows [row_offset, row_offset + rows) of one layer; pointers at the first row
    uint8_t* state;
    float* scale;
    float* v;
    const float* grad_w;
    uint32_t* packed2;         // may be null
    int in_features, rows, row_offset;
};
cudaError_t launch_counter_update_group(const UpdateDesc* d, int n, int C, float lr, float lr_scale, float rms_beta,
                                        float rms_eps, uint32_t seed, const uint32_t* seed_offset, int* err_word, int sm_count,
                                        size_t max_smem, cudaStream_t stream, int* launches);
cudaError_t launch_decode_weight(const uint8_t* state, const float* scale, float* w, int C,
                                 int in_features, int out_features, int sm_count, cudaStream_t stream);
cudaError_t launch_pack2(const uint8_t* state, uint32_t* packed2, int C, int in_features,
                         int out_features, int sm_count, cudaStream_t stream);

// layer_kernels.cu -- one launch per product of a narrow layer, operands converted inside the kernel
bool layer_kernels_fit(size_t tokens, size_t in_features, size_t out_features);
// rather these kernels than the split-once route of tc_gemm.cu: a product [tokens, N] over K; the update, whose other route takes `tiles` row tiles
bool layer_rows_pay(size_t tokens, size_t N, size_t K, int sm_count);
bool layer_update_pays(size_t tokens, size_t in_features, size_t out_features, size_t tiles, int sm_count);
// dx = 0: c[tokens, O] = a (scale T)^T;  dx = 1: c[tokens, I] = (a . scale) T
cudaError_t launch_layer_rows(int dx, const float* a, const uint8_t* state, const float* scale, float* c, int tokens, int I, int O,
                              int C, int* err_word, size_t max_smem, int sm_count, cudaStream_t stream);
// the counter update of a whole layer from its activations (d.grad_w unused, d.row_offset == 0; x 16-byte aligned)
cudaError_t launch_layer_update(const UpdateDesc& d, const float* dy, const float* x, int tokens, int C, float lr, float lr_scale,
                                float rms_beta, float rms_eps, uint32_t seed, const uint32_t* seed_offset, int* err_word, int sm_count,
                                size_t max_smem, cudaStream_t stream);
// the same in the order of the exact kernels (simt_gemm.cu), for layers that fit those kernels and few multiply-adds
cudaError_t launch_exact_update(const UpdateDesc& d, const float* dy, const float* x, int tokens, int C, float lr, float lr_scale,
                                float rms_beta, float rms_eps, uint32_t seed, const uint32_t* seed_offset, int sm_count, size_t max_smem,
                                cudaStream_t stream);

// simt_gemm.cu -- fp32 CUDA-core contractions (any shape; exact fp32 FMA accumulation)
cudaError_t launch_simt_matmul_f32(const float* a, const float* b, float* c, int M, int K, int N,
                                   int transA, int transB, cudaStream_t stream);
cudaError_t launch_simt_counter_forward(const float* x, const uint8_t* state, const float* scale,
                                        float* y, int batch, int in_features, int out_features, int C,
                                        cudaStream_t stream);
cudaError_t launch_simt_counter_backward_input(const uint8_t* state, const float* scale,
                                               const float* grad_out, float* grad_x, int batch,
                                               int in_features, int out_features, int C,
                                               cudaStream_t stream);
cudaError_t launch_simt_ternary_forward(const float* x, const uint32_t* packed2, const float* scale, float* y,
                                        int batch, int in_features, int out_features, cudaStream_t stream);
cudaError_t launch_simt_ternary_backward_input(const uint32_t* packed2, const float* scale, const float* grad_out,
                                               float* grad_x, int batch, int in_features, int out_features,
                                               cudaStream_t stream);
// dW rows [row0, row0+rows) of dY^T X into grad_w[rows, in]
cudaError_t launch_simt_grad_w(const float* grad_out, const float* x, float* grad_w, int batch,
                               int in_features, int out_features, int row0, int rows,
                               cudaStream_t stream);

// tc_gemm.cu -- tcgen05 / TMEM / TMA contractions on fp16 term planes (see the file header)
struct TcPlan { int pair, bn, splits, ktiles_per_split, together; size_t workspace_bytes; double cost; };
TcPlan tc_plan(int M, int N, int K, int nterms, int sm_count, int depth_limit);
TcPlan tc_plan_shared(int M, int N, int K, int nterms, int cg, int depth_limit, int min_items, bool together = false);
// k-tiles of 64 per accumulator for fp32 x fp32 products.  Each instruction that adds into an accumulator truncates it; the
// error is about 2.7e-9 for each on terms of either sign (K = 4096: 2e-6) and half a last bit, 6e-8, for each of the leading
// products where a sum grows in one direction (four per k-tile: 1.5e-5).
constexpr int kGradDepthLimit = 64;
constexpr size_t kTermPad = 1024;  // readable bytes after the last plane of a TcOperand
struct TcOperand {             // fp16 planes [planes][rows][ld] of a row-major tensor with `cols` columns
    const void* ptr;
    int rows, cols, ld;
    int planes;                // 2: hi and lo terms of an fp32 tensor; 1: ternary digits
    int mn_major;              // the contraction runs over the rows (0: over the columns)
    const float* inv;          // K-major and scaled by row: 2^-s of every row (else null)
    const uint32_t* words;     // words of the exponent g, where this operand is the one that carries it (at most one of a product)
};
// C[M,N] = sum over k of A B (b.planes == 1: two products, b.planes == 2: three); with plan.splits > 1 into splitk_ws
// [splits][M][N], which a reduction adds up
struct TcProblem {
    TcOperand a, b;
    float* c;
    int M, N, K;
    TcPlan plan;
    const float* col_scale;    // of the output's columns (plan.splits == 1)
    float* splitk_ws;
    int turned;                // c is [N][M]: a the digits, b the split tensor (scaled by row); col_scale of the rows of the product
};
cudaError_t launch_tc_products(const TcProblem* probs, int n, int* err_word, size_t max_smem, int sm_count, cudaStream_t stream,
                               int* launches);
// fp32 [rows, cols] -> fp16 terms [2][rows][ld] of src (planes) and / or of src . col_scale (planes_s).  planes_s, and planes where
// row_inv is given, are scaled by a power of two 2^s of each row; row_inv / row_inv_s receive 2^-s.  Planes without row_inv are scaled by
// 2^(g - s_t), with 2^-s_t from `comp` (row_inv of the tensor on the other side of a contraction over the rows; null: 1), and
// words receives what g follows from.
struct SplitDesc {
    const float* src;
    int rows, cols, ld;
    const float* col_scale;
    void* planes;
    void* planes_s;
    float* row_inv;
    float* row_inv_s;
    const float* comp;
    uint32_t* words;           // two words
};
cudaError_t launch_split_terms(const SplitDesc* d, int n, int sm_count, cudaStream_t stream, int* launches);
struct ExpandDesc {            // ternary digits as fp16 [O][ld], from the 6-bit state (state != null) or the 2-bit words (I % 16 == 0, ld == I)
    const uint8_t* state;
    const uint32_t* packed2;
    int O, I, ld;
    void* T;
};
cudaError_t launch_expand_ternary(const ExpandDesc* d, int n, int C, int sm_count, cudaStream_t stream, int* launches);
cudaError_t launch_splitk_reduce_group(const float* const* partial, float* const* out, const long long* elements, const int* splits,
                                       int n, int sm_count, cudaStream_t stream, int* launches);
cudaError_t launch_splitk_reduce(const float* partial, float* c, const float* col_scale, int M, int N, int ldc,
                                 int splits, cudaStream_t stream);

// gemv.cu
// M = 1: one CUDA-core launch that streams the 2-bit words (in_features % 16 == 0)
cudaError_t launch_ternary_gemv_stream(const float* x, const uint32_t* packed2, const float* scale, float* y, int M,
                                       int in_features, int out_features, int sm_count, cudaStream_t stream);
cudaError_t launch_ternary_gemv(const float* x, const uint32_t* packed2, const float* scale, float* y,
                                int M, int in_features, int out_features, int sm_count,
                                cudaStream_t stream);

// Decode GEMVs.  A launch takes a list of matrices, M rows of x each (the xs may be one or several).  In a recording, the nodes of a launch
// can take a longer list instead (`nodes`).  follows: the launch before this one on the stream is one of these.
constexpr int kGemvListCap = 48;       // the list is a kernel argument, in gemv_tc.cu with a tensor map for every matrix
constexpr int kGemvXCap = 8;           // different xs of a list of gemv_tc.cu
struct GemvItem {
    const float* x;
    const uint32_t* packed2;
    const float* scale;
    float* y;
    int in_features, out_features;
};
// Slices of K (2^n of them) that up to 8 rows of x have a unit of their own in.  They follow from the length alone, so that a result does
// not depend on the launch that a matrix is part of, nor on the kernel.
int gemv_log_slices(int in_features);
#ifdef __CUDACC__
// Whole numbers of 30 bits and sign below a largest magnitude (given as bits of a float without sign): 2^e above it, and the factor
// 2^(30 - e) in two steps, since it leaves fp32 for magnitudes below 2^-97.
__device__ __forceinline__ int gemv_exponent(unsigned int top) { return (int)(top >> 23) - 126; }
struct GemvUnit { float a, b; };
__device__ __forceinline__ GemvUnit gemv_unit(int e) {
    const int a = min(30 - e, 127);
    return {__uint_as_float((uint32_t)(127 + a) << 23), __uint_as_float((uint32_t)(127 + 30 - e - a) << 23)};
}
#endif
// gemv_mma.cu -- M <= 8, one launch (one node) of integer mma.sync; clusters sized for the shortest rows of a list
bool gemv_mma_supported(int M, int in_features, const void* packed2, size_t max_smem);
bool gemv_mma_takes(const GemvItem* items, int n, int M, size_t max_smem);      // as one list, each of them supported
cudaError_t launch_ternary_gemv_mma(const GemvItem* items, int n, int M, bool follows, const cudaGraphNode_t* nodes, int sm_count,
                                    size_t max_smem, cudaStream_t stream);
// gemv_tc.cu -- M <= 16, two launches (two nodes): digits, integer tcgen05.  parts: bit 0 the first launch, bit 1 the second; with `nodes`,
// the parts whose node takes the list.  nodes[0] null: the first gets a node of `graph` right before nodes[1].
bool gemv_tc_supported(int M, int in_features, const void* packed2);
bool gemv_tc_pays(const GemvItem* items, int n, int M, int sm_count);                    // against gemv_mma.cu
size_t gemv_tc_workspace_bytes(const GemvItem* items, int n, int M, int sm_count);      // ~0: more xs or k-blocks than a launch takes
cudaError_t launch_ternary_gemv_tc(const GemvItem* items, int n, int M, void* workspace, int parts, bool follows, const cudaGraphNode_t* nodes,
                                   cudaGraph_t graph, int* err_word, int sm_count, size_t max_smem, cudaStream_t stream);

// peer_reduce.cu -- one-shot sum of a small vector over the GPUs of a node (peer loads, bounded flag wait)
constexpr int kPeerMaxWorld = 8;
constexpr int kPeerErrCode = 31;
constexpr int kPeerFlagWords = 64;        // a rank's flag area: one word per rank, then the call counter
constexpr int kPeerCounterWord = 32;
struct PeerTable {
    const float* data[kPeerMaxWorld];     // every rank's partial buffers (two parities, parity_stride4 float4 apart)
    uint32_t* flags[kPeerMaxWorld];       // every rank's flag words: flags[r][s] = last partial number rank s announced to rank r
    size_t parity_stride4;
    int rank, world;
};
cudaError_t launch_peer_allreduce(const PeerTable& tab, size_t n, int parity, float* out, int* err_word, cudaStream_t stream);

// eltwise.cu: op 0 add, 1 sub, 2 mul, 3 mul_scalar, 4 add_scalar, 5 zero, 6 a - alpha*b
cudaError_t launch_eltwise_f32(int op, const float* a, const float* b, float* out, size_t n, float alpha,
                               int sm_count, cudaStream_t stream);

// trainer_ops.cu -- the fp32 row ops of the ternary15m block stack around its counter layers
cudaError_t launch_rmsnorm(const float* x, const float* w, float* out, size_t rows, int cols, float eps, int sm_count,
                           cudaStream_t stream);
cudaError_t launch_rmsnorm_backward_x(const float* x, const float* w, const float* dy, float* dx, size_t rows, int cols,
                                      float eps, int sm_count, cudaStream_t stream);
cudaError_t launch_rmsnorm_backward_weight(const float* x, const float* dy, float* row_inv, float* dw, size_t rows,
                                           int cols, float eps, int sm_count, cudaStream_t stream);
cudaError_t launch_mse_loss_partial(const float* pred, const float* target, float* partial, size_t n, cudaStream_t stream);
cudaError_t launch_mean_reduce(const float* partial, float* out, int count, int denominator, cudaStream_t stream);
cudaError_t launch_mse_backward(const float* pred, const float* target, const float* grad_out, float* grad_pred, size_t n,
                                cudaStream_t stream);
cudaError_t launch_swiglu(const float* packed, float* out, size_t rows, int hidden, int sm_count, cudaStream_t stream);
cudaError_t launch_swiglu_backward(const float* packed, const float* dy, float* dpacked, size_t rows, int hidden,
                                   int sm_count, cudaStream_t stream);
cudaError_t launch_softmax_cross_entropy(const float* logits, const int* targets, float* partial, float* out, size_t rows,
                                         int cols, int sm_count, cudaStream_t stream);
cudaError_t launch_softmax_cross_entropy_backward(const float* logits, const int* targets, const float* grad_out,
                                                  float* grad_logits, size_t rows, int cols, int sm_count,
                                                  cudaStream_t stream);
cudaError_t launch_embedding(const float* token_weight, const float* pos_weight, const int* ids, float* out, size_t tokens,
                             int vocab, int seq_len, int dim, int sm_count, cudaStream_t stream);
cudaError_t launch_embedding_scatter(const int* ids, const float* grad_out, float* grad_weight, size_t tokens, int vocab, int dim,
                                     int sm_count, cudaStream_t stream);
cudaError_t launch_position_backward(const float* grad_out, float* grad_position, int batch, int seq_len, int dim, int sm_count,
                                     cudaStream_t stream);
cudaError_t launch_rope(const float* x, float* out, size_t rows, int tokens, int channels, int n_head, int head_dim,
                        int rotary_dim, int token_offset, float theta, int inverse, int split_half, int sm_count,
                        cudaStream_t stream);
cudaError_t launch_adam(float* param, const float* grad, float* m, float* v, size_t n, float lr, float beta1, float beta2,
                        float eps, float weight_decay, float c1, float c2, int sm_count, cudaStream_t stream);
size_t gqa_forward_scratch_floats(int batch, int tq, int tk, int n_head, int hd, int vhd);
cudaError_t launch_gqa_forward(const float* q, const float* k, const float* v, float* out, int batch, int tq, int tk,
                               int key_stride, int n_head, int n_kv, int hd, int vhd, int causal, int q_off, int window,
                               float scale, float* scores_ws, cudaStream_t stream, int* launches);
cudaError_t launch_gqa_backward(const float* q, const float* k, const float* v, const float* dout, float* probs, float* ds,
                                float* dq, float* dk, float* dv, int batch, int tq, int tk, int n_head, int n_kv, int hd,
                                int causal, int q_off, float scale, cudaStream_t stream, int* launches);

}  // namespace mcl
