// Tensor-core contractions of the counter-linear path for sm_100a: tcgen05.mma with fp32
// accumulators in tensor memory (TMEM), operands staged in shared memory by TMA.
//
// One kernel serves the three products of a training step (MotifCL
// src/nn/compact_counter.cpp:233-300 and kernels/matmul.cl:413-563 compute them with fp32
// scalar FMAs) and the dense fp32 matmul:
//     Y  [tokens,out] = X  . T^T          A = terms of X    [tokens,in]     B = T [out,in]
//     dX [tokens,in ] = (dY.s) . T        A = terms of dY.s [tokens,out]    B = T [out,in], read MN-major
//     dW [out,in]     = dY^T . X          A = terms of dY, B = terms of X   both [tokens, .], read MN-major
// (Y and dX also turned, as C^T = T . X^T and T^T . (dY.s)^T with tokens as columns, where the plan wastes less of a tile),
// so every tensor is split once, in its own layout, and T is expanded once: a transposed operand is the
// same shared-memory tile with the MN-major bit of the instruction descriptor.
//
// How an fp32 tensor becomes two fp16 terms (split_terms_kernel): with a power of two f that brings the largest magnitude
// into [2^14, 2^15), hi = fp16(a f) and lo = fp16((a f - hi) 2^12).  hi keeps 11 bits, the residual is at most half a unit of
// hi and keeps 11 more below its sign: |a f - hi - lo 2^-12| <= 2^-23 |a f|, the last bit of fp32 (the first bf16 form of this
// file needed three 8-bit terms for the same bits).  lo is stored 2^12 up so that it stays a normal number wherever hi is:
// elements down to 2^-28 of the largest keep all their bits, smaller ones are off by less than 2^-50 of it.
// What f belongs to:
//   an operand whose rows are rows (or columns) of the product: each row has its own f from its own largest finite element,
//       and the epilogue undoes it.  A row far below the others keeps its bits; an infinity, a NaN or a huge value stays in
//       the rows (columns) of the product that it belongs to.
//   dW and other products along the rows of both: one operand has a scale 2^s_t per row t as above, the other 2^(g - s_t), and
//       the epilogue undoes 2^g.  g follows from the largest |a_t| max|b_t|, so what is lost is below 2^-42 (sampled, see
//       there) of the largest product.  Infinities and NaN stay in their column.
// The lo products go into the accumulator first; the first hi product scales it down by 2^-12 (tcgen05.mma scale-input-d).
// Ternary digits are exact in fp16.  Cost per product of a step in bf16-rate passes: Y, dX 2 (3 before), dW 3
// (hi.hi + hi.lo + lo.hi; 6 before).
// The kernel is bound by the tensor pipe; its time at a stated size stands at tc_gemm_kernel.
#include <cuda.h>
#include <cuda_fp16.h>

#include "counter_codec.cuh"
#include "kernels.h"
#include "sample_rule.h"
#include "tc_ptx.cuh"

namespace mcl {
namespace {

constexpr int BM = 128;          // UMMA M
constexpr int BK = 64;           // 64 fp16 = 128 bytes = one swizzle row
constexpr int kMaxStages = 8;
constexpr int kATileBytes = BM * BK * 2;   // 16 KiB
constexpr int kLoShift = 12;               // lo terms are stored 2^12 up

// One product of a launch's table.
struct TcTile {
    const float* col_scale;   // optional, applied when splits == 1
    const float* a_inv;       // 2^-s of every row of A, of every row of B (column of the product); null: 1
    const float* b_inv;
    const uint32_t* words;    // the product's words of g (null: g = 0)
    int M, N, K;
    int BN, stage_bytes;      // tile width; bytes of one ring slot (A tile and this CTA's share of B, or both terms of them)
    int b_bytes;              // this CTA's share of a B tile
    int a_mn, b_mn;           // operand is stored with M / N contiguous
    int turned;               // C is [N][M]: A are the digits (one plane), B the terms, col_scale belongs to the rows of the product
    int nterms;               // 2: A lo, A hi against one B plane (turned: B's against A); 3: lo.hi, hi.lo, hi.hi
    int ktiles_per_split, splits;
    int tiles_m, tiles_n, group_m;
    int item_begin;           // first work item of the product
};
// The table is a kernel argument: 60 products with their tensor maps are 28 KB.
template <int CAP>
struct TcTable {
    int n, n_items, stages, slot_bytes, acc_cols;
    int* err;
    TcTile p[CAP];
    CUtensorMap maps[3 * CAP];      // A, B, C of product i at 3 i
};
constexpr int kTcCap = 60;

// s of a row (see the file header): its largest magnitude lands in [2^14, 2^15)
__device__ __forceinline__ int term_exp(uint32_t amax_bits) {
    const int e = (int)(amax_bits >> 23);
    const int s = 141 - (e < 1 ? 1 : e);
    return s > 126 ? 126 : s;
}
// g of a tensor that goes with the row scales of another: words hold biased exponents, of an element that is its own plus that of
// its row's 2^-s; 0: no finite element but zeros.  words[0]: what g is first chosen for (the largest of a sample and kSampleRoom, or
// the exact maximum), words[1]: the exact maximum, found while splitting.  words[0] lands in [2^14, 2^15); of the binade above it
// fp16 rounds everything from 65520 up to infinity, so a tensor with a larger exact maximum is split again for it.
constexpr uint32_t kWordBias = 512;
__device__ __forceinline__ int word_g(uint32_t w) { return 141 - (w ? (int)w - (int)kWordBias : 1); }
__device__ __forceinline__ bool terms_redone(uint32_t w0, uint32_t w1) { return w1 > w0; }
__device__ __forceinline__ int terms_g(const uint32_t* words) { return word_g(max(__ldg(words), __ldg(words + 1))); }
__device__ __forceinline__ uint32_t word_of(uint32_t amax_bits, int row_exp) {     // amax_bits: of a finite magnitude
    return amax_bits ? (uint32_t)((int)max(amax_bits >> 23, 1u) + row_exp + (int)kWordBias) : 0u;
}
__device__ __forceinline__ int exp_of(float pow) { return (int)(__float_as_uint(pow) >> 23) - 127; }
__device__ __forceinline__ float pow2(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }

// Instruction descriptor, kind::f16: D = f32 (bits 4-5 = 1), A = B = f16 (bits 7-9, 10-12 = 0), A / B MN-major at bits
// 15 / 16, N >> 3 at bit 17, M >> 4 at bit 24.
__device__ __forceinline__ uint32_t idesc_f16(int m, int n, int a_mn, int b_mn) {
    return (1u << 4) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// MN-major 16-bit tile in the 128-byte swizzle: chunks of 64 MN elements x 64 k rows of 128 bytes; leading byte offset =
// 8192 (next chunk), stride byte offset = 1024 (next 8 k rows).
__device__ __forceinline__ uint64_t smem_desc_mn_sw128(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(8192 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// D = A.B + (accum ? D : 0), and D = A.B + D 2^-12; descriptors as low and high words; CG = 2: issued by the pair's leader for
// both CTAs
template <int CG>
__device__ __forceinline__ void umma_f16(uint32_t tmem_c, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                         uint32_t accum) {
    if (CG == 1)
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %6, 0;\n\tmov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n\t}"
                     ::"r"(tmem_c), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accum) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %6, 0;\n\tmov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %5, p;\n\t}"
                     ::"r"(tmem_c), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accum) : "memory");
}
template <int CG>
__device__ __forceinline__ void umma_f16_down12(uint32_t tmem_c, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc) {
    if (CG == 1)
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, 1, 0;\n\tmov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p, 12;\n\t}"
                     ::"r"(tmem_c), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, 1, 0;\n\tmov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %5, p, 12;\n\t}"
                     ::"r"(tmem_c), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc) : "memory");
}
// arrive on the barrier at this shared-memory offset, in both CTAs of a pair, when the MMAs issued so far are done
template <int CG>
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    if (CG == 1) umma_commit(bar);
    else
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                     ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// tile load whose bytes are counted by `bar`; CG = 2: the barrier may be the other CTA's (a shared::cluster address)
template <int CG>
__device__ __forceinline__ void tc_load(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
    if (CG == 1) tma_load_3d(dst, map, bar, c0, c1, c2);
    else
        asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, %5}], [%2];"
                     ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
template <int CG>
__device__ __forceinline__ void tc_load4(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
    if (CG == 1)
        asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                     ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, %5, %6}], [%2];"
                     ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

// item -> product, output tile and K slice.  Groups of group_m row tiles run through all column tiles before the next group, so
// that the CTAs in flight share both operands' tiles in L2.  `pi` only moves forward.
struct TcItem { int mt, nt, split, kt0, nkt; };
__device__ __forceinline__ TcItem tc_item(const TcTile* tab, int n, int item, int& pi) {
    while (pi + 1 < n && item >= tab[pi + 1].item_begin) ++pi;
    const TcTile& P = tab[pi];
    TcItem t;
    const int per_split = P.tiles_m * P.tiles_n, local = item - P.item_begin;
    t.split = local / per_split;
    int r = local - t.split * per_split;
    const int per_group = P.group_m * P.tiles_n;
    const int g = r / per_group;
    r -= g * per_group;
    const int gm = min(P.group_m, P.tiles_m - g * P.group_m);
    t.nt = r / gm;
    t.mt = g * P.group_m + (r - t.nt * gm);
    t.kt0 = t.split * P.ktiles_per_split;
    t.nkt = min(P.ktiles_per_split, (P.K + BK - 1) / BK - t.kt0);
    return t;
}

// Persistent CTAs of 192 threads (pairs of them with CG = 2); the work items of all products of the table (output tile x split-K slice)
// are drawn from a counter.  A CTA whose SM is taken by another kernel, a collective for instance, then costs its share and not a
// second wave: Y and dX of 21 layers (8192 x 288 -> 768) beside a kernel that holds 16 SMs 786 us, dealt round-robin
// 1055 (660 alone); of 16384 x 2048 -> 2048 517 and 743 (457).
//   warp 0        TMA producer (one elected lane): tiles of A and B into a ring of `stages` shared-memory slots; the leader's draws the
//                 items, one ahead of its copies, and hands them to all other warps through a ring of kDealt words
//   warp 1        MMA issuer (one elected lane): four tcgen05.mma (K = 16 each) per slot; also allocates / frees TMEM
//   warps 2..5    epilogue: tcgen05.ld of 32 lanes x 64 columns, scale, a swizzled 32 x 32 tile in shared memory, TMA store
// Two accumulators live in TMEM (columns [0,BN) and [ACC,ACC+BN)), so the epilogue of one item
// overlaps the main loop of the next.
//
// CG = 2: a cluster of two CTAs shares a 256 x BN tile (tcgen05 cta_group::2).  Each CTA loads its own 128 rows of A and
// its own half of the BN rows of B, the leader's lane issues the MMAs for both tensor cores, and every CTA holds the
// accumulator rows of its own A.  That halves the B bytes a CTA has to write to and read from shared memory: with
// CG = 1 and BN = 256 a k-tile of 64 moves 96 KB through a 128 B/clk pipe (768 cycles) for 512 cycles of MMA; with CG = 2
// 64 KB (512).  All loads count on the leader's barrier.
//
// TOGETHER: a slot holds both terms of A and of B for one k-tile; hi.hi goes into one accumulator, lo.hi and hi.lo into a
// second one beside it, and the epilogue adds the second scaled down by 2^-12.  Every plane is read once (4 tiles per k-tile
// instead of 6): dW of 42 layers at 8192 tokens 456 -> 365 us, memory reads 2.2 -> 1.1 GB, 5.5 GB through L2 (15 TB/s: the bound).
//
// Every mbarrier wait is bounded: on time-out the kernel records an error word, skips the rest of its work, frees
// its TMEM and returns.
constexpr int kTcThreads = 192;
constexpr int kDealt = 4;                  // items between the draw and the epilogue's prefetch: one each in copies, MMAs, epilogue and ahead
constexpr int kQueueWord = 8;              // of the context's words: items drawn, CTAs (pairs) that are done
constexpr int kStageBytes = 8 * 4096;      // epilogue staging: two 32 x 32 float tiles per warp

template <int CG>
__device__ __forceinline__ bool deal_try(uint32_t bar, uint32_t parity) {      // the word may come from the other CTA of a pair
    if (CG == 1) return mbar_try_wait(bar, parity);
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
template <int CG>
__device__ __forceinline__ bool deal_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {      // whole warp, bounded
    if (__all_sync(0xffffffffu, deal_try<CG>(bar, parity))) return true;
    const unsigned long long t0 = clock64();
    unsigned spins = 0;
    while (!__all_sync(0xffffffffu, deal_try<CG>(bar, parity))) {
        if ((++spins & 0x3FFu) == 0) {
            const bool stop = *abort_flag || clock64() - t0 > kWaitCycles;
            if (__any_sync(0xffffffffu, stop)) return false;
        }
    }
    return true;
}
// The word has been read (the arrive takes it as an operand) and nothing was written: no release, which would wait for the warp's
// stores and cost the row products of narrow layers 3 %.
template <int CG>
__device__ __forceinline__ void deal_return(uint32_t bar, int word) {
    if (CG == 1) asm volatile("{\n\t.reg .b32 w;\n\tmov.b32 w, %1;\n\tmbarrier.arrive.relaxed.cta.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar), "r"(word) : "memory");
    else asm volatile("{\n\t.reg .b32 w;\n\tmov.b32 w, %1;\n\tmbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];\n\t}" ::"r"(cluster_addr(bar, 0)), "r"(word) : "memory");
}
// the word to the other CTA of the pair, counted by the barrier there
__device__ __forceinline__ void deal_to_peer(uint32_t word_addr, uint32_t bar, int word) {
    const uint32_t b = cluster_addr(bar, 1);
    asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], 4;" ::"r"(b) : "memory");
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(cluster_addr(word_addr, 1)), "r"(word), "r"(b) : "memory");
}

// TURNED: products of the table may be (a form of its own: the second way out costs the others 1 %)
template <int CG, int CAP, bool TOGETHER, bool TURNED>
__global__ void __launch_bounds__(kTcThreads) tc_gemm_kernel(const __grid_constant__ TcTable<CAP> tab) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kMaxStages + 4 + 2 * kDealt];
    __shared__ int dealt[kDealt];
    __shared__ TcTile sp[CAP];      // the roles walk the table at every item; the constant bank is too small a cache for it
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = tab.stages, n_items = tab.n_items;
    const uint32_t rank = CG == 2 ? (blockIdx.x & 1u) : 0u;      // cluster of two consecutive CTAs
    int* const queue = tab.err + kQueueWord;
    int drawn = n_items;                   // warp 0 of the leader, lane 0
    if (rank == 0 && threadIdx.x == 0) drawn = atomicAdd(queue, 1);
    const uint32_t staging = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t tiles = staging + kStageBytes;
    const uint32_t slot_bytes = (uint32_t)tab.slot_bytes;
    const uint32_t bar0 = smem_u32(bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (kMaxStages + s); };
    auto acc_full = [&](int a) { return bar0 + 8u * (2 * kMaxStages + a); };
    auto acc_empty = [&](int a) { return bar0 + 8u * (2 * kMaxStages + 2 + a); };
    auto deal_full = [&](int i) { return bar0 + 8u * (2 * kMaxStages + 4 + i); };
    auto deal_empty = [&](int i) { return bar0 + 8u * (2 * kMaxStages + 4 + kDealt + i); };
    // the k-th item of this CTA, or -1 after the last; k is the caller's own count
    auto take = [&](uint32_t k) -> int {
        const uint32_t i = k % kDealt;
        if (!deal_wait<CG>(deal_full(i), (k / kDealt) & 1u, &abort_flag)) { abort_flag = 1; if (lane == 0) atomicExch(tab.err, 16); return -1; }
        const int item = *reinterpret_cast<volatile int*>(&dealt[i]);
        __syncwarp();
        if (lane == 0) deal_return<CG>(deal_empty(i), item);
        return item;
    };
    const uint32_t acc_cols = (uint32_t)tab.acc_cols;      // of one accumulator: a power of two >= the widest BN; together: of two
    const uint32_t lo_cols = acc_cols >> 1;                // together: the lo products' accumulator starts here
    const uint32_t tmem_cols = 2 * acc_cols;               // <= 512

    {
        static_assert(sizeof(TcTile) % 4 == 0, "copied word by word");
        const uint32_t* src = reinterpret_cast<const uint32_t*>(tab.p);
        uint32_t* dst = reinterpret_cast<uint32_t*>(sp);
        for (int i = threadIdx.x; i < tab.n * (int)(sizeof(TcTile) / 4); i += kTcThreads) dst[i] = src[i];
    }
    if (threadIdx.x == 0) {
        abort_flag = (*reinterpret_cast<volatile int*>(tab.err) != 0);   // an earlier CTA gave up: do not wait at all
        for (int s = 0; s < S; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(acc_full(a), 1); mbar_init(acc_empty(a), 4 * CG); }
        // readers of a dealt word: MMA warp and four epilogue warps, and the other CTA's producer and four epilogue warps
        for (int i = 0; i < kDealt; ++i) { mbar_init(deal_full(i), 1); mbar_init(deal_empty(i), 5 * CG); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if (CG == 1) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                         ::"r"(smem_u32(&tmem_slot)), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                         ::"r"(smem_u32(&tmem_slot)), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (CG == 2) cluster_sync();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;

    if (warp == 0) {
        // ---- TMA producer ------------------------------------------------------------------
        int s = 0, pi = 0;         // ring slot and its phase, across all items of this CTA
        uint32_t ph = 1;
        bool ok = true;
        for (uint32_t k = 0; ok; ++k) {
            int item;
            if (rank == 0) {
                item = __shfl_sync(0xffffffffu, drawn, 0);
                if (item >= n_items) item = -1;
                const uint32_t i = k % kDealt;
                ok = deal_wait<CG>(deal_empty(i), ((k / kDealt) & 1u) ^ 1u, &abort_flag);
                if (!ok) { abort_flag = 1; if (lane == 0) atomicExch(tab.err, 17); break; }
                if (lane == 0) {
                    *reinterpret_cast<volatile int*>(&dealt[i]) = item;
                    mbar_arrive(deal_full(i));
                    if (CG == 2) deal_to_peer(smem_u32(&dealt[i]), deal_full(i), item);
                }
                __syncwarp();
                if (item >= 0 && lane == 0) drawn = atomicAdd(queue, 1);      // arrives under the copies
            } else {
                item = take(k);
            }
            if (item < 0) break;
            const TcItem t = tc_item(sp, tab.n, item, pi);
            const TcTile& P = sp[pi];
            const CUtensorMap* tmA = &tab.maps[3 * pi];
            const CUtensorMap* tmB = &tab.maps[3 * pi + 1];
            const int BN = P.BN, nterms = P.nterms, a_mn = P.a_mn, b_mn = P.b_mn;
            const bool turned = TURNED && P.turned;
            const uint32_t bytes = (uint32_t)(CG * P.stage_bytes);
            const int m0 = (t.mt * CG + (int)rank) * BM, n0 = t.nt * BN + (int)rank * (BN / CG);
            const uint32_t b_bytes = (uint32_t)P.b_bytes;
            for (int kk = 0; TOGETHER && kk < t.nkt; ++kk) {
                ok = mbar_wait_all(empty_bar(s), ph, &abort_flag);
                if (!ok) { abort_flag = 1; if (lane == 0) atomicExch(tab.err, 1); break; }
                const uint32_t a_dst = tiles + (uint32_t)s * slot_bytes, b_dst = a_dst + 2 * kATileBytes;
                const uint32_t bar = CG == 2 ? cluster_addr(full_bar(s), 0) : full_bar(s);
                const int k0 = (t.kt0 + kk) * BK;
                if (elect_one()) {
                    if (rank == 0) mbar_expect_tx(full_bar(s), bytes);
                    for (int pl = 0; pl < 2; ++pl) {
                        if (a_mn) tc_load4<CG>(a_dst + pl * kATileBytes, tmA, bar, m0, k0, 0, pl);
                        else tc_load<CG>(a_dst + pl * kATileBytes, tmA, bar, k0, m0, pl);
                        if (pl == 1 && nterms == 2) break;
                        if (b_mn) tc_load4<CG>(b_dst + pl * b_bytes, tmB, bar, n0, k0, 0, pl);
                        else tc_load<CG>(b_dst + pl * b_bytes, tmB, bar, k0, n0, pl);
                    }
                }
                __syncwarp();
                if (++s == S) { s = 0; ph ^= 1u; }
            }
            for (int term = 0; !TOGETHER && term < nterms && ok; ++term) {
                // planes: 0 = hi, 1 = lo; products with a lo term first
                const int pa = nterms == 3 ? (term == 0) : !turned && term == 0;
                const int pb = nterms == 3 ? (term == 1) : turned && term == 0;
                for (int kk = 0; kk < t.nkt; ++kk) {
                    ok = mbar_wait_all(empty_bar(s), ph, &abort_flag);
                    if (!ok) { abort_flag = 1; if (lane == 0) atomicExch(tab.err, 1); break; }
                    const uint32_t a_dst = tiles + (uint32_t)s * slot_bytes;
                    const uint32_t bar = CG == 2 ? cluster_addr(full_bar(s), 0) : full_bar(s);
                    const int k0 = (t.kt0 + kk) * BK;
                    if (elect_one()) {
                        if (rank == 0) mbar_expect_tx(full_bar(s), bytes);
                        if (a_mn) tc_load4<CG>(a_dst, tmA, bar, m0, k0, 0, pa);
                        else tc_load<CG>(a_dst, tmA, bar, k0, m0, pa);
                        if (b_mn) tc_load4<CG>(a_dst + kATileBytes, tmB, bar, n0, k0, 0, pb);
                        else tc_load<CG>(a_dst + kATileBytes, tmB, bar, k0, n0, pb);
                    }
                    __syncwarp();
                    if (++s == S) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // ---- MMA issuer ----------------------------------------------------------------
            const uint64_t dk = smem_desc_k_sw128(tiles), dm = smem_desc_mn_sw128(tiles);
            const uint32_t k_hi = (uint32_t)(dk >> 32), m_hi = (uint32_t)(dm >> 32), k_lo = (uint32_t)dk, m_lo = (uint32_t)dm;
            uint32_t n_local = 0, ph = 0;
            int s = 0, pi = 0;
            bool ok = true;
            for (int item = take(0); item >= 0 && ok; item = take(++n_local)) {
                const TcItem t = tc_item(sp, tab.n, item, pi);
                const TcTile& P = sp[pi];
                const uint32_t idesc = idesc_f16(CG * BM, P.BN, P.a_mn, P.b_mn);
                const uint32_t a_step = P.a_mn ? 128u : 2u, b_step = P.b_mn ? 128u : 2u;   // 16 k further, in 16-byte units
                const uint32_t a_hi = P.a_mn ? m_hi : k_hi, b_hi = P.b_mn ? m_hi : k_hi;
                const uint32_t a0 = P.a_mn ? m_lo : k_lo, b0 = (P.b_mn ? m_lo : k_lo) + (kATileBytes >> 4);
                const int total = P.nterms * t.nkt, first_hi = total - t.nkt;
                const uint32_t acc = n_local & 1u, aph = (n_local >> 1) & 1u;
                ok = mbar_wait_all(acc_empty(acc), aph ^ 1u, &abort_flag);
                if (!ok) { abort_flag = 1; if (lane == 0) atomicExch(tab.err, 4); break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * acc_cols;
                for (int j = 0; TOGETHER && j < t.nkt; ++j) {
                    ok = mbar_wait_all(full_bar(s), ph, &abort_flag);
                    if (!ok) { abort_flag = 1; if (lane == 0) atomicExch(tab.err, 2); break; }
                    tc_fence_after();
                    const uint32_t off = ((uint32_t)s * slot_bytes) >> 4;
                    const uint32_t a_lo = a0 + off, b_lo = b0 + off + (kATileBytes >> 4), b_next = (uint32_t)P.b_bytes >> 4;
                    if (elect_one()) {
                        const uint32_t more = j != 0 ? 1u : 0u;
#pragma unroll
                        for (int kk = 0; kk < BK / 16; ++kk)           // hi.hi
                            umma_f16<CG>(d_tmem, a_lo + a_step * kk, a_hi, b_lo + b_step * kk, b_hi, idesc, kk ? 1u : more);
#pragma unroll
                        for (int kk = 0; kk < BK / 16; ++kk)           // lo.hi
                            umma_f16<CG>(d_tmem + lo_cols, a_lo + (kATileBytes >> 4) + a_step * kk, a_hi, b_lo + b_step * kk, b_hi, idesc, kk ? 1u : more);
                        if (P.nterms == 3) {
#pragma unroll
                            for (int kk = 0; kk < BK / 16; ++kk)       // hi.lo
                                umma_f16<CG>(d_tmem + lo_cols, a_lo + a_step * kk, a_hi, b_lo + b_next + b_step * kk, b_hi, idesc, 1u);
                        }
                        tc_commit<CG>(empty_bar(s));
                        if (j == t.nkt - 1) tc_commit<CG>(acc_full(acc));
                    }
                    __syncwarp();
                    if (++s == S) { s = 0; ph ^= 1u; }
                }
                for (int j = 0; !TOGETHER && j < total; ++j) {
                    ok = mbar_wait_all(full_bar(s), ph, &abort_flag);
                    if (!ok) { abort_flag = 1; if (lane == 0) atomicExch(tab.err, 2); break; }
                    tc_fence_after();
                    const uint32_t off = ((uint32_t)s * slot_bytes) >> 4;
                    const uint32_t a_lo = a0 + off, b_lo = b0 + off;
                    if (elect_one()) {
                        if (j == first_hi) umma_f16_down12<CG>(d_tmem, a_lo, a_hi, b_lo, b_hi, idesc);
                        else umma_f16<CG>(d_tmem, a_lo, a_hi, b_lo, b_hi, idesc, j != 0 ? 1u : 0u);
#pragma unroll
                        for (int kk = 1; kk < BK / 16; ++kk)
                            umma_f16<CG>(d_tmem, a_lo + a_step * kk, a_hi, b_lo + b_step * kk, b_hi, idesc, 1u);
                        tc_commit<CG>(empty_bar(s));
                        if (j == total - 1) tc_commit<CG>(acc_full(acc));
                    }
                    __syncwarp();
                    if (++s == S) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else {
        // ---- epilogue warps: TMEM -> registers -> shared memory -> global ---------------------------
        const int q = warp & 3;                        // TMEM lane quarter this warp may read
        const uint32_t my_stage = staging + (uint32_t)q * 8192u;
        uint32_t n_local = 0, n_store = 0;
        int pi = 0, at = -1, g = 0;
        // The row's 2^-s of an item, and the factors of its first 64 columns, lane = column (2^-s of the rows of B, or col_scale: no
        // product has both), are fetched one item ahead, further columns 64 ahead: read where they are used, their latency was 15 to 25 %
        // of products with short main loops.
        auto row_bits = [&](const TcTile& P, const TcItem& t) {
            const int row = (t.mt * CG + (int)rank) * BM + q * 32 + lane;
            const float* f = !(TURNED && P.turned) ? P.a_inv : P.splits == 1 ? P.col_scale : nullptr;
            return f && row < P.M ? __float_as_int(__ldg(f + row)) : 0x3F800000;
        };
        auto columns = [&](const TcTile& P) { return P.b_inv ? P.b_inv : P.splits == 1 ? P.col_scale : nullptr; };
        auto column = [&](const float* f, int c, int N) { return f && c < N ? __ldg(f + c) : 1.0f; };
        TcItem t = {}, t_next = {};
        int inv_bits = 0, inv_next = 0, pi_next = 0;
        float col[2], col_next[2] = {1.0f, 1.0f};
        int item = take(0), item_next = -1;
        auto ahead = [&](int item) {
            if (item < 0) return;
            t_next = tc_item(sp, tab.n, item, pi_next);
            const TcTile& P = sp[pi_next];
            const float* f = columns(P);
            inv_next = row_bits(P, t_next);
            col_next[0] = column(f, t_next.nt * P.BN + lane, P.N);
            col_next[1] = column(f, t_next.nt * P.BN + 32 + lane, P.N);
        };
        ahead(item);
        for (; item >= 0; item = item_next, ++n_local) {
            t = t_next; pi = pi_next; inv_bits = inv_next;
            col[0] = col_next[0]; col[1] = col_next[1];
            item_next = take(n_local + 1);     // drawn when the copies of this item have been issued: before its accumulator is full
            ahead(item_next);
            const TcTile& P = sp[pi];
            const float* factors = columns(P);
            if (pi != at) {
                g = P.words ? terms_g(P.words) : 0;
                at = pi;
            }
            // undo the powers of two of the split: the row's and g in two halves, so that no step leaves fp32 unless the result does
            const int e = max(-252, (inv_bits >> 23) - 127 - g), e1 = e >> 1;
            const bool turned = TURNED && P.turned;
            const float r1 = pow2(e1), r2 = turned ? __int_as_float(inv_bits) : pow2(e - e1);      // turned: the row's scale
            const CUtensorMap* tmC = &tab.maps[3 * pi + 2];
            const uint32_t acc = n_local & 1u, aph = (n_local >> 1) & 1u;
            const bool was = !abort_flag;
            if (!__all_sync(0xffffffffu, was)) break;
            if (!mbar_wait_warp(acc_full(acc), aph, &abort_flag)) { abort_flag = 1; if (lane == 0) atomicExch(tab.err, 3); break; }
            tc_fence_after();
            const int n0 = t.nt * P.BN, row0 = (t.mt * CG + (int)rank) * BM + q * 32;
            const int ncols = min(P.BN, P.N - n0), M = P.M;
            for (int c0 = 0; c0 < ncols; c0 += 64) {
                uint32_t r[2][32];
                float col_later[2] = {1.0f, 1.0f};
                if (c0 + 64 < ncols) {
                    col_later[0] = column(factors, n0 + c0 + 64 + lane, P.N);
                    col_later[1] = column(factors, n0 + c0 + 96 + lane, P.N);
                }
                const uint32_t t_addr = tmem_base + acc * acc_cols + ((uint32_t)(q * 32) << 16) + (uint32_t)c0;
                tmem_ld32(t_addr, r[0]);
                if (c0 + 32 < ncols) tmem_ld32(t_addr + 32, r[1]);
                tmem_ld_wait();
                if (TOGETHER) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (c0 + 32 * h >= ncols) break;
                        uint32_t l[32];
                        tmem_ld32(t_addr + lo_cols + 32 * h, l);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            r[h][j] = __float_as_uint(fmaf(__uint_as_float(l[j]), 1.0f / (1 << kLoShift), __uint_as_float(r[h][j])));
                    }
                }
                if (c0 + 64 >= ncols) {                // the accumulator is in registers: release it
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (CG == 1) mbar_arrive(acc_empty(acc));
                        else asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr(acc_empty(acc), 0)) : "memory");
                    }
                }
                if (row0 >= M) continue;               // rows of the padding: nothing to store
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int cc = c0 + 32 * h;
                    if (cc >= ncols) break;
                    const uint32_t buf = my_stage + (n_store & 1u) * 4096u;
                    ++n_store;
                    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");     // the store before last has read this buffer
                    __syncwarp();
                    if (turned) {
                        // the power of two of a column (a row of C) in two halves around the scale; a lane's values go down a column of the box
                        const int ce = (__float_as_int(col[h]) >> 23) - 127, ce1 = ce >> 1;
                        const float k1 = pow2(ce1), k2 = pow2(ce - ce1);
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            const float v = __uint_as_float(r[h][j]) * __shfl_sync(0xffffffffu, k1, j) * r2 * __shfl_sync(0xffffffffu, k2, j);
                            asm volatile("st.shared.f32 [%0], %1;" ::"r"(buf + (uint32_t)j * 128u + (uint32_t)(((lane >> 2) ^ (j & 7)) << 4) + (uint32_t)((lane & 3) << 2)),
                                         "f"(v) : "memory");
                        }
                    } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) r[h][j] = __float_as_uint(__uint_as_float(r[h][j]) * r1);
                    if (factors) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) r[h][j] = __float_as_uint(__uint_as_float(r[h][j]) * __shfl_sync(0xffffffffu, col[h], j));
                    }
#pragma unroll
                    for (int j = 0; j < 32; ++j) r[h][j] = __float_as_uint(__uint_as_float(r[h][j]) * r2);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                                     ::"r"(buf + (uint32_t)lane * 128u + (uint32_t)((j ^ (lane & 7)) << 4)), "r"(r[h][4 * j]), "r"(r[h][4 * j + 1]),
                                       "r"(r[h][4 * j + 2]), "r"(r[h][4 * j + 3]) : "memory");
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                                     ::"l"(reinterpret_cast<uint64_t>(tmC)), "r"(buf), "r"(turned ? row0 : n0 + cc), "r"(turned ? n0 + cc : row0), "r"(t.split) : "memory");
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                }
                col[0] = col_later[0]; col[1] = col_later[1];
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    __syncwarp();
    if (abort_flag) {
        // gave up: let copies that are still in flight land before the shared memory is released
        const unsigned long long t0 = clock64();
        while (clock64() - t0 < 2000000ull) {}
    }
    tc_fence_before();
    if (CG == 2) cluster_sync();
    else __syncthreads();
    if (warp == 1) {
        if (CG == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
    // the last one to leave sets the counter back for the next launch: everyone has drawn for the last time
    if (rank == 0 && threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(queue + 1, 1) == (int)gridDim.x / CG - 1) { queue[0] = 0; queue[1] = 0; }
    }
}

// C[m,n] = scale[n] * sum_z partial[z][m][n], z ascending (deterministic split-K reduction).
__global__ void splitk_reduce_kernel(const float* __restrict__ partial, float* __restrict__ C,
                                     const float* __restrict__ col_scale, int M, int N, int ldc, int splits) {
    const size_t n4 = (size_t)M * (N / 4);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x) {
        const int m = (int)(i / (N / 4)), c = (int)(i % (N / 4)) * 4;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int z = 0; z < splits; ++z) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(partial + ((size_t)z * M + m) * N + c));
            acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
        if (col_scale) {
            const float4 s = __ldg(reinterpret_cast<const float4*>(col_scale + c));
            acc.x *= s.x; acc.y *= s.y; acc.z *= s.z; acc.w *= s.w;
        }
        *reinterpret_cast<float4*>(C + (size_t)m * ldc + c) = acc;
    }
}

// ---- pre-pass 1: a magnitude for the tensors that complete another's row scales ---------------------------------
// Reading a whole tensor for its maximum costs half of what splitting it does (25 us of 67 us for 16384 x 2048), so the choice is
// made from a sample: the largest of up to 16384 elements spread over rows and columns, raised by 2^kSampleRoom.  The split itself sees every
// element and records the exact maximum; a third launch, empty unless some tensor is larger than fp16 holds, splits those
// again.  Small tensors are sampled whole.  With the room the terms keep all bits of elements down to 2^-20 of the sample's
// maximum and are off by less than 2^-42 of it below.
constexpr int kSampleRoom = 8;
constexpr int kSplitCap = 128;
struct SplitTensor {
    const float* src;
    const float* col_scale;        // of planes_s
    __half* planes;                // terms [2][R][ld] of src, or null
    __half* planes_s;              // terms of src . col_scale, or null
    float* row_inv;                // 2^-s of the rows of planes; null: planes are scaled by 2^(g - s_t) of comp and words
    float* row_inv_s;              // of the rows of planes_s
    const float* comp;             // 2^-s_t of the partner's rows, or null
    uint32_t* words;
    int R, Cc, ld, vec;            // vec: rows of src and col_scale start on 16-byte boundaries
    int rows_per_chunk;            // whole rows, at most SplitShape::kUnits units; 0: a row is larger
    uint32_t magic;                // ceil(2^32 / units per row); 0: one
};
struct SplitGroup {
    int n;
    int chunk_begin[kSplitCap + 1];
    SplitTensor t[kSplitCap];
};
constexpr int kSplitRows = 256;                     // rows per chunk at most
// NT threads per block: units of 8 columns per thread and chunk, chunks in shared memory (0: loaded to registers), blocks per SM
template <int NT> struct SplitShape;
template <> struct SplitShape<256> { static constexpr int kPer = 2, kUnits = 512, kStages = 2, kBlocks = 5, kSmem = 2 * 512 * 32; };
template <> struct SplitShape<1024> { static constexpr int kPer = 4, kUnits = 4096, kStages = 0, kBlocks = 1, kSmem = 0; };

__device__ __forceinline__ uint32_t finite_bits(float v) {
    const uint32_t b = __float_as_uint(v) & 0x7FFFFFFFu;
    return b < 0x7F800000u ? b : 0u;
}

__global__ void __launch_bounds__(512) sample_magnitude_kernel(const __grid_constant__ SplitGroup g) {
    const SplitTensor& T = g.t[blockIdx.x];
    if (!T.words) return;
    const long long total = (long long)T.R * T.Cc;
    const long long units = total >> 2, step = units > kSampleUnits ? units / kSampleUnits : 1;       // units of 4 consecutive elements
    uint32_t m = 0;
    auto row_exp = [&](long long r) { return T.comp ? exp_of(__ldg(T.comp + r)) : 0; };
    const long long used = step > 1 ? min(units / step, 2ll * kSampleUnits) : units;        // (u + 1) * step <= units; at most 8191 where step is 1
    // a thread's loads all at once (taken two at a time, and with four divisions per unit, the launch took 19 us for 84 tensors)
    if (T.vec && used * step * 4 < 0x7fffffffll) {               // a unit lies in one row
        const int n = (int)used;
        for (int u0 = threadIdx.x; u0 < n; u0 += 8 * 512) {
            float4 v[8];
            int x[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int e = 4 * (int)sample_unit(min(u0 + k * 512, n - 1), step);
                v[k] = __ldg(reinterpret_cast<const float4*>(T.src + e));
                x[k] = row_exp((uint32_t)e / (uint32_t)T.Cc);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k)
                m = max(m, word_of(max(max(finite_bits(v[k].x), finite_bits(v[k].y)), max(finite_bits(v[k].z), finite_bits(v[k].w))), x[k]));
        }
    } else {
        for (long long u = threadIdx.x; u < used; u += 512)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const long long e = sample_unit(u, step) * 4 + k;
                m = max(m, word_of(finite_bits(__ldg(T.src + e)), row_exp(e / T.Cc)));
            }
    }
    for (long long e = (units << 2) + threadIdx.x; e < total; e += 512) m = max(m, word_of(finite_bits(__ldg(T.src + e)), row_exp(e / T.Cc)));
    m = __reduce_max_sync(0xffffffffu, m);
    __shared__ uint32_t w0[16];
    if ((threadIdx.x & 31) == 0) w0[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t a = 0;
        for (int w = 0; w < 16; ++w) a = max(a, w0[w]);
        T.words[0] = a && step > 1 ? a + kSampleRoom : a;
        T.words[1] = 0u;
    }
}

// ---- pre-pass 2: fp32 [R, Cc] -> fp16 terms, the rows' scales and the exact maxima -------------------------------
// HBM-bound: 4 bytes read, 4 written per element and output.  A block takes chunks of whole rows, units of 8 columns (one
// 128-bit store per term and unit) that stay in registers between the rows' maxima, found through shared memory, and
// the split.  All tensors of a step in one launch; FIX: only those whose first g did not hold.
//   256 threads, rows up to 4096 columns: the chunk is one contiguous piece of memory that cp.async brings one chunk ahead, five
//       blocks per SM.  42 layers at 8192 tokens: X 160 us at 5.8 TB/s, dY and dY . scale 308 at 5.5 (issue slots 70 % busy).  Larger
//       chunks or three of them in flight with fewer blocks: 1 to 8 % of the step slower; chunks half as large 8 %.
//   1024 threads, rows up to 32768 columns: a chunk is loaded straight to the registers of a block that fills the SM.  4096 rows of 32000:
//       163 us at 6.1 TB/s; with the row read twice, the second time from L2, 235 (five blocks per SM: half of it came from
//       memory again) to 263.
// Still wider rows are read twice.
// eight scaled values as terms; lo of an infinity is NaN
__device__ __forceinline__ void split_terms8(const float (&a)[8], uint4* __restrict__ hi, uint4* __restrict__ lo) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const __half2 hh = __floats2half2_rn(a[2 * k], a[2 * k + 1]);
        const float2 back = __half22float2(hh);
        const __half2 ll = __floats2half2_rn((a[2 * k] - back.x) * (float)(1 << kLoShift), (a[2 * k + 1] - back.y) * (float)(1 << kLoShift));
        h[k] = *reinterpret_cast<const uint32_t*>(&hh);
        l[k] = *reinterpret_cast<const uint32_t*>(&ll);
    }
    *hi = make_uint4(h[0], h[1], h[2], h[3]);
    *lo = make_uint4(l[0], l[1], l[2], l[3]);
}
__device__ __forceinline__ uint32_t max_bits8(const float (&v)[8]) {       // of the largest finite magnitude
    const float m = fmaxf(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))),
                          fmaxf(fmaxf(fabsf(v[4]), fabsf(v[5])), fmaxf(fabsf(v[6]), fabsf(v[7]))));
    uint32_t b = __float_as_uint(m);           // NaN only where all are
    if (b >= 0x7F800000u) {
        b = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) b = max(b, finite_bits(v[q]));
    }
    return b;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void load8(const float* src, int left, bool vec, float (&v)[8]) {
    if (vec && left >= 8) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(src)), b = __ldg(reinterpret_cast<const float4*>(src) + 1);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = q < left ? __ldg(src + q) : 0.0f;
    }
}
__device__ __forceinline__ int tensor_of_chunk(const SplitGroup& g, int from, int ch) {
    while (ch >= g.chunk_begin[from + 1]) ++from;
    return from;
}
// ROWS: every tensor has planes scaled by row and no others
template <bool FIX, bool ROWS, int NT>
__global__ void __launch_bounds__(NT, SplitShape<NT>::kBlocks) split_terms_kernel(const __grid_constant__ SplitGroup g) {
    constexpr int kPer = SplitShape<NT>::kPer, kUnits = SplitShape<NT>::kUnits, kStages = SplitShape<NT>::kStages;
    auto redo = [&](int t) { return g.t[t].words && terms_redone(__ldg(g.t[t].words), __ldg(g.t[t].words + 1)); };
    if (FIX) {
        const int t = threadIdx.x;              // kSplitCap <= 256
        if (!__syncthreads_or(t < g.n && redo(t))) return;
    }
    // maxima of a chunk's rows, of src and of src . col_scale.  Three sets in turn: the one of chunk i + 2 is cleared between the
    // barriers of chunks i and i + 1, when all have read chunk i - 1's and none writes chunk i + 2's.
    extern __shared__ __align__(16) float ring[];      // [kStages][kUnits * 8]
    __shared__ uint32_t row_max[3][2][kSplitRows];
    for (int i = threadIdx.x; i < 3 * 2 * kSplitRows; i += NT) (&row_max[0][0][0])[i] = 0u;
    __syncthreads();
    const int total = g.chunk_begin[g.n], tid = threadIdx.x, lane = tid & 31;
    int pch = blockIdx.x, pti = 0, pslot = 0, slot = 0;    // next chunk to fetch, its tensor and slot; slot of the current chunk
    auto fetch = [&]() {                       // one group per chunk, empty where a chunk is read directly
        if (pch < total) {
            pti = tensor_of_chunk(g, pti, pch);
            const SplitTensor& T = g.t[pti];
            if (T.vec && T.rows_per_chunk && (!FIX || redo(pti))) {
                const int r0 = (pch - g.chunk_begin[pti]) * T.rows_per_chunk, n4 = min(T.rows_per_chunk, T.R - r0) * (T.Cc >> 2);
                const float4* src = reinterpret_cast<const float4*>(T.src + (size_t)r0 * T.Cc) + tid;
                const uint32_t dst = smem_u32(ring + pslot * (kUnits * 8)) + 16u * tid;
#pragma unroll
                for (int k = 0; k < 2 * kPer; ++k)
                    if (tid + NT * k < n4) cp_async16(dst + 16u * NT * k, src + NT * k);
            }
            pch += gridDim.x;
        }
        pslot = pslot == kStages - 1 ? 0 : pslot + 1;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int i = 0; i < kStages - 1; ++i) fetch();
    int ti = -1, first = 0, last = 0, set = 0;         // chunks of tensor ti
    bool skip = false;
    uint32_t chosen = 0, word = 0;             // the word that g was first chosen for; the largest of this thread's share of the tensor
    int gexp = 0;
    auto flush = [&]() {                       // only what is above counts
        if (ROWS || FIX || !__any_sync(0xffffffffu, word > chosen)) return;
        const uint32_t b = __reduce_max_sync(0xffffffffu, word);
        if (lane == 0) atomicMax(g.t[ti].words + 1, b);
    };
    for (int ch = blockIdx.x; ch < total; ch += gridDim.x) {
        if (ch >= last) {
            flush();
            ti = tensor_of_chunk(g, ti < 0 ? 0 : ti, ch);
            first = g.chunk_begin[ti]; last = g.chunk_begin[ti + 1];
            skip = FIX && !redo(ti);
            chosen = word = 0;
            if (!ROWS && g.t[ti].words) {
                word = chosen = __ldg(g.t[ti].words + (FIX ? 1 : 0));
                gexp = word_g(chosen);
            }
        }
        if (kStages) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kStages ? kStages - 2 : 0) : "memory");
            __syncthreads();                   // this chunk has landed for all; the slot before it has been read by all
            fetch();
        }
        const float* landed = ring + slot * (kUnits * 8);
        slot = slot == kStages - 1 ? 0 : slot + 1;
        if (skip) continue;
        const SplitTensor& T = g.t[ti];
        const int n8 = (T.Cc + 7) >> 3, Cc = T.Cc;
        const bool plain = ROWS || T.planes != nullptr, by_row = ROWS || T.row_inv != nullptr, scaled = !ROWS && !FIX && T.planes_s != nullptr;
        const bool maxima = (plain && by_row) || scaled;       // FIX: a tensor that is not scaled by row
        uint32_t (&rm)[2][kSplitRows] = row_max[set];
        const int r0 = T.rows_per_chunk ? (ch - first) * T.rows_per_chunk : ch - first;
        const size_t at0 = (size_t)r0 * n8, ps = (size_t)T.R * n8;       // in units: ld = 8 n8
        uint4* const p0 = reinterpret_cast<uint4*>(T.planes) + at0;
        uint4* const p1 = reinterpret_cast<uint4*>(T.planes_s) + at0;
        auto times_scale = [&](const float (&v)[8], int c, float (&a)[8]) {
            load8(T.col_scale + c, Cc - c, T.vec, a);
#pragma unroll
            for (int q = 0; q < 8; ++q) a[q] = __fmul_rn(v[q], a[q]);
        };
        // scale, split and store unit u of the chunk: columns [c, c + 8) of row r0 + r, whose maxima are m0 and m1
        auto store = [&](const float (&v)[8], int u, int r, int c, uint32_t m0, uint32_t m1) {
            float a[8];
            if (plain) {
                if (by_row) {
                    const int s = term_exp(m0);
                    const float f = pow2(s);
                    if (c == 0) T.row_inv[r0 + r] = pow2(-s);
#pragma unroll
                    for (int q = 0; q < 8; ++q) a[q] = v[q] * f;
                } else {
                    const int x = T.comp ? exp_of(__ldg(T.comp + r0 + r)) : 0;
                    // a row with finite elements other than zeros needs no more than 2^164, and below 2^-252 nothing is left of it
                    const int e = max(-252, min(252, gexp + x)), e0 = e >> 1;
                    const float f0 = pow2(e0), f1 = pow2(e - e0);
                    if (!FIX) word = max(word, word_of(max_bits8(v), x));
#pragma unroll
                    for (int q = 0; q < 8; ++q) a[q] = v[q] * f0 * f1;
                }
                split_terms8(a, p0 + u, p0 + ps + u);
            }
            if (scaled) {
                const int s = term_exp(m1);
                const float f = pow2(s);
                if (c == 0) T.row_inv_s[r0 + r] = pow2(-s);
                times_scale(v, c, a);
#pragma unroll
                for (int q = 0; q < 8; ++q) a[q] *= f;
                split_terms8(a, p1 + u, p1 + ps + u);
            }
        };
        auto unit_maxima = [&](const float (&v)[8], int c, uint32_t* m0, uint32_t* m1) {
            *m0 = *m1 = 0u;
            if (plain && by_row) *m0 = max_bits8(v);
            if (scaled) { float a[8]; times_scale(v, c, a); *m1 = max_bits8(a); }
        };
        if (T.rows_per_chunk) {
            const int units = min(T.rows_per_chunk, T.R - r0) * n8;
            float v[kPer][8];
            int rl[kPer];                 // row in the chunk
#pragma unroll
            for (int k = 0; k < kPer; ++k) {
                const int u = tid + NT * k, uc = min(u, units - 1);
                rl[k] = T.magic ? (int)__umulhi((uint32_t)uc, T.magic) : uc;       // uc n8 < 2^32: exact
                const int c = 8 * (uc - rl[k] * n8);
                if (kStages && T.vec) {
                    const float4* p = reinterpret_cast<const float4*>(landed + rl[k] * Cc + c);
                    const float4 a = p[0], b = c + 8 <= Cc ? p[1] : make_float4(0.f, 0.f, 0.f, 0.f);      // Cc % 4 == 0
                    v[k][0] = a.x; v[k][1] = a.y; v[k][2] = a.z; v[k][3] = a.w; v[k][4] = b.x; v[k][5] = b.y; v[k][6] = b.z; v[k][7] = b.w;
                } else {
                    load8(T.src + (size_t)(r0 + rl[k]) * Cc + c, Cc - c, !kStages && T.vec, v[k]);
                }
            }
            if (maxima) {
#pragma unroll
                for (int k = 0; k < kPer; ++k) {
                    // the 32 units of a warp follow one another: mostly one row, or the end of one and the start of the next
                    const int uc = min(tid + NT * k, units - 1);
                    uint32_t m0, m1;
                    unit_maxima(v[k], 8 * (uc - rl[k] * n8), &m0, &m1);
                    const int ra = __shfl_sync(0xffffffffu, rl[k], 0), rb = __shfl_sync(0xffffffffu, rl[k], 31);
                    if (rb == ra) {
                        if (plain && by_row) { const uint32_t w = __reduce_max_sync(0xffffffffu, m0); if (lane == 0) atomicMax(&rm[0][ra], w); }
                        if (scaled) { const uint32_t w = __reduce_max_sync(0xffffffffu, m1); if (lane == 0) atomicMax(&rm[1][ra], w); }
                    } else if (rb == ra + 1) {
                        const bool in = rl[k] == ra;
                        if (plain && by_row) {
                            const uint32_t w = __reduce_max_sync(0xffffffffu, in ? m0 : 0u), x = __reduce_max_sync(0xffffffffu, in ? 0u : m0);
                            if (lane < 2) atomicMax(&rm[0][ra + lane], lane ? x : w);
                        }
                        if (scaled) {
                            const uint32_t w = __reduce_max_sync(0xffffffffu, in ? m1 : 0u), x = __reduce_max_sync(0xffffffffu, in ? 0u : m1);
                            if (lane < 2) atomicMax(&rm[1][ra + lane], lane ? x : w);
                        }
                    } else {
                        if (plain && by_row) atomicMax(&rm[0][rl[k]], m0);
                        if (scaled) atomicMax(&rm[1][rl[k]], m1);
                    }
                }
                __syncthreads();
            }
#pragma unroll
            for (int k = 0; k < kPer; ++k) {
                const int u = tid + NT * k;
                if (u < units) store(v[k], u, rl[k], 8 * (u - rl[k] * n8), rm[0][rl[k]], rm[1][rl[k]]);
            }
        } else {
            const float* src = T.src + (size_t)r0 * Cc;
            if (maxima) {
                uint32_t m0 = 0, m1 = 0;
#pragma unroll 4
                for (int u = tid; u < n8; u += NT) {
                    float v[8];
                    uint32_t a, b;
                    load8(src + 8 * u, Cc - 8 * u, T.vec, v);
                    unit_maxima(v, 8 * u, &a, &b);
                    m0 = max(m0, a); m1 = max(m1, b);
                }
                m0 = __reduce_max_sync(0xffffffffu, m0); m1 = __reduce_max_sync(0xffffffffu, m1);
                if (lane == 0) { atomicMax(&rm[0][0], m0); atomicMax(&rm[1][0], m1); }
                __syncthreads();
            }
#pragma unroll 2
            for (int u = tid; u < n8; u += NT) {
                float v[8];
                load8(src + 8 * u, Cc - 8 * u, T.vec, v);
                store(v, u, 0, 8 * u, rm[0][0], rm[1][0]);
            }
        }
        if (maxima) {
            const int clear = set == 0 ? 2 : set - 1;
            for (int i = tid; i < 2 * kSplitRows; i += NT) (&row_max[clear][0][0])[i] = 0u;
            set = set == 2 ? 0 : set + 1;
        }
    }
    flush();
}

// ---- pre-pass 3: packed 6-bit state -> fp16 ternary digits T [O][ld] --------------------------------------------
// VEC (in_features % 16 == 0, 4-byte aligned rows): thread = 16 weights = three words in, 32 bytes out, two codes per
// look-up in a 4096-entry table.  16 KB per table and CTA; a 14336 x 4096 layer took 101 us with the transposing
// byte-wise form, HBM needs 25.
__device__ __forceinline__ uint32_t digit_pair(uint32_t two_codes, int lv) {
    const __half2 h = __floats2half2_rn((float)((int)(two_codes & 63u) / lv - 1), (float)((int)(two_codes >> 6) / lv - 1));
    return *reinterpret_cast<const uint32_t*>(&h);
}
constexpr int kExpandCap = 128;
struct ExpandGroup {
    int n, C;
    long long unit_begin[kExpandCap + 1];      // units of 16 weights (VEC) or of 4
    const uint8_t* state[kExpandCap];          // 6-bit state of the layer, or null: then
    const uint32_t* packed2[kExpandCap];       // its 2-bit words (field = t + 1, 16 per word; in_features % 16 == 0)
    __half* T[kExpandCap];
    int I[kExpandCap], ld[kExpandCap];
};
template <bool VEC>
__global__ void __launch_bounds__(256) expand_ternary_kernel(const __grid_constant__ ExpandGroup g) {
    __shared__ uint32_t lut[4096];
    for (int e = threadIdx.x; e < 4096; e += 256) lut[e] = digit_pair((uint32_t)e, 2 * g.C - 1);
    __syncthreads();
    const __half2 off = __floats2half2_rn(1025.0f, 1025.0f);
    const long long total = g.unit_begin[g.n];
    int li = 0;
    for (long long u = (long long)blockIdx.x * 256 + threadIdx.x; u < total; u += (long long)gridDim.x * 256) {
        while (u >= g.unit_begin[li + 1]) ++li;
        const long long i = u - g.unit_begin[li];
        if (VEC) {                                              // rows follow one another: ld == I
            uint4* o = reinterpret_cast<uint4*>(g.T[li] + 16 * i);
            if (g.state[li]) {
                const uint32_t* w = reinterpret_cast<const uint32_t*>(g.state[li]);
                const uint32_t a = __ldg(w + 3 * i), b = __ldg(w + 3 * i + 1), c = __ldg(w + 3 * i + 2);
                const uint32_t g0 = a & 0xFFFFFFu, g1 = (a >> 24) | (b << 8), g2 = (b >> 16) | (c << 16), g3 = c >> 8;
                o[0] = make_uint4(lut[g0 & 4095u], lut[g0 >> 12], lut[g1 & 4095u], lut[(g1 >> 12) & 4095u]);
                o[1] = make_uint4(lut[g2 & 4095u], lut[(g2 >> 12) & 4095u], lut[g3 & 4095u], lut[g3 >> 12]);
            } else {
                const uint32_t w = __ldg(g.packed2[li] + i);
                uint32_t h[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {                   // fp16 1024 + field in both halves, minus 1025
                    const uint32_t two = 0x64006400u | ((w >> (4 * j)) & 3u) | (((w >> (4 * j + 2)) & 3u) << 16);
                    const __half2 t = __hsub2(*reinterpret_cast<const __half2*>(&two), off);
                    h[j] = *reinterpret_cast<const uint32_t*>(&t);
                }
                o[0] = make_uint4(h[0], h[1], h[2], h[3]);
                o[1] = make_uint4(h[4], h[5], h[6], h[7]);
            }
        } else {                                                // byte-wise state access
            const uint8_t* s = g.state[li] + i * 3;
            const uint32_t w = (uint32_t)__ldg(s) | ((uint32_t)__ldg(s + 1) << 8) | ((uint32_t)__ldg(s + 2) << 16);
            const int gpr = g.I[li] >> 2;
            const long long o = i / gpr;
            *reinterpret_cast<uint2*>(g.T[li] + o * g.ld[li] + (i - o * gpr) * 4) = make_uint2(lut[w & 4095u], lut[w >> 12]);
        }
    }
}

// out[i] = sum over z of partial[z][i], z ascending, for the split-K products of a step
constexpr int kReduceCap = 128;
struct ReduceGroup {
    int n;
    long long unit_begin[kReduceCap + 1];      // float4s
    const float* partial[kReduceCap];
    float* out[kReduceCap];
    int splits[kReduceCap];
};
__global__ void __launch_bounds__(256) splitk_reduce_group_kernel(const __grid_constant__ ReduceGroup g) {
    const long long total = g.unit_begin[g.n];
    int li = 0;
    for (long long u = (long long)blockIdx.x * 256 + threadIdx.x; u < total; u += (long long)gridDim.x * 256) {
        while (u >= g.unit_begin[li + 1]) ++li;
        const long long i = u - g.unit_begin[li], n4 = g.unit_begin[li + 1] - g.unit_begin[li];
        const float4* p = reinterpret_cast<const float4*>(g.partial[li]) + i;
        float4 acc = __ldg(p);
        for (int z = 1; z < g.splits[li]; ++z) {
            const float4 v = __ldg(p + z * n4);
            acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
        reinterpret_cast<float4*>(g.out[li])[i] = acc;
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// Map over fp16 planes [P][rows][ld] with `cols` used columns, 128-byte swizzle.  K-major: dims {cols, rows, P}, box
// {64, tile_rows, 1}.  MN-major: a tile of more than 64 columns is several 128-byte wide chunks in shared memory, so a third
// dimension of stride 64 columns walks over the chunks: dims {cols, rows, chunks, P}, box {64, 64 k rows, chunks, 1}, one
// copy per tile (the lane that issues copies was the limit with one copy per chunk: 613 cycles per k-tile against 565).
// Reads beyond cols or rows return zeros; chunks after the first may run past the end of a row into the next (those
// columns of the output are clipped), or past the last row: buffers are padded by kTermPad bytes.
bool make_map(CUtensorMap* map, const TcOperand& o, int tile_rows) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    cuuint32_t estr[4] = {1, 1, 1, 1};
    const cuuint64_t plane = (cuuint64_t)o.rows * o.ld * 2;
    if (o.mn_major) {
        const int chunks = (tile_rows + 63) / 64;
        cuuint64_t dims[4] = {(cuuint64_t)o.cols, (cuuint64_t)o.rows, (cuuint64_t)chunks, (cuuint64_t)o.planes};
        cuuint64_t strides[3] = {(cuuint64_t)o.ld * 2, 128, plane};
        cuuint32_t box[4] = {64, (cuuint32_t)BK, (cuuint32_t)chunks, 1};
        return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(o.ptr), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    }
    cuuint64_t dims[3] = {(cuuint64_t)o.cols, (cuuint64_t)o.rows, (cuuint64_t)o.planes};
    cuuint64_t strides[2] = {(cuuint64_t)o.ld * 2, plane};
    cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)tile_rows, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(o.ptr), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Output [splits][M][N] fp32, written in boxes of 32 rows x 32 columns (128-byte swizzle); boxes are clipped at M and N.
bool make_out_map(CUtensorMap* map, float* c, int M, int N, int splits) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    cuuint64_t dims[3] = {(cuuint64_t)N, (cuuint64_t)M, (cuuint64_t)splits};
    cuuint64_t strides[2] = {(cuuint64_t)N * 4, (cuuint64_t)M * N * 4};
    cuuint32_t box[3] = {32, 32, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, c, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// How a product is cut.  Time of a work item in cycles: per k-tile of 64 and term, the larger of 2 BN (MMA) and the shared-
// memory traffic ((128 + B rows of the CTA) x 128 bytes, written once and read once, at 128 B/clk), plus a fixed part; the
// launch takes that times the number of waves.  Split-K adds the traffic of its partial sums.  The rule takes the cheapest of
// one CTA or a pair per tile, tile widths of 64 to 256 and the K splits.
// Accuracy: tensor-core accumulation into TMEM truncates, and the error of a product of two fp32-split operands grows
// linearly with the accumulation depth.  `depth_limit` (k-tiles of 64) bounds what one accumulator absorbs; deeper
// contractions are cut into slices that the reduction kernel adds in fp32 with round-to-nearest.
TcPlan tc_plan(int M, int N, int K, int nterms, int sm_count, int depth_limit) {
    TcPlan best = {};
    double best_cost = 1e300;
    const int ktiles = (K + BK - 1) / BK;
    const int min_splits = depth_limit > 0 ? (ktiles + depth_limit - 1) / depth_limit : 1;
    for (int cg = 1; cg <= 2; ++cg) {
        if (cg == 2 && M <= BM) break;
        const int tm = (M + cg * BM - 1) / (cg * BM), units = sm_count / cg;
        for (int bn = 64; bn <= 256; bn += 32) {
            const int tiles = tm * ((N + bn - 1) / bn);
            const double cyc = (double)nterms * (2 * bn > 2 * (128 + bn / cg) ? 2 * bn : 2 * (128 + bn / cg));
            for (int s = min_splits; s <= 64; s = s < 4 ? s + 1 : s * 5 / 4) {
                if (s > min_splits && (ktiles < 4 * s || tiles * (s - 1) >= 2 * units)) break;
                const int per = (ktiles + s - 1) / s, real = (ktiles + per - 1) / per;
                const int waves = (tiles * real + units - 1) / units;
                double cost = waves * (per * cyc + 500.0) + 12.0 * bn;
                if (real > 1) cost += ((double)(real + 1) * M * N * 4.0) / 3000.0 + 4000.0;
                if (cost < best_cost) {
                    best_cost = cost;
                    best.pair = cg == 2; best.bn = bn; best.splits = real; best.ktiles_per_split = per; best.cost = cost;
                }
            }
        }
    }
    best.workspace_bytes = best.splits > 1 ? (size_t)best.splits * M * N * sizeof(float) : 0;
    return best;
}

// The same choice for one product among many that share a launch: what counts is the sum of the items' times, so tiles
// waste least and K is split only where the accumulation depth asks for it, or `min_items` for more items.
// `together` (three terms): the three of a k-tile from one slot.  A term after the other over the whole of K reads the hi
// planes twice, and with the slices of 18 layers in flight the second time from memory (dW of 42 layers at 8192 tokens: 2.2 GB
// from memory and 9.4 GB through L2, which was its bound).  Then the lo products cannot wait for the scale-down of the first
// hi product and get an accumulator of their own, so BN stops at 128.
TcPlan tc_plan_shared(int M, int N, int K, int nterms, int cg, int depth_limit, int min_items, bool together) {
    TcPlan best = {};
    double best_cost = 1e300;
    const int ktiles = (K + BK - 1) / BK, tm = (M + cg * BM - 1) / (cg * BM);
    for (int bn = 64; bn <= (together ? 128 : 256); bn += 32) {
        const int tiles = tm * ((N + bn - 1) / bn);
        int s = depth_limit > 0 ? (ktiles + depth_limit - 1) / depth_limit : 1;
        if (depth_limit > 0)
            while (tiles * s < min_items && ktiles >= 16 * (s + 1)) ++s;
        const int per = (ktiles + s - 1) / s, real = (ktiles + per - 1) / per;
        // together: both operands are read MN-major, in whole chunks of 64; an SM takes about 28 bytes per clock out of L2
        const double cyc = together ? 2.0 * (128 + (bn / cg + 63) / 64 * 64) * 128 / 28
                                    : (double)nterms * (2 * bn > 2 * (128 + bn / cg) ? 2 * bn : 2 * (128 + bn / cg));
        const double cost = cg * ((double)tiles * real * (per * cyc + 500.0));
        if (cost < best_cost) {
            best_cost = cost;
            best.pair = cg == 2; best.bn = bn; best.splits = real; best.ktiles_per_split = per; best.together = together;
        }
    }
    best.cost = best_cost;
    best.workspace_bytes = best.splits > 1 ? (size_t)best.splits * M * N * sizeof(float) : 0;
    return best;
}

namespace {
template <int CG, int CAP, bool TOGETHER>
cudaError_t run_tc_table(const TcProblem* probs, int n, int* err_word, size_t max_smem, int sm_count, cudaStream_t stream) {
    static thread_local TcTable<CAP> tab;      // 28 KB: built in place, copied by the launch
    tab.n = n;
    tab.err = err_word;
    tab.slot_bytes = 0;
    int items = 0, bn_max = 64, want = 2;
    for (int i = 0; i < n; ++i) {
        const TcProblem& q = probs[i];
        const TcOperand &a = q.a, &b = q.b;
        const int out_rows = q.turned ? q.N : q.M, out_cols = q.turned ? q.M : q.N;
        if (q.turned ? a.planes != 1 || b.planes != 2 || !b.inv || q.plan.together : a.planes != 2 || b.planes < 1 || b.planes > 2) return cudaErrorInvalidValue;
        if ((a.words && b.words) || (out_cols & 3) || (a.ld & 7) || (b.ld & 7)) return cudaErrorInvalidValue;
        const int bn = q.plan.bn, b_rows = bn / CG;
        float* out = q.plan.splits > 1 ? q.splitk_ws : q.c;
        if (!make_map(&tab.maps[3 * i], a, BM) || !make_map(&tab.maps[3 * i + 1], b, b_rows) ||
            !make_out_map(&tab.maps[3 * i + 2], out, out_rows, out_cols, q.plan.splits)) return cudaErrorInvalidValue;
        TcTile& p = tab.p[i];
        p.col_scale = q.col_scale;
        p.a_inv = a.inv; p.b_inv = b.inv;
        p.words = a.words ? a.words : b.words;
        p.M = q.M; p.N = q.N; p.K = q.K;
        p.BN = bn;
        p.b_bytes = (b.mn_major ? (b_rows + 63) / 64 * 64 : b_rows) * BK * 2;
        p.stage_bytes = q.plan.together ? 2 * kATileBytes + b.planes * p.b_bytes : kATileBytes + p.b_bytes;
        p.a_mn = a.mn_major; p.b_mn = b.mn_major;
        p.turned = q.turned;
        p.nterms = !q.turned && b.planes == 2 ? 3 : 2;
        p.ktiles_per_split = q.plan.ktiles_per_split; p.splits = q.plan.splits;
        p.tiles_m = (q.M + CG * BM - 1) / (CG * BM); p.tiles_n = (q.N + bn - 1) / bn;
        p.group_m = 12 / CG;                   // 12 row tiles x 12 column tiles in flight on 148 SMs
        p.item_begin = items;
        items += p.tiles_m * p.tiles_n * p.splits;
        if (p.stage_bytes > tab.slot_bytes) tab.slot_bytes = p.stage_bytes;
        if (bn > bn_max) bn_max = bn;
        const int slots = (q.plan.together ? 1 : p.nterms) * p.ktiles_per_split;
        if (slots > want) want = slots;
    }
    tab.n_items = items;
    tab.acc_cols = 64;
    while (tab.acc_cols < bn_max) tab.acc_cols *= 2;
    if (TOGETHER) tab.acc_cols *= 2;
    if (tab.acc_cols > 256) return cudaErrorInvalidValue;
    int stages = (int)((max_smem - 1024 - sizeof(TcTile) * CAP - 2048 - kStageBytes) / (size_t)tab.slot_bytes);
    if (stages > kMaxStages) stages = kMaxStages;
    // Two accumulators of one CTA take 2 * pow2(BN) TMEM columns of the SM's 512.  Narrow tiles (BN <= 128) with short main
    // loops leave room for a second resident CTA, which doubles the loads in flight where the loop is latency-bound; then
    // each CTA gets half the shared memory.
    bool two_ctas = false;
    if (CG == 1 && !TOGETHER && bn_max <= 128 && want <= 32 && items > sm_count) {
        const int half = (int)((max_smem / 2 - 2048 - sizeof(TcTile) * CAP - 1024 - kStageBytes) / (size_t)tab.slot_bytes);
        if (half >= 3) { two_ctas = true; if (half < stages) stages = half; }
    }
    if (stages > want) stages = want;
    if (stages < 2) return cudaErrorInvalidConfiguration;
    tab.stages = stages;
    const size_t smem = (size_t)stages * tab.slot_bytes + 1024 + kStageBytes;
    bool turned = false;
    for (int i = 0; i < n; ++i) turned = turned || probs[i].turned;
    const auto kern = turned ? tc_gemm_kernel<CG, CAP, TOGETHER, !TOGETHER> : tc_gemm_kernel<CG, CAP, TOGETHER, false>;
    cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), turned ? 41 + 2 * (CG == 2) + (CAP > 1) : TOGETHER ? (CG == 2 ? 30 : 31) : CG == 2 ? (CAP > 1 ? 24 : 16) : (CAP > 1 ? 25 : 4), max_smem);
    if (e != cudaSuccess) return e;
    int units = (sm_count / CG) * (two_ctas ? 2 : 1);
    if (units > items) units = items;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(units * CG));
    cfg.blockDim = dim3(kTcThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = CG == 2 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, tab);
}
}  // namespace

// Products in launches of up to kTcCap each; all of a launch have the same plan.pair and plan.together.
cudaError_t launch_tc_products(const TcProblem* probs, int n, int* err_word, size_t max_smem, int sm_count, cudaStream_t stream,
                               int* launches) {
    for (int i = 0; i < n;) {
        int k = 1;
        while (i + k < n && k < kTcCap && probs[i + k].plan.pair == probs[i].plan.pair && probs[i + k].plan.together == probs[i].plan.together) ++k;
        const bool pair = probs[i].plan.pair;
        cudaError_t e;
        if (probs[i].plan.together)
            e = pair ? run_tc_table<2, kTcCap, true>(probs + i, k, err_word, max_smem, sm_count, stream)
                     : run_tc_table<1, kTcCap, true>(probs + i, k, err_word, max_smem, sm_count, stream);
        else if (k == 1)
            e = pair ? run_tc_table<2, 1, false>(probs + i, 1, err_word, max_smem, sm_count, stream)
                     : run_tc_table<1, 1, false>(probs + i, 1, err_word, max_smem, sm_count, stream);
        else
            e = pair ? run_tc_table<2, kTcCap, false>(probs + i, k, err_word, max_smem, sm_count, stream)
                     : run_tc_table<1, kTcCap, false>(probs + i, k, err_word, max_smem, sm_count, stream);
        if (e != cudaSuccess) return e;
        ++*launches;
        i += k;
    }
    return cudaSuccess;
}

cudaError_t launch_splitk_reduce_group(const float* const* partial, float* const* out, const long long* elements, const int* splits,
                                       int n, int sm_count, cudaStream_t stream, int* launches) {
    for (int done = 0; done < n;) {
        ReduceGroup g;
        const int take = n - done < kReduceCap ? n - done : kReduceCap;
        long long units = 0;
        for (int j = 0; j < take; ++j) {
            g.unit_begin[j] = units;
            g.partial[j] = partial[done + j]; g.out[j] = out[done + j]; g.splits[j] = splits[done + j];
            units += elements[done + j] / 4;
        }
        g.unit_begin[take] = units;
        g.n = take;
        long long blocks = (units + 255) / 256;
        if (blocks > (long long)sm_count * 8) blocks = (long long)sm_count * 8;
        splitk_reduce_group_kernel<<<(int)blocks, 256, 0, stream>>>(g);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        ++*launches;
        done += take;
    }
    return cudaSuccess;
}

cudaError_t launch_splitk_reduce(const float* partial, float* c, const float* col_scale, int M, int N, int ldc,
                                 int splits, cudaStream_t stream) {
    const size_t n4 = (size_t)M * (N / 4);
    int blocks = (int)((n4 + 255) / 256);
    if (blocks > 148 * 8) blocks = 148 * 8;
    splitk_reduce_kernel<<<blocks, 256, 0, stream>>>(partial, c, col_scale, M, N, ldc, splits);
    return cudaGetLastError();
}

namespace {
template <int NT>
cudaError_t run_split(const SplitGroup& g, bool rows_only, bool sampled, int sm_count, cudaStream_t stream) {
    using S = SplitShape<NT>;
    const int chunks = g.chunk_begin[g.n], grid = chunks < sm_count * S::kBlocks ? chunks : sm_count * S::kBlocks;
    if (rows_only) split_terms_kernel<false, true, NT><<<grid, NT, S::kSmem, stream>>>(g);
    else split_terms_kernel<false, false, NT><<<grid, NT, S::kSmem, stream>>>(g);
    if (sampled) split_terms_kernel<true, false, NT><<<grid, NT, S::kSmem, stream>>>(g);
    return cudaGetLastError();
}
}  // namespace

// Tensors of their own first, then those that complete the row scales of one of these.
cudaError_t launch_split_terms(const SplitDesc* d, int n, int sm_count, cudaStream_t stream, int* launches) {
    for (int dependent = 0; dependent < 2; ++dependent) {
        for (int i = 0; i < n;) {
            SplitGroup g;
            g.n = 0;
            bool words = false, rows_only = true, sampled = false, wide = false;     // a tensor sampled whole needs no second look
            for (; i < n && g.n < kSplitCap; ++i) {
                const SplitDesc& q = d[i];
                if ((q.comp != nullptr) != (dependent == 1)) continue;
                SplitTensor& t = g.t[g.n++];
                t.src = q.src; t.col_scale = q.planes_s ? q.col_scale : nullptr;
                t.planes = static_cast<__half*>(q.planes); t.planes_s = static_cast<__half*>(q.planes_s);
                t.row_inv = q.row_inv; t.row_inv_s = q.row_inv_s; t.comp = q.comp;
                t.words = q.planes && !q.row_inv ? q.words : nullptr;
                t.R = q.rows; t.Cc = q.cols; t.ld = q.ld;
                t.vec = (q.cols & 3) == 0 && (reinterpret_cast<uintptr_t>(q.src) & 15) == 0 &&
                        (t.col_scale == nullptr || (reinterpret_cast<uintptr_t>(t.col_scale) & 15) == 0);
                if ((q.cols + 7) / 8 > SplitShape<256>::kUnits) wide = true;
                if (t.words) words = true;
                if (!t.planes || !t.row_inv || t.planes_s) rows_only = false;
                if (t.words && (long long)q.rows * q.cols / 4 >= 2 * kSampleUnits) sampled = true;
            }
            if (g.n == 0) continue;
            const int units = wide ? SplitShape<1024>::kUnits : SplitShape<256>::kUnits;
            long long chunks = 0;
            for (int j = 0; j < g.n; ++j) {
                SplitTensor& t = g.t[j];
                const int n8 = (t.Cc + 7) / 8;
                t.rows_per_chunk = n8 > units ? 0 : units / n8 < kSplitRows ? units / n8 : kSplitRows;
                t.magic = n8 == 1 ? 0u : (uint32_t)((0x100000000ull + (uint32_t)n8 - 1) / (uint32_t)n8);
                g.chunk_begin[j] = (int)chunks;
                chunks += t.rows_per_chunk ? ((long long)t.R + t.rows_per_chunk - 1) / t.rows_per_chunk : t.R;
                if (chunks > 0x3fffffff) return cudaErrorInvalidValue;
            }
            g.chunk_begin[g.n] = (int)chunks;
            if (words) sample_magnitude_kernel<<<g.n, 512, 0, stream>>>(g);
            const cudaError_t e = wide ? run_split<1024>(g, rows_only, sampled, sm_count, stream) : run_split<256>(g, rows_only, sampled, sm_count, stream);
            if (e != cudaSuccess) return e;
            *launches += 1 + (words ? 1 : 0) + (sampled ? 1 : 0);
        }
    }
    return cudaSuccess;
}

cudaError_t launch_expand_ternary(const ExpandDesc* d, int n, int C, int sm_count, cudaStream_t stream, int* launches) {
    for (int vec = 0; vec < 2; ++vec) {        // layers with aligned rows of whole words, then the others
        for (int i = 0; i < n;) {
            ExpandGroup g;
            g.n = 0; g.C = C;
            long long units = 0;
            for (; i < n && g.n < kExpandCap; ++i) {
                const bool v = d[i].I % 16 == 0 && d[i].ld == d[i].I && (!d[i].state || (reinterpret_cast<uintptr_t>(d[i].state) & 3) == 0);
                if (v != (vec == 0)) continue;
                g.unit_begin[g.n] = units;
                g.state[g.n] = d[i].state; g.packed2[g.n] = d[i].packed2; g.T[g.n] = static_cast<__half*>(d[i].T);
                g.I[g.n] = d[i].I; g.ld[g.n] = d[i].ld;
                units += (long long)d[i].O * (d[i].I / (v ? 16 : 4));
                ++g.n;
            }
            if (g.n == 0) continue;
            g.unit_begin[g.n] = units;
            long long blocks = (units + 255) / 256;
            if (blocks > (long long)sm_count * 8) blocks = (long long)sm_count * 8;
            if (vec == 0) expand_ternary_kernel<true><<<(int)blocks, 256, 0, stream>>>(g);
            else expand_ternary_kernel<false><<<(int)blocks, 256, 0, stream>>>(g);
            const cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) return e;
            ++*launches;
        }
    }
    return cudaSuccess;
}

}  // namespace mcl
