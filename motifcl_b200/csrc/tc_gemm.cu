// Tensor-core contractions of the counter-linear path for sm_100a: tcgen05.mma with fp32
// accumulators in tensor memory (TMEM), operands staged in shared memory by TMA.
//
// One kernel serves the three products of a training step (MotifCL
// src/nn/compact_counter.cpp:233-300 and kernels/matmul.cl:413-563 compute them with fp32
// scalar FMAs) and the dense fp32 matmul:
//     Y  [tokens,out] = X  . T^T          A = terms of X    [tokens,in]     B = T [out,in]
//     dX [tokens,in ] = (dY.s) . T        A = terms of dY.s [tokens,out]    B = T [out,in], read MN-major
//     dW [out,in]     = dY^T . X          A = terms of dY, B = terms of X   both [tokens, .], read MN-major
// so every tensor is split once, in its own layout, and T is expanded once: a transposed operand is the
// same shared-memory tile with the MN-major bit of the instruction descriptor.
//
// How an fp32 tensor becomes two fp16 terms (split_terms_kernel): with m = the largest magnitude of the tensor and
// f = 2^(14 - floor(log2 m)), hi = fp16(a f) and lo = fp16((a f - hi) 2^12).  hi keeps 11 bits, the residual is at most
// half a unit of hi and keeps 11 more below its sign: |a f - hi - lo 2^-12| <= 2^-23 |a f|, the last bit of fp32 (the first
// bf16 form of this file needed three 8-bit terms for the same bits).  lo is stored 2^12 up so that it stays a normal
// number wherever hi is: elements down to 2^-28 of the largest keep all their bits, smaller ones are off by less
// than 2^-50 of it.  The lo products go into the accumulator first; the first hi product scales it down by 2^-12
// (tcgen05.mma scale-input-d), and the epilogue undoes f.  Ternary digits are exact in fp16.  Cost per product of a
// step in bf16-rate passes: Y, dX 2 (3 before), dW 3 (hi.hi + hi.lo + lo.hi; 6 before).
// The kernel is bound by the tensor pipe; its time at a stated size stands at tc_gemm_kernel.
#include <cuda.h>
#include <cuda_fp16.h>

#include "counter_codec.cuh"
#include "kernels.h"
#include "tc_ptx.cuh"

namespace mcl {
namespace {

constexpr int BM = 128;          // UMMA M
constexpr int BK = 64;           // 64 fp16 = 128 bytes = one swizzle row
constexpr int kMaxStages = 8;
constexpr int kATileBytes = BM * BK * 2;   // 16 KiB
constexpr int kLoShift = 12;               // lo terms are stored 2^12 up

struct TcParams {
    const float* col_scale;   // optional, applied when splits == 1
    const uint32_t* a_amax;   // bits of the largest magnitude of the split tensor (null: operand is unscaled)
    const uint32_t* b_amax;
    int M, N, K;
    int BN, stages, b_bytes;   // b_bytes: one CTA's share of a B tile
    int a_mn, b_mn;           // operand is stored with M / N contiguous
    int nterms;               // 2: A lo, A hi against one B plane; 3: lo.hi, hi.lo, hi.hi
    int ktiles_per_split, splits;
    int group_m;
    int* err;
};

// exponent of f (see the file header): the largest magnitude lands in [2^14, 2^15)
__device__ __forceinline__ int term_exp(uint32_t amax_bits) {
    const int e = (int)(amax_bits >> 23);
    const int s = 141 - (e < 1 ? 1 : e);
    return s > 126 ? 126 : s;
}
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

// item -> output tile and K slice.  Groups of group_m row tiles run through all column tiles before the next group, so
// that the CTAs in flight share both operands' tiles in L2.
struct TcItem { int mt, nt, split; };
__device__ __forceinline__ TcItem tc_item(int item, int tiles_m, int tiles_n, int group_m) {
    TcItem t;
    const int per_split = tiles_m * tiles_n;
    t.split = item / per_split;
    int r = item - t.split * per_split;
    const int per_group = group_m * tiles_n;
    const int g = r / per_group;
    r -= g * per_group;
    const int gm = min(group_m, tiles_m - g * group_m);
    t.nt = r / gm;
    t.mt = g * group_m + (r - t.nt * gm);
    return t;
}

// Persistent CTAs of 192 threads; work items (output tile x split-K slice) are dealt round-robin.
//   warp 0        TMA producer (one elected lane): tiles of A and B into a ring of `stages` shared-memory slots
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
// Every mbarrier wait is bounded: on time-out the kernel records an error word, skips the rest of its work, frees
// its TMEM and returns.
constexpr int kTcThreads = 192;
constexpr int kSmemSlotTcPair = 16;       // ensure_dynamic_smem: see there
constexpr int kStageBytes = 8 * 4096;      // epilogue staging: two 32 x 32 float tiles per warp

template <int CG>
__global__ void __launch_bounds__(kTcThreads) tc_gemm_kernel(const __grid_constant__ CUtensorMap tmA,
                                                             const __grid_constant__ CUtensorMap tmB,
                                                             const __grid_constant__ CUtensorMap tmC,
                                                             const TcParams p) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kMaxStages + 4];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int BN = p.BN, S = p.stages;
    const uint32_t rank = CG == 2 ? (blockIdx.x & 1u) : 0u;      // cluster of two consecutive CTAs
    const int unit = (int)blockIdx.x / CG, n_units = (int)gridDim.x / CG;
    const uint32_t staging = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t tiles = staging + kStageBytes;
    const uint32_t stage_bytes = kATileBytes + (uint32_t)p.b_bytes;
    const uint32_t bar0 = smem_u32(bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (kMaxStages + s); };
    auto acc_full = [&](int a) { return bar0 + 8u * (2 * kMaxStages + a); };
    auto acc_empty = [&](int a) { return bar0 + 8u * (2 * kMaxStages + 2 + a); };
    uint32_t acc_cols = 32;                       // columns of one accumulator (power of two >= BN)
    while ((int)acc_cols < BN) acc_cols <<= 1;
    const uint32_t tmem_cols = 2 * acc_cols;      // <= 512

    const int tiles_n = (p.N + BN - 1) / BN, tiles_m = (p.M + CG * BM - 1) / (CG * BM);
    const int ktiles = (p.K + BK - 1) / BK;
    const int n_items = tiles_m * tiles_n * p.splits;

    if (threadIdx.x == 0) {
        abort_flag = (*reinterpret_cast<volatile int*>(p.err) != 0);   // an earlier CTA gave up: do not wait at all
        for (int s = 0; s < S; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(acc_full(a), 1); mbar_init(acc_empty(a), 4 * CG); }
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
    if (CG == 2) cluster_sync();
    else __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;

    if (warp == 0) {
        // ---- TMA producer ------------------------------------------------------------------
        int s = 0;                 // ring slot and its phase, across all items of this CTA
        uint32_t ph = 1;
        bool ok = true;
        for (int item = unit; item < n_items && ok; item += n_units) {
            const TcItem t = tc_item(item, tiles_m, tiles_n, p.group_m);
            const int kt0 = t.split * p.ktiles_per_split;
            const int my_kt = min(p.ktiles_per_split, ktiles - kt0);
            const int m0 = (t.mt * CG + (int)rank) * BM, n0 = t.nt * BN + (int)rank * (BN / CG);
            for (int term = 0; term < p.nterms && ok; ++term) {
                // planes: 0 = hi, 1 = lo; products with a lo term first
                const int pa = p.nterms == 3 ? (term == 0) : (term + 1 < p.nterms);
                const int pb = p.nterms == 3 && term == 1;
                for (int kk = 0; kk < my_kt; ++kk) {
                    ok = mbar_wait_all(empty_bar(s), ph, &abort_flag);
                    if (!ok) { abort_flag = 1; if (lane == 0) atomicExch(p.err, 1); break; }
                    const uint32_t a_dst = tiles + (uint32_t)s * stage_bytes;
                    const uint32_t bar = CG == 2 ? cluster_addr(full_bar(s), 0) : full_bar(s);
                    const int k0 = (kt0 + kk) * BK;
                    if (elect_one()) {
                        if (rank == 0) mbar_expect_tx(full_bar(s), CG * stage_bytes);
                        if (p.a_mn) tc_load4<CG>(a_dst, &tmA, bar, m0, k0, 0, pa);
                        else tc_load<CG>(a_dst, &tmA, bar, k0, m0, pa);
                        if (p.b_mn) tc_load4<CG>(a_dst + kATileBytes, &tmB, bar, n0, k0, 0, pb);
                        else tc_load<CG>(a_dst + kATileBytes, &tmB, bar, k0, n0, pb);
                    }
                    __syncwarp();
                    if (++s == S) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // ---- MMA issuer ----------------------------------------------------------------
            const uint32_t idesc = idesc_f16(CG * BM, BN, p.a_mn, p.b_mn);
            const uint32_t a_step = p.a_mn ? 128u : 2u, b_step = p.b_mn ? 128u : 2u;   // 16 k further, in 16-byte units
            const uint64_t da0 = p.a_mn ? smem_desc_mn_sw128(tiles) : smem_desc_k_sw128(tiles);
            const uint64_t db0 = p.b_mn ? smem_desc_mn_sw128(tiles + kATileBytes) : smem_desc_k_sw128(tiles + kATileBytes);
            const uint32_t a_hi = (uint32_t)(da0 >> 32), b_hi = (uint32_t)(db0 >> 32), a0 = (uint32_t)da0, b0 = (uint32_t)db0;
            uint32_t n_local = 0, ph = 0;
            int s = 0;
            bool ok = true;
            for (int item = unit; item < n_items && ok; item += n_units, ++n_local) {
                const int kt0 = (item / (tiles_m * tiles_n)) * p.ktiles_per_split;
                const int my_kt = min(p.ktiles_per_split, ktiles - kt0);
                const int total = p.nterms * my_kt, first_hi = total - my_kt;
                const uint32_t acc = n_local & 1u, aph = (n_local >> 1) & 1u;
                ok = mbar_wait_all(acc_empty(acc), aph ^ 1u, &abort_flag);
                if (!ok) { abort_flag = 1; if (lane == 0) atomicExch(p.err, 4); break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * acc_cols;
                for (int j = 0; j < total; ++j) {
                    ok = mbar_wait_all(full_bar(s), ph, &abort_flag);
                    if (!ok) { abort_flag = 1; if (lane == 0) atomicExch(p.err, 2); break; }
                    tc_fence_after();
                    const uint32_t off = ((uint32_t)s * stage_bytes) >> 4;
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
        const bool scale = (p.col_scale != nullptr) && p.splits == 1;
        const float fa = p.a_amax ? pow2(-term_exp(__ldg(p.a_amax))) : 1.0f;      // undo the powers of two of the split
        const float fb = p.b_amax ? pow2(-term_exp(__ldg(p.b_amax))) : 1.0f;
        const uint32_t my_stage = staging + (uint32_t)q * 8192u;
        uint32_t n_local = 0, n_store = 0;
        for (int item = unit; item < n_items; item += n_units, ++n_local) {
            const TcItem t = tc_item(item, tiles_m, tiles_n, p.group_m);
            const uint32_t acc = n_local & 1u, aph = (n_local >> 1) & 1u;
            const bool was = !abort_flag;
            if (!__all_sync(0xffffffffu, was)) break;
            if (!mbar_wait_warp(acc_full(acc), aph, &abort_flag)) { abort_flag = 1; if (lane == 0) atomicExch(p.err, 3); break; }
            tc_fence_after();
            const int n0 = t.nt * BN, row0 = (t.mt * CG + (int)rank) * BM + q * 32;
            const int ncols = min(BN, p.N - n0);
            for (int c0 = 0; c0 < ncols; c0 += 64) {
                uint32_t r[2][32];
                const uint32_t t_addr = tmem_base + acc * acc_cols + ((uint32_t)(q * 32) << 16) + (uint32_t)c0;
                tmem_ld32(t_addr, r[0]);
                if (c0 + 32 < ncols) tmem_ld32(t_addr + 32, r[1]);
                tmem_ld_wait();
                if (c0 + 64 >= ncols) {                // the accumulator is in registers: release it
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (CG == 1) mbar_arrive(acc_empty(acc));
                        else asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr(acc_empty(acc), 0)) : "memory");
                    }
                }
                if (row0 >= p.M) continue;             // rows of the padding: nothing to store
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int cc = c0 + 32 * h;
                    if (cc >= ncols) break;
                    const uint32_t buf = my_stage + (n_store & 1u) * 4096u;
                    ++n_store;
                    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");     // the store before last has read this buffer
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float4 o = make_float4(__uint_as_float(r[h][4 * j]), __uint_as_float(r[h][4 * j + 1]),
                                               __uint_as_float(r[h][4 * j + 2]), __uint_as_float(r[h][4 * j + 3]));
                        o.x = o.x * fa * fb; o.y = o.y * fa * fb; o.z = o.z * fa * fb; o.w = o.w * fa * fb;
                        if (scale && cc + 4 * j < ncols) {            // N % 4 == 0
                            const float4 sc = __ldg(reinterpret_cast<const float4*>(p.col_scale + n0 + cc + 4 * j));
                            o.x *= sc.x; o.y *= sc.y; o.z *= sc.z; o.w *= sc.w;
                        }
                        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};"
                                     ::"r"(buf + (uint32_t)lane * 128u + (uint32_t)((j ^ (lane & 7)) << 4)), "f"(o.x), "f"(o.y), "f"(o.z), "f"(o.w) : "memory");
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                                     ::"l"(reinterpret_cast<uint64_t>(&tmC)), "r"(buf), "r"(n0 + cc), "r"(row0), "r"(t.split) : "memory");
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                }
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

// ---- pre-pass 1: largest magnitude of a tensor, and of the tensor times a per-column factor ----------------
// amax[0] = max |src|, amax[1] = max |src . col_scale| (when col_scale != null), as float bits, by atomicMax into zeroed
// words.  HBM-bound: one read.
template <bool VEC>
__global__ void __launch_bounds__(256) amax_kernel(const float* __restrict__ src, size_t R, int Cc,
                                                   const float* __restrict__ col_scale, uint32_t* __restrict__ amax) {
    constexpr int W = VEC ? 4 : 1;
    const int n = Cc / W;                                   // VEC needs Cc % 4 == 0
    const size_t total = R * (size_t)n, stride = (size_t)gridDim.x * 256;
    const size_t i0 = (size_t)blockIdx.x * 256 + threadIdx.x;
    int c = (int)(i0 % (size_t)n);
    const int step = (int)(stride % (size_t)n);
    float m0 = 0.0f, m1 = 0.0f;
#pragma unroll 4
    for (size_t i = i0; i < total; i += stride) {
        if (VEC) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(src) + i);
            m0 = fmaxf(fmaxf(m0, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
            if (col_scale) {
                const float4 s = __ldg(reinterpret_cast<const float4*>(col_scale) + c);
                m1 = fmaxf(fmaxf(m1, fmaxf(fabsf(v.x * s.x), fabsf(v.y * s.y))), fmaxf(fabsf(v.z * s.z), fabsf(v.w * s.w)));
            }
        } else {
            const float v = __ldg(src + i);
            m0 = fmaxf(m0, fabsf(v));
            if (col_scale) m1 = fmaxf(m1, fabsf(v * __ldg(col_scale + c)));
        }
        c += step;
        if (c >= n) c -= n;
    }
    uint32_t b0 = __reduce_max_sync(0xffffffffu, __float_as_uint(m0)), b1 = __reduce_max_sync(0xffffffffu, __float_as_uint(m1));
    __shared__ uint32_t w0[8], w1[8];
    if ((threadIdx.x & 31) == 0) { w0[threadIdx.x >> 5] = b0; w1[threadIdx.x >> 5] = b1; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) { b0 = max(b0, w0[w]); b1 = max(b1, w1[w]); }
        if (b0) atomicMax(amax, b0);
        if (col_scale && b1) atomicMax(amax + 1, b1);
    }
}

// ---- pre-pass 2: fp32 [R, Cc] -> fp16 terms [2][R][ld] of src (planes) and of src . col_scale (planes_s) ----------
// Thread = 8 consecutive columns: two 128-bit loads, one 128-bit store per term.  HBM-bound: 4 bytes read, 4 written per
// element and output.
__device__ __forceinline__ void split_terms8(const float (&v)[8], float f, uint4* hi, uint4* lo) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float a = v[2 * k] * f, b = v[2 * k + 1] * f;
        const __half2 hh = __floats2half2_rn(a, b);
        const float2 back = __half22float2(hh);
        const __half2 ll = __floats2half2_rn((a - back.x) * (float)(1 << kLoShift), (b - back.y) * (float)(1 << kLoShift));
        h[k] = *reinterpret_cast<const uint32_t*>(&hh);
        l[k] = *reinterpret_cast<const uint32_t*>(&ll);
    }
    *hi = make_uint4(h[0], h[1], h[2], h[3]);
    *lo = make_uint4(l[0], l[1], l[2], l[3]);
}
template <bool VEC>
__global__ void __launch_bounds__(256) split_terms_kernel(const float* __restrict__ src, int R, int Cc, int ld,
                                                          const float* __restrict__ col_scale, __half* __restrict__ planes,
                                                          __half* __restrict__ planes_s, const uint32_t* __restrict__ amax) {
    const int n8 = (Cc + 7) >> 3;
    const float f0 = planes ? pow2(term_exp(__ldg(amax))) : 0.0f, f1 = planes_s ? pow2(term_exp(__ldg(amax + 1))) : 0.0f;
    const size_t total = (size_t)R * n8, stride = (size_t)gridDim.x * 256, ps = (size_t)R * ld;
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < total; i += stride) {
        const size_t r = i / (size_t)n8;
        const int c = (int)(i - r * n8) * 8;
        const float* s = src + r * Cc + c;
        float v[8];
        if (VEC && c + 8 <= Cc) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(s)), b = __ldg(reinterpret_cast<const float4*>(s) + 1);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = c + k < Cc ? __ldg(s + k) : 0.0f;
        }
        uint4 hi, lo;
        const size_t at = r * ld + c;                       // ld % 8 == 0
        if (planes) {
            split_terms8(v, f0, &hi, &lo);
            *reinterpret_cast<uint4*>(planes + at) = hi;
            *reinterpret_cast<uint4*>(planes + ps + at) = lo;
        }
        if (planes_s) {
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = __fmul_rn(v[k], c + k < Cc ? __ldg(col_scale + c + k) : 0.0f);
            split_terms8(v, f1, &hi, &lo);
            *reinterpret_cast<uint4*>(planes_s + at) = hi;
            *reinterpret_cast<uint4*>(planes_s + ps + at) = lo;
        }
    }
}

// ---- pre-pass 3: packed 6-bit state -> fp16 ternary digits T [O][ld] --------------------------------------------
// VEC (in_features % 16 == 0, 4-byte aligned rows): thread = 16 weights = three words in, 32 bytes out, two codes per
// look-up in a 4096-entry table.  16 KB per table and CTA; a 14336 x 4096 layer took 101 us with the transposing
// byte-wise form, HBM needs 25.
__device__ __forceinline__ uint32_t digit_pair(uint32_t two_codes, int lv) {
    const __half2 h = __floats2half2_rn((float)((int)(two_codes & 63u) / lv - 1), (float)((int)(two_codes >> 6) / lv - 1));
    return *reinterpret_cast<const uint32_t*>(&h);
}
template <bool VEC>
__global__ void __launch_bounds__(256) expand_ternary_kernel(const uint8_t* __restrict__ state, int C, int O, int I,
                                                             __half* __restrict__ T, int ld) {
    __shared__ uint32_t lut[4096];
    for (int e = threadIdx.x; e < 4096; e += 256) lut[e] = digit_pair((uint32_t)e, 2 * C - 1);
    __syncthreads();
    if (VEC) {
        const size_t total = (size_t)O * (I >> 4);
        const uint32_t* w = reinterpret_cast<const uint32_t*>(state);
        for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (size_t)gridDim.x * 256) {   // ld == I here
            const uint32_t a = __ldg(w + 3 * i), b = __ldg(w + 3 * i + 1), c = __ldg(w + 3 * i + 2);
            const uint32_t g0 = a & 0xFFFFFFu, g1 = (a >> 24) | (b << 8), g2 = (b >> 16) | (c << 16), g3 = c >> 8;
            uint4* o = reinterpret_cast<uint4*>(T + 16 * i);
            o[0] = make_uint4(lut[g0 & 4095u], lut[g0 >> 12], lut[g1 & 4095u], lut[(g1 >> 12) & 4095u]);
            o[1] = make_uint4(lut[g2 & 4095u], lut[(g2 >> 12) & 4095u], lut[g3 & 4095u], lut[g3 >> 12]);
        }
    } else {
        const int gpr = I >> 2;
        const size_t total = (size_t)O * gpr;
        for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (size_t)gridDim.x * 256) {
            const uint8_t* s = state + i * 3;
            const uint32_t g = (uint32_t)__ldg(s) | ((uint32_t)__ldg(s + 1) << 8) | ((uint32_t)__ldg(s + 2) << 16);
            const size_t o = i / (size_t)gpr;
            *reinterpret_cast<uint2*>(T + o * ld + (i - o * gpr) * 4) = make_uint2(lut[g & 4095u], lut[g >> 12]);
        }
    }
}

// Same expansion from the 2-bit packed weights (field = t + 1, 16 per word): what ranks that do
// not own a layer's counter state use after the all-gather of packed weights.
__global__ void __launch_bounds__(256) expand_ternary_p2_kernel(const uint32_t* __restrict__ packed2, size_t words,
                                                                __half* __restrict__ T) {
    const __half2 off = __floats2half2_rn(1025.0f, 1025.0f);
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < words; i += (size_t)gridDim.x * 256) {
        const uint32_t w = __ldg(packed2 + i);
        uint32_t h[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {      // fp16 1024 + field in both halves, minus 1025
            const uint32_t two = 0x64006400u | ((w >> (4 * j)) & 3u) | (((w >> (4 * j + 2)) & 3u) << 16);
            const __half2 t = __hsub2(*reinterpret_cast<const __half2*>(&two), off);
            h[j] = *reinterpret_cast<const uint32_t*>(&t);
        }
        uint4* o = reinterpret_cast<uint4*>(T + 16 * i);       // in_features % 16 == 0, so rows follow one another
        o[0] = make_uint4(h[0], h[1], h[2], h[3]);
        o[1] = make_uint4(h[4], h[5], h[6], h[7]);
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
                    best.pair = cg == 2; best.bn = bn; best.splits = real; best.ktiles_per_split = per;
                }
            }
        }
    }
    best.workspace_bytes = best.splits > 1 ? (size_t)best.splits * M * N * sizeof(float) : 0;
    return best;
}

cudaError_t launch_tc_gemm(const TcOperand& a, const TcOperand& b, float* c, int M, int N, int K, const TcPlan& plan,
                           const float* col_scale, float* splitk_ws, int* err_word, size_t max_smem, int sm_count,
                           cudaStream_t stream, int* launches) {
    if (a.planes != 2 || b.planes < 1 || b.planes > 2 || (N & 3) || (a.ld & 7) || (b.ld & 7)) return cudaErrorInvalidValue;
    const int bn = plan.bn, cg = plan.pair ? 2 : 1, splits = plan.splits, b_rows = bn / cg;
    float* out = splits > 1 ? splitk_ws : c;
    CUtensorMap ma, mb, mc;
    if (!make_map(&ma, a, BM)) return cudaErrorInvalidValue;
    if (!make_map(&mb, b, b_rows)) return cudaErrorInvalidValue;
    if (!make_out_map(&mc, out, M, N, splits)) return cudaErrorInvalidValue;
    TcParams p;
    p.col_scale = col_scale;
    p.M = M; p.N = N; p.K = K;
    p.BN = bn;
    p.a_mn = a.mn_major; p.b_mn = b.mn_major;
    p.a_amax = a.amax; p.b_amax = b.amax;
    p.b_bytes = (b.mn_major ? (b_rows + 63) / 64 * 64 : b_rows) * BK * 2;
    p.group_m = 12 / cg;          // 12 row tiles x 12 column tiles in flight on 148 SMs
    p.nterms = b.planes == 2 ? 3 : 2;
    p.splits = splits;
    p.ktiles_per_split = plan.ktiles_per_split;
    p.err = err_word;
    const size_t stage_bytes = (size_t)kATileBytes + (size_t)p.b_bytes;
    int stages = (int)((max_smem - 2048 - kStageBytes) / stage_bytes);
    if (stages > kMaxStages) stages = kMaxStages;
    const int want = p.nterms * p.ktiles_per_split;   // slots one work item fills
    const int n_items = ((N + bn - 1) / bn) * ((M + cg * BM - 1) / (cg * BM)) * splits;
    // Two accumulators of one CTA take 2 * pow2(BN) TMEM columns of the SM's 512.  Narrow tiles
    // (BN <= 128) with short main loops leave room for a second resident CTA, which doubles the
    // loads in flight where the loop is latency-bound; then each CTA gets half the shared memory.
    bool two_ctas = false;
    if (cg == 1 && bn <= 128 && want <= 32 && n_items > sm_count) {
        const int half = (int)((((max_smem - 4096) / 2) - 1024 - kStageBytes) / stage_bytes);
        if (half >= 3) { two_ctas = true; if (half < stages) stages = half; }
    }
    if (stages > want) stages = want;
    if (stages < 2) stages = 2;
    const size_t smem = (size_t)stages * stage_bytes + 1024 + kStageBytes;
    if (smem > max_smem) return cudaErrorInvalidConfiguration;
    p.stages = stages;
    const void* kern = cg == 2 ? reinterpret_cast<const void*>(tc_gemm_kernel<2>) : reinterpret_cast<const void*>(tc_gemm_kernel<1>);
    cudaError_t e = ensure_dynamic_smem(kern, cg == 2 ? kSmemSlotTcPair : 4, max_smem);
    if (e != cudaSuccess) return e;
    int units = (sm_count / cg) * (two_ctas ? 2 : 1);
    if (units > n_items) units = n_items;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(units * cg));
    cfg.blockDim = dim3(kTcThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cg == 2 ? 1 : 0;
    e = cg == 2 ? cudaLaunchKernelEx(&cfg, tc_gemm_kernel<2>, ma, mb, mc, p) : cudaLaunchKernelEx(&cfg, tc_gemm_kernel<1>, ma, mb, mc, p);
    if (e != cudaSuccess) return e;
    ++*launches;
    if (splits > 1) {
        e = launch_splitk_reduce(splitk_ws, c, col_scale, M, N, N, splits, stream);
        if (e != cudaSuccess) return e;
        ++*launches;
    }
    return cudaSuccess;
}

// K-major use: 2-D {cols, rows}, box {32, box_outer rows}, 128-byte swizzle.  MN-major use (cols % 32 == 0):
// 3-D {32, rows, cols / 32} with the 32-column chunk as the outermost index, box {32, 32, box_outer chunks},
// 128-byte swizzle with 32-byte atoms.  Elements outside the tensor read as zero.
bool tc_encode_map_f32(void* map, const float* base, int cols, int rows, int ld, int mn_major, int box_outer) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    CUtensorMap* m = static_cast<CUtensorMap*>(map);
    void* ptr = const_cast<float*>(base);
    if (!mn_major) {
        cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
        cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
        cuuint32_t box[2] = {32, (cuuint32_t)box_outer};
        cuuint32_t estr[2] = {1, 1};
        return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    }
    if (cols % 32 != 0) return false;
    cuuint64_t dims[3] = {32, (cuuint64_t)rows, (cuuint64_t)(cols / 32)};
    cuuint64_t strides[2] = {(cuuint64_t)ld * 4, 128};
    cuuint32_t box[3] = {32, 32, (cuuint32_t)box_outer};
    cuuint32_t estr[3] = {1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool tc_encode_map_bf16(void* map, const void* base, int cols, int rows, int ld, int box_outer) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_outer};
    cuuint32_t estr[2] = {1, 1};
    return enc(static_cast<CUtensorMap*>(map), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box,
               estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t launch_splitk_reduce(const float* partial, float* c, const float* col_scale, int M, int N, int ldc,
                                 int splits, cudaStream_t stream) {
    const size_t n4 = (size_t)M * (N / 4);
    int blocks = (int)((n4 + 255) / 256);
    if (blocks > 148 * 8) blocks = 148 * 8;
    splitk_reduce_kernel<<<blocks, 256, 0, stream>>>(partial, c, col_scale, M, N, ldc, splits);
    return cudaGetLastError();
}

cudaError_t launch_split_terms(const float* src, int R, int Cc, int ld, const float* col_scale, void* planes, void* planes_s,
                               uint32_t* amax, int sm_count, cudaStream_t stream) {
    const bool vec = (Cc & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0 &&
                     (col_scale == nullptr || (reinterpret_cast<uintptr_t>(col_scale) & 15) == 0);
    __half* p0 = static_cast<__half*>(planes);
    __half* p1 = static_cast<__half*>(planes_s);
    const float* cs = p1 ? col_scale : nullptr;
    auto blocks = [&](size_t work, int per_sm) {
        const size_t b = (work + 255) / 256;
        return (int)(b < (size_t)sm_count * per_sm ? (b ? b : 1) : (size_t)sm_count * per_sm);
    };
    const size_t n = (size_t)R * Cc;
    if (vec) amax_kernel<true><<<blocks(n / 4, 8), 256, 0, stream>>>(src, R, Cc, cs, amax);
    else amax_kernel<false><<<blocks(n, 8), 256, 0, stream>>>(src, R, Cc, cs, amax);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const int nb = blocks((size_t)R * ((Cc + 7) / 8), 8);
    if (vec) split_terms_kernel<true><<<nb, 256, 0, stream>>>(src, R, Cc, ld, cs, p0, p1, amax);
    else split_terms_kernel<false><<<nb, 256, 0, stream>>>(src, R, Cc, ld, cs, p0, p1, amax);
    return cudaGetLastError();
}

cudaError_t launch_expand_ternary(const uint8_t* state, const uint32_t* packed2, int C, int O, int I, void* T, int ld,
                                  int sm_count, cudaStream_t stream) {
    __half* t = static_cast<__half*>(T);
    const size_t units = (size_t)O * ((I + 15) / 16);
    int blocks = (int)((units + 255) / 256 < (size_t)sm_count * 8 ? (units + 255) / 256 : (size_t)sm_count * 8);
    if (!state)
        expand_ternary_p2_kernel<<<blocks, 256, 0, stream>>>(packed2, (size_t)O * (I / 16), t);
    else if (I % 16 == 0 && ld == I && (reinterpret_cast<uintptr_t>(state) & 3) == 0)
        expand_ternary_kernel<true><<<blocks, 256, 0, stream>>>(state, C, O, I, t, ld);
    else
        expand_ternary_kernel<false><<<blocks, 256, 0, stream>>>(state, C, O, I, t, ld);
    return cudaGetLastError();
}

}  // namespace mcl
