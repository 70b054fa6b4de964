// Single-layer kernels of narrow counter linears: one launch each for Y, for dX and for the memory-native update.
//
// MotifCL's autograd asks for one product of one layer at a time (src/nn/compact_counter.cpp:40-50,158-300), and a layer of a
// few hundred features is a few microseconds of arithmetic: what a call costs is its launches, its passes over scratch memory
// and the latency of each.  So the operands are made where they are used: threads load fp32 activations and packed
// 6-bit codes, split and expand them in registers, and store bf16 tiles straight into the swizzled shared-memory layouts that
// tcgen05.mma reads.  An fp32 value is three bf16 terms (24 bits: exact up to the smallest exponents); a ternary digit is one.
//   Y, dX   three products per k (term x digit)
//   dW      six products per k (terms x terms, those above 2^-24)
// Tensor-core accumulation truncates in proportion to what the accumulator holds, so the products of leading terms have an
// accumulator of their own and all smaller ones share a second; the epilogue adds the two in fp32 (one accumulator for
// all: 1.1e-6 relative error at K = 512).
// Loads run two k-tiles ahead in registers (one tile ahead left 1000 of 1550 cycles per k-tile waiting for them); two shared-memory
// stages let the tensor core work on one while the threads fill the other.  These kernels are latency-bound (tens of CTAs, a
// handful of k-tiles each).
//
// Every wait on an mbarrier is bounded; on time-out the error word is set and the results are invalid.
#include <cuda_bf16.h>

#include <cfloat>
#include <type_traits>

#include "counter_codec.cuh"
#include "counter_update_body.cuh"
#include "kernels.h"
#include "tc_ptx.cuh"

namespace mcl {
namespace {

constexpr int kLThreads = 512;
constexpr int kErrLayer = 41;

// two fp32 values -> their three bf16 terms, packed two per word
__device__ __forceinline__ void split3(float a, float b, uint32_t (&t)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        t[i] = *reinterpret_cast<const uint32_t*>(&h);
        if (i < 2) { a -= __uint_as_float(t[i] << 16); b -= __uint_as_float(t[i] & 0xFFFF0000u); }
    }
}
__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b) {
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void sts128u(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// MN-major bf16 tile in the 128-byte swizzle: chunks of 64 MN elements, `chunk` bytes apart, each k rows of 128 bytes
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr, uint32_t chunk) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(chunk >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// kind::f16, D = f32, A = B = bf16, major bits 15 / 16 as given
__device__ __forceinline__ uint32_t idesc_bf16(int m, int n, uint32_t a_mn, uint32_t b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn << 15) | (b_mn << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_peer(uint32_t addr, uint32_t rank) {      // 16 bytes of a cluster peer's shared memory
    uint32_t a;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
// four consecutive floats of a row of n, zero beyond its end
__device__ __forceinline__ float4 load4(const float* row, int c, int n, bool vec) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (vec) {
        if (c < n) v = load_behind(reinterpret_cast<const float4*>(row + c));
    } else {
        if (c < n) v.x = load_behind(row + c);
        if (c + 1 < n) v.y = load_behind(row + c + 1);
        if (c + 2 < n) v.z = load_behind(row + c + 2);
        if (c + 3 < n) v.w = load_behind(row + c + 3);
    }
    return v;
}
__device__ __forceinline__ void tmem_alloc(uint32_t slot_addr, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_addr), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

// ---- Y = X (s T)^T and dX = (dY s) T ----------------------------------------------------------------------------
// CTA = 128 rows x BN columns, k-tiles of 64.  Shared memory per stage: A terms 3 x [128 rows][64 k] (K-major), digits
// [BN rows][64 k] for Y (K-major) or [64 k][BN] in chunks of 64 columns for dX (MN-major): both are the state's own order.
struct RowParams {
    const float* a;           // [M, K]
    const uint8_t* state;     // [out, in] packed
    const float* scale;       // [out]
    float* c;                 // [M, N]
    int M, N, K, in_features, C;
    int BN, stage_bytes;
    int parts, kt_per;        // CTAs of a cluster along K and k-tiles of each
    int vec;                  // rows of a start on 16-byte boundaries
    int* err;
};
constexpr int kRowATerm = 128 * 128;          // bytes of one A term per stage

// CUT: K is cut over the CTAs of a cluster (a form of its own: with both ways out in it the other one lost 1 us a launch)
template <bool DX, bool CUT>
__global__ void __launch_bounds__(kLThreads, 1) layer_rows_kernel(const RowParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ uint32_t tmem_slot, digit[64], lut[4096];
    __shared__ int abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t stage0 = (smem_u32(smem) + 1023u) & ~1023u;
    const uint32_t bar0 = smem_u32(bars);
    const int BN = p.BN, I = p.in_features;
    const int m0 = blockIdx.x * 128, n0 = blockIdx.y * BN;
    const bool words = (I & 15) == 0 && (reinterpret_cast<uintptr_t>(p.state) & 3) == 0;     // 16 weights = 3 aligned words
    uint32_t cols = 32;
    while ((int)cols < BN) cols <<= 1;
    if (tid == 0) {
        mbar_init(bar0, 1); mbar_init(bar0 + 8, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(smem_u32(&tmem_slot), 2 * cols);       // leading terms, smaller terms
    if (tid < 64) {
        const __nv_bfloat16 h = __float2bfloat16_rn((float)(tid / (2 * p.C - 1) - 1));
        digit[tid] = __bfloat16_as_ushort(h);
    }
    // A: 4 float4 of a k-tile per thread: rows tid / 16 + 32 j, the same 4 k in each.  Digits: units of 16 weights, up to 2 per
    // thread.  All addresses are formed once and advance by a constant per k-tile.
    struct Regs { float4 a[4], sc4; uint32_t w[2][3]; };
    const int kt0 = CUT ? (int)blockIdx.z * p.kt_per : 0, nkt = CUT ? min((p.K + 63) / 64 - kt0, p.kt_per) : (p.K + 63) / 64, nu = 4 * BN;         // units per k-tile: BN rows x 4 (Y) or 64 rows x BN / 16 (dX)
    const int rb = I / 4 * 3, ka = (tid & 15) * 4, arow = tid >> 4;
    const float* ap = p.a + (size_t)(m0 + arow) * p.K + ka;
    const size_t astep = (size_t)32 * p.K;
    uint32_t arows = 0;                                    // bit j: row m0 + arow + 32 j exists
#pragma unroll
    for (int j = 0; j < 4; ++j) arows |= (m0 + arow + 32 * j < p.M ? 1u : 0u) << j;
    const uint32_t a_at = (uint32_t)arow * 128u + (uint32_t)(((ka >> 3) ^ (arow & 7)) << 4) + (uint32_t)((ka & 4) << 1);
    uint32_t u_off[2], u_at[2];                            // byte offset of the unit's codes, shared-memory address of its first 8 digits
    int u_row[2], u_left[2];                               // row (Y: constant, dX: k within the tile) and groups of 4 up to the row's end
    const uint8_t* sp = DX ? p.state + (size_t)(n0 / 4) * 3 : p.state + (size_t)n0 * rb;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int u = tid + kLThreads * j;
        if (DX) {
            const int per = BN >> 4, kr = u / per, cu = u - kr * per;
            u_row[j] = u < nu ? kr : 1 << 30;
            u_left[j] = (I - n0) / 4 - 4 * cu;
            u_off[j] = (uint32_t)(kr * rb + 12 * cu);
            u_at[j] = (uint32_t)(cu >> 2) * 8192u + (uint32_t)kr * 128u + ((uint32_t)((2 * (cu & 3)) ^ (kr & 7)) << 4);
        } else {
            const int r = u >> 2, ku = u & 3;
            u_row[j] = u < nu && n0 + r < p.N ? 0 : 1 << 30;
            u_left[j] = I / 4 - 4 * ku;
            u_off[j] = (uint32_t)(r * rb + 12 * ku);
            u_at[j] = (uint32_t)r * 128u + ((uint32_t)((2 * ku) ^ (r & 7)) << 4);
        }
    }
    const size_t ustep = DX ? (size_t)64 * rb : 48;
    auto load = [&](int kt, Regs& r) {
        const int k = kt * 64 + ka;
        const float* q = ap + kt * 64;
        if (p.vec) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                r.a[j] = ((arows >> j) & 1u) && k < p.K ? load_behind(reinterpret_cast<const float4*>(q + j * astep)) : make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) r.a[j] = load4(q + j * astep - k, k, (arows >> j) & 1u ? p.K : 0, false);
        }
        if (DX) r.sc4 = load4(p.scale, k, p.K, false);
        const uint8_t* g = sp + kt * ustep;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            r.w[j][0] = r.w[j][1] = r.w[j][2] = 0;
            const bool in = DX ? u_row[j] + kt * 64 < p.K && u_left[j] > 0 : u_row[j] == 0 && u_left[j] > 16 * kt;
            if (in) {
                if (words) {
                    const uint32_t* s = reinterpret_cast<const uint32_t*>(g + u_off[j]);
                    r.w[j][0] = load_behind(s); r.w[j][1] = load_behind(s + 1); r.w[j][2] = load_behind(s + 2);
                } else {
                    const int nb = 3 * min(4, u_left[j] - (DX ? 0 : 16 * kt));
#pragma unroll
                    for (int b = 0; b < 12; ++b)
                        if (b < nb) r.w[j][b >> 2] |= (uint32_t)load_behind(g + u_off[j] + b) << (8 * (b & 3));
                }
            }
        }
    };
    Regs r0, r1;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_release();
    for (int e = tid; e < 4096; e += kLThreads) lut[e] = digit[e & 63] | (digit[e >> 6] << 16);
    grid_wait();
    load(kt0, r0);
    if (nkt > 1) load(kt0 + 1, r1);
    __syncthreads();
    const uint32_t tmem = tmem_slot;
    const uint32_t idesc = idesc_bf16(128, BN, 0, DX ? 1u : 0u);
    bool ok = true;
    auto step = [&](int i, Regs& r) {
        const int s = i & 1, kt = kt0 + i;
        const uint32_t st = stage0 + (uint32_t)s * (uint32_t)p.stage_bytes, sb = st + 3u * kRowATerm;
        if (i >= 2 && ok) ok = mbar_wait(bar0 + 8u * s, ((uint32_t)(i >> 1) - 1u) & 1u, &abort_flag);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float4 v = r.a[j];
            if (DX) {                                      // grad_out times the scale of its column, rounded to fp32
                v.x = __fmul_rn(v.x, r.sc4.x); v.y = __fmul_rn(v.y, r.sc4.y);
                v.z = __fmul_rn(v.z, r.sc4.z); v.w = __fmul_rn(v.w, r.sc4.w);
            }
            uint32_t t0[3], t1[3];
            split3(v.x, v.y, t0); split3(v.z, v.w, t1);
#pragma unroll
            for (int t = 0; t < 3; ++t) sts64(st + a_at + (uint32_t)(4096 * j + kRowATerm * t), t0[t], t1[t]);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            if (tid + kLThreads * j < nu) {
                // groups of 4 that exist (the others, and rows outside, were loaded as zero codes and must become zero digits)
                const int left = DX ? (u_row[j] + kt * 64 < p.K ? u_left[j] : 0) : (u_row[j] == 0 ? u_left[j] - 16 * kt : 0);
                uint32_t h[8];
                const uint32_t g[4] = {r.w[j][0] & 0xFFFFFFu, (r.w[j][0] >> 24) | ((r.w[j][1] & 0xFFFFu) << 8),
                                       (r.w[j][1] >> 16) | ((r.w[j][2] & 0xFFu) << 16), r.w[j][2] >> 8};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    h[2 * q] = q < left ? lut[g[q] & 4095u] : 0u;
                    h[2 * q + 1] = q < left ? lut[g[q] >> 12] : 0u;
                }
                sts128u(sb + u_at[j], h[0], h[1], h[2], h[3]);
                sts128u(sb + (u_at[j] ^ 16u), h[4], h[5], h[6], h[7]);
            }
        }
        if (i + 2 < nkt) load(kt + 2, r);
        fence_proxy_async();
        __syncthreads();
        if (warp == 0) {
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int t = 2; t >= 0; --t) {              // smallest term first
                    const uint64_t da = smem_desc_k_sw128(st + (uint32_t)t * kRowATerm);
                    const uint64_t db = DX ? desc_mn(sb, 8192) : smem_desc_k_sw128(sb);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        umma_bf16(t == 0 ? tmem : tmem + cols, da + 2u * kk, db + (DX ? 128u : 2u) * kk, idesc,
                                  (i | kk) != 0 || t == 1 ? 1u : 0u);
                }
                umma_commit(bar0 + 8u * s);
            }
            __syncwarp();
        }
    };
    for (int i = 0; i < nkt; i += 2) {
        step(i, r0);
        if (i + 1 < nkt) step(i + 1, r1);
    }
    if (ok) ok = mbar_wait(bar0 + 8u * ((nkt - 1) & 1), (uint32_t)((nkt - 1) >> 1) & 1u, &abort_flag);
    if (!ok && tid == 0) atomicExch(p.err, kErrLayer);
    tc_fence_after();
    if constexpr (CUT) {
        // K is cut over the CTAs of a cluster: each publishes both accumulators, then adds its share of the rows over all of them in rank
        // order, the leading ones with their rounding errors carried along (a plain sum of rounded parts: error 4.3 -> 5.8e-8)
        const int q = warp & 3, pitch = (BN + 4) * 4;
        const uint32_t small = stage0 + 128u * (uint32_t)pitch;
        for (int c0 = (warp >> 2) * 32; c0 < BN; c0 += 128) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t r[32];
                tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (half ? cols : 0u) + (uint32_t)c0, r);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    sts128u((half ? small : stage0) + (uint32_t)((q * 32 + lane) * pitch + (c0 + 4 * j) * 4), r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
            }
        }
        cluster_sync_all();
        const int share = 128 / p.parts, quads = BN >> 2, row0 = (int)cluster_rank() * share;
        const bool wide = (p.N & 3) == 0 && (reinterpret_cast<uintptr_t>(p.c) & 15) == 0;
        auto add = [](float& s, float& e, float v, float w) {      // s + e += v + w, s rounded, e what that loses
            const float t = __fadd_rn(s, v), u = __fsub_rn(t, s), lost = __fadd_rn(__fsub_rn(s, __fsub_rn(t, u)), __fsub_rn(v, u));
            e = __fadd_rn(e, __fadd_rn(fabsf(t) <= FLT_MAX ? lost : 0.0f, w));      // a sum that left fp32 is an infinity and loses nothing
            s = t;
        };
        for (int i = tid; i < share * quads; i += kLThreads) {
            const int row = row0 + i / quads, c = (i % quads) * 4, m = m0 + row, n = n0 + c;
            if (m >= p.M || n >= p.N) continue;
            const uint32_t at = (uint32_t)(row * pitch + c * 4);
            float4 sum = make_float4(0.f, 0.f, 0.f, 0.f), e = sum;
            for (int k = 0; k < p.parts; k += 2) {                 // four remote loads in flight
                const float4 v0 = ld_peer(stage0 + at, (uint32_t)k), w0 = ld_peer(small + at, (uint32_t)k);
                const float4 v1 = ld_peer(stage0 + at, (uint32_t)k + 1), w1 = ld_peer(small + at, (uint32_t)k + 1);
                add(sum.x, e.x, v0.x, w0.x); add(sum.y, e.y, v0.y, w0.y); add(sum.z, e.z, v0.z, w0.z); add(sum.w, e.w, v0.w, w0.w);
                add(sum.x, e.x, v1.x, w1.x); add(sum.y, e.y, v1.y, w1.y); add(sum.z, e.z, v1.z, w1.z); add(sum.w, e.w, v1.w, w1.w);
            }
            sum.x += e.x; sum.y += e.y; sum.z += e.z; sum.w += e.w;
            if (!DX) {
                const float4 sc = load4(p.scale, n, p.N, false);
                sum.x *= sc.x; sum.y *= sc.y; sum.z *= sc.z; sum.w *= sc.w;
            }
            float* out = p.c + (size_t)m * p.N + n;
            if (wide) *reinterpret_cast<float4*>(out) = sum;
            else {
                out[0] = sum.x;
                if (n + 1 < p.N) out[1] = sum.y;
                if (n + 2 < p.N) out[2] = sum.z;
                if (n + 3 < p.N) out[3] = sum.w;
            }
        }
        cluster_sync_all();                                // before this CTA's shared memory goes
    } else {
        // epilogue: warp = 32 rows x a quarter of the columns; a 32 x 33 tile in shared memory turns lane = row into lane = column
        const int q = warp & 3, part = warp >> 2;
        float* tile = reinterpret_cast<float*>(smem) + warp * 32 * 33;
        for (int c0 = part * 32; c0 < BN && n0 + c0 < p.N; c0 += 128) {
            uint32_t r[32], r1[32];
            tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, r);
            tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + cols + (uint32_t)c0, r1);
            tmem_ld_wait();
            const int col = n0 + c0 + lane;
            const float sc = !DX && col < p.N ? load_behind(p.scale + col) : 1.0f;
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 32; ++j) tile[lane * 33 + j] = __uint_as_float(r[j]) + __uint_as_float(r1[j]);
            __syncwarp();
            const int rows = min(32, p.M - m0 - q * 32);
            if (col < p.N) {
                float* out = p.c + (size_t)(m0 + q * 32) * p.N + col;
#pragma unroll 8
                for (int i = 0; i < rows; ++i) out[(size_t)i * p.N] = DX ? tile[i * 33 + lane] : tile[i * 33 + lane] * sc;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * cols) : "memory");
}

// ---- memory-native update: dW = dY^T X of 128 rows in tensor memory, then the counter update, in one launch ----------------
// A cluster of CTAs owns 128 rows of the layer; each CTA contracts a slice of the tokens into its own tensor memory (all
// columns of the rows, in passes of up to 256).  The slices are added through distributed shared memory, 128 columns at a
// time: every CTA publishes its partial tile, then sums its share of the rows over all CTAs in rank order (deterministic) into its
// own shared memory, where the update runs on whole rows.  grad_w never exists outside the chip.
struct LayerUpdParams {
    const float* dy;          // [tokens, O]
    const float* x;           // [tokens, I]
    int tokens, O, slice;     // slice: tokens per CTA, a multiple of 32
    int mr;                   // rows of the layer that a cluster owns (at most 128)
    int np, pw;               // passes over the columns and their width (a multiple of 64, at most 256)
    int off_stage, stage_bytes;
    int vec_dy;
    uint32_t magic;
    int* err;
    UpdParams u;              // of the whole layer; rows_per_batch = rows of a CTA
};
constexpr int kDwK = 32;                      // tokens per k-tile: two MMA steps
constexpr int kDwDepth = kGradDepthLimit * 64 / kDwK;      // k-tiles that one accumulator takes before it is added up in fp32
constexpr int kDwChunk = kDwK * 128;          // bytes of 64 columns x 32 tokens
constexpr int kDwATerm = 2 * kDwChunk;

// the update for in_features % 16 != 0: groups of four weights read and written as bytes
template <bool WITH_Q>
__device__ __forceinline__ void update_rows_by_group(const UpdParams& p, const int nrows, unsigned char* smem, const U16Layout& L) {
    DecodeLut* lut = reinterpret_cast<DecodeLut*>(smem);
    RowK* rowc = reinterpret_cast<RowK*>(smem + L.off_rowc);
    float* part = reinterpret_cast<float*>(smem + L.off_part);
    const float4* gw_s = reinterpret_cast<const float4*>(smem + L.off_gw);
    const int tid = threadIdx.x, lane = tid & 31, pair = tid >> 6, vlane = tid & 63;
    const int I = p.in_features, gpr = I >> 2, lv = 2 * p.C - 1;
    const uint32_t seed = p.seed + (p.seed_offset ? load_behind(p.seed_offset) : 0u);
    auto group = [&](int r, int g) -> uint32_t {
        const uint8_t* s = p.state + ((size_t)r * gpr + g) * 3;
        return (uint32_t)s[0] | ((uint32_t)s[1] << 8) | ((uint32_t)s[2] << 16);
    };
    build_decode_lut(lut, p.C, tid, kLThreads);
    __syncthreads();
    for (int r = pair; r < nrows; r += kLThreads / 64) {
        float a = 0.0f, b = 0.0f;
        for (int g = vlane; g < gpr; g += 64) {
            const float4 gw = gw_s[r * gpr + g];
            a = __fadd_rn(a, __fmul_rn(gw.x, gw.x)); a = __fadd_rn(a, __fmul_rn(gw.y, gw.y));
            a = __fadd_rn(a, __fmul_rn(gw.z, gw.z)); a = __fadd_rn(a, __fmul_rn(gw.w, gw.w));
            if (WITH_Q) {
                const uint32_t w = group(r, g);
                b = __fadd_rn(b, __fmul_rn(gw.x, lut->e[w & 63u].x)); b = __fadd_rn(b, __fmul_rn(gw.y, lut->e[(w >> 6) & 63u].x));
                b = __fadd_rn(b, __fmul_rn(gw.z, lut->e[(w >> 12) & 63u].x)); b = __fadd_rn(b, __fmul_rn(gw.w, lut->e[(w >> 18) & 63u].x));
            }
        }
        if (vlane >= 32) { part[pair * 64 + lane] = a; part[pair * 64 + 32 + lane] = b; }
        asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory");
        if (vlane < 32) {
            a = __fadd_rn(a, part[pair * 64 + lane]); b = __fadd_rn(b, part[pair * 64 + 32 + lane]);
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) {
                a = __fadd_rn(a, __shfl_down_sync(0xffffffffu, a, s)); b = __fadd_rn(b, __shfl_down_sync(0xffffffffu, b, s));
            }
            if (lane == 0) rowc[r] = finish_row_stats<WITH_Q>(p, r, a, b, (float)p.C, p.scale[r], p.v[r]);
        }
        asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory");
    }
    __syncthreads();
    for (int i = tid; i < nrows * gpr; i += kLThreads) {
        const int r = i / gpr, g = i - r * gpr;
        const RowK rc = rowc[r];
        const float4 gw = gw_s[i];
        const float gv[4] = {gw.x, gw.y, gw.z, gw.w};
        const uint32_t w = group(r, g), e0 = (uint32_t)(p.row_offset + r) * (uint32_t)I + 4u * (uint32_t)g;
        uint32_t nw = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 tc = lut->e[(w >> (6 * k)) & 63u];
            uint32_t fld;
            nw |= (counter_tick(gv[k], tc.x, tc.y, e0 + (uint32_t)k, seed, -p.lr, rc.dn, rc.k_tick, rc.k_reb, (float)p.C, p.C, lv, &fld) & 0x3Fu) << (6 * k);
        }
        uint8_t* s = p.state + (size_t)i * 3;
        s[0] = (uint8_t)nw; s[1] = (uint8_t)(nw >> 8); s[2] = (uint8_t)(nw >> 16);
    }
}

// DEEP: slices of more than kDwDepth k-tiles.  A form of its own: with the segments in it the loop spills, which cost 2 to 9 %.
template <bool WITH_Q, bool U16, bool DEEP>
__global__ void __launch_bounds__(kLThreads, 1) layer_update_kernel(const __grid_constant__ LayerUpdParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    uint32_t cs;
    asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(cs));
    const int rank = (int)cluster_rank(), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int I = p.u.in_features, gpr = I >> 2, R = p.u.rows_per_batch;
    const U16Layout L = u16_layout(I, R, WITH_Q, kLThreads / 64);
    const int m0 = ((int)blockIdx.x / (int)cs) * p.mr;
    const int valid = min(p.mr, p.O - m0), rpc = (valid + (int)cs - 1) / (int)cs;
    const int my_row0 = rank * rpc, my_rows = max(0, min(rpc, valid - my_row0));
    const int t0 = rank * p.slice, t1 = min(p.tokens, t0 + p.slice);
    const int nkt = t1 > t0 ? (t1 - t0 + kDwK - 1) / kDwK : 0;
    const uint32_t stage0 = ((smem_u32(smem) + 1023u) & ~1023u) + (uint32_t)p.off_stage;
    const uint32_t bar0 = smem_u32(bars);
    float4* gw_s = reinterpret_cast<float4*>(smem + L.off_gw);
    uint32_t cols = 32;
    while ((int)cols < p.pw) cols <<= 1;
    if (tid == 0) {
        mbar_init(bar0, 1); mbar_init(bar0 + 8, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(smem_u32(&tmem_slot), 2 * cols);       // leading products, smaller products
    UpdParams u = p.u;                            // of this CTA's rows
    {
        const int row = m0 + my_row0;
        u.state += (size_t)row * gpr * 3;
        u.scale += row; u.v += row;
        if (u.packed2) u.packed2 += (size_t)row * (I >> 4);
        u.rows = my_rows; u.row_offset = row;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_release();
    if (U16 && my_rows > 0) {                     // what the update needs beside the gradient is in place before it
        build_decode_lut(reinterpret_cast<DecodeLut*>(smem), u.C, tid, kLThreads);
        build_tick_table(reinterpret_cast<uint32_t*>(smem + L.off_tick), u.C, tid, kLThreads);
    }
    grid_wait();
    if (U16 && my_rows > 0) {
        u16_load_state<kLThreads>(u, L, smem, 0, my_rows);
        if (tid < my_rows) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(u.scale + tid));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(u.v + tid));
        }
    }
    const uint32_t tmem = tmem_slot;
    bool ok = true;
    int it = 0;                                   // k-tiles so far: stage = it & 1
    const int nseg = DEEP ? (p.slice / kDwK + kDwDepth - 1) / kDwDepth : 1;
    for (int pass = 0; pass < p.np; ++pass) {
        const int n0 = pass * p.pw, nw = min(p.pw, I - n0), nwp = (nw + 15) & ~15, per = nwp >> 2;
        const uint32_t bterm = (uint32_t)((nwp + 63) / 64) * kDwChunk;
        // this thread's float4s of a k-tile: 2 of dY (tokens tid / 32 + 16 j, the same 4 columns), up to 4 of x; addresses are
        // formed once and advance by a constant per k-tile
        struct Regs { float4 a[2], b[4]; };
        int b_off[4], b_tok[4];
        uint32_t b_at[4];
        const int ac = m0 + lane * 4;
        const bool a_in = lane * 4 < valid;
        const float* ap = p.dy + (size_t)(t0 + warp) * p.O + ac;
        const float* bp = p.x + (size_t)t0 * I + n0;
        auto place = [](int row, int col) -> uint32_t {        // shared-memory offset of four columns of one token
            return (uint32_t)(col >> 6) * kDwChunk + (uint32_t)row * 128u + (uint32_t)((((col & 63) >> 3) ^ (row & 7)) << 4) + (uint32_t)((col & 4) << 1);
        };
        const uint32_t a_at = place(warp, lane * 4);           // rows 16 further: + 2048, the swizzle repeats
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int idx = tid + kLThreads * j, row = idx / per, col = 4 * (idx - row * per);
            b_tok[j] = row < kDwK ? row : 1 << 30;
            b_off[j] = n0 + col < I ? row * I + col : -1;
            b_at[j] = place(row, col);
        }
        auto load = [&](int kt, Regs& r) {
            const int left = t1 - t0 - kt * kDwK;              // tokens from this k-tile on
            const float* q = ap + (size_t)kt * kDwK * p.O;
            if (p.vec_dy) {
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    r.a[j] = warp + 16 * j < left && a_in ? load_behind(reinterpret_cast<const float4*>(q + (size_t)(16 * j) * p.O)) : make_float4(0.f, 0.f, 0.f, 0.f);
            } else {
#pragma unroll
                for (int j = 0; j < 2; ++j) r.a[j] = load4(q + (size_t)(16 * j) * p.O - ac, ac, warp + 16 * j < left && a_in ? p.O : 0, false);
            }
            const float* g = bp + (size_t)kt * kDwK * I;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                r.b[j] = b_tok[j] < left && b_off[j] >= 0 ? load_behind(reinterpret_cast<const float4*>(g + b_off[j])) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        for (int seg = 0; seg < nseg; ++seg) {
            const int k0 = DEEP ? seg * kDwDepth : 0, k1 = DEEP ? min(nkt, k0 + kDwDepth) : nkt;
            Regs r0, r1;
            if (k0 < k1) load(k0, r0);
            if (k0 + 1 < k1) load(k0 + 1, r1);
            auto step = [&](int kt, Regs& r) {
                const uint32_t st = stage0 + (uint32_t)(it & 1) * (uint32_t)p.stage_bytes, sb = st + 3u * kDwATerm;
                if (it >= 2 && ok) ok = mbar_wait(bar0 + 8u * (it & 1), ((uint32_t)(it >> 1) - 1u) & 1u, &abort_flag);
                auto put = [&](uint32_t at, uint32_t term, float4 v) {     // four columns of one token, three terms
                    uint32_t u0[3], u1[3];
                    split3(v.x, v.y, u0); split3(v.z, v.w, u1);
#pragma unroll
                    for (int t = 0; t < 3; ++t) sts64(at + (uint32_t)t * term, u0[t], u1[t]);
                };
#pragma unroll
                for (int j = 0; j < 2; ++j) put(st + a_at + 2048u * j, kDwATerm, r.a[j]);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (b_tok[j] < kDwK) put(sb + b_at[j], bterm, r.b[j]);
                if (kt + 2 < k1) load(kt + 2, r);
                fence_proxy_async();
                __syncthreads();
                if (warp == 0) {
                    tc_fence_after();
                    if (elect_one()) {
                        // terms: 0 = hi .. 2 = lo, smallest products first
                        const int pa[6] = {2, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
                        for (int q = 0; q < 6; ++q) {
                            const uint64_t da = desc_mn(st + (uint32_t)pa[q] * kDwATerm, kDwChunk), db = desc_mn(sb + (uint32_t)pb[q] * bterm, kDwChunk);
#pragma unroll
                            for (int kk = 0; kk < kDwK / 16; ++kk)         // 16 tokens = 2048 bytes further
                                umma_bf16(q == 5 ? tmem : tmem + cols, da + 128u * kk, db + 128u * kk, idesc_bf16(128, nwp, 1, 1),
                                          ((kt - k0) | kk) != 0 || (q > 0 && q < 5) ? 1u : 0u);
                        }
                        umma_commit(bar0 + 8u * (it & 1));
                    }
                    __syncwarp();
                }
                ++it;
            };
            for (int kt = k0; kt < k1; kt += 2) {
                step(kt, r0);
                if (kt + 1 < k1) step(kt + 1, r1);
            }
            if (it > 0 && ok) ok = mbar_wait(bar0 + 8u * ((it - 1) & 1), (uint32_t)((it - 1) >> 1) & 1u, &abort_flag);
            tc_fence_after();
            // sum over the cluster, 128 columns at a time; the exchange tile lies over the (finished) stages
            for (int c0 = 0; c0 < nw; c0 += 128) {
                const int q = warp & 3, cc = (warp >> 2) * 32, row = q * 32 + lane;
                if (c0 + cc < nw && q * 32 < valid) {
                    uint32_t r[32], r1[32];
                    if (k0 < k1) {
                        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(c0 + cc), r);
                        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + cols + (uint32_t)(c0 + cc), r1);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(r1[j]));
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j) r[j] = 0;
                    }
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        sts128u(stage0 + (uint32_t)row * 512u + (uint32_t)(((cc >> 2) + j) ^ (row & 7)) * 16u, r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
                }
                tc_fence_before();
                cluster_sync_all();
                for (int i = tid; i < my_rows * 32; i += kLThreads) {
                    const int r = i >> 5, c = i & 31, g = ((n0 + c0) >> 2) + c;
                    if (c0 + 4 * c < nw) {
                        const int mr = my_row0 + r;
                        const uint32_t at = stage0 + (uint32_t)mr * 512u + (uint32_t)(c ^ (mr & 7)) * 16u;
                        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
                        for (uint32_t k = 0; k < cs; k += 4) {             // four remote loads in flight
                            float4 v[4];
#pragma unroll
                            for (uint32_t i4 = 0; i4 < 4; ++i4) v[i4] = ld_peer(at, k + i4);
#pragma unroll
                            for (uint32_t i4 = 0; i4 < 4; ++i4) {
                                sum.x = __fadd_rn(sum.x, v[i4].x); sum.y = __fadd_rn(sum.y, v[i4].y);
                                sum.z = __fadd_rn(sum.z, v[i4].z); sum.w = __fadd_rn(sum.w, v[i4].w);
                            }
                        }
                        float4& to = gw_s[r * gpr + (U16 ? swz4(g) : g)];
                        if (DEEP && seg > 0) {
                            sum.x = __fadd_rn(to.x, sum.x); sum.y = __fadd_rn(to.y, sum.y);
                            sum.z = __fadd_rn(to.z, sum.z); sum.w = __fadd_rn(to.w, sum.w);
                        }
                        to = sum;
                    }
                }
                cluster_sync_all();
                tc_fence_after();
            }
        }
    }
    if (!ok && tid == 0) atomicExch(p.err, kErrLayer);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * cols) : "memory");
    if (my_rows == 0) return;
    if (U16) update_u16_body<WITH_Q, true, kLThreads>(u, p.magic, 1u << 16, 1u << 17, 0, 1, false);
    else update_rows_by_group<WITH_Q>(u, my_rows, smem, L);
}

// ---- memory-native update of a small layer in the order of the exact kernels ----------------------------------------------
// A CTA owns a few rows: a thread forms four columns of one of them, tokens ascending, multiply and add rounded separately (the sum of
// simt_gemm.cu, bit for bit), into shared memory, where the update runs on whole rows.  Before, grad_w went through memory in up to eight row
// tiles of two launches each, 5 to 19 us a launch: 64 x 64 at 32 tokens 66 us, 128 x 200 at 128 132 us.  Bound: the chain of loads and sums.
// Forward, backward and update, before and now: 64 x 64 at 32 tokens 110 and 22 us, at 1000 907 and 61; 128 -> 200 at 128 195 and 31; 1000 -> 33 at
// 100 333 and 55.
template <bool WITH_Q, bool U16>
__global__ void __launch_bounds__(kLThreads, 1) exact_update_kernel(const __grid_constant__ LayerUpdParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x, I = p.u.in_features, gpr = I >> 2, R = p.u.rows_per_batch;
    const int row0 = (int)blockIdx.x * R, my_rows = min(R, p.O - row0);
    const U16Layout L = u16_layout(I, R, WITH_Q, kLThreads / 64);
    float4* gw_s = reinterpret_cast<float4*>(smem + L.off_gw);
    UpdParams u = p.u;
    u.state += (size_t)row0 * gpr * 3;
    u.scale += row0; u.v += row0;
    if (u.packed2) u.packed2 += (size_t)row0 * (I >> 4);
    u.rows = my_rows; u.row_offset = row0;
    grid_release();
    if (U16) {
        build_decode_lut(reinterpret_cast<DecodeLut*>(smem), u.C, tid, kLThreads);
        build_tick_table(reinterpret_cast<uint32_t*>(smem + L.off_tick), u.C, tid, kLThreads);
    }
    grid_wait();
    if (U16) u16_load_state<kLThreads>(u, L, smem, 0, my_rows);
    constexpr int AHEAD = 8;                  // tokens loaded at a time, one such set ahead of the sums
    struct Set { float4 x[AHEAD]; float d[AHEAD]; };
    for (int i = tid; i < my_rows * gpr; i += kLThreads) {
        const int r = i / gpr, g = i - r * gpr;
        const float4* xp = reinterpret_cast<const float4*>(p.x) + g;
        const float* dp = p.dy + row0 + r;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        auto load = [&](int t0, Set& s) {
#pragma unroll
            for (int j = 0; j < AHEAD; ++j) {
                const int t = min(t0 + j, p.tokens - 1);
                s.x[j] = load_behind(xp + (size_t)t * gpr);
                s.d[j] = load_behind(dp + (size_t)t * p.O);
            }
        };
        auto sum = [&](int t0, const Set& s) {
#pragma unroll
            for (int j = 0; j < AHEAD; ++j) {
                if (t0 + j >= p.tokens) break;
                acc.x = __fadd_rn(acc.x, __fmul_rn(s.d[j], s.x[j].x)); acc.y = __fadd_rn(acc.y, __fmul_rn(s.d[j], s.x[j].y));
                acc.z = __fadd_rn(acc.z, __fmul_rn(s.d[j], s.x[j].z)); acc.w = __fadd_rn(acc.w, __fmul_rn(s.d[j], s.x[j].w));
            }
        };
        Set a, b;
        load(0, a);
        for (int t0 = 0; t0 < p.tokens; t0 += 2 * AHEAD) {
            if (t0 + AHEAD < p.tokens) load(t0 + AHEAD, b);
            sum(t0, a);
            if (t0 + 2 * AHEAD < p.tokens) load(t0 + 2 * AHEAD, a);
            sum(t0 + AHEAD, b);
        }
        gw_s[r * gpr + (U16 ? swz4(g) : g)] = acc;
    }
    __syncthreads();
    if (U16) update_u16_body<WITH_Q, true, kLThreads>(u, p.magic, 1u << 16, 1u << 17, 0, 1, false);
    else update_rows_by_group<WITH_Q>(u, my_rows, smem, L);
}

}  // namespace

bool layer_kernels_fit(size_t tokens, size_t in_features, size_t out_features) {
    return in_features % 4 == 0 && in_features <= 1024 && out_features <= 2048 && tokens <= (1u << 20);
}

namespace {
constexpr int kCutColumns = 192;              // both accumulators of a tile, published in shared memory: 200 KB
// Column tile of the row kernels and CTAs that share its K: waves of CTAs times the time of a k-tile (conversion of A, then digits and MMAs per
// column), in ns.  K is cut where that fits one wave: a cluster pays two barriers and the exchange of its tile, each CTA leaves out
// k-tiles of a microsecond.  Forward, backward and update of one layer, us, uncut and cut: 128 -> 1200 at 200 rows 47 and 28, 1024 -> 1024 at 64
// 78 and 51, 512 -> 128 at 128 42 and 32 (5 to 7 of each from launches that overlap); cut in four, 288 -> 288 at 256 would lose 2 of 30.
double rows_cost(int tokens, int N, int K, int sm_count, int* bn_out, int* parts_out) {
    const int tm = (tokens + 127) / 128, nkt = (K + 63) / 64;
    double best = 1e30;
    for (int bn = 32; bn <= 256; bn += 32)
        for (int parts = 1; parts <= (bn <= kCutColumns ? 8 : 1); parts *= 2) {
            const int tiles = tm * ((N + bn - 1) / bn), per = (nkt + parts - 1) / parts;
            // clusters of 8 fit the GPCs 15 at a time, of 4 about 34
            if (parts > 1 && ((parts - 1) * per >= nkt || tiles > (parts == 8 ? sm_count * 15 / 148 : parts == 4 ? sm_count * 34 / 148 : sm_count * 70 / 148))) continue;
            const double cost = (double)((tiles * parts + sm_count - 1) / sm_count) * (per * (900.0 + 5.0 * bn) + 4000.0 + 6.0 * bn) + (parts > 1 ? 1500.0 + 40.0 * bn : 0.0);
            if (cost < best) { best = cost; *bn_out = bn; *parts_out = parts; }
        }
    return best;
}
// Rows per cluster and CTAs per cluster of the update: a CTA contracts its slice of the tokens (all columns, whatever the rows),
// then moves its rows x columns through the exchange once.  More CTAs shorten the slices, fewer rows per cluster shorten the
// exchange; all CTAs should be resident at once.  Times in cycles from the stamps of both phases.
struct UpdateShape { int np, pw, mr, cs, ktiles; double exchange; };
UpdateShape update_shape(int tokens, int I, int O, int sm_count) {
    UpdateShape u = {(I + 255) / 256, 0, 128, 8, 0, 0.0};
    u.pw = ((I + u.np - 1) / u.np + 63) / 64 * 64;
    double best = 1e30;
    for (int c = 4; c <= 8; c *= 2)            // clusters of 16 need two waves where eights need one: 288 x 288 at 256 rows 55 us, not 40
        for (int m = 128; m >= 32; m /= 2) {
            const int ctas = (O + m - 1) / m * c, kt = ((tokens + c - 1) / c + kDwK - 1) / kDwK;
            const double exchange = (double)m * I * 4 / 16.0 + u.np * ((u.pw + 127) / 128) * 1500.0 + 4000.0 + (double)(m / c) * I * 0.6;
            const double cost = (double)((ctas + sm_count - 1) / sm_count) * ((double)u.np * kt * (400.0 + 5.0 * (m + u.pw)) + exchange);
            if (cost < best) { best = cost; u.mr = m; u.cs = c; u.ktiles = kt; u.exchange = exchange; }
        }
    return u;
}
}  // namespace

// Which route a product of one layer takes, by its shape alone: the one-launch kernels, or terms split once (tc_gemm.cu), which need
// activation-sized workspace and have to be a fifth faster to be worth that.  Models in us, fitted to 36 shapes of 64 to 2048
// features at 32 to 262144 tokens (B200), within 10 % for nearly all.  One launch against split: 288 x 288 forward 27 / 30 us at
// 16384 tokens, 92 / 79 at 65536, 346 / 256 at 262144 (the line: about 100000); 288 x 1536 17 / 22 at 2048, 48 / 38 at 8192 (6000);
// 1024 x 1024 23 / 26 at 1024, 42 / 36 at 4096, 81 / 53 at 8192 (5000).
namespace { bool worth_workspace(double layer, double split) { return layer > 1.2 * split + 2.0; } }
bool layer_rows_pay(size_t tokens, size_t N, size_t K, int sm_count) {
    int bn = 0, parts = 0;
    const double layer = 1.8 + 1.864 / 1900.0 * rows_cost((int)tokens, (int)N, (int)K, sm_count, &bn, &parts);
    const double bytes = (double)tokens * (12.0 * K + 4.0 * N), flops = 4.0 * tokens * N * K;
    // split by the terms' kernels: launches, the pass over the digits, then memory or the tensor pipe
    const double split = 13.8 + 0.0075 * K + 1.5e-6 * N * K + (bytes / 4.7e6 > flops / 1.1e9 ? bytes / 4.7e6 : flops / 1.1e9);
    return !worth_workspace(layer, split);
}
// The same for the update, whose other route forms grad_w in `tiles` row tiles (288 x 768: 165 / 241 us at 16384 tokens, 610 / 406 at
// 65536; 512 x 512: 121 / 179 at 4096, 386 / 240 at 16384).  Clusters of 8 fit the GPCs 15 at a time, of 4 about 34.
bool layer_update_pays(size_t tokens, size_t I, size_t O, size_t tiles, int sm_count) {
    const UpdateShape u = update_shape((int)tokens, (int)I, (int)O, sm_count);
    const int clusters = ((int)O + u.mr - 1) / u.mr, fit = u.cs == 8 ? sm_count * 15 / 148 : sm_count * 34 / 148;
    const double layer = 5.0 + (clusters + fit - 1) / fit * (u.np * u.ktiles * (0.85 + 0.002 * u.pw) + u.exchange / 1900.0);
    const double split = 60.0 + 18.0 * tiles + (double)tokens * (8.0 * (I + O) + 4.0 * tiles * I + 4.0 * O) / 4.4e6;
    return !worth_workspace(layer, split);
}

cudaError_t launch_layer_rows(int dx, const float* a, const uint8_t* state, const float* scale, float* c, int tokens, int I, int O,
                              int C, int* err_word, size_t max_smem, int sm_count, cudaStream_t stream) {
    RowParams p;
    p.a = a; p.state = state; p.scale = scale; p.c = c;
    p.M = tokens; p.N = dx ? I : O; p.K = dx ? O : I; p.in_features = I; p.C = C;
    p.vec = (p.K & 3) == 0 && (reinterpret_cast<uintptr_t>(a) & 15) == 0;
    p.err = err_word;
    rows_cost(tokens, p.N, p.K, sm_count, &p.BN, &p.parts);
    p.kt_per = ((p.K + 63) / 64 + p.parts - 1) / p.parts;
    const int tm = (tokens + 127) / 128;
    p.stage_bytes = 3 * kRowATerm + (dx ? (p.BN + 63) / 64 * 8192 : p.BN * 128);
    const bool cut = p.parts > 1;
    const size_t stages = 2 * (size_t)p.stage_bytes, sums = cut ? (size_t)2 * 128 * (p.BN + 4) * 4 : 0, smem = (stages > sums ? stages : sums) + 1024;
    const auto kern = dx ? (cut ? layer_rows_kernel<true, true> : layer_rows_kernel<true, false>) : (cut ? layer_rows_kernel<false, true> : layer_rows_kernel<false, false>);
    cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), (cut ? 45 : 17) + (dx ? 1 : 0), max_smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)tm, (unsigned)((p.N + p.BN - 1) / p.BN), (unsigned)p.parts);
    cfg.blockDim = dim3(kLThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // launch_chained, with clusters
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = (unsigned)p.parts;
    cfg.attrs = attr;
    cfg.numAttrs = cut ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, p);
}

namespace {
void fill_update(LayerUpdParams& p, const UpdateDesc& d, const float* dy, const float* x, int tokens, int C, float lr, float lr_scale, float rms_beta,
                 float rms_eps, uint32_t seed, const uint32_t* seed_offset, int* err_word, int rows) {
    const int I = d.in_features, O = d.rows;
    p.dy = dy; p.x = x; p.tokens = tokens; p.O = O;
    p.vec_dy = (O & 3) == 0 && (reinterpret_cast<uintptr_t>(dy) & 15) == 0;
    const uint32_t upr = (uint32_t)(I / 16);
    p.magic = upr <= 1 ? 0u : (uint32_t)((0x100000000ull + upr - 1) / upr);
    p.err = err_word;
    UpdParams& u = p.u;
    u.state = d.state; u.scale = d.scale; u.v = d.v; u.grad_w = nullptr; u.packed2 = d.packed2;
    u.C = C; u.in_features = I; u.rows = O; u.row_offset = 0; u.rows_per_batch = rows;
    u.state_align = (I % 64 == 0 && (reinterpret_cast<uintptr_t>(d.state) & 15) == 0 && (reinterpret_cast<uintptr_t>(d.packed2) & 15) == 0) ? 16 : 4;
    u.lr = lr; u.lr_scale = lr_scale; u.rms_beta = rms_beta; u.rms_eps = rms_eps; u.seed = seed; u.seed_offset = seed_offset;
}
}  // namespace

cudaError_t launch_exact_update(const UpdateDesc& d, const float* dy, const float* x, int tokens, int C, float lr, float lr_scale,
                                float rms_beta, float rms_eps, uint32_t seed, const uint32_t* seed_offset, int sm_count, size_t max_smem,
                                cudaStream_t stream) {
    const int I = d.in_features, O = d.rows, gpr = I / 4;
    const bool with_q = lr_scale != 0.0f, u16 = I % 16 == 0 && (reinterpret_cast<uintptr_t>(d.state) & 3) == 0;
    // rows of a CTA: all SMs first, then as many as its threads take at once
    int R = (O + sm_count - 1) / sm_count;
    if (R > kLThreads / gpr) R = kLThreads / gpr;
    if (R < 1) R = 1;
    LayerUpdParams p = {};
    fill_update(p, d, dy, x, tokens, C, lr, lr_scale, rms_beta, rms_eps, seed, seed_offset, nullptr, R);
    const auto kern = u16 ? (with_q ? exact_update_kernel<true, true> : exact_update_kernel<false, true>)
                          : (with_q ? exact_update_kernel<true, false> : exact_update_kernel<false, false>);
    const cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), 48 + (u16 ? 2 : 0) + (with_q ? 1 : 0), max_smem);
    if (e != cudaSuccess) return e;
    return launch_chained(kern, dim3((unsigned)((O + R - 1) / R)), dim3(kLThreads), u16_layout(I, R, with_q, kLThreads / 64).total, stream, p);
}

cudaError_t launch_layer_update(const UpdateDesc& d, const float* dy, const float* x, int tokens, int C, float lr, float lr_scale,
                                float rms_beta, float rms_eps, uint32_t seed, const uint32_t* seed_offset, int* err_word, int sm_count,
                                size_t max_smem, cudaStream_t stream) {
    const int I = d.in_features, O = d.rows;
    const bool with_q = lr_scale != 0.0f;
    const bool u16 = I % 16 == 0 && (reinterpret_cast<uintptr_t>(d.state) & 3) == 0;
    const UpdateShape shape = update_shape(tokens, I, O, sm_count);
    const int mr = shape.mr, cs = shape.cs;
    const int slice = ((tokens + cs - 1) / cs + kDwK - 1) / kDwK * kDwK;
    const bool deep = slice > kDwDepth * kDwK;
    const auto pick = [&](auto d) {
        constexpr bool D = decltype(d)::value;
        return u16 ? (with_q ? layer_update_kernel<true, true, D> : layer_update_kernel<false, true, D>)
                   : (with_q ? layer_update_kernel<true, false, D> : layer_update_kernel<false, false, D>);
    };
    const auto kern = deep ? pick(std::true_type()) : pick(std::false_type());
    cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), (deep ? 32 : 20) + (u16 ? 2 : 0) + (with_q ? 1 : 0), max_smem);
    if (e != cudaSuccess) return e;
    {
        const int tiles = (O + mr - 1) / mr;
        LayerUpdParams p;
        p.mr = mr;
        const int R = mr / cs;
        const size_t base = (u16_layout(I, R, with_q, kLThreads / 64).total + 1023) & ~size_t(1023);
        size_t smem = 0;
        for (p.np = shape.np; p.np <= 16; ++p.np) {
            p.pw = ((I + p.np - 1) / p.np + 63) / 64 * 64;
            p.stage_bytes = 3 * kDwATerm + 3 * (p.pw / 64) * kDwChunk;
            const size_t area = 2 * (size_t)p.stage_bytes > 65536 ? 2 * (size_t)p.stage_bytes : 65536;
            smem = base + area + 1024;
            if (smem + 1024 <= max_smem) break;
        }
        if (p.np > 16) return cudaErrorInvalidConfiguration;
        p.off_stage = (int)base;
        fill_update(p, d, dy, x, tokens, C, lr, lr_scale, rms_beta, rms_eps, seed, seed_offset, err_word, R);
        p.slice = slice;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(tiles * cs));
        cfg.blockDim = dim3(kLThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)cs; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // launch_chained, with clusters
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        return cudaLaunchKernelEx(&cfg, kern, p);
    }
}

}  // namespace mcl
