// The 16-weight form of the counter update as a device function over rows in shared memory: the narrow-row kernels of
// counter_update.cu and the layer kernel that forms the gradient itself (layer_kernels.cu) run the same code.
#pragma once

#include "counter_codec.cuh"
#include "kernels.h"

namespace mcl {
namespace {

constexpr int kUpdThreads = 256;             // 4 warp pairs

struct UpdParams {
    uint8_t* state;          // [rows, in/4*3]
    float* scale;            // [rows]
    float* v;                // [rows]
    const float* grad_w;     // [rows, in]
    uint32_t* packed2;       // [rows, in/16] or null
    int C, in_features, rows, row_offset;
    int rows_per_batch;
    int state_align;         // 16, 4 or 1: widest access every state / packed2 row start allows
    float lr, lr_scale, rms_beta, rms_eps;
    uint32_t seed;
    const uint32_t* seed_offset;   // optional device word added to seed (a step counter for recorded batches)
};

// Per-row table indexed by the OLD code: x = float(c) * (s_old / s_new) (the rebased counter),
// y = index of the tail-table row of the code's ternary digit, pre-offset by kTailK.
struct RowEntry {
    float creb;
    int tail_base;
};

// ---------------------------------------------------------------------------------------------
// Fast variant for in_features % 16 == 0 (every benchmark shape): same phases, but
//   * a batch holds up to kMaxRowsU16 rows, so narrow layers still give each CTA thousands of
//     weights between barriers; a warp pair walks its rows of the batch one after another and
//     pairs meet on their own named barrier, not a CTA-wide one;
//   * the tick works on units of 16 weights = 3 aligned state words in, 3 state words + one
//     2-bit word out, all 32-bit shared-memory accesses; units of all rows of the batch are
//     flattened over the threads;
//   * the gradient tile in shared memory is XOR-swizzled at 16-byte granularity so that the
//     unit-strided 128-bit reads are bank-conflict free;
//   * the right shifts of the integer hash are issued as mul.hi (FMA pipe) because the ALU
//     pipe is the busiest one in this kernel.
constexpr int kMaxRowsU16 = 64;
#ifndef MCL_UPD_CTAS_PER_SM
#define MCL_UPD_CTAS_PER_SM 4         // resident CTAs per SM the 16-weight kernel is compiled and sized for
#endif
constexpr int kUpdCtasPerSm = MCL_UPD_CTAS_PER_SM;
constexpr int kPairs = kUpdThreads / 64;

__device__ __forceinline__ int swz4(int f) {          // float4 index -> swizzled float4 index
    return (f & ~3) | ((f & 3) ^ ((f >> 3) & 3));
}
__device__ __forceinline__ uint32_t shr_mulhi(uint32_t x, uint32_t pow2) {   // x >> (32 - log2(pow2))
    return pow2 == 65536u ? x >> 16 : x >> 15;
}

__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
    uint32_t v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a)); return v;
}
__device__ __forceinline__ float2 lds_f2(uint32_t a) {
    float2 v; asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a)); return v;
}
__device__ __forceinline__ float4 lds_f4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts_u32(uint32_t a, uint32_t v) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

__device__ __forceinline__ float fmax_nan(float a, float b) {          // max that keeps a NaN operand
    float r; asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b)); return r;
}

// Per-row constants of the tick (32 bytes).  gw / dn is formed without a division: yh = RN(1 / dn) and
// yl = RN((1 - dn * yh) * yh) make yh + yl equal 1 / dn to ~2^-47, so p = RN(gw * yh + RN(gw * yl)) is one of the
// two floats next to gw / dn, and one residual step  q = RN(p + (gw - dn * p) * yh)  (the residual is exact in an
// FMA) is the correctly rounded quotient -- the value the reference's IEEE division gives (Markstein's theorem:
// a faithful quotient, a reciprocal within 2^-24 relative, one FMA correction).  The argument needs no underflow:
// it holds for dn in [2^-32, 2^32] and |q| >= 2^-64; `qlo` is that bound for rows whose dn is in range and NaN for
// the others, and a unit whose smallest |q| fails  qmin >= qlo  is looked at again and, unless its small quotients
// are exact zeros, redone with the division.
struct RowK {
    float yh, yl, dn, k_tick, k_reb, qlo, pad0, pad1;
};

// Tick table of the 16-weight kernel: for weight position k in its group, old ternary digit t in {-1,0,1,2} and
// rounded counter ccv in [-64, 63]:  new code << 6k  |  (new digit + 1) << (24 + 2k), so that the four look-ups of
// a group ADD UP to its 24-bit state word and its byte of 2-bit fields.
constexpr int kTickN = 128;                      // entries per (k, t)
constexpr int kTickHalf = kTickN / 2;
constexpr int kTickBytes = 4 * 4 * kTickN * 4;   // 8 KiB
constexpr float kTickValMax = (float)(kTickHalf - 2);   // |counter + tick| below this stays inside the table

// The tick of one 16-weight unit (3 state words in, 3 state words and one word of 2-bit fields out), shared by the
// kernels below.  All operands are shared-memory addresses: sa_rowk the row's RowK, rt its 64-entry row table, sw the
// unit's three state words, g4 the first of its four gradient float4s (swizzled by jsw).  e_unit = global element
// index of the unit's first weight.
__device__ __forceinline__ void tick_unit16(const uint32_t sa_rowk, const uint32_t rt, const uint32_t sw, const uint32_t g4,
                                            const uint32_t jsw, const uint32_t e_unit, const uint32_t seed, const float neg_lr,
                                            const float Cf, const int C, const int lv, const uint32_t pow16,
                                            const uint32_t pow17, const DecodeLut* lut, uint32_t (&nwd)[4], uint32_t& fields) {
    const float4 rcv = lds_f4(sa_rowk);            // yh, yl, dn, k_tick
    const float2 rcw = lds_f2(sa_rowk + 16u);      // k_reb, qlo
    const float ndn = -rcv.z;
    const uint32_t s0 = lds_u32(sw), s1 = lds_u32(sw + 4), s2 = lds_u32(sw + 8);
    const uint32_t gwd[4] = {s0 & 0xFFFFFFu, (s0 >> 24) | ((s1 & 0xFFFFu) << 8),
                             (s1 >> 16) | ((s2 & 0xFFu) << 16), s2 >> 8};
    fields = 0;
    float vmax = 0.0f;                              // largest |counter + tick| of the unit (NaN if any is)
    float qmin = __int_as_float(0x7f800000);        // smallest |gw / dn| of the unit
#pragma unroll
    for (int gg = 0; gg < 4; ++gg) {
        const float4 gw = lds_f4(g4 + (((uint32_t)gg ^ jsw) << 4));
        const float gwv[4] = {gw.x, gw.y, gw.z, gw.w};
        const uint32_t w = gwd[gg];
        const uint32_t e0 = e_unit + 4u * gg;
        const uint32_t e0x = e0 ^ shr_mulhi(e0, pow16);
        uint32_t acc = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            // byte offset of the row-table entry of the old code: code * 8
            const uint32_t c8 = (k == 0 ? (w << 3) : (w >> (6 * k - 3))) & 0x1F8u;
            const float2 re = lds_f2(rt + c8);            // x = rebased counter, y = tick-table address (int bits)
            const float g = gwv[k];
            const float pq = __fmaf_rn(g, rcv.x, __fmul_rn(g, rcv.y));
            const float q = __fmaf_rn(__fmaf_rn(ndn, pq, g), rcv.x, pq);      // = RN(g / dn), see RowK
            qmin = fminf(qmin, fabsf(q));
            const float tick = __fmul_rn(__fmul_rn(neg_lr, q), rcv.w);
            const float val = __fadd_rn(re.x, tick);
            vmax = fmax_nan(vmax, fabsf(val));
            uint32_t x = (e0x ^ (uint32_t)k) * 0x7feb352du;
            x ^= shr_mulhi(x, pow17);            // x >> 15
            x *= 0x846ca68bu;
            x = seed ^ x ^ shr_mulhi(x, pow16);  // seed ^ hash(elem)
            x ^= shr_mulhi(x, pow16);
            x *= 0x7feb352du;
            x ^= shr_mulhi(x, pow17);
            x *= 0x846ca68bu;
            const uint32_t h = (x ^ shr_mulhi(x, pow16)) & 0x00ffffffu;
            const float f = floorf(val);
            const float rnd = __fmul_rn((float)h, 1.0f / 16777216.0f);
            int iccv;           // saturating conversion: a wild value still gives an address inside this CTA's shared memory
            asm("cvt.rni.sat.s8.f32 %0, %1;" : "=r"(iccv) : "f"(f));
            iccv += (rnd < __fsub_rn(val, f)) ? 1 : 0;
            acc += lds_u32((uint32_t)(__float_as_int(re.y) + 4 * iccv) + (uint32_t)(k * 4 * kTickN * 4));
        }
        nwd[gg] = acc & 0xFFFFFFu;
        fields |= (acc >> 24) << (8 * gg);
    }
    bool redo = !(vmax < kTickValMax);      // a rounded counter beyond the table, a code outside it, or a NaN
    if (!(qmin >= rcw.y)) {
        // a quotient below the range in which the division-free form is proven (or a row outside it): exact
        // zeros are fine, anything else goes to the formulas
        redo = redo || (rcw.y != rcw.y);
        for (int gg = 0; gg < 4 && !redo; ++gg) {
            const float4 gw = lds_f4(g4 + (((uint32_t)gg ^ jsw) << 4));
            const float gwv[4] = {gw.x, gw.y, gw.z, gw.w};
            for (int k = 0; k < 4; ++k)
                if (gwv[k] != 0.0f && !(fabsf(__fdiv_rn(gwv[k], rcv.z)) >= rcw.y)) redo = true;
        }
    }
    if (redo) {
        // rare: redo the unit with the reference formulas
        fields = 0;
        for (int gg = 0; gg < 4; ++gg) {
            const float4 gw = lds_f4(g4 + (((uint32_t)gg ^ jsw) << 4));
            const float gwv[4] = {gw.x, gw.y, gw.z, gw.w};
            uint32_t nw = 0;
            for (int k = 0; k < 4; ++k) {
                const float2 tc = lut->e[(gwd[gg] >> (6 * k)) & 63u];
                uint32_t fld;
                const uint32_t code = counter_tick(gwv[k], tc.x, tc.y, e_unit + (uint32_t)(4 * gg + k), seed,
                                                   neg_lr, rcv.z, rcv.w, rcw.x, Cf, C, lv, &fld);
                nw += (code & 0x3Fu) << (6 * k);
                fields += (fld & 3u) << (2 * (4 * gg + k));
            }
            nwd[gg] = nw;
        }
    }
}

// kernels/compact_counter.cl:129-136 evaluated for every (old digit, rounded counter) the table covers
__device__ __forceinline__ void build_tick_table(uint32_t* tick_tab, const int C, const int tid, const int nthreads) {
    const int lv = 2 * C - 1;
    const float Cf = (float)C;
    for (int e = tid; e < 4 * kTickN; e += nthreads) {
        const int t = e / kTickN - 1;
        const float ccv = (float)(e % kTickN - kTickHalf);
        const float carry = truncf(__fdiv_rn(ccv, Cf));
        float rem = __fsub_rn(ccv, __fmul_rn(carry, Cf));
        const int nt = t + (int)carry;
        const int ct = nt < -1 ? -1 : (nt > 1 ? 1 : nt);
        if (ct != nt) rem = __fmul_rn(ccv > 0.0f ? 1.0f : (ccv < 0.0f ? -1.0f : 0.0f), __fsub_rn(Cf, 1.0f));
        int ri = (int)rem;
        ri = ri < -(C - 1) ? -(C - 1) : (ri > C - 1 ? C - 1 : ri);
        const uint32_t code = (uint32_t)(((ct + 1) * lv + (ri + (C - 1))) & 0x3F);
        const uint32_t fld = (uint32_t)(ct + 1);
#pragma unroll
        for (int k = 0; k < 4; ++k) tick_tab[k * 4 * kTickN + e] = (code << (6 * k)) | (fld << (24 + 2 * k));
    }
}

// Row constants from the two row sums (kernels/compact_counter.cl:92-99); writes v and the new scale of the row.
template <bool WITH_Q>
__device__ __forceinline__ RowK finish_row_stats(const UpdParams& p, const int row, const float a, const float b, const float Cf,
                                                 const float s_old, const float v_old) {
    const int I = p.in_features;
    const float gsq = __fdiv_rn(a, (float)I);
    float s_new = s_old;
    if (WITH_Q) {
        const float gs = __fdiv_rn(b, __fsqrt_rn((float)I));
        s_new = __fsub_rn(s_old, __fmul_rn(p.lr_scale, gs));
    }
    s_new = fminf(fmaxf(s_new, 1e-5f), 10.0f);
    const float vv = __fadd_rn(__fmul_rn(p.rms_beta, v_old), __fmul_rn(__fsub_rn(1.0f, p.rms_beta), gsq));
    p.v[row] = vv;
    RowK rc;
    rc.dn = fmaxf(__fsqrt_rn(vv), p.rms_eps);
    rc.k_tick = __fdiv_rn(Cf, s_new);
    rc.k_reb = __fdiv_rn(s_old, s_new);
    rc.yh = __frcp_rn(rc.dn);
    rc.yl = __fmul_rn(__fmaf_rn(-rc.dn, rc.yh, 1.0f), rc.yh);
    const bool in_range = rc.dn >= 2.3283064365386963e-10f && rc.dn <= 4294967296.0f;     // 2^-32 .. 2^32
    rc.qlo = in_range ? 5.421010862427522e-20f : __int_as_float(0x7fc00000);                 // 2^-64 or NaN
    rc.pad0 = rc.pad1 = 0.0f;
    p.scale[row] = s_new;           // scale commit (kernels/basic.cl:6-9)
    return rc;
}

// Row-table entry of old code value `code`: the rebased counter and the shared-memory address of the tick-table entry
// of (k = 0, the code's digit, rounded counter 0).  A code whose ternary digit the tick table lacks gets an infinite
// counter, which sends its unit down the formula path.
__device__ __forceinline__ RowEntry row_entry(const DecodeLut* lut, const int code, const float k_reb, const uint32_t sa_tick) {
    const float2 tc = lut->e[code];
    const int ti = (int)tc.x + 1;
    const bool ok = ti >= 0 && ti < 4;
    RowEntry re;
    re.creb = ok ? __fmul_rn(tc.y, k_reb) : __int_as_float(0x7f800000);
    re.tail_base = (int)(sa_tick + 4u * (uint32_t)((ok ? ti : 0) * kTickN + kTickHalf));
    return re;
}

struct U16Layout {
    int sb, off_tick, off_rowc, off_part, off_rowtab, off_gw, off_st, off_so, off_p2;
    size_t total;
};
__host__ __device__ inline U16Layout u16_layout(int I, int R, bool with_q, int pairs = kPairs) {
    (void)with_q;
    U16Layout L;
    const int row_bytes = (I >> 2) * 3;
    L.sb = (row_bytes + 15) & ~15;
    size_t o = sizeof(DecodeLut);
    L.off_tick = (int)o; o += kTickBytes;
    L.off_rowc = (int)o; o += sizeof(RowK) * R;
    L.off_part = (int)o; o += sizeof(float) * 64 * pairs;
    L.off_rowtab = (int)o; o += sizeof(RowEntry) * 64 * (size_t)R;
    L.off_gw = (int)o; o += sizeof(float) * (size_t)R * I;
    L.off_st = (int)o; o += (size_t)R * L.sb + 16;
    L.off_so = (int)o; o += (size_t)R * L.sb + 16;
    L.off_p2 = (int)o; o += (size_t)R * (I >> 2);
    L.total = (o + 15) & ~size_t(15);
    return L;
}

// state rows row0 .. row0 + nrows - 1 into shared memory
template <int NT>
__device__ __forceinline__ void u16_load_state(const UpdParams& p, const U16Layout& L, unsigned char* smem, const int row0, const int nrows) {
    const int row_bytes = (p.in_features >> 2) * 3, tid = threadIdx.x;
    unsigned char* st_s = smem + L.off_st;
    const uint8_t* src = p.state + (size_t)row0 * row_bytes;
    if (p.state_align >= 16) {        // row_bytes % 16 == 0: one flat copy, smem row stride == row_bytes
        const uint4* s4 = reinterpret_cast<const uint4*>(src);
        uint4* d4 = reinterpret_cast<uint4*>(st_s);
        for (int i = tid; i < nrows * (row_bytes >> 4); i += NT) d4[i] = load_behind(s4 + i);
    } else {                          // rows are 4-byte aligned; smem rows padded to L.sb
        const uint32_t* s1 = reinterpret_cast<const uint32_t*>(src);
        const int wpr = row_bytes >> 2;
        for (int i = tid; i < nrows * wpr; i += NT) {
            const int r = i / wpr, w = i - r * wpr;
            reinterpret_cast<uint32_t*>(st_s + (size_t)r * L.sb)[w] = load_behind(s1 + i);
        }
    }
}

// Body shared by the single-layer and the grouped kernel: batches batch0, batch0 + batch_step, ... of the
// layer `p`.  The decode and tick tables depend on C alone; `build_tables` is false when an earlier call
// of the same CTA already built them for this C.
// GW_READY: state and gradient rows of the one batch already lie in shared memory as the load phase leaves them.
// NT: threads of the CTA.
template <bool WITH_Q, bool GW_READY = false, int NT = kUpdThreads>
__device__ __forceinline__ void update_u16_body(const UpdParams& p, const uint32_t unit_magic, const uint32_t pow16,
                                                const uint32_t pow17, const int batch0, const int batch_step,
                                                const bool build_tables) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int I = p.in_features;
    const int gpr = I >> 2;               // packed groups (float4s) per row
    const int upr = I >> 4;               // 16-weight units per row
    const int row_bytes = gpr * 3;
    const int R = p.rows_per_batch;
    const U16Layout L = u16_layout(I, R, WITH_Q, NT / 64);

    DecodeLut* lut = reinterpret_cast<DecodeLut*>(smem);
    uint32_t* tick_tab = reinterpret_cast<uint32_t*>(smem + L.off_tick);
    RowK* rowc = reinterpret_cast<RowK*>(smem + L.off_rowc);
    float* part = reinterpret_cast<float*>(smem + L.off_part);
    RowEntry* rowtab = reinterpret_cast<RowEntry*>(smem + L.off_rowtab);
    float4* gw_s = reinterpret_cast<float4*>(smem + L.off_gw);
    unsigned char* st_s = smem + L.off_st;
    unsigned char* so_s = smem + L.off_so;
    uint32_t* p2_s = reinterpret_cast<uint32_t*>(smem + L.off_p2);
    const uint32_t sa0 = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t sa_tick = sa0 + L.off_tick, sa_rowc = sa0 + L.off_rowc, sa_rowtab = sa0 + L.off_rowtab;
    const uint32_t sa_gw = sa0 + L.off_gw, sa_st = sa0 + L.off_st, sa_so = sa0 + L.off_so, sa_p2 = sa0 + L.off_p2;

    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int lv = 2 * p.C - 1;
    const float Cf = (float)p.C;
    const float neg_lr = -p.lr;
    const uint32_t seed = p.seed + (p.seed_offset ? load_behind(p.seed_offset) : 0u);
    const bool aligned16 = p.state_align >= 16;

    if (build_tables) {
        __syncthreads();                  // an earlier layer's batches may still read the old tables
        build_decode_lut(lut, p.C, tid, NT);
        build_tick_table(tick_tab, p.C, tid, NT);
    }
    __syncthreads();

    const int nbatches = (p.rows + R - 1) / R;
    for (int batch = batch0; batch < nbatches; batch += batch_step) {
        const int row0 = batch * R;
        const int nrows = min(R, p.rows - row0);
        const float s_old = tid < nrows ? p.scale[row0 + tid] : 0.0f, v_old = tid < nrows ? p.v[row0 + tid] : 0.0f;

        // ---- load: the batch's rows are contiguous in global memory ------------------------
        {
            if (!GW_READY) u16_load_state<NT>(p, L, smem, row0, nrows);
            if (!GW_READY) {
            const float4* gsrc = reinterpret_cast<const float4*>(p.grad_w + (size_t)row0 * I);
            const int n4 = nrows * gpr;
            if ((gpr & 31) == 0) {  // rows start on a period of the swizzle: the flat float4 index can be swizzled as it is
                int i = tid;
                for (; i + 3 * NT < n4; i += 4 * NT) {       // four loads in flight per thread
                    const float4 v0 = load_behind(gsrc + i), v1 = load_behind(gsrc + i + NT), v2 = load_behind(gsrc + i + 2 * NT),
                                 v3 = load_behind(gsrc + i + 3 * NT);
                    gw_s[swz4(i)] = v0; gw_s[swz4(i + NT)] = v1;
                    gw_s[swz4(i + 2 * NT)] = v2; gw_s[swz4(i + 3 * NT)] = v3;
                }
                for (; i < n4; i += NT) gw_s[swz4(i)] = load_behind(gsrc + i);
            } else {                // flat over the batch; row = i / gpr by multiply-high (gpr = 4 * units per row)
                for (int i = tid; i < n4; i += NT) {
                    const int r = unit_magic ? (int)__umulhi((uint32_t)i >> 2, unit_magic) : (i >> 2);
                    const int g = i - r * gpr;
                    gw_s[r * gpr + swz4(g)] = load_behind(gsrc + i);
                }
            }
            }
        }
        __syncthreads();

        // ---- stats: a warp per row, two of the 64 lanes of the reduction per thread; then the constants of all rows at once ------
        // (a pair of warps that finished each row before its next one spent 1500 clocks a row on one lane's divisions)
        for (int r = warp; r < nrows; r += NT / 32) {
            float a0 = 0.0f, a1 = 0.0f, b0 = 0.0f, b1 = 0.0f;
            const float4* g4 = gw_s + r * gpr;
            const uint32_t* raw = reinterpret_cast<const uint32_t*>(st_s + (size_t)r * L.sb);
            auto add = [&](const int g, float& a, float& b) {
                const float4 gw = g4[swz4(g)];
                a = __fadd_rn(a, __fmul_rn(gw.x, gw.x));
                a = __fadd_rn(a, __fmul_rn(gw.y, gw.y));
                a = __fadd_rn(a, __fmul_rn(gw.z, gw.z));
                a = __fadd_rn(a, __fmul_rn(gw.w, gw.w));
                if (WITH_Q) {
                    const uint32_t w = load_group24(raw, (uint32_t)g * 3u);
                    b = __fadd_rn(b, __fmul_rn(gw.x, lut->e[w & 63u].x));
                    b = __fadd_rn(b, __fmul_rn(gw.y, lut->e[(w >> 6) & 63u].x));
                    b = __fadd_rn(b, __fmul_rn(gw.z, lut->e[(w >> 12) & 63u].x));
                    b = __fadd_rn(b, __fmul_rn(gw.w, lut->e[(w >> 18) & 63u].x));
                }
            };
            for (int g = lane; g < gpr; g += 64) {
                add(g, a0, b0);
                if (g + 32 < gpr) add(g + 32, a1, b1);
            }
            float a = __fadd_rn(a0, a1), b = __fadd_rn(b0, b1);
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) {
                a = __fadd_rn(a, __shfl_down_sync(0xffffffffu, a, s));
                if (WITH_Q) b = __fadd_rn(b, __shfl_down_sync(0xffffffffu, b, s));
            }
            if (lane == 0) { part[2 * r] = a; part[2 * r + 1] = b; }
        }
        __syncthreads();
        if (tid < nrows) rowc[tid] = finish_row_stats<WITH_Q>(p, row0 + tid, part[2 * tid], part[2 * tid + 1], Cf, s_old, v_old);
        __syncthreads();
        for (int e = tid; e < nrows * 64; e += NT) rowtab[e] = row_entry(lut, e & 63, rowc[e >> 6].k_reb, sa_tick);     // one entry per old code value
        __syncthreads();

        // ---- tick: 16 weights per thread-iteration, units of the whole batch flattened --------
        // Shared memory is addressed with 32-bit shared-space addresses (ld.shared / st.shared), which
        // keeps the address arithmetic of the data-dependent table look-ups to one add each.
        const int nunits = nrows * upr;
        for (int u = tid; u < nunits; u += NT) {
            const int r = unit_magic ? (int)__umulhi((uint32_t)u, unit_magic) : u;       // u / upr (magic 0: upr == 1)
            const int j = u - r * upr;
            const uint32_t g4 = sa_gw + ((uint32_t)(r * gpr + 4 * j) << 4);
            const uint32_t e_unit = (uint32_t)(p.row_offset + row0 + r) * (uint32_t)I + (uint32_t)(16 * j);
            uint32_t nwd[4], fields;
            tick_unit16(sa_rowc + (uint32_t)r * 32u, sa_rowtab + (uint32_t)r * 512u,
                        sa_st + (uint32_t)r * (uint32_t)L.sb + 12u * (uint32_t)j, g4, (uint32_t)((j >> 1) & 3), e_unit, seed,
                        neg_lr, Cf, p.C, lv, pow16, pow17, lut, nwd, fields);
            const uint32_t so = sa_so + (uint32_t)r * (uint32_t)L.sb + 12u * (uint32_t)j;
            sts_u32(so, nwd[0] | (nwd[1] << 24));
            sts_u32(so + 4, (nwd[1] >> 8) | (nwd[2] << 16));
            sts_u32(so + 8, (nwd[2] >> 16) | (nwd[3] << 8));
            sts_u32(sa_p2 + 4u * (uint32_t)(r * upr + j), fields);
        }
        __syncthreads();

        // ---- store (the next batch's loads follow without a barrier: they touch other arrays) ------------
        {
            uint8_t* dst = p.state + (size_t)row0 * row_bytes;
            if (aligned16) {
                const uint4* s4 = reinterpret_cast<const uint4*>(so_s);
                uint4* d4 = reinterpret_cast<uint4*>(dst);
                for (int i = tid; i < nrows * (row_bytes >> 4); i += NT) d4[i] = s4[i];
            } else {
                uint32_t* d1 = reinterpret_cast<uint32_t*>(dst);
                const int wpr = row_bytes >> 2;
                for (int i = tid; i < nrows * wpr; i += NT) {
                    const int r = i / wpr, w = i - r * wpr;
                    d1[i] = reinterpret_cast<const uint32_t*>(so_s + (size_t)r * L.sb)[w];
                }
            }
            if (p.packed2 != nullptr) {
                uint32_t* d = p.packed2 + (size_t)row0 * upr;
                if (aligned16) {
                    const uint4* s4 = reinterpret_cast<const uint4*>(p2_s);
                    uint4* d4 = reinterpret_cast<uint4*>(d);
                    for (int i = tid; i < (nrows * upr) >> 2; i += NT) d4[i] = s4[i];
                } else {
                    for (int i = tid; i < nrows * upr; i += NT) d[i] = p2_s[i];
                }
            }
        }
    }
}

}  // namespace
}  // namespace mcl
