// Grouped-query attention on tensor cores, for heads up to 64, where the grid fills the GPU or one tile holds all keys (attention.cuh serves the others): every fp32
// operand is three bf16 terms of eight bits each (cut off, not rounded: the three are the fp32 value exactly), a product is the
// six term products above 2^-24 (mma.sync m16n8k16; a tile of 16 x 64 by 64 is too small for tcgen05's round trips).  The leading products
// of every step have an accumulator of their own and are added in fp32, so that tensor-core rounding never sees a sum.
//
// A warp owns 16 queries of one head (the key kernel: 16 keys) and keeps their terms in registers; a CTA of four walks over tiles of 64
// keys, whose terms lie in shared memory, split once per CTA.  Scores turn into the next product's operand in registers.  The next tile
// comes by cp.async under the products of this one.
//   forward   online softmax: S -> P -> O = O alpha + P V
//   backward  kernel 1 (queries): S and dP, kept in the caller's scratch, with maximum, sum and sum of P dP; then P, dS from them
//             (written, as the reference leaves them) and dq += dS K.
//             kernel 2 (keys): dv = P^T dO, dk = dS^T Q, summed over the query heads of the kv head; P and dS are read in
//             operand order, 32 bytes of a row by eight lanes.
// What bounds it: a warp's chain of loads, products and exponentials; the tensor pipe is busy for a quarter to a third of the time (m16n8k16 takes 8
// cycles of a quarter SM here: 1016 multiply-adds per clock and SM, a sixth of that for fp32; the FMAs of attention.cuh could do 256).  Causal, us with FMAs and here: 16 sequences of 256 tokens, 6 heads of
// 48: forward 37 and 28, backward 111 and 80; 16 of 512, 12 heads of 64: 316 and 184, 798 and 557; one of 33 tokens, 8 heads of 48: 14 and 8, 40
// and 24; a grid of 192 CTAs with eight key tiles each (2 of 512, 12 of 64) 50 and 68, 206 and 268.  Error against float64 1.5 to 2.5e-7 (2.1 to 5.1e-7).
#pragma once

// two fp32 values -> their three bf16 terms, packed two per word
__device__ __forceinline__ void terms3(float a, float b, uint32_t (&t)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const uint32_t x = __float_as_uint(a), y = __float_as_uint(b);
        t[i] = __byte_perm(x, y, 0x7632);
        if (i < 2) { a -= __uint_as_float(x & 0xFFFF0000u); b -= __uint_as_float(y & 0xFFFF0000u); }
    }
}
template <int NC>
struct AttTile {                                     // 64 rows of HDP columns, three planes of bf16 terms; the pitch keeps ldmatrix free of conflicts
    static constexpr int HDP = 16 * NC, kPitch = HDP + 8, kPlane = 64 * kPitch * 2, kBytes = 3 * kPlane;
    static constexpr int kRaw = 64 * HDP * 4;        // the fp32 rows as they come
};
__device__ __forceinline__ uint32_t sm_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// staging rows -> terms; thread t of NT
template <int NC, int NT>
__device__ __forceinline__ void split_tile(unsigned char* dst, const float* raw, int t) {
    using T = AttTile<NC>;
#pragma unroll
    for (int i0 = 0; i0 < 64 * T::HDP / 4; i0 += NT) {
        const int i = i0 + t, row = i / (T::HDP / 4), d = (i - row * (T::HDP / 4)) * 4;
        const float4 v = *reinterpret_cast<const float4*>(raw + row * T::HDP + d);
        uint32_t a[3], b[3];
        terms3(v.x, v.y, a); terms3(v.z, v.w, b);
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint2*>(dst + k * T::kPlane + (row * T::kPitch + d) * 2) = make_uint2(a[k], b[k]);
    }
}
__device__ __forceinline__ void ldm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16_first(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {      // onto zero
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}
// c[n] (two column tiles) = sum over KS steps of 16 of the six term products of a[k] and the operand that `load` brings for step k (three
// planes, both tiles: [plane][0..1] and [2..3]).  The leading products of every step and the two orders of small ones each have
// accumulators of their own, added in fp32: short chains (of two of 18 MMAs before, a warp waited for most of them), and an error
// below that of fp32 sums.
template <int KS, class Load>
__device__ __forceinline__ void term_products(float (&c)[2][4], const uint32_t (&a)[KS][3][4], const Load& load) {
    float s1[2][4], s2[2][4];
#pragma unroll
    for (int k = 0; k < KS; ++k) {
        uint32_t b[3][4];
        float h[2][4];
#pragma unroll
        for (int t = 0; t < 3; ++t) load(b[t], t, k);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            if (k == 0) mma_bf16_first(s2[n], a[k][2], b[0][2 * n], b[0][2 * n + 1]);
            else mma_bf16(s2[n], a[k][2], b[0][2 * n], b[0][2 * n + 1]);
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            if (k == 0) mma_bf16_first(s1[n], a[k][1], b[0][2 * n], b[0][2 * n + 1]);
            else mma_bf16(s1[n], a[k][1], b[0][2 * n], b[0][2 * n + 1]);
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) mma_bf16_first(h[n], a[k][0], b[0][2 * n], b[0][2 * n + 1]);
#pragma unroll
        for (int n = 0; n < 2; ++n) mma_bf16(s2[n], a[k][0], b[2][2 * n], b[2][2 * n + 1]);
#pragma unroll
        for (int n = 0; n < 2; ++n) mma_bf16(s1[n], a[k][0], b[1][2 * n], b[1][2 * n + 1]);
#pragma unroll
        for (int n = 0; n < 2; ++n) mma_bf16(s2[n], a[k][1], b[1][2 * n], b[1][2 * n + 1]);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) c[n][i] = k == 0 ? h[n][i] : c[n][i] + h[n][i];
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) c[n][i] += s1[n][i] + s2[n][i];
}
// c[n] = sum over d of a[16 rows][d] b[8 n' + .][d] for rows b0 .. b0 + 15 of a tile (two column tiles)
template <int NC>
__device__ __forceinline__ void rows_product(float (&c)[2][4], const uint32_t (&a)[NC][3][4], uint32_t tile, int b0, int lane) {
    using T = AttTile<NC>;
    const uint32_t at = tile + (uint32_t)(((b0 + ((lane >> 4) << 3) + (lane & 7)) * T::kPitch + ((lane >> 3) & 1) * 8) * 2);
    term_products<NC>(c, a, [&](uint32_t (&b)[4], int t, int k) { ldm4(b, at + t * T::kPlane + k * 32); });
}
// c[n] = sum over 16 KS rows r of a[16][r] b[r][8 (n0 + n) + .]: rows from r0 on of a tile, column tiles n0 and n0 + 1
template <int NC, int KS>
__device__ __forceinline__ void cols_product(float (&c)[2][4], const uint32_t (&a)[KS][3][4], uint32_t tile, int r0, int n0, int lane) {
    using T = AttTile<NC>;
    const uint32_t at = tile + (uint32_t)(((r0 + ((lane >> 3) & 1) * 8 + (lane & 7)) * T::kPitch + (n0 + (lane >> 4)) * 8) * 2);
    term_products<KS>(c, a, [&](uint32_t (&b)[4], int t, int k) { ldm4t(b, at + t * T::kPlane + k * 16 * T::kPitch * 2); });
}
// scores of 16 rows x 16 columns (two column tiles) -> terms of the operand of a product along those columns
__device__ __forceinline__ void as_operand(uint32_t (&a)[3][4], const float (&c)[2][4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {                    // (row g, columns 2 tq), (g + 8, .), then the second tile
        uint32_t t[3];
        terms3(c[i >> 1][2 * (i & 1)], c[i >> 1][2 * (i & 1) + 1], t);
#pragma unroll
        for (int k = 0; k < 3; ++k) a[k][i] = t[k];
    }
}
// terms of 16 rows of a [*, ld] matrix as the row operand
template <int NC>
__device__ __forceinline__ void load_rows(uint32_t (&a)[NC][3][4], const float* __restrict__ src, long long ld, int r0, int rmax, int hd, int lane) {
    const int g = lane >> 2, tq = lane & 3;
#pragma unroll
    for (int k = 0; k < NC; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = r0 + g + (i & 1) * 8, d = k * 16 + (i >> 1) * 8 + 2 * tq;
            const float* s = src + (long long)row * ld + d;
            const float x = row < rmax && d < hd ? __ldg(s) : 0.0f, y = row < rmax && d + 1 < hd ? __ldg(s + 1) : 0.0f;
            uint32_t t[3];
            terms3(x, y, t);
#pragma unroll
            for (int j = 0; j < 3; ++j) a[k][j][i] = t[j];
        }
}
__device__ __forceinline__ float quad_max(float v) { v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1)); return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2)); }
__device__ __forceinline__ float quad_sum(float v) { v += __shfl_xor_sync(0xffffffffu, v, 1); return v + __shfl_xor_sync(0xffffffffu, v, 2); }

// Terms of an infinity are an infinity and NaNs.  A warp whose results are not all finite does its rows again as plain fp32 sums over the
// keys that they attend to: an infinity or NaN in an operand shows in the result.
template <int N>
__device__ __forceinline__ bool beyond_fp32(const float (&c)[N][4]) {
    bool b = false;
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) b = b || !(fabsf(c[n][i]) <= FLT_MAX);
    return __any_sync(0xffffffffu, b);
}
__device__ __forceinline__ float row_dot(const float* a, const float* b, int n) {
    float s = 0.0f;
    for (int d = 0; d < n; ++d) s = fmaf(a[d], b[d], s);
    return s;
}
// c (columns lane and lane + 32) += sum over 32 lanes of w times that lane's row; rows: the first of them, ld apart
__device__ __forceinline__ void add_rows(float (&c)[2], float w, const float* rows, long long ld, int count, int n, int lane) {
    for (int j = 0; j < count; ++j) {
        const float f = __shfl_sync(0xffffffffu, w, j);
        for (int i = 0; i < 2; ++i)
            if (lane + 32 * i < n) c[i] = fmaf(f, rows[j * ld + lane + 32 * i], c[i]);
    }
}
// rows r0 .. r0 + 15: q and out at row 0 of the head
__device__ __noinline__ void fwd_again(const float* q, const float* k, const float* v, float* out, const GqaDims& p, int r0) {
    const int lane = threadIdx.x & 31;
    const long long qld = (long long)p.n_head * p.hd, kld = (long long)p.n_kv * p.hd;
    for (int r = r0; r < min(r0 + 16, p.tq); ++r) {
        const int lo = row_lo(p, r), hi = row_hi(p, r);
        float m = -FLT_MAX, l = 0.0f, c[2] = {};
        for (int k0 = lo; k0 < hi; k0 += 32)
            if (k0 + lane < hi) m = fmaxf(m, row_dot(q + r * qld, k + (k0 + lane) * kld, p.hd) * p.scale);
        m = warp_max(m);
        for (int k0 = lo; k0 < hi; k0 += 32) {
            const float e = k0 + lane < hi ? expf(row_dot(q + r * qld, k + (k0 + lane) * kld, p.hd) * p.scale - m) : 0.0f;
            l += e;
            add_rows(c, e, v + k0 * kld, kld, min(32, hi - k0), p.hd, lane);
        }
        l = warp_sum(l);
        for (int i = 0; i < 2; ++i)
            if (lane + 32 * i < p.hd) out[r * qld + lane + 32 * i] = c[i] * (l > 0.0f ? 1.0f / l : 0.0f);
    }
}
// rows r0 .. r0 + 15 of probs, ds (of this head) and dq
__device__ __noinline__ void bwd_q_again(const float* q, const float* k, const float* v, const float* dout, float* probs, float* ds, float* dq, const GqaDims& p, int r0) {
    const int lane = threadIdx.x & 31;
    const long long qld = (long long)p.n_head * p.hd, kld = (long long)p.n_kv * p.hd;
    __syncwarp();                                          // other lanes wrote to these rows
    for (int r = r0; r < min(r0 + 16, p.tq); ++r) {
        const int hi = row_hi(p, r);
        float* pr = probs + (long long)r * p.tk;
        float* dr = ds + (long long)r * p.tk;
        float m = -FLT_MAX, l = 0.0f, dot = 0.0f, c[2] = {};
        for (int j = lane; j < hi; j += 32) {              // this lane reads them back
            pr[j] = row_dot(q + r * qld, k + j * kld, p.hd) * p.scale;
            dr[j] = row_dot(dout + r * qld, v + j * kld, p.hd);
            m = fmaxf(m, pr[j]);
        }
        m = warp_max(m);
        for (int j = lane; j < hi; j += 32) {
            const float e = expf(pr[j] - m);
            l += e;
            dot = fmaf(e, dr[j], dot);
        }
        l = warp_sum(l);
        l = l > 0.0f ? 1.0f / l : 0.0f;
        dot = warp_sum(dot) * l;
        for (int k0 = 0; k0 < p.tk; k0 += 32) {
            const int j = k0 + lane;
            const float e = j < hi ? expf(pr[j] - m) * l : 0.0f, w = j < hi ? e * (dr[j] - dot) : 0.0f;
            if (j < p.tk) { pr[j] = e; dr[j] = w; }
            if (k0 < hi) add_rows(c, w, k + k0 * kld, kld, min(32, hi - k0), p.hd, lane);
        }
        for (int i = 0; i < 2; ++i)
            if (lane + 32 * i < p.hd) dq[r * qld + lane + 32 * i] = c[i] * p.scale;
    }
}
// keys k0 .. k0 + 15 of a kv head: q, dout, probs and ds at the first query head of its group
__device__ __noinline__ void bwd_k_again(const float* q, const float* dout, const float* probs, const float* ds, float* dk, float* dv, const GqaDims& p, int k0) {
    const int lane = threadIdx.x & 31;
    const long long qld = (long long)p.n_head * p.hd, kld = (long long)p.n_kv * p.hd;
    for (int key = k0; key < min(k0 + 16, p.tk); ++key) {
        float cv[2] = {}, ck[2] = {};
        for (int h = 0; h < p.n_head / p.n_kv; ++h)
            for (int r = p.causal ? max(key - p.q_off, 0) : 0; r < p.tq; ++r) {
                const long long at = ((long long)h * p.tq + r) * p.tk + key;
                for (int i = 0; i < 2; ++i)
                    if (lane + 32 * i < p.hd) {
                        cv[i] = fmaf(probs[at], dout[r * qld + h * p.hd + lane + 32 * i], cv[i]);
                        ck[i] = fmaf(ds[at], q[r * qld + h * p.hd + lane + 32 * i], ck[i]);
                    }
            }
        for (int i = 0; i < 2; ++i)
            if (lane + 32 * i < p.hd) { dv[key * kld + lane + 32 * i] = cv[i]; dk[key * kld + lane + 32 * i] = ck[i] * p.scale; }
    }
}

template <int NC>
__global__ void __launch_bounds__(128, 2) gqa_fwd_mma_kernel(const float* __restrict__ q, const float* __restrict__ k,
                                                                       const float* __restrict__ v, float* __restrict__ out, const __grid_constant__ GqaDims p) {
    grid_release();
    extern __shared__ __align__(16) unsigned char smb[];
    using T = AttTile<NC>;
    constexpr int NT = 128, BQ = 64;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, tq = lane & 3;
    unsigned char *ks = smb, *vs = smb + T::kBytes;
    float *kr = reinterpret_cast<float*>(smb + 2 * T::kBytes), *vr = kr + T::kRaw / 4;
    const int tiles = (p.tq + BQ - 1) / BQ, q0 = (tiles - 1 - (int)blockIdx.y) * BQ;
    const int b = blockIdx.x / p.n_head, h = blockIdx.x % p.n_head, gr = h / (p.n_head / p.n_kv);
    const long long qld = (long long)p.n_head * p.hd, kld = (long long)p.n_kv * p.hd;
    const float* kb_ = k + (long long)b * p.key_stride * kld + gr * p.hd;
    const float* vb = v + (long long)b * p.key_stride * kld + gr * p.hd;
    int kbeg, kend;
    tile_range<BQ>(p, q0, kbeg, kend);
    const bool vec = rows16(kb_, kld, p.hd) && rows16(vb, kld, p.hd);
    auto copy = [&](int k0) {
        copy_rows<kKT, NT, T::HDP, T::HDP>(kr, kb_, kld, k0, p.tk, p.hd, vec, t);
        copy_rows<kKT, NT, T::HDP, T::HDP>(vr, vb, kld, k0, p.tk, p.hd, vec, t);
    };
    copy(kbeg);
    const int r0 = q0 + 16 * warp;
    uint32_t qf[NC][3][4];
    load_rows<NC>(qf, q + (long long)b * p.tq * qld + h * p.hd, qld, r0, p.tq, p.hd, lane);
    float m[2] = {-FLT_MAX, -FLT_MAX}, l[2] = {0.0f, 0.0f}, o[2 * NC][4];
#pragma unroll
    for (int n = 0; n < 2 * NC; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[n][i] = 0.0f;
    const int lo[2] = {row_lo(p, r0 + g), row_lo(p, r0 + g + 8)}, hi[2] = {row_hi(p, r0 + g), row_hi(p, r0 + g + 8)};
    for (int k0 = kbeg; k0 < kend; k0 += kKT) {
        copies_wait<0>();
        __syncthreads();
        split_tile<NC, NT>(ks, kr, t);
        split_tile<NC, NT>(vs, vr, t);
        __syncthreads();
        if (k0 + kKT < kend) copy(k0 + kKT);
        float s[4][2][4], mx[2] = {m[0], m[1]};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            rows_product<NC>(s[j], qf, sm_addr(ks), 16 * j, lane);
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int key = k0 + 16 * j + 8 * n + 2 * tq + (i & 1);
                    s[j][n][i] = key < lo[i >> 1] || key >= hi[i >> 1] ? -FLT_MAX : s[j][n][i] * p.scale;
                    mx[i >> 1] = fmaxf(mx[i >> 1], s[j][n][i]);
                }
        }
        float alpha[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            mx[r] = quad_max(mx[r]);
            alpha[r] = expf(m[r] - mx[r]);
            l[r] *= alpha[r];                      // this lane's keys: added over the four lanes at the end
            m[r] = mx[r];
        }
        uint32_t pf[4][3][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    s[j][n][i] = s[j][n][i] == -FLT_MAX ? 0.0f : expf(s[j][n][i] - mx[i >> 1]);
                    l[i >> 1] += s[j][n][i];
                }
            as_operand(pf[j], s[j]);
        }
#pragma unroll
        for (int n = 0; n < 2 * NC; n += 2) {
            float c[2][4];
            cols_product<NC, 4>(c, pf, sm_addr(vs), 0, n, lane);
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int i = 0; i < 4; ++i) o[n + e][i] = fmaf(o[n + e][i], alpha[i >> 1], c[e][i]);
        }
    }
    copies_wait<0>();
    if (beyond_fp32(o)) {
        fwd_again(q + (long long)b * p.tq * qld + h * p.hd, kb_, vb, out + (long long)b * p.tq * qld + h * p.hd, p, r0);
        return;
    }
    float* ob = out + (long long)b * p.tq * qld + h * p.hd;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const float sum = quad_sum(l[r]), inv = sum > 0.0f ? 1.0f / sum : 0.0f;
        const int row = r0 + g + 8 * r;
        if (row >= p.tq) continue;
#pragma unroll
        for (int n = 0; n < 2 * NC; ++n)
#pragma unroll
            for (int i = 0; i < 2; ++i)
                if (8 * n + 2 * tq + i < p.hd) ob[(long long)row * qld + 8 * n + 2 * tq + i] = o[n][2 * r + i] * inv;
    }
}

// probs, ds [B, n_head, tq, tk]; dq
template <int NC>
__global__ void __launch_bounds__(128, 2) gqa_bwd_q_mma_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                                                           const float* __restrict__ dout, float* __restrict__ probs, float* __restrict__ ds,
                                                           float* __restrict__ dq, const __grid_constant__ GqaDims p) {
    grid_release();
    extern __shared__ __align__(16) unsigned char smb[];
    using T = AttTile<NC>;
    constexpr int NT = 128, BQ = 64;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, tq = lane & 3;
    unsigned char *ks = smb, *vs = smb + T::kBytes;
    float *kr = reinterpret_cast<float*>(smb + 2 * T::kBytes), *vr = kr + T::kRaw / 4;
    const int tiles = (p.tq + BQ - 1) / BQ, q0 = (tiles - 1 - (int)blockIdx.y) * BQ;
    const int b = blockIdx.x / p.n_head, h = blockIdx.x % p.n_head, gr = h / (p.n_head / p.n_kv);
    const long long qld = (long long)p.n_head * p.hd, kld = (long long)p.n_kv * p.hd, at = (long long)b * p.tq * qld + h * p.hd;
    const float* kb_ = k + (long long)b * p.tk * kld + gr * p.hd;
    const float* vb = v + (long long)b * p.tk * kld + gr * p.hd;
    int kbeg, kend;
    tile_range<BQ>(p, q0, kbeg, kend);
    const bool vec = rows16(kb_, kld, p.hd) && rows16(vb, kld, p.hd);
    auto copy = [&](int k0) {
        copy_rows<kKT, NT, T::HDP, T::HDP>(kr, kb_, kld, k0, p.tk, p.hd, vec, t);
        copy_rows<kKT, NT, T::HDP, T::HDP>(vr, vb, kld, k0, p.tk, p.hd, vec, t);
    };
    copy(0);
    const int r0 = q0 + 16 * warp;
    uint32_t qf[NC][3][4], gf[NC][3][4];
    load_rows<NC>(qf, q + at, qld, r0, p.tq, p.hd, lane);
    load_rows<NC>(gf, dout + at, qld, r0, p.tq, p.hd, lane);
    float m[2] = {-FLT_MAX, -FLT_MAX}, l[2] = {0.0f, 0.0f}, dot[2] = {0.0f, 0.0f};
    const int end[2] = {r0 + g < p.tq ? row_hi(p, r0 + g) : 0, r0 + g + 8 < p.tq ? row_hi(p, r0 + g + 8) : 0};
    const long long plane = ((long long)blockIdx.x * p.tq + r0 + g) * p.tk;
    const bool pairs = ((p.tk | (int)(reinterpret_cast<uintptr_t>(probs) >> 2) | (int)(reinterpret_cast<uintptr_t>(ds) >> 2)) & 1) == 0;
    // two column tiles of rows g and g + 8 from key0 on, what of them exists
    auto store = [&](float* to, const float (&c)[2][4], int key0) {
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const int key = key0 + 8 * n + 2 * tq;
                float* w = to + plane + (long long)(8 * r) * p.tk + key;
                if (r0 + g + 8 * r >= p.tq || key >= p.tk) continue;
                if (pairs) *reinterpret_cast<float2*>(w) = make_float2(c[n][2 * r], c[n][2 * r + 1]);
                else { w[0] = c[n][2 * r]; if (key + 1 < p.tk) w[1] = c[n][2 * r + 1]; }
            }
    };
    auto fetch = [&](const float* from, float (&c)[2][4], int key0) {
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const int key = key0 + 8 * n + 2 * tq;
                const float* w = from + plane + (long long)(8 * r) * p.tk + key;
                c[n][2 * r] = c[n][2 * r + 1] = 0.0f;
                if (r0 + g + 8 * r >= p.tq || key >= p.tk) continue;
                if (pairs) { const float2 f = *reinterpret_cast<const float2*>(w); c[n][2 * r] = f.x; c[n][2 * r + 1] = f.y; }
                else { c[n][2 * r] = w[0]; if (key + 1 < p.tk) c[n][2 * r + 1] = w[1]; }
            }
    };
    for (int k0 = 0; k0 < kend; k0 += kKT) {
        copies_wait<0>();
        __syncthreads();
        split_tile<NC, NT>(ks, kr, t);
        split_tile<NC, NT>(vs, vr, t);
        __syncthreads();
        if (k0 + kKT < kend) copy(k0 + kKT);
        else if (kend > kKT) copy_rows<kKT, NT, T::HDP, T::HDP>(kr, kb_, kld, 0, p.tk, p.hd, vec, t);      // the second pass begins
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
            float s[2][4], d[2][4], mx[2] = {m[0], m[1]};
            rows_product<NC>(s, qf, sm_addr(ks), 16 * j, lane);
            rows_product<NC>(d, gf, sm_addr(vs), 16 * j, lane);
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    s[n][i] *= p.scale;
                    if (k0 + 16 * j + 8 * n + 2 * tq + (i & 1) < end[i >> 1]) mx[i >> 1] = fmaxf(mx[i >> 1], s[n][i]);
                }
            store(probs, s, k0 + 16 * j);              // this thread reads them back in the second pass
            store(ds, d, k0 + 16 * j);
#pragma unroll
            for (int r = 0; r < 2; ++r) {              // this lane's keys with this lane's maximum: put together at the end
                const float alpha = expf(m[r] - mx[r]);
                l[r] *= alpha; dot[r] *= alpha; m[r] = mx[r];
            }
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float e = k0 + 16 * j + 8 * n + 2 * tq + (i & 1) < end[i >> 1] ? expf(s[n][i] - mx[i >> 1]) : 0.0f;
                    l[i >> 1] += e;
                    dot[i >> 1] += e * d[n][i];
                }
        }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const float mx = quad_max(m[r]), c = expf(m[r] - mx), sum = quad_sum(l[r] * c);
        l[r] = sum > 0.0f ? 1.0f / sum : 0.0f;
        dot[r] = quad_sum(dot[r] * c) * l[r];
        m[r] = mx;
    }
    float acc[2 * NC][4];
#pragma unroll
    for (int n = 0; n < 2 * NC; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] = 0.0f;
    for (int k0 = 0; k0 < kend; k0 += kKT) {
        float s[4][2][4], d[4][2][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) { fetch(probs, s[j], k0 + 16 * j); fetch(ds, d[j], k0 + 16 * j); }
        if (kend > kKT) {                              // with one tile of keys its terms are still in place
            copies_wait<0>();
            __syncthreads();
            split_tile<NC, NT>(ks, kr, t);
            __syncthreads();
            if (k0 + kKT < kend) copy_rows<kKT, NT, T::HDP, T::HDP>(kr, kb_, kld, k0 + kKT, p.tk, p.hd, vec, t);
        }
        uint32_t sf[4][3][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int r = i >> 1;
                    const bool in = k0 + 16 * j + 8 * n + 2 * tq + (i & 1) < end[r];
                    s[j][n][i] = in ? expf(s[j][n][i] - m[r]) * l[r] : 0.0f;
                    d[j][n][i] = in ? s[j][n][i] * (d[j][n][i] - dot[r]) : 0.0f;
                }
            store(probs, s[j], k0 + 16 * j);
            store(ds, d[j], k0 + 16 * j);
            as_operand(sf[j], d[j]);
        }
#pragma unroll
        for (int n = 0; n < 2 * NC; n += 2) {
            float c[2][4];
            cols_product<NC, 4>(c, sf, sm_addr(ks), 0, n, lane);
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[n + e][i] += c[e][i];
        }
    }
    copies_wait<0>();
    if (beyond_fp32(acc)) {
        const long long head = (long long)blockIdx.x * p.tq * p.tk;
        bwd_q_again(q + at, kb_, vb, dout + at, probs + head, ds + head, dq + at, p, r0);
        return;
    }
    // beyond every query of the tile: zeros
    {
        const float zero[2][4] = {};
        for (int k0 = (kend + kKT - 1) / kKT * kKT; k0 < p.tk; k0 += 16) { store(probs, zero, k0); store(ds, zero, k0); }
    }
    float* o = dq + at;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int row = r0 + g + 8 * r;
        if (row >= p.tq) continue;
#pragma unroll
        for (int n = 0; n < 2 * NC; ++n)
#pragma unroll
            for (int i = 0; i < 2; ++i)
                if (8 * n + 2 * tq + i < p.hd) o[(long long)row * qld + 8 * n + 2 * tq + i] = acc[n][2 * r + i] * p.scale;
    }
}

// CTA = 64 keys of one kv head, a warp 16 of them
template <int NC>
__global__ void __launch_bounds__(128, 2) gqa_bwd_k_mma_kernel(const float* __restrict__ q, const float* __restrict__ dout, const float* __restrict__ probs,
                                                        const float* __restrict__ ds, float* __restrict__ dk, float* __restrict__ dv, const __grid_constant__ GqaDims p) {
    grid_release();
    extern __shared__ __align__(16) unsigned char smb[];
    using T = AttTile<NC>;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, tq = lane & 3;
    unsigned char *gs = smb, *qs = smb + T::kBytes;
    float *raw_g = reinterpret_cast<float*>(smb + 2 * T::kBytes), *raw_q = raw_g + T::kRaw / 4;
    const int k0 = (int)blockIdx.y * kKT, b = blockIdx.x / p.n_kv, gr = blockIdx.x % p.n_kv, group = p.n_head / p.n_kv;
    const long long qld = (long long)p.n_head * p.hd, kld = (long long)p.n_kv * p.hd;
    const int qbeg = p.causal && k0 > p.q_off ? (k0 - p.q_off) / kKT : 0, qtiles = (p.tq + kKT - 1) / kKT;      // earlier queries see none of these keys
    const int per = max(qtiles - qbeg, 0), count = group * per;
    const bool vec = rows16(dout, qld, p.hd) && rows16(q, qld, p.hd);
    // tile n of this key block: a query head of the group and 64 queries
    auto head = [&](int n) { return gr * group + n / per; };
    auto copy = [&](int n) {
        const long long at = (long long)b * p.tq * qld + head(n) * p.hd;
        const int q0 = (qbeg + n % per) * kKT;
        copy_rows<kKT, 128, T::HDP, T::HDP>(raw_g, dout + at, qld, q0, p.tq, p.hd, vec, t);
        copy_rows<kKT, 128, T::HDP, T::HDP>(raw_q, q + at, qld, q0, p.tq, p.hd, vec, t);
    };
    float av[2 * NC][4], ak[2 * NC][4];
#pragma unroll
    for (int n = 0; n < 2 * NC; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) av[n][i] = ak[n][i] = 0.0f;
    if (count > 0) copy(0);
    const int key = k0 + 16 * warp + g;
    // the warp's part of a tile of P or dS: rows = keys g, g + 8; columns = queries 2 tq, + 1, then + 8
    auto fetch = [&](float (&x)[4][4][2], const float* src, int n) {
        const int q0 = (qbeg + n % per) * kKT;
        src += (((long long)b * p.n_head + head(n)) * p.tq + q0) * p.tk + key;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int row = 16 * j + (i >> 1) * 8 + 2 * tq + e, kk = (i & 1) * 8;
                    x[j][i][e] = q0 + row < p.tq && key + kk < p.tk ? __ldg(src + (long long)row * p.tk + kk) : 0.0f;
                }
    };
    float xp[4][4][2], xs[4][4][2];
    if (count > 0) fetch(xp, probs, 0);
    for (int n = 0; n < count; ++n) {
        uint32_t f[4][3][4];
        auto operand = [&](const float (&x)[4][4][2]) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint32_t w[3];
                    terms3(x[j][i][0], x[j][i][1], w);
#pragma unroll
                    for (int k = 0; k < 3; ++k) f[j][k][i] = w[k];
                }
        };
        auto add = [&](float (&a)[2 * NC][4], const unsigned char* tile) {
#pragma unroll
            for (int m = 0; m < 2 * NC; m += 2) {
                float c[2][4];
                cols_product<NC, 4>(c, f, sm_addr(tile), 0, m, lane);
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int i = 0; i < 4; ++i) a[m + e][i] += c[e][i];
            }
        };
        fetch(xs, ds, n);
        copies_wait<0>();
        __syncthreads();
        split_tile<NC, 128>(gs, raw_g, t);
        split_tile<NC, 128>(qs, raw_q, t);
        __syncthreads();
        if (n + 1 < count) copy(n + 1);
        operand(xp);
        if (n + 1 < count) fetch(xp, probs, n + 1);
        add(av, gs);
        operand(xs);
        add(ak, qs);
    }
    copies_wait<0>();
    if (beyond_fp32(av) || beyond_fp32(ak)) {
        const long long first = (long long)b * p.tq * qld + gr * group * p.hd, head = ((long long)b * p.n_head + gr * group) * p.tq * p.tk, to = (long long)b * p.tk * kld + gr * p.hd;
        bwd_k_again(q + first, dout + first, probs + head, ds + head, dk + to, dv + to, p, k0 + 16 * warp);
        return;
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        if (key + 8 * r >= p.tk) continue;
        const long long at = ((long long)b * p.tk + key + 8 * r) * kld + gr * p.hd;
#pragma unroll
        for (int n = 0; n < 2 * NC; ++n)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int d = 8 * n + 2 * tq + i;
                if (d < p.hd) { dv[at + d] = av[n][2 * r + i]; dk[at + d] = ak[n][2 * r + i] * p.scale; }
            }
    }
}
