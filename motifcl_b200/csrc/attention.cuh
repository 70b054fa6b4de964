// Grouped-query attention, forward and backward, for head sizes up to 64 and grids that do not fill the GPU (attention_mma.cuh takes
// those that do): exact fp32 FMAs on tiles in shared memory (tf32 would not hold the reference's accuracy), scores never written by
// the forward pass.  Included by trainer_ops.cu.
//
// A CTA owns 32 queries of one head and walks over tiles of 64 keys with TWO groups of 64 threads that take alternate tiles
// (a training step has few query tiles: one group left 10 warps on an SM, each issuing every 5.6 cycles) and merge at the end.
// Thread (ty, tx) of a group holds 8 queries x 4 keys (keys tx + 16 j) of a score tile and 8 queries x NC columns (tx + 16 j) of
// the output.  Products run on the two-lane FMA (fma.rn.f32x2, the rounding of two FMAs in one issue slot) over pairs of queries:
// queries lie transposed in shared memory, keys and values row-major.  Row maxima and sums
// are reduced over the 16 lanes that share a ty.
//   forward   online softmax: S tile -> P tile (transposed through shared memory) -> O += P V
//   backward  kernel 1 (queries): S and dP tiles, kept in the caller's scratch, with the running maximum, sum and sum of P dP;
//             then P, dS from them (written, as the reference leaves them) and dq += dS K.
//             kernel 2 (keys): dv = P^T dO, dk = dS^T Q, summed over the query heads of the kv head.
// Tiles come by cp.async into one buffer each: the copy of the next tile starts as soon as the product that read the last one
// is done and runs under the other product (waiting for them took half of the time).
// Grids run over the heads first and over the tiles with the longest rows before the short ones.
// 16 sequences of 256 tokens, 6 heads of 48, causal, before (seven batched products and two row passes): forward 82 us,
// backward 232 us.
#pragma once

constexpr int kKT = 64;               // keys per tile
constexpr int kBQ = 32;               // queries per tile

__device__ __forceinline__ float half_sum(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float half_max(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ void copy16(float* dst, const float* src, bool in) {      // 16 bytes, or zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// rows r0 .. r0 + R - 1 of a [*, ld] matrix, W columns of which n exist -> dst[row * S + d], zero outside; thread t of NT.  vec: rows
// start on 16-byte boundaries and n % 4 == 0 (copied in the background), else plain loads.
template <int R, int NT, int W, int S>
__device__ __forceinline__ void copy_rows(float* dst, const float* __restrict__ src, long long ld, int r0, int rmax, int n, bool vec, int t) {
#pragma unroll
    for (int i0 = 0; i0 < R * (W / 4); i0 += NT) {
        const int i = i0 + t, row = i / (W / 4), d = (i - row * (W / 4)) * 4;
        if (R * (W / 4) % NT != 0 && i >= R * (W / 4)) break;
        const bool in = r0 + row < rmax && d < n;
        const float* s = in ? src + (long long)(r0 + row) * ld + d : src;
        if (vec) {
            copy16(dst + row * S + d, s, in);
        } else {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (in) {
                v.x = __ldg(s);
                if (d + 1 < n) v.y = __ldg(s + 1);
                if (d + 2 < n) v.z = __ldg(s + 2);
                if (d + 3 < n) v.w = __ldg(s + 3);
            }
            *reinterpret_cast<float4*>(dst + row * S + d) = v;
        }
    }
    copies_commit();
}
__device__ __forceinline__ bool rows16(const void* p, long long ld, int n) { return ((ld | n) & 3) == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
// the same rows transposed: dst[d * (R + 4) + row]; all loads of a thread in flight at once, a warp stores 32 rows of one column
template <int R, int NT, int HDP>
__device__ __forceinline__ void load_cols(float* dst, const float* __restrict__ src, long long ld, int r0, int rmax, int hd, bool vec, int t) {
    constexpr int N = (R * (HDP / 4) + NT - 1) / NT;
    float4 v[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const int i = n * NT + t, row = i & (R - 1), d = (i / R) * 4;
        v[n] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r0 + row < rmax && d < hd) {
            const float* s = src + (long long)(r0 + row) * ld + d;
            if (vec) v[n] = __ldg(reinterpret_cast<const float4*>(s));
            else {
                v[n].x = __ldg(s);
                if (d + 1 < hd) v[n].y = __ldg(s + 1);
                if (d + 2 < hd) v[n].z = __ldg(s + 2);
                if (d + 3 < hd) v[n].w = __ldg(s + 3);
            }
        }
    }
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const int i = n * NT + t, row = i & (R - 1), d = (i / R) * 4;
        if (d < HDP) {
            dst[d * (R + 4) + row] = v[n].x; dst[(d + 1) * (R + 4) + row] = v[n].y;
            dst[(d + 2) * (R + 4) + row] = v[n].z; dst[(d + 3) * (R + 4) + row] = v[n].w;
        }
    }
}
__device__ __forceinline__ void fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ float2 halves(unsigned long long v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
// s[i][j] = sum over d of a[d][8 ty + i] b[tx + 16 j][d]; a: kBQ + 4 floats per d, b: HDP + 4 per row
template <int HDP>
__device__ __forceinline__ void scores(float (&s)[8][4], const float* a, const float* b, int ty, int tx) {
    const float* pa = a + 8 * ty;
    const float* pb = b + tx * (HDP + 4);
    unsigned long long c[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) c[i][j] = 0ull;
#pragma unroll 2
    for (int d = 0; d < HDP; d += 4) {
        float bv[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(bv[j]) = *reinterpret_cast<const float4*>(pb + 16 * j * (HDP + 4) + d);
#pragma unroll
        for (int dd = 0; dd < 4; ++dd) {
            const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(pa + (d + dd) * (kBQ + 4)), a1 = *reinterpret_cast<const ulonglong2*>(pa + (d + dd) * (kBQ + 4) + 4);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                unsigned long long bb;
                asm("mov.b64 %0, {%1, %1};" : "=l"(bb) : "f"(bv[j][dd]));
                fma2(c[0][j], a0.x, bb); fma2(c[1][j], a0.y, bb); fma2(c[2][j], a1.x, bb); fma2(c[3][j], a1.y, bb);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) { const float2 h = halves(c[i][j]); s[2 * i][j] = h.x; s[2 * i + 1][j] = h.y; }
}
// acc (pairs of queries 8 ty + 2 i, + 1) += sum over n rows r of a[r][8 ty + .] b[r][tx + 16 j]
template <int NC>
__device__ __forceinline__ void outer(unsigned long long (&acc)[4][NC], const float* a, int as, const float* b, int bs, int n, int ty, int tx) {
    const float* pa = a + 8 * ty;
    const float* pb = b + tx;
#pragma unroll 4
    for (int r = 0; r < n; ++r) {
        const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(pa + r * as), a1 = *reinterpret_cast<const ulonglong2*>(pa + r * as + 4);
        const unsigned long long av[4] = {a0.x, a0.y, a1.x, a1.y};
#pragma unroll
        for (int j = 0; j < NC; ++j) {
            const float v = pb[r * bs + 16 * j];
            unsigned long long bb;
            asm("mov.b64 %0, {%1, %1};" : "=l"(bb) : "f"(v));
#pragma unroll
            for (int i = 0; i < 4; ++i) fma2(acc[i][j], av[i], bb);
        }
    }
}
__device__ __forceinline__ void group_sync(int group, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(threads) : "memory"); }

// floats of shared memory: rows of HDP + 4 for tiles, of kBQ + 4 for transposed probability tiles
template <int NC>
__host__ __device__ constexpr size_t fwd_group_floats() { return (size_t)2 * kKT * (16 * NC + 4) + kKT * (kBQ + 4); }
template <int NC>
__host__ __device__ constexpr size_t fwd_floats() { return (size_t)16 * NC * (kBQ + 4) + 2 * fwd_group_floats<NC>(); }
template <int NC>
__host__ __device__ constexpr size_t bwd_q_group_floats() {      // k and v tiles, or k and dS tiles
    return (size_t)kKT * (16 * NC + 4) + ((size_t)kKT * (16 * NC + 4) > (size_t)kKT * (kBQ + 4) ? (size_t)kKT * (16 * NC + 4) : (size_t)kKT * (kBQ + 4));
}
template <int NC>
__host__ __device__ constexpr size_t bwd_q_floats() { return (size_t)2 * 16 * NC * (kBQ + 4) + 2 * bwd_q_group_floats<NC>() + 6 * kBQ; }
template <int NC>
__host__ __device__ constexpr size_t bwd_k_group_floats() { return (size_t)2 * 32 * (kKT + 4) + 2 * (size_t)32 * (16 * NC + 4); }
template <int NC>
__host__ __device__ constexpr size_t bwd_k_floats() { return 2 * bwd_k_group_floats<NC>(); }

// first and one-past-last key of query row r, without a table in registers
__device__ __forceinline__ int row_hi(const GqaDims& p, int r) { return p.causal ? min(p.q_off + r + 1, p.tk) : p.tk; }
__device__ __forceinline__ int row_lo(const GqaDims& p, int r) { return p.window ? max(p.q_off + r + 1 - p.window, 0) : 0; }
// keys a tile of queries can see
template <int BQ>
__device__ __forceinline__ void tile_range(const GqaDims& p, int q0, int& kb, int& ke) {
    const int last = min(q0 + BQ, p.tq) - 1;
    int a0, a1, b0, b1;
    key_range(p, q0, a0, a1);
    key_range(p, last, b0, b1);
    kb = a0 / kKT * kKT;
    ke = b1;
}

template <int NC>
__global__ void __launch_bounds__(4 * kBQ, 128 / kBQ) gqa_fwd_kernel(const float* __restrict__ q, const float* __restrict__ k,
                                                         const float* __restrict__ v, float* __restrict__ out, GqaDims p) {
    grid_release();
    extern __shared__ __align__(16) float sm[];
    constexpr int BQ = kBQ, HDP = 16 * NC, HS = HDP + 4, QS = BQ + 4, NT = 2 * BQ;
    const int grp = threadIdx.x / NT, t = threadIdx.x % NT, tx = t & 15, ty = t >> 4;
    float* qs = sm;                                                        // [HDP][QS]
    float* ks = qs + HDP * QS + grp * fwd_group_floats<NC>();           // this group's k [64][HS], v [64][HS], P^T [64][QS]
    float* vs = ks + kKT * HS;
    float* pt = vs + kKT * HS;
    const int tiles = (p.tq + BQ - 1) / BQ, q0 = (tiles - 1 - (int)blockIdx.y) * BQ;
    const int b = blockIdx.x / p.n_head, h = blockIdx.x % p.n_head, g = h / (p.n_head / p.n_kv);
    const long long qld = (long long)p.n_head * p.hd, kld = (long long)p.n_kv * p.hd;
    const float* kb_ = k + (long long)b * p.key_stride * kld + g * p.hd;
    const float* vb = v + (long long)b * p.key_stride * kld + g * p.hd;
    const float* qb = q + (long long)b * p.tq * qld + h * p.hd;
    load_cols<BQ, 2 * NT, HDP>(qs, qb, qld, q0, p.tq, p.hd, rows16(qb, qld, p.hd), threadIdx.x);
    float m[8], l[8];
    unsigned long long o[4][NC];
#pragma unroll
    for (int i = 0; i < 8; ++i) { m[i] = -FLT_MAX; l[i] = 0.0f; }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NC; ++j) o[i][j] = 0ull;
    int kbeg, kend;
    tile_range<BQ>(p, q0, kbeg, kend);
    const bool vec = rows16(kb_, kld, p.hd) && rows16(vb, kld, p.hd);
    int k0 = kbeg + grp * kKT;
    copy_rows<kKT, NT, HDP, HS>(ks, kb_, kld, k0, p.tk, p.hd, vec, t);
    copy_rows<kKT, NT, HDP, HS>(vs, vb, kld, k0, p.tk, p.hd, vec, t);
    __syncthreads();
    for (; k0 < kend; k0 += 2 * kKT) {
        copies_wait<1>();
        group_sync(grp, NT);
        float s[8][4];
        scores<HDP>(s, qs, ks, ty, tx);
        group_sync(grp, NT);
        copy_rows<kKT, NT, HDP, HS>(ks, kb_, kld, k0 + 2 * kKT, p.tk, p.hd, vec, t);
        float alpha[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int lo = row_lo(p, q0 + 8 * ty + i), hi = row_hi(p, q0 + 8 * ty + i);
            float mx = m[i];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = k0 + tx + 16 * j;
                s[i][j] = key < lo || key >= hi ? -FLT_MAX : s[i][j] * p.scale;
                mx = fmaxf(mx, s[i][j]);
            }
            mx = half_max(mx);
            alpha[i] = expf(m[i] - mx);
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[i][j] = s[i][j] == -FLT_MAX ? 0.0f : expf(s[i][j] - mx);
                sum += s[i][j];
            }
            l[i] = l[i] * alpha[i] + sum;          // this lane's keys: added over the 16 lanes at the end
            m[i] = mx;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            unsigned long long a2;
            asm("mov.b64 %0, {%1, %2};" : "=l"(a2) : "f"(alpha[2 * i]), "f"(alpha[2 * i + 1]));
#pragma unroll
            for (int j = 0; j < NC; ++j) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(o[i][j]) : "l"(a2));
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float* d = pt + (tx + 16 * j) * QS + 8 * ty;
            *reinterpret_cast<float4*>(d) = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
            *reinterpret_cast<float4*>(d + 4) = make_float4(s[4][j], s[5][j], s[6][j], s[7][j]);
        }
        copies_wait<1>();
        group_sync(grp, NT);
        outer<NC>(o, pt, QS, vs, HS, kKT, ty, tx);
        group_sync(grp, NT);
        copy_rows<kKT, NT, HDP, HS>(vs, vb, kld, k0 + 2 * kKT, p.tk, p.hd, vec, t);
    }
    copies_wait<0>();
#pragma unroll
    for (int i = 0; i < 8; ++i) l[i] = half_sum(l[i]);
    // merge the groups: the second leaves maximum, sum and accumulator in its tiles
    float* mg = qs + HDP * QS + fwd_group_floats<NC>();      // [8 + 8 + 8 NC][NT] floats
    static_assert(fwd_group_floats<NC>() >= (size_t)(16 + 8 * NC) * NT, "merge area");
    __syncthreads();
    if (grp == 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) { mg[i * NT + t] = m[i]; mg[(8 + i) * NT + t] = l[i]; }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                const float2 f = halves(o[i][j]);
                mg[(16 + (2 * i) * NC + j) * NT + t] = f.x;
                mg[(16 + (2 * i + 1) * NC + j) * NT + t] = f.y;
            }
    }
    __syncthreads();
    if (grp == 1) return;
    float* ob = out + (long long)b * p.tq * qld + h * p.hd;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int row = q0 + 8 * ty + i;
        const float m1 = mg[i * NT + t], mx = fmaxf(m[i], m1), c0 = expf(m[i] - mx), c1 = expf(m1 - mx);
        const float sum = l[i] * c0 + mg[(8 + i) * NT + t] * c1, inv = sum > 0.0f ? 1.0f / sum : 0.0f;
#pragma unroll
        for (int j = 0; j < NC; ++j) {
            const float2 f = halves(o[i >> 1][j]);
            if (row < p.tq && tx + 16 * j < p.hd)
                ob[(long long)row * qld + tx + 16 * j] = ((i & 1 ? f.y : f.x) * c0 + mg[(16 + i * NC + j) * NT + t] * c1) * inv;
        }
    }
}

// probs, ds [B, n_head, tq, tk]; dq
template <int NC>
__global__ void __launch_bounds__(4 * kBQ, 128 / kBQ) gqa_bwd_q_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                                                           const float* __restrict__ dout, float* __restrict__ probs, float* __restrict__ ds,
                                                           float* __restrict__ dq, GqaDims p) {
    grid_release();
    extern __shared__ __align__(16) float sm[];
    constexpr int BQ = kBQ, HDP = 16 * NC, HS = HDP + 4, QS = BQ + 4, NT = 2 * BQ;
    const int grp = threadIdx.x / NT, t = threadIdx.x % NT, tx = t & 15, ty = t >> 4;
    float* qs = sm;                       // [HDP][QS]
    float* gs = qs + HDP * QS;            // dO
    float* ks = gs + HDP * QS + grp * bwd_q_group_floats<NC>();      // this group's k [64][HS]
    float* vs = ks + kKT * HS;            // pass 1: v [64][HS]; pass 2: dS^T [64][QS]
    float* st = gs + HDP * QS + 2 * bwd_q_group_floats<NC>();        // [2][3][BQ]: maximum, sum, sum of P dP of each group
    const int tiles = (p.tq + BQ - 1) / BQ, q0 = (tiles - 1 - (int)blockIdx.y) * BQ;
    const int b = blockIdx.x / p.n_head, h = blockIdx.x % p.n_head, g = h / (p.n_head / p.n_kv);
    const long long qld = (long long)p.n_head * p.hd, kld = (long long)p.n_kv * p.hd;
    const float* kb_ = k + (long long)b * p.tk * kld + g * p.hd;
    const float* vb = v + (long long)b * p.tk * kld + g * p.hd;
    const float* qb = q + (long long)b * p.tq * qld + h * p.hd;
    load_cols<BQ, 2 * NT, HDP>(qs, qb, qld, q0, p.tq, p.hd, rows16(qb, qld, p.hd), threadIdx.x);
    const float* gb = dout + (long long)b * p.tq * qld + h * p.hd;
    load_cols<BQ, 2 * NT, HDP>(gs, gb, qld, q0, p.tq, p.hd, rows16(gb, qld, p.hd), threadIdx.x);
    float m[8], l[8], dot[8];
    auto row_end = [&](int i) { return q0 + 8 * ty + i < p.tq ? row_hi(p, q0 + 8 * ty + i) : 0; };
#pragma unroll
    for (int i = 0; i < 8; ++i) { m[i] = -FLT_MAX; l[i] = 0.0f; dot[i] = 0.0f; }
    int kbeg, kend;
    tile_range<BQ>(p, q0, kbeg, kend);
    float* pr = probs + ((long long)blockIdx.x * p.tq + q0 + 8 * ty) * p.tk + tx;
    float* dr = ds + ((long long)blockIdx.x * p.tq + q0 + 8 * ty) * p.tk + tx;
    const bool vec = rows16(kb_, kld, p.hd) && rows16(vb, kld, p.hd);
    int k0 = kbeg + grp * kKT;
    copy_rows<kKT, NT, HDP, HS>(ks, kb_, kld, k0, p.tk, p.hd, vec, t);
    copy_rows<kKT, NT, HDP, HS>(vs, vb, kld, k0, p.tk, p.hd, vec, t);
    __syncthreads();
    for (; k0 < kend; k0 += 2 * kKT) {
        float s[8][4], d[8][4];
        copies_wait<1>();
        group_sync(grp, NT);
        scores<HDP>(s, qs, ks, ty, tx);
        group_sync(grp, NT);
        copy_rows<kKT, NT, HDP, HS>(ks, kb_, kld, k0 + 2 * kKT, p.tk, p.hd, vec, t);
        copies_wait<1>();
        group_sync(grp, NT);
        scores<HDP>(d, gs, vs, ty, tx);
        group_sync(grp, NT);
        copy_rows<kKT, NT, HDP, HS>(vs, vb, kld, k0 + 2 * kKT, p.tk, p.hd, vec, t);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int hi = row_end(i);
            float mx = m[i];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[i][j] *= p.scale;
                if (k0 + tx + 16 * j < hi) {      // this thread reads them back in pass 2
                    pr[(long long)i * p.tk + k0 + 16 * j] = s[i][j];
                    dr[(long long)i * p.tk + k0 + 16 * j] = d[i][j];
                    mx = fmaxf(mx, s[i][j]);
                }
            }
            mx = half_max(mx);
            const float alpha = expf(m[i] - mx);
            float sum = 0.0f, pd = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float e = k0 + tx + 16 * j < hi ? expf(s[i][j] - mx) : 0.0f;
                sum += e;
                pd += e * d[i][j];
            }
            l[i] = l[i] * alpha + sum;             // this lane's keys: added over the 16 lanes at the end
            dot[i] = dot[i] * alpha + pd;
            m[i] = mx;
        }
    }
    copies_wait<0>();
#pragma unroll
    for (int i = 0; i < 8; ++i) { l[i] = half_sum(l[i]); dot[i] = half_sum(dot[i]); }
    if (tx == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float* w = st + grp * 3 * BQ + 8 * ty + i;
            w[0] = m[i]; w[BQ] = l[i]; w[2 * BQ] = dot[i];
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float* w = st + (grp ^ 1) * 3 * BQ + 8 * ty + i;
        const float mx = fmaxf(m[i], w[0]), c0 = expf(m[i] - mx), c1 = expf(w[0] - mx);
        const float sum = l[i] * c0 + w[BQ] * c1;
        l[i] = sum > 0.0f ? 1.0f / sum : 0.0f;
        dot[i] = (dot[i] * c0 + w[2 * BQ] * c1) * l[i];
        m[i] = mx;
    }
    unsigned long long acc[4][NC];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NC; ++j) acc[i][j] = 0ull;
    copy_rows<kKT, NT, HDP, HS>(ks, kb_, kld, grp * kKT, p.tk, p.hd, vec, t);
    for (k0 = grp * kKT; k0 < p.tk; k0 += 2 * kKT) {
        if (k0 >= kend) {                      // beyond every query of the tile: zeros
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (q0 + 8 * ty + i < p.tq && k0 + tx + 16 * j < p.tk) {
                        pr[(long long)i * p.tk + k0 + 16 * j] = 0.0f;
                        dr[(long long)i * p.tk + k0 + 16 * j] = 0.0f;
                    }
            continue;
        }
#pragma unroll
        for (int jp = 0; jp < 4; ++jp) {               // a quarter of a tile's values in flight at a time
            constexpr int J = 1;
            float pv[8][J], dv[8][J];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    const int key = k0 + tx + 16 * (jp + j);
                    const bool in = key < row_end(i);
                    pv[i][j] = in ? pr[(long long)i * p.tk + k0 + 16 * (jp + j)] : -FLT_MAX;
                    dv[i][j] = in ? dr[(long long)i * p.tk + k0 + 16 * (jp + j)] : 0.0f;
                }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    const bool in = k0 + tx + 16 * (jp + j) < row_end(i);
                    pv[i][j] = in ? expf(pv[i][j] - m[i]) * l[i] : 0.0f;
                    dv[i][j] = in ? pv[i][j] * (dv[i][j] - dot[i]) : 0.0f;
                    if (q0 + 8 * ty + i < p.tq && k0 + tx + 16 * (jp + j) < p.tk) {
                        pr[(long long)i * p.tk + k0 + 16 * (jp + j)] = pv[i][j];
                        dr[(long long)i * p.tk + k0 + 16 * (jp + j)] = dv[i][j];
                    }
                }
#pragma unroll
            for (int j = 0; j < J; ++j) {
                float* d = vs + (tx + 16 * (jp + j)) * QS + 8 * ty;
                *reinterpret_cast<float4*>(d) = make_float4(dv[0][j], dv[1][j], dv[2][j], dv[3][j]);
                *reinterpret_cast<float4*>(d + 4) = make_float4(dv[4][j], dv[5][j], dv[6][j], dv[7][j]);
            }
        }
        copies_wait<0>();
        group_sync(grp, NT);
        outer<NC>(acc, vs, QS, ks, HS, kKT, ty, tx);
        group_sync(grp, NT);
        copy_rows<kKT, NT, HDP, HS>(ks, kb_, kld, k0 + 2 * kKT, p.tk, p.hd, vec, t);
    }
    copies_wait<0>();
    float* mg = gs + HDP * QS + bwd_q_group_floats<NC>();      // the second group's tiles
    static_assert(bwd_q_group_floats<NC>() >= (size_t)8 * NC * NT, "merge area");
    __syncthreads();
    if (grp == 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                const float2 f = halves(acc[i][j]);
                mg[((2 * i) * NC + j) * NT + t] = f.x;
                mg[((2 * i + 1) * NC + j) * NT + t] = f.y;
            }
    }
    __syncthreads();
    if (grp == 1) return;
    float* o = dq + (long long)b * p.tq * qld + h * p.hd;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < NC; ++j) {
            const float2 f = halves(acc[i >> 1][j]);
            if (q0 + 8 * ty + i < p.tq && tx + 16 * j < p.hd)
                o[(long long)(q0 + 8 * ty + i) * qld + tx + 16 * j] = ((i & 1 ? f.y : f.x) + mg[(i * NC + j) * NT + t]) * p.scale;
        }
}

constexpr int kQT = 32;               // queries per tile of the key kernel
// CTA = 64 keys of one kv head, two groups of 128 threads that take alternate tiles of 32 queries
template <int NC>
__global__ void __launch_bounds__(256, 2) gqa_bwd_k_kernel(const float* __restrict__ q, const float* __restrict__ dout, const float* __restrict__ probs,
                                                        const float* __restrict__ ds, float* __restrict__ dk, float* __restrict__ dv, GqaDims p) {
    grid_release();
    extern __shared__ __align__(16) float sm[];
    constexpr int HDP = 16 * NC, HS = HDP + 4, KS = kKT + 4;
    const int grp = threadIdx.x >> 7, t = threadIdx.x & 127, tx = t & 15, ty = t >> 4;
    float* ps = sm + grp * bwd_k_group_floats<NC>();      // P [32 queries][KS]
    float* ss = ps + kQT * KS;            // dS
    float* gs = ss + kQT * KS;            // dO [32 queries][HS]
    float* qs = gs + kQT * HS;            // Q
    const int k0 = (int)blockIdx.y * kKT, b = blockIdx.x / p.n_kv, g = blockIdx.x % p.n_kv, group = p.n_head / p.n_kv;
    const long long qld = (long long)p.n_head * p.hd, kld = (long long)p.n_kv * p.hd;
    unsigned long long av[4][NC], ak[4][NC];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NC; ++j) av[i][j] = ak[i][j] = 0ull;
    const int qbeg = p.causal && k0 > p.q_off ? (k0 - p.q_off) / kQT : 0, qtiles = (p.tq + kQT - 1) / kQT;      // earlier queries see none of these keys
    const int per = max(qtiles - qbeg, 0), count = group * per, nk = min(kKT, p.tk - k0);
    const bool vec = rows16(probs + k0, p.tk, nk) && rows16(ds + k0, p.tk, nk) && rows16(dout, qld, p.hd) && rows16(q, qld, p.hd);
    // tile n of this key block: a query head of the group and 32 queries; beyond the last one nothing is loaded
    auto first = [&](int n) {      // P and dO
        const int h = g * group + (n < count ? n / per : 0), q0 = n < count ? (qbeg + n % per) * kQT : 0, rows = n < count ? p.tq : 0;
        copy_rows<kQT, 128, kKT, KS>(ps, probs + ((long long)b * p.n_head + h) * p.tq * (long long)p.tk + k0, p.tk, q0, rows, nk, vec, t);
        copy_rows<kQT, 128, HDP, HS>(gs, dout + (long long)b * p.tq * qld + h * p.hd, qld, q0, rows, p.hd, vec, t);
    };
    auto second = [&](int n) {     // dS and Q
        const int h = g * group + (n < count ? n / per : 0), q0 = n < count ? (qbeg + n % per) * kQT : 0, rows = n < count ? p.tq : 0;
        copy_rows<kQT, 128, kKT, KS>(ss, ds + ((long long)b * p.n_head + h) * p.tq * (long long)p.tk + k0, p.tk, q0, rows, nk, vec, t);
        copy_rows<kQT, 128, HDP, HS>(qs, q + (long long)b * p.tq * qld + h * p.hd, qld, q0, rows, p.hd, vec, t);
    };
    first(grp);
    second(grp);
    for (int n = grp; n < count; n += 2) {
        copies_wait<2>();
        group_sync(grp, 128);
        outer<NC>(av, ps, KS, gs, HS, kQT, ty, tx);
        group_sync(grp, 128);
        first(n + 2);
        copies_wait<2>();
        group_sync(grp, 128);
        outer<NC>(ak, ss, KS, qs, HS, kQT, ty, tx);
        group_sync(grp, 128);
        second(n + 2);
    }
    copies_wait<0>();
    float* mg = sm + bwd_k_group_floats<NC>();
    static_assert(bwd_k_group_floats<NC>() >= (size_t)16 * NC * 128, "merge area");
    __syncthreads();
    if (grp == 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                const float2 f = halves(av[i][j]), e = halves(ak[i][j]);
                mg[((4 * i) * NC + j) * 128 + t] = f.x; mg[((4 * i + 1) * NC + j) * 128 + t] = f.y;
                mg[((4 * i + 2) * NC + j) * 128 + t] = e.x; mg[((4 * i + 3) * NC + j) * 128 + t] = e.y;
            }
    }
    __syncthreads();
    if (grp == 1) return;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int key = k0 + 8 * ty + i;
#pragma unroll
        for (int j = 0; j < NC; ++j)
            if (key < p.tk && tx + 16 * j < p.hd) {
                const float2 f = halves(av[i >> 1][j]), e = halves(ak[i >> 1][j]);
                const long long at = ((long long)b * p.tk + key) * kld + g * p.hd + tx + 16 * j;
                const int r = 4 * (i >> 1) + (i & 1);
                dv[at] = (i & 1 ? f.y : f.x) + mg[(r * NC + j) * 128 + t];
                dk[at] = ((i & 1 ? e.y : e.x) + mg[((r + 2) * NC + j) * 128 + t]) * p.scale;
            }
    }
}
