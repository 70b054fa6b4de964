// Ternary decode GEMV in one launch, M <= 8 activation rows: y[m,o] = scale[o] * sum_k x[m,k] * t[o,k], t from the 2-bit words.
//
// What bounds it: the words are 0.25 byte a weight, so at 6.5 TB/s an SM has to take 90 weights per clock, and a whole
// matrix is 1 to 3 us.  Three things follow.  (1) No instruction per weight: a warp's m16n8k32 int8 MMA takes 512 weights
// straight from registers, and a 16-weight word becomes four operand registers with seven logic operations ((w >> 2i) &
// 0x03030303 holds the fields 4j + i as bytes; the order of k inside a group of 16 does not matter as long as both operands
// share it).  A unit is 32 rows, so that the digits read from shared memory serve two MMAs (with 16 rows that pipe was the
// bound: 510 clocks per 256 weights of 16 rows and 16 warps against 256 for the MMAs).  (2) No second launch: the CTAs of a cluster split K,
// each forms the int8 digits of its own slice of x (with its own power-of-two scale, so nothing has to be known of the rest of
// the row), and the slices of an output meet through distributed shared memory in slice order.  (3) Bytes in flight: a
// warp's next units are loaded into registers while it works on one, the first ones before the activations are touched at all.
// Where the launch before this one in a recorded batch is a decode GEMV too, those first loads even pass under its tail
// (programmatic dependent launch): the words of a matrix are no output of such a launch; x may be, and is read after the wait.
//
// A recording puts matrices that do not depend on one another into one launch (a list): set-up, digits and hand-over of a launch are 2 to 4
// us, as long as the words of a small matrix take.  One row of x, launches apart and as a list: q, k, v of 2048 x 2048 (three
// launches of 4.0 us) 7.8 us, w1 and w3 of 14336 x 4096 21 us (two of 10.7); 4 blocks of 1280 / 5120, 20 matrices, 60 and 21 us.  Long lists
// are quicker on gemv_tc.cu (gemv_tc_pays).
//
// x is scaled to whole numbers of 30 bits and sign below the slice's largest magnitude and written as four signed digits of
// base 256; one row alone (M = 1) has columns to spare and gets the 31 bits of the remainder as a second row.  Integer sums are
// exact; the offset of the fields (f = t + 1) is taken off as a digit sum; slices are put together in double precision.
// Legacy integer MMAs run at 2025 multiply-adds per clock and SM here (measured): 128 weights per clock for M <= 4 and 63 for
// M = 8; beyond that the tcgen05 kernel is the faster one.
#include <algorithm>

#include "kernels.h"

namespace mcl {
namespace {

constexpr int MV_THREADS = 256;
constexpr int MV_WARPS = MV_THREADS / 32;
constexpr int MV_CHUNK = 256;          // weights of a row per unit: 64 bytes, 16 for each of the four lanes that share the row
constexpr int MV_ROWS = 32;            // rows of a unit
constexpr int MV_MAX_S = 8;

// One launch takes a list of matrices; their groups of 32 rows are numbered through.
struct MvMat {
    const uint4* words;
    const float* x;
    const float* scale;
    float* y;
    long long cost;                    // of everything before it, in chunks
    int I, O;
    int first;                         // number of its first group
    int next;                          // the first matrix behind it that has another x
    int log_k;                         // slices of K that a CTA takes (one, or two in a cluster of half as many CTAs as slices)
};
template <int CAP>         // one matrix, or kGemvListCap
struct MvTable {
    long long cost;
    int n, groups, M;
    int log_s, log_p;                  // CTAs of a cluster; slices of the matrix that has most
    int groups_q, groups_r;            // one matrix: groups of a cluster (the first groups_r clusters take one more)
    int block;                         // groups whose partial sums are held at a time
    int owned;                         // of them, the most that one CTA of the cluster finishes
    int xq_bytes;                      // the digits of the widest slice
    MvMat m[CAP];
};
constexpr int MV_GROUP_COST = 1;       // chunks that the end of a group counts for
constexpr int MV_X_COST = 64;          // and the digits of another x, in the cluster whose run goes over to it: 1.6 us
__host__ __device__ inline int mv_chunks(int I) { return (I + MV_CHUNK - 1) / MV_CHUNK; }

// The first group at or behind cluster c's share of the cost, and its matrix (m: one at or before it).
template <int CAP>
__host__ __device__ inline int mv_cut(const MvTable<CAP>& p, int c, int clusters, int& m) {
    if (c == clusters) return p.groups;
    const long long t = p.cost * c / clusters;
    while (m + 1 < p.n && t >= p.m[m + 1].cost) ++m;
    const int per = mv_chunks(p.m[m].I) + MV_GROUP_COST, end = m + 1 < p.n ? p.m[m + 1].first : p.groups;
    const int f = p.m[m].first + (int)((t - p.m[m].cost + per - 1) / per);
    if (f >= end && m + 1 < p.n) ++m;
    return f < end ? f : end;
}

__device__ __forceinline__ uint4 mv_load(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 mv_load_x(const float* p) {       // never before the wait on the grid this one depends on
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void mv_mma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t mv_word(const uint4& v, int q) { return q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w; }

// FORM: 1 for more than one matrix, 2 where a CTA has two slices of some.  A cluster takes a run of groups, cut so that all clusters have the same number of chunks whatever the matrices are.  Matrices with
// one x are neighbours in the list (a segment): their digits are formed once.  The words are loaded ahead across groups, rounds
// (a barrier) and segments (new digits) alike.
// NT: tiles of eight digit columns (two rows of x each); R: units a warp has in registers
template <int NT, int R, int FORM>
__global__ void __launch_bounds__(MV_THREADS, 2) gemv_mma_kernel(const __grid_constant__ MvTable<FORM ? kGemvListCap : 1> p) {
    constexpr bool LIST = FORM > 0;
    extern __shared__ __align__(128) unsigned char mv_smem[];
    constexpr int KS = FORM == 2 ? 2 : 1;           // slices of a CTA, at most
    __shared__ unsigned int amax[KS][8];
    __shared__ int corr[KS][NT * 8];
    __shared__ double xscale[2][MV_MAX_S][8];       // of every slice: the value of one unit of its whole numbers; two segments
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tq = lane & 3;
    const int lg_s = p.log_s, S = 1 << lg_s, rank = blockIdx.x & (S - 1), cid = blockIdx.x >> lg_s;
    const int M = p.M, Mp = M == 1 ? 2 : M;
    int mat = 0, g_begin, g_end;                    // matrix of the group at hand; this cluster's groups
    if (LIST) {
        const int clusters = gridDim.x >> lg_s;
        int behind = 0;
        g_begin = mv_cut(p, cid, clusters, mat);
        g_end = mv_cut(p, cid + 1, clusters, behind);
    } else {
        g_begin = cid * p.groups_q + min(cid, p.groups_r);
        g_end = g_begin + p.groups_q + (cid < p.groups_r ? 1 : 0);
    }
    auto segment_end = [&](int m) -> int {
        if (!LIST) return g_end;
        const int k = p.m[m].next;
        return min(g_end, k < p.n ? p.m[k].first : p.groups);
    };

    uint4 w[R][4];
    // load cursor: group lf of matrix lm, its chunk lc; the warp takes every MV_WARPS-th group of a segment
    int lm = mat, lf = g_begin + warp, lc = 0, l_end = g_begin < g_end ? segment_end(mat) : g_begin, l_c0 = 0, l_nc = 1, l_row16 = 0;
    const uint4* l_words = nullptr;                 // this lane's piece of the group's first row, in the slice's first chunk
    uint32_t l_off[4];                              // from there to its four rows, in pieces
    auto seek = [&](bool segment) {                 // lf has moved
        if constexpr (LIST) {
            while (lf >= l_end && l_end < g_end) {
                lm = p.m[lm].next;
                lf = l_end + warp;
                l_end = segment_end(lm);
                segment = true;
            }
            if (lf >= l_end) return;
            while (lm + 1 < p.n && lf >= p.m[lm + 1].first) ++lm;
            if (segment) {
                const int NC = mv_chunks(p.m[lm].I);
                l_c0 = (rank * NC) >> lg_s;
                l_nc = (((rank + 1) * NC) >> lg_s) - l_c0;
                l_row16 = p.m[lm].I >> 6;               // 16-byte pieces of a row
            }
            const int row = (lf - p.m[lm].first) * MV_ROWS, last = p.m[lm].O - 1 - row;
            l_words = p.m[lm].words + (size_t)row * l_row16 + l_c0 * 4 + tq;
#pragma unroll
            for (int h = 0; h < 4; ++h) l_off[h] = (uint32_t)(min(h * 8 + g, last) * l_row16);
        }
    };
    auto load = [&](uint4 (&u)[4]) {
        if (lf >= l_end) return;
        const int piece = (l_c0 + lc) * 4 + tq;
        if (piece < l_row16) {
#pragma unroll
            for (int h = 0; h < 4; ++h)
                u[h] = mv_load(LIST ? l_words + lc * 4 + l_off[h] : p.m[0].words + (size_t)min(lf * MV_ROWS + h * 8 + g, p.m[0].O - 1) * l_row16 + piece);
        } else {
#pragma unroll
            for (int h = 0; h < 4; ++h) u[h] = make_uint4(0, 0, 0, 0);       // beyond the row: the digits there are zero as well
        }
        if (++lc == l_nc) { lc = 0; lf += MV_WARPS; seek(false); }
    };
    if (LIST) {
        seek(true);
    } else {
        const int NC = mv_chunks(p.m[0].I);
        l_c0 = (rank * NC) >> lg_s;
        l_nc = (((rank + 1) * NC) >> lg_s) - l_c0;
        l_row16 = p.m[0].I >> 6;
    }
#pragma unroll
    for (int j = 0; j < R; ++j) load(w[j]);
    if (threadIdx.x < KS * 8) amax[0][threadIdx.x] = 0u;
    if (threadIdx.x < KS * NT * 8) corr[0][threadIdx.x] = 0;
    if (S > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");    // only "this CTA runs": nothing to publish
    grid_release();
    grid_wait();
    const uint32_t part0 = (uint32_t)__cvta_generic_to_shared(mv_smem) + (uint32_t)p.xq_bytes;
    const uint32_t part_bytes = (uint32_t)(p.owned * Mp) * (MV_ROWS * 8u);      // one slice's sums for the groups a CTA finishes
    int parity = 0;
    bool first = true;
#pragma unroll 1
    for (int seg = 0, s_begin = g_begin; LIST ? s_begin < g_end : seg == 0; ++seg) {
    const int s_end = segment_end(mat), I = p.m[mat].I, NC = mv_chunks(I);
    const float* const x = p.m[mat].x;
    const int c0 = (rank * NC) >> lg_s, nc = (((rank + 1) * NC) >> lg_s) - c0;
    const int lg_k = KS > 1 ? p.m[mat].log_k : 0, slice0 = rank << lg_k;
    const int mid = lg_k ? (((slice0 + 1) * NC) >> (lg_s + 1)) - c0 : nc;       // chunks of the first of two slices
    if (LIST && seg > 0) {
        if (threadIdx.x < KS * 8) amax[0][threadIdx.x] = 0u;
        if (threadIdx.x < KS * NT * 8) corr[0][threadIdx.x] = 0;
    }
    __syncthreads();

    // -- the digits of this slice: a warp takes 128 activations of one row at a time, four a lane --------------------
    const int k0 = c0 * MV_CHUNK, per_row = nc * 2;
#pragma unroll 4
    for (int unit = warp; unit < M * per_row; unit += MV_WARPS) {
        const int m = unit / per_row, k = k0 + (unit - m * per_row) * 128 + lane * 4;
        unsigned int top = 0u;
        if (k < I) {
            const float4 v = mv_load_x(x + (size_t)m * I + k);
            top = max(max(__float_as_uint(v.x) & 0x7FFFFFFFu, __float_as_uint(v.y) & 0x7FFFFFFFu),
                      max(__float_as_uint(v.z) & 0x7FFFFFFFu, __float_as_uint(v.w) & 0x7FFFFFFFu));
        }
        top = __reduce_max_sync(0xffffffffu, top);
        if (lane == 0) atomicMax(&amax[KS > 1 && (unit - m * per_row) >> 1 >= mid][m], top);
    }
    __syncthreads();
#pragma unroll 2
    for (int unit = warp; unit < Mp * per_row; unit += MV_WARPS) {
        const int mp = unit / per_row, quad = (unit - mp * per_row) * 32 + lane, k = k0 + quad * 4;
        const int m = M == 1 ? 0 : mp;
        const int sl = KS > 1 && (unit - mp * per_row) >> 1 >= mid;
        const unsigned int top = amax[sl][m];
        const GemvUnit inv = gemv_unit(top >= 0x7F800000u ? 0 : gemv_exponent(top));
        const float4 t = k < I ? mv_load_x(x + (size_t)m * I + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float f[4] = {t.x * inv.a * inv.b, t.y * inv.a * inv.b, t.z * inv.a * inv.b, t.w * inv.a * inv.b};
        uint32_t r[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            int n = __float2int_rn(f[a]);
            // what the 30 bits leave over: nothing from 2^23 on, where f is a whole number itself
            if (M == 1 && mp == 1) n = __float2int_rn((f[a] - (float)n) * 1073741824.0f);
            r[a] = ((uint32_t)n + 0x80808080u) ^ 0x80808080u;        // four signed bytes, base 256
        }
        // Four lanes hold a group of 16 activations, element 4 j + a in register a of lane j; the MMA wants, for every digit, a
        // word of the elements a, 4 + a, 8 + a, 12 + a.  Two exchanges of bytes leave lane j with the four words of byte j.
        int sum = 0;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const uint32_t o1 = __shfl_xor_sync(0xffffffffu, r[a], 1);
            const uint32_t h = (lane & 1) ? __byte_perm(r[a], o1, 0x3715) : __byte_perm(r[a], o1, 0x6240);   // bytes j & 1 and (j & 1) + 2 of the pair
            const uint32_t o2 = __shfl_xor_sync(0xffffffffu, h, 2);
            r[a] = (lane & 2) ? __byte_perm(o2, h, 0x7632) : __byte_perm(h, o2, 0x5410);
            sum = __dp4a((int)r[a], 0x01010101, sum);
        }
        const int grp16 = quad >> 2, d = 3 - tq;    // byte 3 is the leading digit
        *reinterpret_cast<uint4*>(mv_smem + (size_t)(((grp16 >> 4) * 4 + (grp16 & 3)) * NT + (mp >> 1)) * 512 + (mp & 1) * 256 + d * 64 +
                                  ((grp16 >> 2) & 3) * 16) = make_uint4(r[0], r[1], r[2], r[3]);
#pragma unroll
        for (int s = 4; s < 32; s <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
        if (lane < 4) atomicAdd(&corr[sl][mp * 4 + d], sum);
    }
    __syncthreads();
    if (S > 1 && first) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");      // every CTA of the cluster runs
    first = false;
    if ((int)threadIdx.x < 8 * S && (int)(threadIdx.x & 7) < M) {
        const int m = threadIdx.x & 7;
        for (int sl = 0; sl < 1 << lg_k; ++sl) {
            const unsigned int top = amax[sl][m];
            const int e = gemv_exponent(top);
            const double v = top >= 0x7F800000u ? __longlong_as_double(0x7FF8000000000000ll)       // an infinity or NaN: so is the row
                                                : __longlong_as_double((long long)(1023 + e - 30) << 52);
            uint32_t to;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to)
                         : "r"((uint32_t)__cvta_generic_to_shared(&xscale[seg & 1][slice0 + sl][m])), "r"(threadIdx.x >> 3));
            asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(to), "d"(v) : "memory");
        }
    }

    // -- the contraction ---------------------------------------------------------------------------------------------
    int grp = s_begin + warp;
#pragma unroll 1
    for (int gb = s_begin; gb < s_end; gb += p.block, parity ^= 1) {
        const int ge = min(gb + p.block, s_end);
        const uint32_t part = (uint32_t)(parity << p.log_p) * part_bytes;
        int acc[2][NT][4] = {};
        int cc = 0;
#pragma unroll 1
        while (grp < ge) {
            int used = 0;
#pragma unroll
            for (int j = 0; j < R; ++j) {
                if (grp < ge) {
                    used = j + 1;
                    const uint4* bx = reinterpret_cast<const uint4*>(mv_smem) + cc * (NT * 128) + lane;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint32_t a[4];
#pragma unroll
                        for (int h = 0; h < 4; ++h) a[h] = mv_word(w[j][h], q);
#pragma unroll
                        for (int t = 0; t < NT; ++t) {
                            const uint4 v = bx[(q * NT + t) * 32];
#pragma unroll
                            for (int h = 0; h < 2; ++h)
                                mv_mma(acc[h][t], a[2 * h] & 0x03030303u, a[2 * h + 1] & 0x03030303u, (a[2 * h] >> 2) & 0x03030303u,
                                       (a[2 * h + 1] >> 2) & 0x03030303u, v.x, v.y);
#pragma unroll
                            for (int h = 0; h < 2; ++h)
                                mv_mma(acc[h][t], (a[2 * h] >> 4) & 0x03030303u, (a[2 * h + 1] >> 4) & 0x03030303u, (a[2 * h] >> 6) & 0x03030303u,
                                       (a[2 * h + 1] >> 6) & 0x03030303u, v.z, v.w);
                        }
                    }
                    load(w[j]);
                    ++cc;
                    if (cc == nc || (KS > 1 && cc == mid)) {
                        // a slice of this group is complete: its sums, two digits to a word, go to the CTA that finishes the group
                        const int li = grp - gb, sl = KS > 1 && cc > mid;
                        uint32_t dst;
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst)
                                     : "r"(part0 + part + (slice0 + sl) * part_bytes + (uint32_t)((li >> lg_s) * Mp) * (MV_ROWS * 8u)), "r"(li & (S - 1)));
#pragma unroll
                        for (int t = 0; t < NT; ++t) {
                            const int s0 = corr[sl][t * 8 + 2 * tq], s1 = corr[sl][t * 8 + 2 * tq + 1], m = 2 * t + (tq >> 1);
#pragma unroll
                            for (int h = 0; h < 4; ++h) {
                                const int a0 = acc[h >> 1][t][2 * (h & 1)] - s0, a1 = acc[h >> 1][t][2 * (h & 1) + 1] - s1;
                                if (m < Mp)
                                    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(dst + (uint32_t)((m * MV_ROWS + h * 8 + g) * 8 + (tq & 1) * 4)),
                                                 "r"(a0 * 256 + a1) : "memory");
                            }
#pragma unroll
                            for (int i = 0; i < 4; ++i) acc[0][t][i] = acc[1][t][i] = 0;
                        }
                        if (cc == nc) {
                            cc = 0;
                            grp += MV_WARPS;
                        }
                    }
                }
            }
            // a round may end inside the ring of registers: the next unit has to stand in front again
#pragma unroll 1
            for (; used < R && ge < g_end; --used) {
                if (used == 0) break;
                uint4 t[4];
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    t[h] = w[0][h];
#pragma unroll
                    for (int j = 0; j + 1 < R; ++j) w[j][h] = w[j + 1][h];
                    w[R - 1][h] = t[h];
                }
            }
        }
        const int nb = ge - gb, cnt = nb > rank ? (nb - rank + S - 1) >> lg_s : 0, per = M * MV_ROWS;
        if (S > 1) {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else {
            __syncthreads();
        }
        // two buffers: sums of the block after the next land here only after the barrier that follows these reads
        const unsigned char* src = mv_smem + p.xq_bytes + part;
        for (int i = threadIdx.x; i < cnt * per; i += MV_THREADS) {
            const int slot = i / per, j = i - slot * per, m = j / MV_ROWS, f = gb + (slot << lg_s) + rank;
            int k = mat;
            while (LIST && k + 1 < p.n && f >= p.m[k + 1].first) ++k;
            const int o = (f - p.m[k].first) * MV_ROWS + (j & (MV_ROWS - 1)), O = p.m[k].O;
            if (o >= O) continue;
            const float sc = load_behind(p.m[k].scale + o);
            const size_t at = (size_t)(slot * Mp * MV_ROWS + j) * 8;
            double sum = 0.0, rest = 0.0;
#pragma unroll 4
            for (int s = 0; s < S << lg_k; ++s) {
                const int2 v = *reinterpret_cast<const int2*>(src + s * part_bytes + at);
                sum += xscale[seg & 1][s][m] * ((double)v.x * 65536.0 + (double)v.y);
                if (M == 1) {
                    const int2 u = *reinterpret_cast<const int2*>(src + s * part_bytes + at + MV_ROWS * 8);
                    rest += xscale[seg & 1][s][m] * ((double)u.x * 65536.0 + (double)u.y);
                }
            }
            if (M == 1) sum += rest * (1.0 / 1073741824.0);
            p.m[k].y[(size_t)m * O + o] = (float)((double)sc * sum);
        }
    }
    if (s_end < g_end) mat = p.m[mat].next;
    s_begin = s_end;
    }
    if (S > 1 && first) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int NT, int R, int CAP>
cudaError_t mv_launch(MvTable<CAP>& p, int sm_count, size_t max_smem, int slot, bool follows, const cudaGraphNode_t* nodes, cudaStream_t stream) {
    constexpr bool LIST = CAP > 1;
    const int Mp = p.M == 1 ? 2 : p.M, S = 1 << p.log_s;
    const size_t group_bytes = ((size_t)Mp << p.log_p) * MV_ROWS * 8;
    int nc = 1;
    for (int i = 0; i < p.n; ++i) nc = std::max(nc, (mv_chunks(p.m[i].I) + S - 1) / S);
    p.xq_bytes = nc * NT * 2048;
    // Clusters of 8 do not tile the GPCs: of sm_count / 8 the last ones share SMs with others, which then hold the whole launch up.
    // Seven eighths of the SMs (16 clusters of 8): 20 matrices of an 8B-scale model 88 -> 81 us for one row, 118 -> 106 for four, 181 -> 166
    // for eight with other work beside them (one row alone 164 -> 162); 12 clusters 84 and 204, 30 (two CTAs on every SM) 109 and 139: one
    // setting for all rows, which is not the best one for eight.
    int clusters = sm_count * 7 / 8 / S;
    if (clusters < 1) clusters = 1;
    if (clusters > p.groups) clusters = p.groups;
    p.groups_q = p.groups / clusters; p.groups_r = p.groups % clusters;
    const size_t budget = max_smem - 4096;
    const size_t room = p.xq_bytes < budget ? budget - p.xq_bytes : 0;
    // The longest run of one cluster with one x.  Two buffers where a cluster takes more than one.  Room for more than that would keep the CTAs of
    // the launch behind this one off the SMs until it ends: blocks of 14336 x 4096 whose w3 and w2 share a list, one row, 41.6 us with the room for
    // all groups, 36.0 so, 35.8 with MV_X_COST (38.6 as single launches); of 5632 x 2048 17.4, 16.1, 15.7 (19.5).
    int most = 1, bufs = 1;
    if (!LIST) most = p.groups_q + (p.groups_r ? 1 : 0);
    for (int c = 0; LIST && c < clusters; ++c) {
        int m = 0, behind = 0;
        int begin = mv_cut(p, c, clusters, m);
        const int end = mv_cut(p, c + 1, clusters, behind);
        for (int k = m; begin < end; k = p.m[k].next) {
            const int stop = std::min(end, p.m[k].next < p.n ? p.m[p.m[k].next].first : p.groups);
            most = std::max(most, stop - begin);
            if (stop < end) bufs = 2;
            begin = stop;
        }
    }
    p.owned = (most + S - 1) / S;
    if (p.log_p > p.log_s) { p.owned = (p.owned + 1) / 2; bufs = 2; }           // twice the slices in the same room
    if ((size_t)p.owned * bufs * group_bytes > room) {
        bufs = 2;
        const int fit = (int)std::min((size_t)1 << 20, room / (2 * group_bytes));
        p.owned = std::min(p.owned, std::max(fit, 1));
    }
    p.block = p.owned * S;
    const size_t smem = p.xq_bytes + bufs * p.owned * group_bytes;
    if (smem > max_smem - 4096) return cudaErrorInvalidConfiguration;
    const bool two = LIST && p.log_p > p.log_s;
    void (*const kernel)(MvTable<CAP>) = two ? gemv_mma_kernel<NT, R, 2 * LIST> : gemv_mma_kernel<NT, R, LIST>;
    const void* kern = reinterpret_cast<const void*>(kernel);
    cudaError_t e = ensure_dynamic_smem(kern, two ? slot + 32 : LIST ? slot + 10 : slot, max_smem);
    if (e != cudaSuccess) return e;
    if (nodes) {
        void* args[] = {&p};
        cudaKernelNodeParams kp = {};
        kp.func = const_cast<void*>(kern);
        kp.gridDim = dim3(clusters * S); kp.blockDim = dim3(MV_THREADS); kp.sharedMemBytes = (unsigned)smem;
        kp.kernelParams = args;
        cudaKernelNodeAttrValue cluster = {};
        cluster.clusterDim.x = S; cluster.clusterDim.y = cluster.clusterDim.z = 1;
        e = cudaGraphKernelNodeSetAttribute(nodes[0], cudaLaunchAttributeClusterDimension, &cluster);      // first: a list's clusters only shrink
        return e == cudaSuccess ? cudaGraphKernelNodeSetParams(nodes[0], &kp) : e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(clusters * S); cfg.blockDim = dim3(MV_THREADS); cfg.stream = stream;
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[2];
    int n = 0;
    if (S > 1) { at[n].id = cudaLaunchAttributeClusterDimension; at[n].val.clusterDim.x = S; at[n].val.clusterDim.y = 1; at[n].val.clusterDim.z = 1; ++n; }
    if (follows) { at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[n].val.programmaticStreamSerializationAllowed = 1; ++n; }
    cfg.attrs = at; cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, p);
}

}  // namespace

// The widest portable cluster: the fixed part of a call (digits of a slice, sums of an output) shrinks with the slice (20 matrices
// of an 8B-scale model, four rows of x: 379 / 262 / 206 us with 2 / 4 / 8).  A slice has one chunk at least.
int gemv_log_slices(int in_features) {
    const int NC = (in_features + MV_CHUNK - 1) / MV_CHUNK;
    int s = 3;
    while ((1 << s) > NC) --s;
    return s;
}
bool gemv_mma_supported(int M, int in_features, const void* packed2, size_t max_smem) {
    if (M < 1 || M > 8 || in_features % 64 != 0 || in_features < 64 || reinterpret_cast<uintptr_t>(packed2) % 16 != 0) return false;
    const int S = 1 << gemv_log_slices(in_features), NC = (in_features + MV_CHUNK - 1) / MV_CHUNK;
    return (size_t)((NC + S - 1) / S) * ((M + 1) / 2) * 2048 + 2 * (size_t)S * (M == 1 ? 2 : M) * MV_ROWS * 8 + 4096 <= max_smem;
}

// A list's clusters are those of its shortest rows, a CTA then takes two slices of longer ones (15 matrices of 1280 and 5120, one row: 18.6 us; in clusters of
// eight, of which short rows leave three CTAs idle, 23).
bool gemv_mma_takes(const GemvItem* items, int n, int M, size_t max_smem) {
    int low = 3, high = 0, chunks = 1;
    long long groups = 0;
    for (int i = 0; i < n; ++i) {
        low = std::min(low, gemv_log_slices(items[i].in_features));
        high = std::max(high, gemv_log_slices(items[i].in_features));
        chunks = std::max(chunks, mv_chunks(items[i].in_features));
        groups += (items[i].out_features + (long long)MV_ROWS - 1) / MV_ROWS;
    }
    const size_t digits = (size_t)((chunks + (1 << low) - 1) >> low) * ((M + 1) / 2) * 2048, sums = 2 * ((size_t)(M == 1 ? 2 : M) << high) * MV_ROWS * 8;
    return high - low <= 1 && groups <= 0x3fffffff && digits + sums + 4096 <= max_smem;
}

namespace {
template <int CAP>
cudaError_t mv_list(const GemvItem* items, int n, int M, bool follows, const cudaGraphNode_t* nodes, int sm_count, size_t max_smem,
                    cudaStream_t stream) {
    MvTable<CAP> p;
    p.n = n; p.M = M; p.log_s = 3; p.log_p = 0;
    for (int i = 0; i < n; ++i) { p.log_s = std::min(p.log_s, gemv_log_slices(items[i].in_features)); p.log_p = std::max(p.log_p, gemv_log_slices(items[i].in_features)); }
    // one x after the other
    bool taken[CAP] = {};
    int k = 0;
    long long groups = 0;
    p.cost = 0;
    for (int i = 0; i < n; ++i) {
        if (taken[i]) continue;
        const int begin = k;
        if (k > 0) p.cost += MV_X_COST;
        for (int j = i; j < n; ++j) {
            if (taken[j] || items[j].x != items[i].x || items[j].in_features != items[i].in_features) continue;
            taken[j] = true;
            const GemvItem& it = items[j];
            MvMat& m = p.m[k++];
            m.words = reinterpret_cast<const uint4*>(it.packed2); m.x = it.x; m.scale = it.scale; m.y = it.y;
            m.I = it.in_features; m.O = it.out_features;
            m.log_k = gemv_log_slices(it.in_features) - p.log_s;
            m.first = (int)groups; m.cost = p.cost;
            const long long g = (it.out_features + (long long)MV_ROWS - 1) / MV_ROWS;
            groups += g;
            p.cost += g * (mv_chunks(m.I) + MV_GROUP_COST);
        }
        for (int j = begin; j < k; ++j) p.m[j].next = k;
    }
    if (groups > 0x3fffffff) return cudaErrorInvalidValue;
    p.groups = (int)groups;
    switch ((M + 1) / 2) {
        case 1: return mv_launch<1, 4, CAP>(p, sm_count, max_smem, 26, follows, nodes, stream);
        case 2: return mv_launch<2, 3, CAP>(p, sm_count, max_smem, 27, follows, nodes, stream);
        case 3: return mv_launch<3, 2, CAP>(p, sm_count, max_smem, 28, follows, nodes, stream);
        default: return mv_launch<4, 2, CAP>(p, sm_count, max_smem, 29, follows, nodes, stream);
    }
}

}  // namespace

cudaError_t launch_ternary_gemv_mma(const GemvItem* items, int n, int M, bool follows, const cudaGraphNode_t* nodes, int sm_count,
                                    size_t max_smem, cudaStream_t stream) {
    return n == 1 ? mv_list<1>(items, n, M, follows, nodes, sm_count, max_smem, stream)
                  : mv_list<kGemvListCap>(items, n, M, follows, nodes, sm_count, max_smem, stream);
}

}  // namespace mcl
