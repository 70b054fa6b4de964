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
// Where the launch before this one in a recorded batch is a launch of this kernel, those first loads even pass under its tail
// (programmatic dependent launch): the words of a matrix are no output of such a launch; x may be, and is read after the wait.
//
// x is scaled to whole numbers of 30 bits and sign below the slice's largest magnitude and written as four signed digits of
// base 256; one row alone (M = 1) has columns to spare and gets the 31 bits of the remainder as a second row.  Integer sums are
// exact; the offset of the fields (f = t + 1) is taken off as a digit sum; slices are put together in double precision.
// Legacy integer MMAs run at 2025 multiply-adds per clock and SM here (measured): 128 weights per clock for M <= 4 and 63 for
// M = 8; beyond that the tcgen05 kernel is the faster one.
#include "kernels.h"

namespace mcl {
namespace {

constexpr int MV_THREADS = 256;
constexpr int MV_WARPS = MV_THREADS / 32;
constexpr int MV_CHUNK = 256;          // weights of a row per unit: 64 bytes, 16 for each of the four lanes that share the row
constexpr int MV_ROWS = 32;            // rows of a unit
constexpr int MV_MAX_S = 8;

struct MvParams {
    const float* x;
    const uint32_t* packed2;
    const float* scale;
    float* y;
    int M, I, O;
    int log_s;                         // CTAs of a cluster
    int groups_q, groups_r;            // row groups of a cluster (the first groups_r clusters take one more)
    int block;                         // groups whose partial sums are held at a time
    int owned;                         // of them, the most that one CTA of the cluster finishes
    int xq_bytes;                      // the digits of the widest slice
};

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

// NT: tiles of eight digit columns (two rows of x each); R: units a warp has in registers
template <int NT, int R>
__global__ void __launch_bounds__(MV_THREADS, 2) gemv_mma_kernel(const MvParams p) {
    extern __shared__ __align__(128) unsigned char mv_smem[];
    __shared__ unsigned int amax[8];
    __shared__ int corr[NT * 8];
    __shared__ double xscale[MV_MAX_S][8];          // of every slice: the value of one unit of its whole numbers
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tq = lane & 3;
    const int lg_s = p.log_s, S = 1 << lg_s, rank = blockIdx.x & (S - 1), cid = blockIdx.x >> lg_s;
    const int M = p.M, Mp = M == 1 ? 2 : M, I = p.I, O = p.O;
    const int g_begin = cid * p.groups_q + min(cid, p.groups_r);
    const int g_end = g_begin + p.groups_q + (cid < p.groups_r ? 1 : 0);
    const int NC = (I + MV_CHUNK - 1) / MV_CHUNK;
    const int c0 = (rank * NC) >> lg_s, nc = (((rank + 1) * NC) >> lg_s) - c0;
    const int row16 = I >> 6;                       // 16-byte pieces of a row

    uint4 w[R][4];
    const uint4* words = reinterpret_cast<const uint4*>(p.packed2);
    int fg = g_begin + warp, fc = 0;                // load cursor: group, chunk
    auto load = [&](int end, uint4 (&u)[4]) {
        if (fg >= end) return;
        const int piece = (c0 + fc) * 4 + tq;
        if (piece < row16) {
#pragma unroll
            for (int h = 0; h < 4; ++h) u[h] = mv_load(words + (size_t)min(fg * MV_ROWS + h * 8 + g, O - 1) * row16 + piece);
        } else {
#pragma unroll
            for (int h = 0; h < 4; ++h) u[h] = make_uint4(0, 0, 0, 0);       // beyond the row: the digits there are zero as well
        }
        if (++fc == nc) { fc = 0; fg += MV_WARPS; }
    };
#pragma unroll
    for (int j = 0; j < R; ++j) load(min(g_begin + p.block, g_end), w[j]);
    if (threadIdx.x < 8) amax[threadIdx.x] = 0u;
    if (threadIdx.x < NT * 8) corr[threadIdx.x] = 0;
    if (S > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");    // only "this CTA runs": nothing to publish
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __syncthreads();

    // -- the digits of this slice: a warp takes 128 activations of one row at a time, four a lane --------------------
    const int k0 = c0 * MV_CHUNK, per_row = nc * 2;
#pragma unroll 4
    for (int unit = warp; unit < M * per_row; unit += MV_WARPS) {
        const int m = unit / per_row, k = k0 + (unit - m * per_row) * 128 + lane * 4;
        unsigned int top = 0u;
        if (k < I) {
            const float4 v = mv_load_x(p.x + (size_t)m * I + k);
            top = max(max(__float_as_uint(v.x) & 0x7FFFFFFFu, __float_as_uint(v.y) & 0x7FFFFFFFu),
                      max(__float_as_uint(v.z) & 0x7FFFFFFFu, __float_as_uint(v.w) & 0x7FFFFFFFu));
        }
        top = __reduce_max_sync(0xffffffffu, top);
        if (lane == 0) atomicMax(&amax[m], top);
    }
    __syncthreads();
#pragma unroll 2
    for (int unit = warp; unit < Mp * per_row; unit += MV_WARPS) {
        const int mp = unit / per_row, quad = (unit - mp * per_row) * 32 + lane, k = k0 + quad * 4;
        const int m = M == 1 ? 0 : mp;
        const unsigned int top = amax[m];
        int e = max((int)(top >> 23) - 126, -90);   // 2^e above every magnitude (of the smallest ones: 2^-90)
        if (top >= 0x7F800000u) e = 0;
        const float inv = __uint_as_float((uint32_t)(127 + 30 - e) << 23);
        const float4 t = k < I ? mv_load_x(p.x + (size_t)m * I + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float f[4] = {t.x * inv, t.y * inv, t.z * inv, t.w * inv};
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
        if (lane < 4) atomicAdd(&corr[mp * 4 + d], sum);
    }
    __syncthreads();
    if (S > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");      // every CTA of the cluster runs
    if ((int)threadIdx.x < 8 * S && (int)(threadIdx.x & 7) < M) {
        const int m = threadIdx.x & 7;
        const unsigned int top = amax[m];
        const int e = max((int)(top >> 23) - 126, -90);
        const double v = top >= 0x7F800000u ? __longlong_as_double(0x7FF8000000000000ll)       // an infinity or NaN: so is the row
                                            : __longlong_as_double((long long)(1023 + e - 30) << 52);
        uint32_t to;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to)
                     : "r"((uint32_t)__cvta_generic_to_shared(&xscale[rank][m])), "r"(threadIdx.x >> 3));
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(to), "d"(v) : "memory");
    }

    // -- the contraction ---------------------------------------------------------------------------------------------
    const uint32_t part0 = (uint32_t)__cvta_generic_to_shared(mv_smem) + (uint32_t)p.xq_bytes;
    const uint32_t part_bytes = (uint32_t)(p.owned * Mp) * (MV_ROWS * 8u);      // one slice's sums for the groups a CTA finishes
    int parity = 0;
    for (int gb = g_begin; gb < g_end; gb += p.block, parity ^= 1) {
        const int ge = min(gb + p.block, g_end);
        if (gb != g_begin) {
            fg = gb + warp; fc = 0;
#pragma unroll
            for (int j = 0; j < R; ++j) load(ge, w[j]);
        }
        const uint32_t part = (uint32_t)(parity * S) * part_bytes;
        int acc[2][NT][4] = {};
        int cc = 0;
#pragma unroll 1
        for (int grp = gb + warp; grp < ge;) {
#pragma unroll
            for (int j = 0; j < R; ++j) {
                if (grp < ge) {
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
                    load(ge, w[j]);
                    if (++cc == nc) {
                        // the slice of this group is complete: its sums, two digits to a word, go to the CTA that finishes the group
                        const int li = grp - gb;
                        uint32_t dst;
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst)
                                     : "r"(part0 + part + rank * part_bytes + (uint32_t)((li >> lg_s) * Mp) * (MV_ROWS * 8u)), "r"(li & (S - 1)));
#pragma unroll
                        for (int t = 0; t < NT; ++t) {
                            const int s0 = corr[t * 8 + 2 * tq], s1 = corr[t * 8 + 2 * tq + 1], m = 2 * t + (tq >> 1);
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
                        cc = 0;
                        grp += MV_WARPS;
                    }
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
            const int slot = i / per, j = i - slot * per, m = j / MV_ROWS, o = (gb + (slot << lg_s) + rank) * MV_ROWS + (j & (MV_ROWS - 1));
            if (o >= O) continue;
            const float sc = __ldg(p.scale + o);
            const size_t at = (size_t)(slot * Mp * MV_ROWS + j) * 8;
            double sum = 0.0;
#pragma unroll 4
            for (int s = 0; s < S; ++s) {
                const int2 v = *reinterpret_cast<const int2*>(src + s * part_bytes + at);
                double t = (double)v.x * 65536.0 + (double)v.y;
                if (M == 1) {
                    const int2 u = *reinterpret_cast<const int2*>(src + s * part_bytes + at + MV_ROWS * 8);
                    t += ((double)u.x * 65536.0 + (double)u.y) * (1.0 / 1073741824.0);
                }
                sum += xscale[s][m] * t;
            }
            p.y[(size_t)m * O + o] = (float)((double)sc * sum);
        }
    }
}

template <int NT, int R>
cudaError_t mv_launch(MvParams p, int sm_count, size_t max_smem, int slot, bool follows, cudaStream_t stream) {
    const int groups = (p.O + MV_ROWS - 1) / MV_ROWS, Mp = p.M == 1 ? 2 : p.M, NC = (p.I + MV_CHUNK - 1) / MV_CHUNK, S = 1 << p.log_s;
    const size_t group_bytes = (size_t)S * Mp * MV_ROWS * 8;
    // Clusters of 8 do not tile the GPCs: of sm_count / 8 the last ones share SMs with others, which then hold the whole launch up.
    // Seven eighths of the SMs (16 clusters of 8): 20 matrices of an 8B-scale model 88 -> 81 us for one row, 118 -> 106 for four, 181 -> 166
    // for eight with other work beside them (one row alone 164 -> 162); 12 clusters 84 and 204, 30 (two CTAs on every SM) 109 and 139: one
    // setting for all rows, which is not the best one for eight.
    int clusters = sm_count * 7 / 8 / S;
    if (clusters < 1) clusters = 1;
    if (clusters > groups) clusters = groups;
    p.groups_q = groups / clusters; p.groups_r = groups % clusters;
    p.block = p.groups_q + (p.groups_r ? 1 : 0);
    p.owned = (p.block + S - 1) / S;
    p.xq_bytes = ((NC + S - 1) / S) * NT * 2048;
    const size_t budget = max_smem - 4096;
    if ((size_t)p.xq_bytes + 2 * group_bytes > budget) return cudaErrorInvalidConfiguration;
    int bufs = 1;
    while (p.xq_bytes + bufs * p.owned * group_bytes > budget) { bufs = 2; p.owned = (p.owned + 1) / 2; p.block = p.owned * S; }
    cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(gemv_mma_kernel<NT, R>), slot, max_smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(clusters * S); cfg.blockDim = dim3(MV_THREADS); cfg.stream = stream;
    cfg.dynamicSmemBytes = p.xq_bytes + bufs * p.owned * group_bytes;
    cudaLaunchAttribute at[2];
    int n = 0;
    if (S > 1) { at[n].id = cudaLaunchAttributeClusterDimension; at[n].val.clusterDim.x = S; at[n].val.clusterDim.y = 1; at[n].val.clusterDim.z = 1; ++n; }
    if (follows) { at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[n].val.programmaticStreamSerializationAllowed = 1; ++n; }
    cfg.attrs = at; cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, gemv_mma_kernel<NT, R>, p);
}

// The widest portable cluster: the fixed part of a call (digits of a slice, sums of an output) shrinks with the slice (20 matrices
// of an 8B-scale model, four rows of x: 379 / 262 / 206 us with 2 / 4 / 8).  A slice has one chunk at least.
int mv_log_s(int in_features) {
    const int NC = (in_features + MV_CHUNK - 1) / MV_CHUNK;
    int s = 3;
    while ((1 << s) > NC) --s;
    return s;
}

}  // namespace

bool gemv_mma_supported(int M, int in_features, const void* packed2, size_t max_smem) {
    if (M < 1 || M > 8 || in_features % 64 != 0 || in_features < 64 || reinterpret_cast<uintptr_t>(packed2) % 16 != 0) return false;
    const int S = 1 << mv_log_s(in_features), NC = (in_features + MV_CHUNK - 1) / MV_CHUNK;
    return (size_t)((NC + S - 1) / S) * ((M + 1) / 2) * 2048 + 2 * (size_t)S * (M == 1 ? 2 : M) * MV_ROWS * 8 + 4096 <= max_smem;
}

cudaError_t launch_ternary_gemv_mma(const float* x, const uint32_t* packed2, const float* scale, float* y, int M, int in_features,
                                    int out_features, bool follows, int sm_count, size_t max_smem, cudaStream_t stream) {
    MvParams p = {};
    p.x = x; p.packed2 = packed2; p.scale = scale; p.y = y; p.M = M; p.I = in_features; p.O = out_features;
    p.log_s = mv_log_s(in_features);
    switch ((M + 1) / 2) {
        case 1: return mv_launch<1, 4>(p, sm_count, max_smem, 26, follows, stream);
        case 2: return mv_launch<2, 3>(p, sm_count, max_smem, 27, follows, stream);
        case 3: return mv_launch<3, 2>(p, sm_count, max_smem, 28, follows, stream);
        default: return mv_launch<4, 2>(p, sm_count, max_smem, 29, follows, stream);
    }
}

}  // namespace mcl
