// Ternary decode GEMV on tensor cores (sm_100a): y[m,o] = scale[o] * sum_k x[m,k] * t[o,k],
// M <= 16, with t read from the 2-bit packed weights.  HBM-bound on out*in/4 bytes of weights.
//
// CUDA cores cannot keep up with 4 weights per byte (one multiply-add per weight and
// activation row), so the contraction runs as integer MMA, exactly:
//   * each activation row is written as whole numbers of 30 bits and sign below its largest magnitude, four signed
//     digits of base 256; digit d of row m is row 4m+d of an int8 matrix Xq [N, in] (N = 16, 32, 48 or 64).  One row alone is two: the second
//     holds the 30 bits that the first leaves over;
//   * up to 8 rows have 30 bits below the largest magnitude of each slice of K (gemv_mma.cu's slices and, bit for bit, its results).  As long as those
//     magnitudes lie within 2^8 of one another, all slices are written in the unit of the finest, which takes a fifth digit, and the whole of K
//     is one exact sum (which a double holds, so that gemv_mma.cu's sum of slices is exact as well).  For an x where they do not, every
//     slice keeps its unit and is taken from the accumulator by itself;
//   * a CTA streams [RT * 128 rows x 256 weights] tiles of packed 2-bit fields (f = t + 1) through TMA, four warps per 128 rows expand
//     the fields to int8 in TENSOR MEMORY, and one thread issues kind::i8 MMAs  acc[128, N] += F . Xq^T  with the A operand from there;
//   * sum_k x t = sum_k x f - sum_k x, so a per-row digit sum is subtracted at the end; digits are put together in whole numbers.
//
// One launch takes a list of matrices.  Its k-blocks are numbered through, tile by tile, and every CTA takes the
// same number of them in a row: nothing is left idle whatever the shapes are.  A tile that lies in one CTA is finished from tensor
// memory; one that a cut runs through is added up by atomics (whole numbers: any order gives the same sum) in a slot of the
// workspace, and the last CTA to arrive finishes it.  The launch before it writes the digits of every x once and clears slots and tickets; the
// first weights are on their way meanwhile (programmatic dependent launch).
//
// What bounds it: an SM has to take 90 weights per clock at 6.5 TB/s (the copies alone run at 5.1 to 5.9 TB/s in these boxes).  20 matrices
// of an 8B-scale model (210 MB) as one list take 65 us for one row of x, 68 for 4, 77 for 8 and 83 for 16 (2.5 to 3.2 TB/s; 50, 52, 62 and 69 with
// other work beside them), where a launch or three per matrix took 157, 333 and 368.  The fifth digit costs 4 rows 4 % and 8 rows 13 % (16
// more digit columns; without it, in the unit of the largest slice, the others would lose bits); an x in slices takes 100 us for one row, 167 for 8.
// MMAs issued from a single-lane branch took most of the time, whatever their N; 64 digit columns bring 16 KB of digits beside 16 KB of words
// per k-block, so two accumulators (RT = 2) share them: 16 rows 82 -> 80 us, one row 70 -> 60.  The epilogue of a tile is not overlapped
// within a CTA: what it loads (scales, sums of x) is loaded under the wait for the accumulator (16 rows 82.9 -> 79.5).
#include <cuda.h>

#include <algorithm>
#include <vector>

#include "kernels.h"
#include "tc_ptx.cuh"

namespace mcl {
namespace {

constexpr int GV_ROWS = 128;       // rows of an accumulator (UMMA M)
constexpr int GV_KB = 256;         // weights per k-block = 64 packed bytes per row
constexpr int GV_RAW = GV_ROWS * (GV_KB / 4);          // 8 KiB of packed bytes
constexpr int GV_MAX_STAGES = 8;       // slots of the raw ring (packed weights + activation digits)
constexpr int GV_ACOLS = 64;           // a [128 rows x 256 int8] tile = 64 32-bit columns
constexpr int GV_TMEM = 256;           // columns of a CTA, half of an SM's: accumulators (64 each), then expanded tiles

struct GvMat {
    const float* scale;
    float* y;
    const long long* sums;     // of x: [slice][16 rows] its whole numbers added up
    const double* units;       // and the value of one
    int O, kblocks, x, log_s;
    int first, tile;   // numbers of its first unit (k-block of a tile) and tile
};
struct GvTable {
    int n, xs, tiles, M, Nq, stages;
    int extra;         // first row of fifth digits
    int cut_q, cut_r;  // units / CTAs, and what is over
    int share;         // CTAs of a cluster
    int* err;
    int* acc;          // slots of [RT][Nq][128] sums for tiles that a cut runs through, by tile or by the CTA that begins it, whichever are fewer
    double* part;      // an x in slices: [CTA][not begun or begun][slice][row][RT * 128] sums of the tile at hand
    int* tickets;
    const int* wide;   // [x][8]: whether a row of it has to be taken in slices
    GvMat m[kGemvListCap];
    CUtensorMap maps[kGemvListCap], xmaps[kGemvXCap];
};

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
}

// Instruction descriptor, kind::i8: D = s32 (bits 4-5 = 2), A = B = signed 8-bit (bits 7-9,
// 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__device__ __forceinline__ uint32_t idesc_i8(int m, int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// D += A.B, A in tensor memory, B's descriptor as low and high words
__device__ __forceinline__ void umma_i8_tsu(uint32_t tmem_c, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accum) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 b;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 b, {%2, %3};\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], b, %4, p;\n\t}"
                 ::"r"(tmem_c), "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accum) : "memory");
}

__device__ __forceinline__ int gv_slice_at(int s, int kblocks, int log_s) { return (int)(((long long)s * kblocks) >> log_s); }
// A CTA's units as parts: of one tile, or (SLICED, for the xs in `wide`) of one slice of K of a tile.  One division at the start.
template <bool SLICED>
struct GvParts {
    const GvTable& p;
    const uint32_t wide;
    int u, end;                            // the next unit, and the one behind the last
    int m = 0, kbs, log_s;                 // matrix of the part
    int tile, kb0, nkb = 0, slice = 0, slice_end;
    __device__ __forceinline__ GvParts(const GvTable& p, int begin, int end, uint32_t wide = 0) : p(p), wide(wide), u(begin), end(end) {
        while (m + 1 < p.n && u >= p.m[m + 1].first) ++m;
        open();
        const int local = u - p.m[m].first;
        tile = local / kbs;
        kb0 = local - tile * kbs;
        if (SLICED) skip();
    }
    __device__ __forceinline__ void open() {
        kbs = p.m[m].kblocks;
        log_s = SLICED && (wide >> p.m[m].x & 1) ? p.m[m].log_s : 0;
        slice_end = SLICED ? gv_slice_at(1, kbs, log_s) : kbs;
    }
    __device__ __forceinline__ void skip() { while (slice_end <= kb0) slice_end = gv_slice_at(++slice + 1, kbs, log_s); }      // to the slice of kb0
    __device__ __forceinline__ bool next() {           // false: no more
        if (u >= end) return false;
        if (nkb > 0) {
            kb0 += nkb;
            if (kb0 == kbs) {
                kb0 = 0;
                slice = 0;
                ++tile;
                if (m + 1 < p.n && u >= p.m[m + 1].first) { ++m; tile = 0; }
                open();
            }
            if (SLICED) skip();
        }
        nkb = min(slice_end - kb0, end - u);
        u += nkb;
        return true;
    }
};
// the first unit of a CTA: units * cta / CTAs
__device__ __forceinline__ int gv_cut(const GvTable& p, int cta) { return p.cut_q * cta + (int)((uint32_t)(p.cut_r * cta) / gridDim.x); }
// the CTAs that share the units from `begin` to `end`, one of which is `cta`
__device__ __forceinline__ int gv_first_cta(const GvTable& p, int cta, int begin) { while (gv_cut(p, cta) > begin) --cta; return cta; }
__device__ __forceinline__ int gv_last_cta(const GvTable& p, int cta, int end) { while (gv_cut(p, cta + 1) < end) ++cta; return cta; }

// all threads of a cluster; what was written to shared memory before can be read behind it
__device__ __forceinline__ void gv_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__host__ __device__ inline int gv_rows(int M) { return M == 1 ? 2 : M; }        // rows of whole numbers
// the xs to be taken in slices; a whole warp, after the wait for the launch before
__device__ __forceinline__ uint32_t gv_wide(const GvTable& p) {
    const int lane = threadIdx.x & 31, row = lane & 7;
    uint32_t mask = 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int x = 4 * i + (lane >> 3);
        const uint32_t b = __ballot_sync(0xffffffffu, x < p.xs && row < p.M && *reinterpret_cast<const volatile int*>(p.wide + 8 * x + row) != 0);
        for (int k = 0; k < 4; ++k) mask |= (b >> (8 * k) & 255u) ? 1u << (4 * i + k) : 0u;
    }
    return mask;
}

// RT: accumulators (128 rows each) of a tile, which share the digits that a k-block loads
// ROWS: 4 or 8, for up to so many rows of x; 0 for more, which have one unit for the whole of K and four digits
// SHARED: one matrix whose tiles a cluster of p.share CTAs has each (RT = 1)
template <int RT, int ROWS, bool SHARED>
__global__ void __launch_bounds__(192 + 128 * RT, 2) gemv_tc_kernel(const __grid_constant__ GvTable p) {
    constexpr int EXP = (GV_TMEM - 64 * RT) / GV_ACOLS;        // expanded tiles in flight in tensor memory
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * GV_MAX_STAGES + 2 * EXP + 2 * RT];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag, last_ticket;
    __shared__ struct alignas(16) { long long sum; double unit; } x_of[8 * 16];       // of the x at hand: of a slice, or of the whole of K

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = p.stages, Nq = p.Nq;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t b_tile = (uint32_t)Nq * 128u;
    // Shared memory holds only what TMA delivers (a raw slot = packed weights | the two digit tiles).  The
    // expanded int8 weight tile is four times larger than its packed form; it is written to TENSOR MEMORY
    // (tcgen05.st, thread = row = TMEM lane) and the MMA takes its A operand from there, so neither the
    // expansion nor the operand fetch uses shared-memory bandwidth.
    const uint32_t stage_bytes = RT * GV_RAW + 2 * b_tile;
    const uint32_t bar0 = smem_u32(bars);
    auto raw_full = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (GV_MAX_STAGES + s); };
    auto a_full = [&](int e) { return bar0 + 8u * (2 * GV_MAX_STAGES + e); };
    auto a_empty = [&](int e) { return bar0 + 8u * (2 * GV_MAX_STAGES + EXP + e); };
    auto acc_full = [&](int h) { return bar0 + 8u * (2 * GV_MAX_STAGES + 2 * EXP + h); };
    auto acc_empty = [&](int h) { return bar0 + 8u * (2 * GV_MAX_STAGES + 2 * EXP + RT + h); };
    const int u_begin = gv_cut(p, blockIdx.x), u_end = gv_cut(p, blockIdx.x + 1);

    if (threadIdx.x == 0) {
        abort_flag = (*reinterpret_cast<volatile int*>(p.err) != 0);
        for (int s = 0; s < S; ++s) { mbar_init(raw_full(s), 1); mbar_init(empty_bar(s), 1); }
        for (int e = 0; e < EXP; ++e) { mbar_init(a_full(e), 4); mbar_init(a_empty(e), 1); }
        for (int h = 0; h < RT; ++h) { mbar_init(acc_full(h), 1); mbar_init(acc_empty(h), 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_slot)), "r"(GV_TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    grid_release();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // ---- TMA producer: packed weights and the two digit tiles of a k-block.  The weights of the first slots do not
            // wait for the kernel before this one, which writes the digits ----
            bool waited = false;
            int it = 0;
            int late[GV_MAX_STAGES], late_x[GV_MAX_STAGES];        // k-blocks whose digits are still to be asked for
            auto digits = [&](int s, int x, int kb) {
                const uint32_t st = base + (uint32_t)s * stage_bytes + RT * GV_RAW;
                tma_load_2d(st, &p.xmaps[x], raw_full(s), kb * GV_KB, 0);
                tma_load_2d(st + b_tile, &p.xmaps[x], raw_full(s), kb * GV_KB + 128, 0);
            };
            auto wait_before = [&] {
                grid_wait();
                for (int i = 0; i < it && i < S; ++i) digits(i, late_x[i], late[i]);
                waited = true;
            };
            for (GvParts<false> t(p, u_begin, u_end); !abort_flag && t.next();) {
                const int m = t.m, x = p.m[m].x;
                for (int j = 0; j < t.nkb; ++j, ++it) {
                    const int s = it % S, kb = t.kb0 + j;
                    if (it == S) wait_before();
                    if (!mbar_wait(empty_bar(s), ((it / S) & 1) ^ 1, &abort_flag)) { abort_flag = 1; atomicExch(p.err, 11); break; }
                    mbar_expect_tx(raw_full(s), stage_bytes);
                    tma_load_2d(base + (uint32_t)s * stage_bytes, &p.maps[m], raw_full(s), kb * (GV_KB / 4), t.tile * (RT * GV_ROWS));
                    if (waited) digits(s, x, kb);
                    else { late[s] = kb; late_x[s] = x; }
                }
            }
            if (!waited) wait_before();
        }
    } else if (warp == 1) {
        // ---- MMA issuer: RT x 8 x (128 x Nq x 32) int8 MMAs per k-block.  The whole warp runs the loop and one lane is elected around
        // the instructions: descriptors are warp-uniform then ----
        const uint32_t idesc = idesc_i8(GV_ROWS, Nq);
        const uint64_t db0 = smem_desc_k_sw128(base + RT * GV_RAW);
        const uint32_t db_hi = (uint32_t)(db0 >> 32), db_lo = (uint32_t)db0, db_stage = stage_bytes >> 4, db_half = b_tile >> 4;
        int n_local = 0, s = 0, e = 0;
        uint32_t e_ph = 0;
        bool ok = true;
        if (ROWS) grid_wait();
        for (GvParts<ROWS != 0> t(p, u_begin, u_end, ROWS ? gv_wide(p) : 0u); ok && t.next(); ++n_local) {
            for (int j = 0; j < t.nkb && ok; ++j) {
#pragma unroll
                for (int h = 0; h < RT; ++h) {
                    if (j == 0 && !mbar_wait_all(acc_empty(h), (n_local & 1) ^ 1, &abort_flag)) { abort_flag = 1; if (lane == 0) atomicExch(p.err, 14); ok = false; break; }
                    // the expanders arrive after they have seen the raw slot: this wait covers the digit tiles too
                    if (!mbar_wait_all(a_full(e), e_ph, &abort_flag)) { abort_flag = 1; if (lane == 0) atomicExch(p.err, 12); ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_tm = tmem_base + 64 * RT + (uint32_t)e * GV_ACOLS, d_tm = tmem_base + 64 * h, db = db_lo + (uint32_t)s * db_stage;
                    if (elect_one()) {
                        const uint32_t more = j != 0 ? 1u : 0u;
#pragma unroll
                        for (int i = 0; i < 8; ++i)             // 32 int8 of k = 8 TMEM columns of A, 32 bytes (+2) of B
                            umma_i8_tsu(d_tm, a_tm + 8 * i, db + (i >> 2) * db_half + 2 * (i & 3), db_hi, idesc, i ? 1u : more);
                        umma_commit(a_empty(e));
                        if (h + 1 == RT) umma_commit(empty_bar(s));
                        if (j + 1 == t.nkb) umma_commit(acc_full(h));
                    }
                    __syncwarp();
                    if (++e == EXP) { e = 0; e_ph ^= 1u; }
                }
                if (++s == S) s = 0;
            }
        }
    } else if (warp < 2 + 4 * RT) {
        // ---- expanders: 2-bit fields -> int8, written to tensor memory; thread = tile row = TMEM lane ----
        // a warp may touch the TMEM lanes of its quarter (warp % 4) only: that quarter is its 32 tile rows
        const int h = (warp - 2) >> 2, r = ((warp & 3) << 5) | lane;         // 0..127
        const uint32_t rsw64 = (uint32_t)((r >> 1) & 3);
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        for (int it = 0; it < u_end - u_begin; ++it) {
            const int s = it % S, e = (it * RT + h) % EXP;
            if (!mbar_wait_all(raw_full(s), (it / S) & 1, &abort_flag) ||
                !mbar_wait_all(a_empty(e), (((it * RT + h) / EXP) & 1) ^ 1, &abort_flag)) { abort_flag = 1; if (lane == 0) atomicExch(p.err, 13); break; }
            tc_fence_after();      // the MMAs that read this TMEM slot have completed (a_empty)
            const unsigned char* st = smem_raw + (base - smem_u32(smem_raw)) + (size_t)s * stage_bytes + h * GV_RAW;
            const uint4* raw = reinterpret_cast<const uint4*>(st + r * 64);
            const uint32_t a_tm = tmem_base + lane_base + 64 * RT + (uint32_t)e * GV_ACOLS;
#pragma unroll
            for (int half = 0; half < 2; ++half) {           // half a row: 32 packed bytes = 128 weights = 32 TMEM columns
                uint32_t v[32];
#pragma unroll
                for (int cc = 0; cc < 2; ++cc) {
                    const uint4 pk = raw[(2 * half + cc) ^ rsw64];    // staging was written with the 64-byte swizzle
                    const uint32_t w[4] = {pk.x, pk.y, pk.z, pk.w};
                    // One packed word (16 fields) into 16 bytes costs seven logic operations when output word i takes the fields
                    // 4j + i (j = byte index): (w >> 2i) & 0x03030303.  That permutes k inside every group of 16; the digits are
                    // stored in the same order.
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        v[cc * 16 + q * 4 + 0] = w[q] & 0x03030303u;
                        v[cc * 16 + q * 4 + 1] = (w[q] >> 2) & 0x03030303u;
                        v[cc * 16 + q * 4 + 2] = (w[q] >> 4) & 0x03030303u;
                        v[cc * 16 + q * 4 + 3] = (w[q] >> 6) & 0x03030303u;
                    }
                }
                tmem_st32(a_tm + (uint32_t)(32 * half), v);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(a_full(e));
        }
    } else {
        // ---- epilogue warps -------------------------------------------------------------------
        grid_wait();       // sums and units of the xs, cleared slots
        const int q = warp & 3, lrow = q * 32 + lane, M = p.M, rows = gv_rows(M);
        const uint32_t wide = ROWS ? gv_wide(p) : 0u, tmem = tmem_base + ((uint32_t)(q * 32) << 16);
        const int chunks = ROWS ? ROWS / 4 : Nq / 16;        // of sixteen digit columns: four rows of x
        const size_t pitch = RT * GV_ROWS;
        auto slice_sums = [&](int cta, bool begun, int slice) { return p.part + (size_t)(((cta * 2 + begun) * 8 + slice) * rows) * pitch; };
        auto number = [](int a, int b, int c, int d) { return ((long long)a * 256 + b) * 65536 + ((long long)c * 256 + d); };
        // of an output row, loaded under the wait for its sums; late where that would spill (8 rows of x, two accumulators)
        constexpr bool EARLY = ROWS < 8 || RT == 1;
        auto scale_of = [&](const GvMat& A, int row) { return row < A.O ? (double)load_behind(A.scale + row) : 0.0; };
        // four rows of x, from row 4 c on, of an output row
        auto write = [&](const GvMat& A, int row, int c, double sc, const double (&v)[4]) {
            if (row >= A.O) return;
            if (!EARLY) sc = scale_of(A, row);
            if (M == 1) {
                A.y[row] = (float)(sc * (v[0] + v[1] * (1.0 / 1073741824.0)));
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (4 * c + j < M) A.y[(size_t)(4 * c + j) * A.O + row] = (float)(sc * v[j]);
            }
        };
        auto finish = [&](const GvMat& A, int row, int c, double sc, const uint32_t* v, const int* fifth) {
            double n[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const auto x = x_of[4 * c + j];                    // beyond the rows there are: zeros
                n[j] = x.unit * (double)(number((int)v[4 * j], (int)v[4 * j + 1], (int)v[4 * j + 2], (int)v[4 * j + 3]) +
                                         (ROWS ? (long long)fifth[j] * 4294967296ll : 0ll) - x.sum);
            }
            write(A, row, c, sc, n);
        };
        int n_local = 0, x = -1;
        bool ok = true, begun = false;
        // A warp that gives up (ok) goes on through the parts and passes every barrier of the four: the others may not have seen it yet
        for (GvParts<ROWS != 0> t(p, u_begin, u_end, wide); t.next(); ++n_local) {
            const GvMat& A = p.m[t.m];
            const bool sliced = ROWS && (wide >> A.x & 1);
            if (t.kb0 == 0 || n_local == 0) begun = t.kb0 == 0;
            if (A.x != x) {
                x = A.x;
                asm volatile("bar.sync 1, 128;" ::: "memory");
                const int i = threadIdx.x - (64 + 128 * RT);
                const bool in = (i & 15) < rows && i >> 4 < 1 << A.log_s;
                long long sum = in ? A.sums[i] : 0ll;
                if (in && !sliced && i < 16)
                    for (int k = 1; k < 1 << A.log_s; ++k) sum += A.sums[16 * k + i];
                x_of[i].sum = sum;
                x_of[i].unit = in ? A.units[i] : 0.0;
                asm volatile("bar.sync 1, 128;" ::: "memory");
            }
            const bool whole = begun && t.kb0 + t.nkb == t.kbs;          // with this part all of the tile has been here
            const int tile_u = A.first + t.tile * t.kbs, from = whole ? blockIdx.x : gv_first_cta(p, blockIdx.x, tile_u);
            const int slot_i = p.tiles < (int)gridDim.x ? A.tile + t.tile : from;
            int* slot = p.acc + (size_t)slot_i * (RT * Nq * GV_ROWS);
#pragma unroll 1
            for (int h = 0; h < RT && ok; ++h) {
                const int row = (t.tile * RT + h) * GV_ROWS + lrow;
                const double sc = EARLY && whole ? scale_of(A, row) : 0.0;
                ok = !abort_flag;
                if (ok && !mbar_wait(acc_full(h), n_local & 1, &abort_flag)) { abort_flag = 1; atomicExch(p.err, 15); ok = false; }
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < (ROWS ? ROWS / 4 : 4); ++c) {
                    if (!ROWS && c == chunks) break;
                    uint32_t v[16];
                    int fifth[4] = {};
                    if (ROWS && !sliced) {
                        tmem_ld16(tmem + 64 * h + (p.extra & ~15), v);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            fifth[j] = (int)((p.extra & 15) ? v[16 - ROWS + 4 * c + j] : v[4 * c + j]);
                            if (SHARED) {
                                if (4 * c + j < rows) asm volatile("st.shared.u32 [%0], %1;" ::"r"(base + (uint32_t)((rows * 16 + (4 * c + j) * 4) * GV_ROWS + lrow * 4)), "r"(fifth[j]) : "memory");
                            } else if (!whole && row < A.O && 4 * c + j < rows) {
                                atomicAdd(slot + (h * Nq + p.extra + 4 * c + j) * GV_ROWS + lrow, fifth[j]);
                            }
                        }
                    }
                    tmem_ld16(tmem + 64 * h + 16 * c, v);
                    tmem_ld_wait();
                    if (sliced) {
                        const bool first = t.kb0 == gv_slice_at(t.slice, t.kbs, t.log_s);
                        double* to = slice_sums(blockIdx.x, begun, t.slice) + h * GV_ROWS + lrow;
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            if (4 * c + j < rows)
                                to[(4 * c + j) * pitch] = (double)(number((int)v[4 * j], (int)v[4 * j + 1], (int)v[4 * j + 2], (int)v[4 * j + 3]) -
                                                                   (first ? x_of[16 * t.slice + 4 * c + j].sum : 0ll));
                    } else if (whole) {
                        finish(A, row, c, sc, v, fifth);
                    } else if (SHARED) {                     // the CTA's one part: the slots of the ring are free
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            if (4 * c + j < rows) asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(base + (uint32_t)(((4 * c + j) * GV_ROWS + lrow) * 16)),
                                         "r"(v[4 * j]), "r"(v[4 * j + 1]), "r"(v[4 * j + 2]), "r"(v[4 * j + 3]) : "memory");
                    } else if (row < A.O) {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (16 * c + j < 4 * rows) atomicAdd(slot + (h * Nq + c * 16 + j) * GV_ROWS + lrow, (int)v[j]);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty(h));
            }
            if (((SHARED || whole) && !sliced) || (t.kb0 + t.nkb != t.kbs && t.u != u_end)) continue;
            if (!whole) {                 // the last of the CTAs that share the tile finishes it
                __threadfence();
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (threadIdx.x == 64 + 128 * RT) last_ticket = ok && atomicAdd(p.tickets + slot_i, 1) == gv_last_cta(p, blockIdx.x, tile_u + t.kbs) - from;
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (!last_ticket) continue;
                __threadfence();
            }
#pragma unroll 1
            for (int h = 0; h < RT && ok; ++h) {
                const int row = (t.tile * RT + h) * GV_ROWS + lrow;
                const double sc = EARLY ? scale_of(A, row) : 0.0;
                if (sliced) {
#pragma unroll 1
                    for (int c = 0; c < chunks; ++c) {
                        double total[4] = {};
                        for (int slice = 0, cta = from; slice < 1 << t.log_s; ++slice) {
                            const int k0 = gv_slice_at(slice, t.kbs, t.log_s), k1 = gv_slice_at(slice + 1, t.kbs, t.log_s);
                            while (gv_cut(p, cta + 1) - tile_u <= k0) ++cta;
                            double n[4] = {};
                            for (int i = cta; ; ++i) {
                                const double* src = slice_sums(i, i == from, slice) + h * GV_ROWS + lrow;
#pragma unroll
                                for (int j = 0; j < 4; ++j)
                                    if (4 * c + j < rows) n[j] += __ldcg(src + (4 * c + j) * pitch);
                                if (gv_cut(p, i + 1) - tile_u >= k1) break;
                            }
#pragma unroll
                            for (int j = 0; j < 4; ++j) total[j] += x_of[16 * slice + 4 * c + j].unit * n[j];
                        }
                        write(A, row, c, sc, total);
                    }
                    continue;
                }
                constexpr int AT_ONCE = ROWS || RT == 2 ? 1 : 2;         // of the widest list, half in flight where registers allow
#pragma unroll
                for (int c = 0; c < (ROWS ? ROWS / 4 : 4); c += AT_ONCE) {
                    if (!ROWS && c >= chunks) break;
                    uint32_t v[16 * AT_ONCE];
                    int fifth[4] = {};
#pragma unroll
                    for (int j = 0; j < 4 && ROWS; ++j) fifth[j] = 4 * c + j < rows ? __ldcg(slot + (h * Nq + p.extra + 4 * c + j) * GV_ROWS + lrow) : 0;
#pragma unroll
                    for (int j = 0; j < 16 * AT_ONCE; ++j) v[j] = 16 * c + j < 4 * rows ? (uint32_t)__ldcg(slot + (h * Nq + c * 16 + j) * GV_ROWS + lrow) : 0u;
                    finish(A, row, c, sc, v, fifth);
                    if (AT_ONCE == 2 && c + 1 < chunks) finish(A, row, c + 1, sc, v + 16 * (AT_ONCE - 1), fifth);
                }
            }
        }
        if (SHARED) {
            // every CTA finishes some rows of x: it adds up their digits' sums over the cluster
            const GvMat& A = p.m[0];
            const int rank = (int)(blockIdx.x % p.share), row = (int)(blockIdx.x / p.share) * GV_ROWS + lrow;
            const bool in = ok && row < A.O && !(wide & 1u);
            const double sc = in ? scale_of(A, row) : 0.0;
            auto sum = [&](int m) {
                int d[5] = {};
#pragma unroll 4
                for (int k = 0; k < p.share; ++k) {
                    uint32_t from;
                    int v[4];
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(from) : "r"(base), "r"(k));
                    asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                                 : "r"(from + (uint32_t)((m * GV_ROWS + lrow) * 16)) : "memory");
#pragma unroll
                    for (int i = 0; i < 4; ++i) d[i] += v[i];
                    if (ROWS) {
                        asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v[0]) : "r"(from + (uint32_t)((rows * 16 + m * 4) * GV_ROWS + lrow * 4)) : "memory");
                        d[4] += v[0];
                    }
                }
                return x_of[m].unit * (double)(number(d[0], d[1], d[2], d[3]) + (ROWS ? (long long)d[4] * 4294967296ll : 0ll) - x_of[m].sum);
            };
            gv_cluster_sync();
            if (in && M == 1) {
                if (rank == 0) A.y[row] = (float)(sc * (sum(0) + sum(1) * (1.0 / 1073741824.0)));
            } else if (in) {
                for (int m = rank; m < M; m += p.share) A.y[(size_t)m * A.O + row] = (float)(sc * sum(m));
            }
            gv_cluster_sync();             // before this CTA's shared memory goes
        }
    }
    __syncwarp();
    if (SHARED && warp < 2 + 4 * RT) { gv_cluster_sync(); gv_cluster_sync(); }
    if (abort_flag) {
        const unsigned long long t0 = clock64();
        while (clock64() - t0 < 2000000ull) {}
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(GV_TMEM) : "memory");
    }
}

__device__ __forceinline__ float4 gv_load_x(const float4* p) {       // never before the wait on the grid this one depends on
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}

// ---- activation rows -> int8 digit rows, their sums, power-of-two units; slots and tickets of the contraction cleared ----
// blocks: one per row of an x (up to 8 rows: per slice and row), then those that clear
constexpr int GQ_THREADS = 512;
struct GqTable {
    int n, M, rows, extra;
    int I[kGemvXCap], log_s[kGemvXCap], spread[kGemvXCap];      // spread: how far apart the units of slices may be for one of all
    int first[kGemvXCap + 1];              // number of an x's first block
    const float* x[kGemvXCap];
    signed char* xq[kGemvXCap];
    long long* sums[kGemvXCap];            // [slice][16]
    double* units[kGemvXCap];
    int* wide;                             // [x][8]
    int4* clear;
    size_t clear_n;
};
__device__ __forceinline__ bool gq_clear(const GqTable& p) {
    if (blockIdx.x < p.first[p.n]) return false;
    const size_t nthr = (size_t)(gridDim.x - p.first[p.n]) * GQ_THREADS;
    for (size_t i = (size_t)(blockIdx.x - p.first[p.n]) * GQ_THREADS + threadIdx.x; i < p.clear_n; i += nthr) p.clear[i] = make_int4(0, 0, 0, 0);
    return true;
}
// up to 8 rows
__global__ void __launch_bounds__(GQ_THREADS) gemv_quantize_slices_kernel(const __grid_constant__ GqTable p) {
    __shared__ unsigned int top[8];
    __shared__ unsigned long long total;
    const int tid = threadIdx.x;
    grid_release();
    grid_wait();
    if (gq_clear(p)) return;
    int xi = 0;
    while (blockIdx.x >= p.first[xi + 1]) ++xi;
    const int at = blockIdx.x - p.first[xi], slice = at / p.rows, slot = at - slice * p.rows;
    const int M = p.M, I = p.I[xi], lg = p.log_s[xi], chunks = (I + GV_KB - 1) / GV_KB;
    const int k0 = (int)(((long long)slice * chunks) >> lg) * GV_KB, k1 = min((int)(((long long)(slice + 1) * chunks) >> lg) * GV_KB, I);
    const float* x = p.x[xi] + (size_t)(M == 1 ? 0 : slot) * I;
    const int warp = tid >> 5, lane = tid & 31;
    auto quad = [&](int k) { return k < k1 ? gv_load_x(reinterpret_cast<const float4*>(x + k)) : make_float4(0.f, 0.f, 0.f, 0.f); };
    float4 v = quad(k0 + 4 * tid);            // the slice's own, under the search for the largest magnitudes
    if (tid < 8) top[tid] = 0u;
    if (tid == 0) total = 0ull;
    __syncthreads();
    // the largest magnitude of every slice, half a chunk of K per warp; eight loads in flight
    constexpr int WARPS = GQ_THREADS / 32, FLIGHT = 8;
    for (int u0 = warp; u0 * 128 < I; u0 += FLIGHT * WARPS) {
        unsigned int t[FLIGHT];
#pragma unroll
        for (int i = 0; i < FLIGHT; ++i) {
            const int k = (u0 + i * WARPS) * 128 + lane * 4;
            const float4 f = k < I ? gv_load_x(reinterpret_cast<const float4*>(x + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
            t[i] = max(max(__float_as_uint(f.x) & 0x7FFFFFFFu, __float_as_uint(f.y) & 0x7FFFFFFFu), max(__float_as_uint(f.z) & 0x7FFFFFFFu, __float_as_uint(f.w) & 0x7FFFFFFFu));
        }
#pragma unroll
        for (int i = 0; i < FLIGHT; ++i) {
            const int u = u0 + i * WARPS;
            if (u * 128 >= I) break;
            t[i] = __reduce_max_sync(0xffffffffu, t[i]);
            if (lane == 0) atomicMax(&top[((((u >> 1) + 1) << lg) - 1) / chunks], t[i]);
        }
    }
    __syncthreads();
    int low = 1 << 20, high = -(1 << 20);
    bool finite = true;
    for (int k = 0; k < 1 << lg; ++k) {
        const unsigned int t = top[k];
        finite = finite && t < 0x7F800000u;
        if (t == 0u || t >= 0x7F800000u) continue;
        low = min(low, gemv_exponent(t));
        high = max(high, gemv_exponent(t));
    }
    const unsigned int mine = top[slice];
    const int e = mine >= 0x7F800000u || low > high ? 0 : gemv_exponent(mine);
    const bool wide = high - low > p.spread[xi];
    const int shift = wide || mine == 0u || mine >= 0x7F800000u ? 0 : e - low;
    const GemvUnit inv = gemv_unit(e);
    signed char* const q = p.xq[xi] + (size_t)(4 * slot) * I + k0;
    signed char* const q5 = p.xq[xi] + (size_t)(p.extra + slot) * I + k0;
    // Four lanes hold a group of 16 activations, element 4 j + a in register a of lane j; word i of a digit row takes the elements i, 4 + i,
    // 8 + i, 12 + i.  Two exchanges of bytes leave lane j with byte j of the four.
    auto turn = [&](uint32_t w) {
        const uint32_t o1 = __shfl_xor_sync(0xffffffffu, w, 1);
        const uint32_t h = (lane & 1) ? __byte_perm(w, o1, 0x3715) : __byte_perm(w, o1, 0x6240);
        const uint32_t o2 = __shfl_xor_sync(0xffffffffu, h, 2);
        return (lane & 2) ? __byte_perm(o2, h, 0x7632) : __byte_perm(h, o2, 0x5410);
    };
    long long sum = 0;
    for (int g0 = 32 * warp; k0 + 4 * g0 < k1; g0 += GQ_THREADS) {
        const int g = g0 + lane;
        if (g0 >= GQ_THREADS) v = quad(k0 + 4 * g);
        const float f[4] = {v.x * inv.a * inv.b, v.y * inv.a * inv.b, v.z * inv.a * inv.b, v.w * inv.a * inv.b};
        uint32_t r[4], r5 = 0;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            int n = __float2int_rn(f[a]);
            // what the 30 bits leave over: nothing from 2^23 on, where f is a whole number itself
            if (M == 1 && slot == 1) n = __float2int_rn((f[a] - (float)n) * 1073741824.0f);
            sum += n;
            const long long b = ((long long)n << shift) + 0x80808080ll;          // signed bytes, base 256
            r[a] = turn((uint32_t)b ^ 0x80808080u);
            r5 |= ((uint32_t)(b >> 32) & 255u) << (8 * a);
        }
        r5 = turn(r5);
        if (k0 + 4 * g < k1) {
            const size_t to = (size_t)(g >> 2) * 16;
            *reinterpret_cast<uint4*>(q + (size_t)(3 - (lane & 3)) * I + to) = make_uint4(r[0], r[1], r[2], r[3]);        // byte 3 is the leading one of four
            *reinterpret_cast<uint32_t*>(q5 + to + 4 * (lane & 3)) = r5;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((tid & 31) == 0) atomicAdd(&total, (unsigned long long)sum);
    __syncthreads();
    if (tid == 0) {
        const int unit = (wide || low > high ? e : low) - 30;
        p.sums[xi][16 * slice + slot] = (long long)total << shift;
        p.units[xi][16 * slice + slot] = __longlong_as_double(finite ? (long long)(1023 + unit) << 52 : 0x7FF8000000000000ll);       // an infinity or NaN: so is the row
        if (slice == 0 && slot < M) p.wide[8 * xi + slot] = wide;
    }
}

// more than 8 rows: one unit for the whole of K
__global__ void __launch_bounds__(GQ_THREADS) gemv_quantize_kernel(const __grid_constant__ GqTable p) {
    __shared__ unsigned int top_s;
    __shared__ int isum[4];
    const int tid = threadIdx.x;
    grid_release();
    grid_wait();
    if (gq_clear(p)) return;
    const int xi = blockIdx.x / p.rows, row = blockIdx.x - xi * p.rows, I = p.I[xi], pitch = I >> 4;
    uint4* q = reinterpret_cast<uint4*>(p.xq[xi] + (size_t)(4 * row) * I);
    const float4* x = reinterpret_cast<const float4*>(p.x[xi] + (size_t)row * I);
    if (tid == 0) top_s = 0u;
    if (tid < 4) isum[tid] = 0;
    __syncthreads();
    unsigned int top = 0u;
    float4 own[4];                 // this thread's first group of 16, all there are up to 8192
    for (int g = tid; g < pitch; g += GQ_THREADS) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 v = gv_load_x(x + 4 * g + j);
            if (g == tid) own[j] = v;
            top = max(max(max(top, __float_as_uint(v.x) & 0x7FFFFFFFu), max(__float_as_uint(v.y) & 0x7FFFFFFFu, __float_as_uint(v.z) & 0x7FFFFFFFu)),
                      __float_as_uint(v.w) & 0x7FFFFFFFu);
        }
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if ((tid & 31) == 0) atomicMax(&top_s, top);
    __syncthreads();
    top = top_s;
    const int e = top >= 0x7F800000u ? 0 : gemv_exponent(top);
    const GemvUnit inv = gemv_unit(e);
    int sum[4] = {0, 0, 0, 0};
    for (int g = tid; g < pitch; g += GQ_THREADS) {
        uint32_t r[16];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 v = g == tid ? own[j] : gv_load_x(x + 4 * g + j);
            const float f[4] = {v.x * inv.a * inv.b, v.y * inv.a * inv.b, v.z * inv.a * inv.b, v.w * inv.a * inv.b};
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                r[4 * j + a] = ((uint32_t)__float2int_rn(f[a]) + 0x80808080u) ^ 0x80808080u;        // four signed bytes, base 256
            }
        }
#pragma unroll
        for (int d = 0; d < 4; ++d) {                // byte 3 is the leading digit; word i of a digit row takes the elements 4 j + i
            uint32_t o[4];
            const uint32_t pick = (uint32_t)(3 - d) | ((uint32_t)(7 - d) << 4);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                o[i] = __byte_perm(__byte_perm(r[i], r[4 + i], pick), __byte_perm(r[8 + i], r[12 + i], pick), 0x5410);
                sum[d] = __dp4a((int)o[i], 0x01010101, sum[d]);
            }
            q[(size_t)d * pitch + g] = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        sum[d] = __reduce_add_sync(0xffffffffu, sum[d]);
        if ((tid & 31) == 0) atomicAdd(&isum[d], sum[d]);
    }
    __syncthreads();
    if (tid == 0) {       // an infinity or NaN: so is the row
        p.sums[xi][row] = ((long long)isum[0] * 256 + isum[1]) * 65536 + ((long long)isum[2] * 256 + isum[3]);
        p.units[xi][row] = __longlong_as_double(top >= 0x7F800000u ? 0x7FF8000000000000ll : (long long)(1023 + e - 30) << 52);
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);
EncodeTiledFn gv_encode_tiled() {
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
bool gv_map_2d(CUtensorMap* map, const void* basep, size_t inner_bytes, size_t rows, size_t pitch_bytes,
               int box_inner, int box_rows, CUtensorMapSwizzle sw) {
    EncodeTiledFn enc = gv_encode_tiled();
    if (!enc) return false;
    cuuint64_t dims[2] = {(cuuint64_t)inner_bytes, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)pitch_bytes};
    cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(basep), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}


// digit rows of a launch, and where the fifth digits begin: each of up to 8 rows' stand in sixteen columns of their own or the last of a group's
int gv_extra(int M) { return M <= 3 ? 12 : M == 4 ? 16 : M <= 6 ? 24 : M <= 8 ? 32 : 0; }
int gv_nq(int M) { return M <= 3 ? 16 : M <= 6 ? 32 : M <= 8 ? 48 : (4 * M + 15) / 16 * 16; }
size_t round_up(size_t n) { return (n + 1023) & ~size_t(1023); }
constexpr size_t kGvUnits = 1024, kGvXBytes = 2048;      // of an x: 128 sums, 128 units
long long gv_blocks(const GemvItem* items, int n) {        // k-blocks of 128 rows
    long long u = 0;
    for (int i = 0; i < n; ++i) u += (items[i].out_features + (long long)GV_ROWS - 1) / GV_ROWS * ((items[i].in_features + GV_KB - 1) / GV_KB);
    return u;
}

}  // namespace

bool gemv_tc_supported(int M, int in_features, const void* packed2) {
    return M >= 1 && M <= 16 && in_features % 64 == 0 && in_features >= 256 && in_features <= (1 << 22) && reinterpret_cast<uintptr_t>(packed2) % 16 == 0;      // 32-bit sums of digits times fields
}

namespace {
struct GvPlan { int RT, ctas, share; long long units, tiles; size_t slots, slices; };      // bytes for tiles that a cut runs through
GvPlan gv_plan(const GemvItem* items, int n, int M, int sm_count) {
    GvPlan g;
    // Two CTAs on every SM and tiles of 256 rows, or one and 128.  One row: 2100 k-blocks 22.6 and 20.8 us, 5760 26.8 and 35.0, 25600 60 and 118; 16
    // rows, alone and with other work beside them: 5760 35 / 26.8 and 43 / 19.7, 25600 80 / 68 and 141 / 66.
    const bool large = gv_blocks(items, n) >= (long long)sm_count * (M <= 8 ? 24 : 64);
    g.RT = large ? 2 : 1;
    g.units = g.tiles = 0;
    for (int i = 0; i < n; ++i) {
        const long long of = (items[i].out_features + (long long)g.RT * GV_ROWS - 1) / (g.RT * GV_ROWS);
        g.tiles += of;
        g.units += of * ((items[i].in_features + GV_KB - 1) / GV_KB);
    }
    // One matrix of few tiles: no CTA has parts of two (4096 x 4096, 16 rows: 16.2 -> 13.1 us), and a tile is cut only where that saves more
    // than adding up its parts costs (six k-blocks, about 4 us; 1024 -> 4096 and back: 11.2 -> 10.1 us a matrix).  Up to 8 CTAs are a cluster
    // then and read one another's sums: atomics, a fence and a ticket cost 2 us more (4096 x 4096
    // in a chain, 9 rows: 12.0 -> 10.9 us, 16: 13.6 -> 11.8).
    int per = g.RT * sm_count;
    g.share = 1;
    if (n == 1 && g.tiles <= sm_count) {
        const int kbs = (items[0].in_features + GV_KB - 1) / GV_KB, cut = std::max(1, std::min(kbs / 2, (int)(sm_count / g.tiles)));
        per = (int)g.tiles * (kbs - kbs / cut > 6 ? cut : 1);
        if (g.RT == 1 && per <= 8 * g.tiles) g.share = per / (int)g.tiles;
    }
    g.ctas = (int)std::min<long long>(per, g.units);
    g.slots = (size_t)std::min<long long>(g.ctas, g.tiles) * g.RT * gv_nq(M) * GV_ROWS * sizeof(int);
    g.slices = M <= 8 ? (size_t)g.ctas * 16 * gv_rows(M) * g.RT * GV_ROWS * sizeof(double) : 0;
    return g;
}
// more than 8 rows: room for the longest list, which a single matrix may become the first of
size_t gv_slot_room(const GvPlan& g, int M, int sm_count) { return round_up(M <= 8 ? g.slots : (size_t)2 * sm_count * 2 * gv_nq(M) * GV_ROWS * sizeof(int)); }
}  // namespace

// tickets | flags of the xs | slots | sums of slices | per x: Xq [Nq][in] int8, sums, units
size_t gemv_tc_workspace_bytes(const GemvItem* items, int n, int M, int sm_count) {
    const GvPlan g = gv_plan(items, n, M, sm_count);
    size_t bytes = round_up(2 * sm_count * sizeof(int)) + 1024 + gv_slot_room(g, M, sm_count) + round_up(g.slices);
    int xs = 0;
    for (int i = 0; i < n; ++i) {
        bool known = false;
        for (int j = 0; j < i; ++j) known = known || (items[j].x == items[i].x && items[j].in_features == items[i].in_features);
        if (known) continue;
        bytes += round_up((size_t)gv_nq(M) * items[i].in_features) + kGvXBytes;
        ++xs;
    }
    return xs <= kGemvXCap && gv_blocks(items, n) <= 0x3fffffff ? bytes : ~size_t(0);
}

// Against gemv_mma.cu (M <= 8), by k-blocks an SM has: that one needs no second launch and starts 5 us earlier, this one takes eight rows almost as
// fast as one and many xs as fast as few, which there are a round and new digits each.  Lists as launches of a dependent chain, us as gemv_mma /
// gemv_tc (A: 4096 x 4096, 512 blocks; B: 14336 x 4096, C: 4096 x 14336, 1792 each).  One x:
//   1 or 2 rows  10 A 25.5 / 26.6, 2 B 18.5 / 22.2      3 or 4  6 A 20.2 / 23.5, 2 B 23.0 / 23.5, 8 A 25.8 / 24.2
//   5 or 6       B 16.7 / 16.9, 4 A 18.7 / 24, 6 A 26.0 / 25.8, 2 B 31 / 28     7 or 8  3 A 18.7 / 22.2, B 20.1 / 17.5, C 25.2 / 20.4, 4 A 23.6 / 24.0
// Several xs:
//   1 or 2 rows  8 A of 4 21.3 / 24.5, B C 21.3 / 23.3, B B C 36 / 28          3 or 4  5 A of 5 20.1 / 23.5, 6 A of 6 26 / 25, B C 35 / 24.2
//   5 or 6       4 A of 4 19.5 / 24, 5 A of 5 31 / 25                            7 or 8  2 A of 2 15.0 / 18.4, 3 A of 3 25.4 / 22.5
bool gemv_tc_pays(const GemvItem* items, int n, int M, int sm_count) {
    static const int blocks[4][2] = {{37, 32}, {25, 20}, {20, 16}, {12, 10}};       // by pairs of rows; one x or several
    bool several = false;
    for (int i = 1; i < n; ++i) several = several || items[i].x != items[0].x || items[i].in_features != items[0].in_features;
    return M <= 8 && gv_blocks(items, n) >= (long long)sm_count * blocks[(M - 1) / 2][several];
}

namespace {
// A kernel node between `node` and what it depended on: `node` comes right behind it, overlapping at the seam.
cudaError_t put_before(cudaGraph_t graph, cudaGraphNode_t node, const cudaKernelNodeParams& kp) {
    size_t n = 0;
    cudaError_t e = cudaGraphNodeGetDependencies_v2(node, nullptr, nullptr, &n);
    if (e != cudaSuccess) return e;
    std::vector<cudaGraphNode_t> from(n), to(n, node);
    std::vector<cudaGraphEdgeData> edges(n);
    if (n > 0) e = cudaGraphNodeGetDependencies_v2(node, from.data(), edges.data(), &n);
    if (e != cudaSuccess) return e;
    cudaGraphNodeParams np = {};
    np.type = cudaGraphNodeTypeKernel;
    np.kernel.func = kp.func; np.kernel.gridDim = kp.gridDim; np.kernel.blockDim = kp.blockDim;
    np.kernel.sharedMemBytes = kp.sharedMemBytes; np.kernel.kernelParams = kp.kernelParams;
    cudaGraphNode_t made = nullptr;
    e = cudaGraphAddNode_v2(&made, graph, from.data(), edges.data(), n, &np);
    if (e == cudaSuccess && n > 0) e = cudaGraphRemoveDependencies_v2(graph, from.data(), to.data(), edges.data(), n);
    if (e != cudaSuccess) return e;
    cudaGraphEdgeData seam = {};
    seam.from_port = cudaGraphKernelNodePortProgrammatic;
    seam.type = cudaGraphDependencyTypeProgrammatic;
    return cudaGraphAddDependencies_v2(graph, &made, &node, &seam, 1);
}
}  // namespace

cudaError_t launch_ternary_gemv_tc(const GemvItem* items, int n, int M, void* workspace, int parts, bool follows, const cudaGraphNode_t* nodes,
                                   cudaGraph_t graph, int* err_word, int sm_count, size_t max_smem, cudaStream_t stream) {
    const int Nq = gv_nq(M);
    const GvPlan plan = gv_plan(items, n, M, sm_count);
    const int RT = plan.RT, ctas = plan.ctas;
    if (plan.units > 0x3fffffff) return cudaErrorInvalidValue;
    char* w = static_cast<char*>(workspace);
    GvTable p;
    GqTable g;
    p.n = n; p.M = M; p.Nq = Nq; p.err = err_word; p.extra = gv_extra(M);
    p.cut_q = (int)(plan.units / ctas); p.cut_r = (int)(plan.units % ctas);
    p.tiles = (int)plan.tiles;
    p.share = plan.share;
    g.wide = reinterpret_cast<int*>(w);
    p.wide = g.wide;
    w += 1024;
    p.tickets = reinterpret_cast<int*>(w);
    w += round_up(2 * sm_count * sizeof(int));
    p.acc = reinterpret_cast<int*>(w);
    w += gv_slot_room(plan, M, sm_count);
    p.part = reinterpret_cast<double*>(w);
    w += round_up(plan.slices);
    g.n = 0; g.M = M; g.rows = gv_rows(M); g.extra = p.extra; g.first[0] = 0;
    long long units = 0, tiles = 0;
    for (int i = 0; i < n; ++i) {
        const GemvItem& it = items[i];
        int x = 0;
        while (x < g.n && (g.x[x] != it.x || g.I[x] != it.in_features)) ++x;
        if (x == g.n) {
            if (x == kGemvXCap) return cudaErrorInvalidValue;
            ++g.n;
            g.x[x] = it.x; g.I[x] = it.in_features;
            g.xq[x] = reinterpret_cast<signed char*>(w);
            w += round_up((size_t)Nq * it.in_features);
            g.sums[x] = reinterpret_cast<long long*>(w);
            g.units[x] = reinterpret_cast<double*>(w + kGvUnits);
            w += kGvXBytes;
            g.log_s[x] = M <= 8 ? gemv_log_slices(it.in_features) : 0;
            // 30 bits, the spread and the carry of a sum of in_features fit the 53 bits of a double
            g.spread[x] = 8;
            while (g.spread[x] > 0 && (1ll << (23 - g.spread[x])) < it.in_features) --g.spread[x];
            g.first[g.n] = g.first[x] + (g.rows << g.log_s[x]);
            if (!gv_map_2d(&p.xmaps[x], g.xq[x], it.in_features, Nq, it.in_features, 128, Nq, CU_TENSOR_MAP_SWIZZLE_128B)) return cudaErrorInvalidValue;
        }
        GvMat& m = p.m[i];
        m.scale = it.scale; m.y = it.y; m.sums = g.sums[x]; m.units = g.units[x];
        m.O = it.out_features; m.x = x; m.log_s = g.log_s[x];
        m.kblocks = (it.in_features + GV_KB - 1) / GV_KB;
        m.first = (int)units;
        m.tile = (int)tiles;
        const long long of = (it.out_features + (long long)RT * GV_ROWS - 1) / (RT * GV_ROWS);
        tiles += of;
        units += of * m.kblocks;
        if (!gv_map_2d(&p.maps[i], it.packed2, (size_t)it.in_features / 4, it.out_features, (size_t)it.in_features / 4, GV_KB / 4, RT * GV_ROWS,
                       CU_TENSOR_MAP_SWIZZLE_64B)) return cudaErrorInvalidValue;
    }
    p.xs = g.n;
    const size_t stage_bytes = (size_t)RT * GV_RAW + 2 * (size_t)Nq * 128;
    p.stages = std::min(GV_MAX_STAGES, (int)((max_smem / 2 - 4608) / stage_bytes));
    if (p.stages < 2) return cudaErrorInvalidConfiguration;
    const size_t smem = p.stages * stage_bytes + 1024;
    // the tickets stand before the slots: one range
    g.clear = reinterpret_cast<int4*>(p.tickets);
    g.clear_n = (round_up(2 * sm_count * sizeof(int)) + (plan.share > 1 ? 0 : plan.slots)) / 16;
    const int q_blocks = g.first[g.n] + (int)std::min<size_t>(sm_count, (g.clear_n + 4 * GQ_THREADS - 1) / (4 * GQ_THREADS));

    // by rows (up to 4, up to 8, more); one accumulator, the same with clusters, two accumulators
    static void (*const kernels[3][3])(GvTable) = {{gemv_tc_kernel<1, 4, false>, gemv_tc_kernel<1, 4, true>, gemv_tc_kernel<2, 4, false>},
                                                   {gemv_tc_kernel<1, 8, false>, gemv_tc_kernel<1, 8, true>, gemv_tc_kernel<2, 8, false>},
                                                   {gemv_tc_kernel<1, 0, false>, gemv_tc_kernel<1, 0, true>, gemv_tc_kernel<2, 0, false>}};
    const int rows = M <= 4 ? 0 : M <= 8 ? 1 : 2, form = RT == 2 ? 2 : plan.share > 1 ? 1 : 0;
    void (*const kernel)(GvTable) = kernels[rows][form];
    const void* kern = reinterpret_cast<const void*>(kernel);
    cudaError_t e = ensure_dynamic_smem(kern, (form == 1 ? 62 : 52 + form / 2) + (form == 1 ? rows : 2 * rows), max_smem);
    if (e != cudaSuccess) return e;
    cudaKernelNodeParams kp = {};
    cudaLaunchConfig_t cfg = {};
    cfg.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = plan.share; at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    if (parts & 1) {
        void* args[] = {&g};
        void (*const digits)(GqTable) = M <= 8 ? gemv_quantize_slices_kernel : gemv_quantize_kernel;
        kp.func = reinterpret_cast<void*>(digits);
        kp.gridDim = cfg.gridDim = dim3(q_blocks); kp.blockDim = cfg.blockDim = dim3(GQ_THREADS);
        kp.kernelParams = args;
        cfg.numAttrs = follows ? 1 : 0;
        e = !nodes ? cudaLaunchKernelEx(&cfg, digits, g) : nodes[0] ? cudaGraphKernelNodeSetParams(nodes[0], &kp) : put_before(graph, nodes[1], kp);
        if (e != cudaSuccess) return e;
    }
    if (parts & 2) {
        void* args[] = {&p};
        kp.func = const_cast<void*>(kern);
        kp.gridDim = cfg.gridDim = dim3(ctas); kp.blockDim = cfg.blockDim = dim3(192 + 128 * RT);
        kp.sharedMemBytes = (unsigned)smem; cfg.dynamicSmemBytes = smem;
        kp.kernelParams = args;
        cfg.numAttrs = plan.share > 1 ? 2 : 1;
        if (nodes) {
            cudaKernelNodeAttrValue cluster = {};
            cluster.clusterDim.x = cluster.clusterDim.y = cluster.clusterDim.z = 1;        // the clusters of what the node was go first
            e = cudaGraphKernelNodeSetAttribute(nodes[1], cudaLaunchAttributeClusterDimension, &cluster);
            if (e == cudaSuccess) e = cudaGraphKernelNodeSetParams(nodes[1], &kp);
            cluster.clusterDim.x = plan.share;
            if (e == cudaSuccess && plan.share > 1) e = cudaGraphKernelNodeSetAttribute(nodes[1], cudaLaunchAttributeClusterDimension, &cluster);
        } else {
            e = cudaLaunchKernelEx(&cfg, kernel, p);
        }
    }
    return e;
}

}  // namespace mcl
