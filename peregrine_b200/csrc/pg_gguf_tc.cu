// Dequantising product y = x . dequant(W)^T for GGUF Q4_0 / Q8_0 weights and several rows of x on the 5th-generation tensor cores
// (few rows: csrc/pg_gguf_stream.cu, which also describes the layout of the weights).
//
// Arithmetic, per 32-element block:
//   * x * 2^s (s per row: the largest element lies in [2^14, 2^15)) = h1 + h2, two f16 numbers: 22 significant bits, and more than
//     that of the row's largest element for all of them.  `gguf_planes_kernel` writes the two planes once per call.
//   * the quants become f16 exactly.  Each product (at most 11 + 8 bits) is exact in f32; the block's sum in the tensor core is the
//     sum of 64 of them, smaller plane first.
//   * the block's f16 scale is applied in f32 by the warps that take the sum out of TMEM: sum += d * block, rounded once per block.
//   * a row that holds a NaN or an infinity gives NaN, as in the streaming form (2^-s is then a NaN).
//
// Weights are the M side of the instruction (128 rows of W), rows of x the N side (MT): a lane of the epilogue owns a row of W, so
// that a block's scale is one register, and 32 lanes store 128 contiguous bytes of a row of y.  With few tiles K is divided over CTAs;
// the last part of a tile to finish adds all parts in their order.
//
// Up to 32 rows, gguf_tc_kernel (19 warps):
//   warps 0, 10   copies: blocks of 128 k of both planes by TMA; slices of W as they lie in memory (eight fills of 16 rows x 256 k)
//   warp 1        products: two steps of 16 k per block of W into an accumulator of its own; the planes lie side by side in one product,
//                 whose issue (not its time in the tensor core) is what counts here
//   warps 2-9     two per TMEM quarter, half of the columns each: sum += d * accumulator
//   warps 11-     quants -> f16 in the 128-byte-swizzled tiles that the products read, 128 k at a time, two such buffers
//
// Above, gguf_tc_wide_kernel (23 warps): the quants go to TMEM as f16 and the products take them from there, which leaves shared memory to
// the planes and makes a product of few columns cheaper (M 128, N 64: 37 cycles, 55 with the weights in shared memory).
//   warps 0, 1    one copy per stage of the planes, one per slice of W (a copy costs its thread 250 ... 600 cycles, whatever it brings)
//   warp 2        products: two planes x two steps of 16 k per block of W
//   warps 3-6     quants -> f16, a lane per row of W, 128 k at a time, two such buffers
//   warps 7-22    sum += d * accumulator, four warps per TMEM quarter
//
// What bounds it: the epilogue's chain per block -- barrier, some 100 cycles to read 32 columns of TMEM, back to the products -- at two or
// three accumulators in flight; at MT = 160 a block takes 685 cycles, 320 of them products.  Waits by the whole warp that end in one
// vote (pg_mbar_wait_warp) took a third off it.  Q4_0, N 14336, K 4096, us, 9 / 16 / 33 / 64 / 128 / 300 / 512 rows: 25 / 26 / 37 / 37 / 47 / 100 / 160
// (33 rows and more with the quants in shared memory and two warps per quarter: 39 / 42 / 53 / 126 / 194).
// Error against 64 bits (2-norm, of either type, plain inputs or 1 % of the channels x 20), which follows from the longest chain of rounded
// sums, by rows 9 ... 32 / 33 ... 64 / 128 / 300: N 14336, K 4096 2.9e-7 / 1.6e-7 / 2.1e-7 / 2.1e-7; N 4096, K 14336 2.8e-7 / 1.6e-7 / 2.1e-7 /
// 2.8e-7; N 4096, K 1024 0.9e-7 / 0.9e-7 / 1.0e-7 / 1.2e-7.  (Tiles of 64 rows with an accumulator to each plane and one chain of sums: 2.9e-7,
// 2.8e-7, 0.9e-7.  N 4096, K 1024 with K in four and two parts, as the form before took it at 128 and 300 rows: 0.95e-7, 1.03e-7.)
// Every mbarrier wait is bounded (pg_async.cuh).
#include <algorithm>

#include "pg_async.cuh"
#include "pg_gguf_f16.cuh"
#include "pg_internal.cuh"
#include "pg_launch.cuh"
#include "pg_tcgen05.cuh"

namespace {

constexpr int GT_N = 128;                         // rows of W per tile
constexpr int GT_ROWS = 64;                       // rows for which the planes always find room (pgk_gguf_tc_reserve)
constexpr size_t GT_TICKET_BYTES = 64 * 1024;     // as in the int8 kernel: tickets, zero between calls, then slabs
constexpr int64_t GT_PLANES = 100 << 20;          // most bytes of planes (they stay in L2; longer calls go in portions)

// ---- up to 32 rows ----------------------------------------------------------------------------------------------------------
template <int TYPE, int MT>
struct GtCfg {
    static constexpr int SEG = TYPE == PG_GGUF_Q4_0 ? 128 : 256;   // quant bytes per row and slice
    static constexpr int FILL = 16 * SEG + 256;
    static constexpr int RAW = 8 * FILL;                           // a slice (256 k) of 128 rows
    static constexpr int A_TILE = GT_N * 64 * 2;                   // 64 k of 128 rows in f16
    static constexpr int A_BYTES = 4 * A_TILE;                     // two buffers of 128 k
    static constexpr int COLS = 2 * MT;                            // accumulator columns of a block: one product for both planes, added up in the epilogue
    static constexpr int PLANE = MT * 64 * 2;
    static constexpr int BK64 = 2;                                 // 64-k blocks of the planes per stage
    static constexpr int B_STAGE = BK64 * 2 * PLANE;
    static constexpr int ROOM = 232448 - 1024 - 512;
    static constexpr int BST = MT == 32 ? 4 : 6;
    static constexpr int FIT = (ROOM - A_BYTES - BST * B_STAGE) / RAW;
    static constexpr int RST = FIT > 7 ? 7 : FIT;
    static constexpr int GB = 4;                                   // blocks per group of accumulators
    static constexpr int NBUF = 512 / (GB * COLS) > 4 ? 4 : 512 / (GB * COLS);
    static constexpr int HALF = MT / 2;                            // rows of x per warp of the epilogue
    static constexpr int DW = 8;                                   // warps that turn quants into f16
    static constexpr int THREADS = (11 + DW) * 32;
    static constexpr size_t SMEM = (size_t)A_BYTES + BST * B_STAGE + RST * RAW + 1024 + 512;
    static_assert(RST >= 2 && NBUF >= 2, "shared memory or TMEM too small");
};

struct GtParts {
    int parts, slices;       // K in `parts` parts of `slices` 256-element slices
    float *slabs;            // [unit][MT][128]
    unsigned int *tickets;   // one per (tile, TMEM quarter, half of the columns), zero between calls
};

// ---- planes of rows row0 .. row0 + rows - 1 of x: [2][rows][K] f16, and 2^-s per row.  grid (rows, parts of K) -----------------
template <bool Q4>
__global__ void __launch_bounds__(256)
    gguf_planes_kernel(const float *__restrict__ x, int row0, int rows, int K, uint4 *__restrict__ planes, float *__restrict__ us)
{
    __shared__ float red[16];
    pg_pdl_begin();
    const int r = blockIdx.x, tid = threadIdx.x, eights = K / 8;
    const float4 *src = reinterpret_cast<const float4 *>(x + (int64_t)(row0 + r) * K);
    float top = 0.0f, poison = 0.0f;              // every part looks at the whole row: it comes from L2
    for (int c = tid; c < K / 4; c += 256) {
        const float4 v = __ldcg(src + c);
        top = fmaxf(top, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
        poison += (v.x - v.x) + (v.y - v.y) + (v.z - v.z) + (v.w - v.w);   // 0, or NaN
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        poison += __shfl_xor_sync(0xffffffffu, poison, o);
    }
    if ((tid & 31) == 0) {
        red[tid >> 5] = top;
        red[8 + (tid >> 5)] = poison;
    }
    __syncthreads();
    for (int i = 0; i < 8; i++) {
        top = fmaxf(top, red[i]);
        poison += red[8 + i];
    }
    // (a row that is not finite has NaN for 2^-s, and zeros)
    const bool fine = poison == 0.0f;
    const int e = fine ? gguf_exponent(top) : 0;
    const float sc = scalbnf(1.0f, 14 - e);
    if (tid == 0 && blockIdx.y == 0) us[r] = fine ? scalbnf(1.0f, e - 14) : NAN;
    const int per = (eights + gridDim.y - 1) / gridDim.y, hi = min(eights, (int)(blockIdx.y + 1) * per);
    for (int c = blockIdx.y * per + tid; c < hi; c += 256) {
        const float4 a = __ldcg(src + 2 * c), b = __ldcg(src + 2 * c + 1);
        const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint4 h1, h2;
        gguf_split8<Q4>(v, sc, h1, h2);
        if (!fine) h1 = h2 = make_uint4(0u, 0u, 0u, 0u);
        planes[(int64_t)r * eights + c] = h1;
        planes[((int64_t)rows + r) * eights + c] = h2;
    }
}

// ---- pieces of the product ------------------------------------------------------------------------------------------------
// kind::f16 with f16 operands (0 at bits 7 and 10), f32 sums, both K-major
__host__ __device__ constexpr uint32_t gt_idesc(int m, int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24); }

// sum[0 .. NC) += d * the next NC columns of this lane's TMEM row
template <int NC>
__device__ __forceinline__ void gt_add(uint32_t taddr, float d, float *sum)
{
    constexpr int P = NC >= 32 ? 32 : NC;
    static_assert(P == 8 || P == 16 || P == 32, "pieces of 32, 16 or 8 columns");
    uint32_t t[P];
    if constexpr (P == 32) {
        tmem_ld32_async(taddr, t);
    } else if constexpr (P == 16) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
            : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7]), "=r"(t[8]), "=r"(t[9]), "=r"(t[10]),
              "=r"(t[11]), "=r"(t[12]), "=r"(t[13]), "=r"(t[14]), "=r"(t[15])
            : "r"(taddr)
            : "memory");
    } else {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7])
                     : "r"(taddr)
                     : "memory");
    }
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < P; i++) sum[i] = fmaf(d, __uint_as_float(t[i]), sum[i]);
    if constexpr (NC > P) gt_add<NC - P>(taddr + P, d, sum + P);
}
__device__ __forceinline__ void gt_sts128(uint32_t addr, const uint32_t (&v)[4])
{
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
// gives copies that are still in flight a bounded time to land before a CTA that gives up exits
__device__ __forceinline__ void gt_settle()
{
    const unsigned long long t0 = pg_globaltimer_ns();
    while (pg_globaltimer_ns() - t0 < 2000000ull) {
    }
}

template <int TYPE, int MT>
__global__ void __launch_bounds__(GtCfg<TYPE, MT>::THREADS, 1)
    gguf_tc_kernel(const __grid_constant__ CUtensorMap tmap_x, const uint8_t *__restrict__ qs, int64_t N, int nslices, int M, const float *__restrict__ us,
                   float *__restrict__ y, const GtParts kp, int32_t *status, unsigned long long limit_ns)
{
    using C = GtCfg<TYPE, MT>;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = pg_smem(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    const uint32_t a_at = base, b_at = a_at + C::A_BYTES, r_at = b_at + C::BST * C::B_STAGE;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_raw + (r_at - raw_addr) + C::RST * C::RAW);
    const uint32_t bar = pg_smem(bars);
    // full and empty of: slices, blocks of the planes, f16 buffers, groups of accumulators
    const uint32_t r_full = bar, r_empty = r_full + 8 * C::RST, b_full = r_empty + 8 * C::RST, b_empty = b_full + 8 * C::BST;
    const uint32_t a_full = b_empty + 8 * C::BST, a_empty = a_full + 16, t_full = a_empty + 16, t_empty = t_full + 8 * C::NBUF;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * C::RST + 2 * C::BST + 4 + 2 * C::NBUF);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < C::RST; i++) {
            pg_mbar_init(r_full + 8 * i, 1);
            pg_mbar_init(r_empty + 8 * i, 8 + C::DW);   // the scales, the quants
        }
        for (int i = 0; i < C::BST; i++) {
            pg_mbar_init(b_full + 8 * i, 1);
            pg_mbar_init(b_empty + 8 * i, 1);
        }
        for (int i = 0; i < 2; i++) {
            pg_mbar_init(a_full + 8 * i, C::DW);
            pg_mbar_init(a_empty + 8 * i, 1);
        }
        for (int i = 0; i < C::NBUF; i++) {
            pg_mbar_init(t_full + 8 * i, 1);
            pg_mbar_init(t_empty + 8 * i, 8);
        }
        *abort_flag = 0;
        pg_mbar_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(pg_smem(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int tiles_m = (M + MT - 1) / MT, tiles_n = (int)((N + GT_N - 1) / GT_N);
    const int sp = kp.parts, total = tiles_m * tiles_n * sp;   // unit u: part u % sp of tile u / sp; the tiles of a row of W follow each other
    auto s_first = [&](int u) { return (u % sp) * kp.slices; };
    auto s_end = [&](int u) { return min(nslices, (u % sp + 1) * kp.slices); };
    bool ok = true;

    if (warp == 0) {
        // ---------------------------------------------------------------- planes of x
        if (lane == 0) {
            uint32_t bs = 0, bp = 0;
            asm volatile("griddepcontrol.wait;" ::: "memory");
            for (int u = blockIdx.x; ok && u < total; u += gridDim.x) {
                const int m0 = (u / sp % tiles_m) * MT;
                for (int kb = 4 * s_first(u), end = 4 * s_end(u); kb < end; kb += C::BK64) {
                    if (!(ok = pg_mbar_wait(b_empty + 8 * bs, bp ^ 1, abort_flag, status, limit_ns))) break;
                    pg_mbar_expect(b_full + 8 * bs, C::B_STAGE);
#pragma unroll
                    for (int i = 0; i < C::BK64; i++)
                        tma_load_3d(b_at + bs * C::B_STAGE + i * 2 * C::PLANE, &tmap_x, b_full + 8 * bs, (kb + i) * 64, m0, 0);
                    if (++bs == C::BST) {
                        bs = 0;
                        bp ^= 1;
                    }
                }
            }
            if (!ok) gt_settle();
        }
    } else if (warp == 10) {
        // ---------------------------------------------------------------- slices of W, which no kernel writes: no wait for the preceding one
        if (lane == 0) {
            const int64_t fills = (N + 15) >> 4;               // (fills behind the last one do not exist)
            uint32_t rs = 0, rp = 0;
            for (int u = blockIdx.x; ok && u < total; u += gridDim.x) {
                const int64_t f0 = (int64_t)(u / sp / tiles_m) * (GT_N / 16);
                const int n = (int)min((int64_t)8, fills - f0);
                for (int s = s_first(u), end = s_end(u); s < end; s++) {
                    if (!(ok = pg_mbar_wait(r_empty + 8 * rs, rp ^ 1, abort_flag, status, limit_ns))) break;
                    pg_mbar_expect(r_full + 8 * rs, (uint32_t)n * C::FILL);
                    for (int i = 0; i < n; i++)
                        pg_bulk_load(r_at + rs * C::RAW + i * C::FILL, qs + ((f0 + i) * nslices + s) * (int64_t)C::FILL, C::FILL, r_full + 8 * rs);
                    if (++rs == C::RST) {
                        rs = 0;
                        rp ^= 1;
                    }
                }
            }
            if (!ok) gt_settle();
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- products (the whole warp; one lane's count)
        const uint32_t on = pg_elect();
        constexpr uint32_t idesc = gt_idesc(GT_N, C::COLS);
        const uint64_t desc_a = make_smem_desc(a_at), desc_b = make_smem_desc(b_at);
        uint32_t bs = 0, bp = 0, as = 0, ap = 0, ts = 0, tp = 0;
        auto wait = [&](uint32_t b, uint32_t parity) { return (bool)__all_sync(0xffffffffu, pg_mbar_wait(b, parity, abort_flag, status, limit_ns)); };
        for (int u = blockIdx.x; ok && u < total; u += gridDim.x)
            for (int h = 2 * s_first(u), end = 2 * s_end(u); ok && h < end; h++) {
                if (!(ok = wait(a_full + 8 * as, ap))) break;
#pragma unroll
                for (int blk = 0; blk < 4; blk++) {             // blocks of the 128 k
                    constexpr int PER_B = 2 * C::BK64;          // blocks per stage of the planes
                    if (blk % PER_B == 0 && !(ok = wait(b_full + 8 * bs, bp))) break;
                    if (blk % C::GB == 0 && !(ok = wait(t_empty + 8 * ts, tp ^ 1))) break;
                    tc_fence_after();
                    const uint32_t d = tmem + (ts * C::GB + blk % C::GB) * C::COLS;
                    const uint64_t da = desc_a + (uint64_t)((as * 2 + (blk >> 1)) * (C::A_TILE >> 4) + (blk & 1) * 4);
                    const uint64_t db = desc_b + (uint64_t)(bs * (C::B_STAGE >> 4) + (blk % PER_B >> 1) * (2 * C::PLANE >> 4) + (blk & 1) * 4);
#pragma unroll
                    for (int j = 0; j < 2; j++) umma_f16(d, da + (uint64_t)(j * 2), db + (uint64_t)(j * 2), idesc, j != 0 ? 1u : 0u, on);
                    if ((blk + 1) % C::GB == 0) {
                        umma_commit(t_full + 8 * ts, on);
                        if (++ts == C::NBUF) {
                            ts = 0;
                            tp ^= 1;
                        }
                    }
                    if ((blk + 1) % PER_B == 0) {
                        umma_commit(b_empty + 8 * bs, on);
                        if (++bs == C::BST) {
                            bs = 0;
                            bp ^= 1;
                        }
                    }
                }
                if (!ok) break;
                umma_commit(a_empty + 8 * as, on);
                as ^= 1;
                if (as == 0) ap ^= 1;
            }
    } else if (warp > 10) {
        // ---------------------------------------------------------------- quants -> f16: 128 / DW rows of W per warp, eight at a time
        constexpr int ROUNDS = GT_N / C::DW / 8, LOADS = TYPE == PG_GGUF_Q4_0 ? 1 : 2;
        const int row0 = (warp - 11) * (GT_N / C::DW) + (lane >> 2), t = lane & 3;
        // lane: row r, quarter t of the blocks; rows of odd number take their blocks in the other order, so that two rows never write
        // to the same banks (and the layout has them read from different ones)
        const int odd = row0 & 1, sw = (odd << 2) | ((row0 >> 1) & 3);   // (rows eight apart have the same)
        uint32_t rs = 0, rp = 0, as = 0, ap = 0;
        for (int u = blockIdx.x; ok && u < total; u += gridDim.x)
            for (int s = s_first(u), end = s_end(u); ok && s < end; s++) {
                ok = __all_sync(0xffffffffu, pg_mbar_wait(r_full + 8 * rs, rp, abort_flag, status, limit_ns));
                for (int h = 0; ok && h < 2; h++) {
                    // Q4_0: word t of four blocks; Q8_0: eight bytes of two blocks, twice
                    uint4 q[ROUNDS][LOADS];
#pragma unroll
                    for (int i = 0; i < ROUNDS; i++) {
                        const int r = row0 + i * 8;
                        const uint32_t src = r_at + rs * C::RAW + (uint32_t)(r >> 4) * C::FILL + (uint32_t)(r & 15) * C::SEG;
#pragma unroll
                        for (int p = 0; p < LOADS; p++) q[i][p] = pg_lds128(src + (uint32_t)((((h * LOADS + p) * 4 + t) ^ sw) * 16));
                    }
                    ok = __all_sync(0xffffffffu, pg_mbar_wait(a_empty + 8 * as, ap ^ 1, abort_flag, status, limit_ns));
                    if (!ok) break;
#pragma unroll
                    for (int i = 0; i < ROUNDS; i++) {
                        const int r = row0 + i * 8;
                        const uint32_t dst = a_at + as * (2 * C::A_TILE) + (uint32_t)r * 128;
                        auto put = [&](int blk, const uint32_t (&v)[4]) {   // block blk of the 128 k
                            gt_sts128(dst + (blk >> 1) * C::A_TILE + (uint32_t)((((blk & 1) * 4 + t) ^ (r & 7)) * 16), v);
                        };
                        uint32_t v[4];
#pragma unroll
                        for (int p = 0; p < 2; p++) {           // blocks 2 p and 2 p + 1
                            if constexpr (TYPE == PG_GGUF_Q4_0) {
                                const uint32_t w0 = p ? q[i][0].z : q[i][0].x, w1 = p ? q[i][0].w : q[i][0].y;
                                gguf_nibbles_f16(odd ? w1 : w0, v);
                                put(2 * p + odd, v);
                                gguf_nibbles_f16(odd ? w0 : w1, v);
                                put(2 * p + (odd ^ 1), v);
                            } else {
                                const uint4 w = q[i][p < LOADS ? p : 0];
                                gguf_bytes_f16(odd ? w.z : w.x, odd ? w.w : w.y, v);
                                put(2 * p + odd, v);
                                gguf_bytes_f16(odd ? w.x : w.z, odd ? w.y : w.w, v);
                                put(2 * p + (odd ^ 1), v);
                            }
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        pg_mbar_arrive(a_full + 8 * as);
                        if (h == 1) pg_mbar_arrive(r_empty + 8 * rs);
                    }
                    as ^= 1;
                    if (as == 0) ap ^= 1;
                }
                if (++rs == C::RST) {
                    rs = 0;
                    rp ^= 1;
                }
            }
    } else {
        // ---------------------------------------------------------------- sums and outputs: lane = row of W
        const int q = warp & 3, half = (warp - 2) >> 2, row = q * 32 + lane;
        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + half * C::HALF;
        asm volatile("griddepcontrol.wait;" ::: "memory");     // y may still be read by the predecessor
        uint32_t rs = 0, rp = 0, ts = 0, tp = 0;
        for (int u = blockIdx.x; ok && u < total; u += gridDim.x) {
            const int tile = u / sp;
            float sum[C::HALF];
#pragma unroll
            for (int j = 0; j < C::HALF; j++) sum[j] = 0.0f;
            for (int s = s_first(u), end = s_end(u); ok && s < end; s++) {
                ok = __all_sync(0xffffffffu, pg_mbar_wait(r_full + 8 * rs, rp, abort_flag, status, limit_ns));
                if (!ok) break;
                const uint4 sc = pg_lds128(r_at + rs * C::RAW + (uint32_t)(row >> 4) * C::FILL + 16 * C::SEG + (uint32_t)(row & 15) * 16);
                const uint32_t scw[4] = {sc.x, sc.y, sc.z, sc.w};
                __syncwarp();
                if (lane == 0) pg_mbar_arrive(r_empty + 8 * rs);
                if (++rs == C::RST) {
                    rs = 0;
                    rp ^= 1;
                }
#pragma unroll
                for (int b = 0; b < 8; b++) {
                    if (b % C::GB == 0) {
                        ok = ok && pg_mbar_wait(t_full + 8 * ts, tp, abort_flag, status, limit_ns);
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                        tc_fence_after();
                    }
                    const __half2 hh = *reinterpret_cast<const __half2 *>(&scw[b >> 1]);
                    const float d = (b & 1) ? __high2float(hh) : __low2float(hh);
                    const uint32_t at = taddr + (ts * C::GB + b % C::GB) * C::COLS;
                    gt_add<C::HALF>(at + MT, d, sum);
                    gt_add<C::HALF>(at, d, sum);
                    if ((b + 1) % C::GB == 0) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) pg_mbar_arrive(t_empty + 8 * ts);
                        if (++ts == C::NBUF) {
                            ts = 0;
                            tp ^= 1;
                        }
                    }
                }
            }
            if (!ok) break;
            if (sp > 1) {
                float *slab = kp.slabs + ((int64_t)u * MT + half * C::HALF) * GT_N + row;
#pragma unroll
                for (int j = 0; j < C::HALF; j++) __stcg(slab + j * GT_N, sum[j]);
                unsigned int *ticket = kp.tickets + tile * 8 + half * 4 + q;
                __threadfence();
                __syncwarp();
                const unsigned int before = __shfl_sync(0xffffffffu, lane == 0 ? atomicAdd(ticket, 1u) : 0u, 0);
                if (before != (unsigned)(sp - 1)) continue;
                __threadfence();
                if (lane == 0) *ticket = 0;
                slab = kp.slabs + ((int64_t)tile * sp * MT + half * C::HALF) * GT_N + row;
#pragma unroll
                for (int j = 0; j < C::HALF; j++) sum[j] = __ldcg(slab + j * GT_N);
                for (int p = 1; p < sp; p++) {
                    slab += MT * GT_N;
#pragma unroll
                    for (int j = 0; j < C::HALF; j++) sum[j] += __ldcg(slab + j * GT_N);
                }
            }
            const int64_t n = (int64_t)(tile / tiles_m) * GT_N + row;
            const int m0 = (tile % tiles_m) * MT + half * C::HALF;
            if (n < N) {
                float *dst = y + (int64_t)m0 * N + n;
#pragma unroll
                for (int j = 0; j < C::HALF; j++)
                    if (m0 + j < M) dst[j * N] = sum[j] * __ldcg(us + m0 + j);
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// asks for NC columns of this lane's TMEM row (8, 16, 32, or pieces of them)
template <int NC>
__device__ __forceinline__ void gt_ask(uint32_t taddr, uint32_t *t)
{
    if constexpr (NC >= 32) {
        tmem_ld32_async(taddr, *reinterpret_cast<uint32_t (*)[32]>(t));
        if constexpr (NC > 32) gt_ask<NC - 32>(taddr + 32, t + 32);
    } else if constexpr (NC >= 16) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
            : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7]), "=r"(t[8]), "=r"(t[9]), "=r"(t[10]),
              "=r"(t[11]), "=r"(t[12]), "=r"(t[13]), "=r"(t[14]), "=r"(t[15])
            : "r"(taddr)
            : "memory");
        if constexpr (NC > 16) gt_ask<NC - 16>(taddr + 16, t + 16);
    } else {
        static_assert(NC == 8, "pieces of 32, 16 and 8 columns");
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7])
                     : "r"(taddr)
                     : "memory");
    }
}
__device__ __forceinline__ void gt_load_4d(uint32_t dst, const CUtensorMap *tmap, uint32_t bar, int x, int y, int z, int w)
{
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(dst),
                 "l"(tmap), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(w)
                 : "memory");
}
// ---- more than 32 rows -------------------------------------------------------------------------------------------------------
template <int TYPE, int MT>
struct GwCfg {
    static constexpr int SEG = TYPE == PG_GGUF_Q4_0 ? 128 : 256;   // quant bytes per row and slice
    static constexpr int FILL = 16 * SEG + 256;
    static constexpr int RAW = 8 * FILL;                           // a slice (256 k) of 128 rows
    static constexpr int PLANE = MT * 128;                         // 64 k of a plane
    static constexpr int BK64 = MT == 64 ? 2 : 1;                  // 64-k blocks of the planes per stage
    static constexpr int PER_B = 2 * BK64;                         // blocks of W per stage
    static constexpr int B_STAGE = BK64 * 2 * PLANE;
    static constexpr int GB = MT == 64 ? 2 : 1;                    // blocks of W per group of accumulators
    static constexpr int SETS = GB;                                // groups go to SETS sets of 4 / SETS warps per TMEM quarter in turn
    static constexpr int PART = MT * SETS / 4;                     // rows of x per warp of the epilogue
    static constexpr int COMB = SETS == 1 ? 0 : 2 * PART * GT_N * 4;   // where the sets' sums meet
    static constexpr int ROOM = 232448 - 1024 - 512 - COMB;
    static constexpr int BST = TYPE == PG_GGUF_Q8_0 && MT == 64 ? 2 : 3;
    static constexpr int FIT = (ROOM - BST * B_STAGE) / RAW;
    static constexpr int RST = FIT > 8 ? 8 : FIT;
    static constexpr int NA = 2;                                   // f16 buffers: 64 columns of TMEM, 128 k of 128 rows of W
    static constexpr int A_COL = 512 - 64 * NA;
    static constexpr int NBUF = A_COL / (GB * MT);
    static constexpr int DW0 = 3, EW0 = 7;                         // first warps of the quants (four), of the epilogue (sixteen)
    static constexpr int THREADS = (EW0 + 16) * 32;
    static constexpr int BARS = 2 * (RST + BST + NA + NBUF) + 8;
    static constexpr size_t SMEM = (size_t)BST * B_STAGE + RST * RAW + COMB + 1024 + 512;
    static_assert(RST >= 2 && NBUF >= 2 && BARS * 8 + 8 <= 512, "shared memory or TMEM too small");
};

template <int TYPE, int MT>
__global__ void __launch_bounds__(GwCfg<TYPE, MT>::THREADS, 1)
    gguf_tc_wide_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, int64_t N, int nslices, int M,
                   const float *__restrict__ us, float *__restrict__ y, const GtParts kp, int32_t *status, unsigned long long limit_ns)
{
    using C = GwCfg<TYPE, MT>;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = pg_smem(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    const uint32_t b_at = base, r_at = b_at + C::BST * C::B_STAGE, c_at = r_at + C::RST * C::RAW;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_raw + (c_at - raw_addr) + C::COMB);
    const uint32_t bar = pg_smem(bars);
    // full and empty of: slices, blocks of the planes, f16 buffers, groups of accumulators; then the meeting of sums, by quarter
    const uint32_t r_full = bar, r_empty = r_full + 8 * C::RST, b_full = r_empty + 8 * C::RST, b_empty = b_full + 8 * C::BST;
    const uint32_t a_full = b_empty + 8 * C::BST, a_empty = a_full + 8 * C::NA, t_full = a_empty + 8 * C::NA, t_empty = t_full + 8 * C::NBUF;
    const uint32_t c_full = t_empty + 8 * C::NBUF, c_free = c_full + 32;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + C::BARS);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < C::RST; i++) {
            pg_mbar_init(r_full + 8 * i, 1);
            pg_mbar_init(r_empty + 8 * i, 16 + 4);   // the scales, the quants
        }
        for (int i = 0; i < C::BST; i++) {
            pg_mbar_init(b_full + 8 * i, 1);
            pg_mbar_init(b_empty + 8 * i, 1);
        }
        for (int i = 0; i < C::NA; i++) {
            pg_mbar_init(a_full + 8 * i, 4);
            pg_mbar_init(a_empty + 8 * i, 1);
        }
        for (int i = 0; i < C::NBUF; i++) {
            pg_mbar_init(t_full + 8 * i, 1);
            pg_mbar_init(t_empty + 8 * i, 16 / C::SETS);
        }
        for (int i = 0; i < 4; i++) {
            pg_mbar_init(c_full + 8 * i, 2);
            pg_mbar_init(c_free + 8 * i, 2);
        }
        *abort_flag = 0;
        pg_mbar_fence();
    }
    __syncwarp();
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(pg_smem(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int tiles_m = (M + MT - 1) / MT, tiles_n = (int)((N + GT_N - 1) / GT_N);
    const int sp = kp.parts, total = tiles_m * tiles_n * sp;   // unit u: part u % sp of tile u / sp; the tiles of a row of W follow each other
    auto s_first = [&](int u) { return (u % sp) * kp.slices; };
    auto s_end = [&](int u) { return min(nslices, (u % sp + 1) * kp.slices); };
    auto wait = [&](uint32_t b, uint32_t parity) { return pg_mbar_wait_warp(b, parity & 1, abort_flag, status, limit_ns); };
    bool ok = true;

    if (warp == 0) {
        // ---------------------------------------------------------------- planes of x: a copy per stage
        if (lane == 0) {
            uint32_t bs = 0, bp = 1;
            asm volatile("griddepcontrol.wait;" ::: "memory");
            for (int u = blockIdx.x; ok && u < total; u += gridDim.x) {
                const int m0 = (u / sp % tiles_m) * MT;
                for (int kb = 4 * s_first(u), end = 4 * s_end(u); kb < end; kb += C::BK64) {
                    if (!(ok = pg_mbar_wait(b_empty + 8 * bs, bp, abort_flag, status, limit_ns))) break;
                    pg_mbar_expect(b_full + 8 * bs, C::B_STAGE);
                    gt_load_4d(b_at + bs * C::B_STAGE, &tmap_x, b_full + 8 * bs, 0, m0, 0, kb);
                    if (++bs == C::BST) {
                        bs = 0;
                        bp ^= 1;
                    }
                }
            }
            if (!ok) gt_settle();
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- slices of W, which no kernel writes: no wait for the preceding one
        if (lane == 0) {
            uint32_t rs = 0, rp = 1;
            for (int u = blockIdx.x; ok && u < total; u += gridDim.x) {
                const int f0 = u / sp / tiles_m * (GT_N / 16);      // (fills behind the last one are zeros)
                for (int s = s_first(u), end = s_end(u); s < end; s++) {
                    if (!(ok = pg_mbar_wait(r_empty + 8 * rs, rp, abort_flag, status, limit_ns))) break;
                    pg_mbar_expect(r_full + 8 * rs, C::RAW);
                    gt_load_4d(r_at + rs * C::RAW, &tmap_w, r_full + 8 * rs, 0, 0, s, f0);
                    if (++rs == C::RST) {
                        rs = 0;
                        rp ^= 1;
                    }
                }
            }
            if (!ok) gt_settle();
        }
    } else if (warp == 2) {
        // ---------------------------------------------------------------- products (the whole warp; one lane's count)
        const uint32_t on = pg_elect();
        constexpr uint32_t idesc = gt_idesc(GT_N, MT);
        const uint64_t desc_b = make_smem_desc(b_at);
        uint32_t bs = 0, bp = 0, as = 0, ap = 0, ts = 0, tp = 0;
        for (int u = blockIdx.x; ok && u < total; u += gridDim.x)
            for (int h = 2 * s_first(u), end = 2 * s_end(u); ok && h < end; h++) {
                if (!(ok = wait(a_full + 8 * as, ap))) break;
#pragma unroll
                for (int blk = 0; blk < 4; blk++) {             // blocks of the 128 k
                    if (blk % C::PER_B == 0 && !(ok = wait(b_full + 8 * bs, bp))) break;
                    if (blk % C::GB == 0) {
                        if (!(ok = wait(t_empty + 8 * ts, tp ^ 1))) break;
                        tc_fence_after();
                    }
                    const uint32_t d = tmem + (ts * C::GB + blk % C::GB) * MT;
                    const uint32_t a = tmem + C::A_COL + as * 64 + blk * 16;
                    const uint64_t db = desc_b + (uint64_t)(bs * (C::B_STAGE >> 4) + (blk % C::PER_B >> 1) * (2 * C::PLANE >> 4) + (blk & 1) * 4);
#pragma unroll
                    for (int l = 1; l >= 0; l--)
#pragma unroll
                        for (int j = 0; j < 2; j++)
                            umma_f16_ta(d, a + j * 8, db + (uint64_t)(l * (C::PLANE >> 4) + j * 2), idesc, l != 1 || j != 0 ? 1u : 0u, on);
                    if ((blk + 1) % C::GB == 0) {
                        umma_commit(t_full + 8 * ts, on);
                        if (++ts == C::NBUF) {
                            ts = 0;
                            tp ^= 1;
                        }
                    }
                    if ((blk + 1) % C::PER_B == 0) {
                        umma_commit(b_empty + 8 * bs, on);
                        if (++bs == C::BST) {
                            bs = 0;
                            bp ^= 1;
                        }
                    }
                }
                if (!ok) break;
                umma_commit(a_empty + 8 * as, on);
                as ^= 1;
                if (as == 0) ap ^= 1;
            }
    } else if (warp < C::EW0) {
        // ---------------------------------------------------------------- quants -> f16 in TMEM: lane = row of W.  A chunk of 128 k is announced
        // when the next one's quants have been read: its stores take some 200 cycles to arrive.
        const int q = warp & 3, row = q * 32 + lane, sw = ((row & 1) << 2) | ((row >> 1) & 3);
        const uint32_t src0 = r_at + (uint32_t)(row >> 4) * C::FILL + (uint32_t)(row & 15) * C::SEG;
        const uint32_t dst0 = tmem + ((uint32_t)(q * 32) << 16) + C::A_COL;
        uint32_t rs = 0, rp = 0, as = 0, ap = 1;
        bool stored = false;                                    // a chunk in the other buffer waits to be announced
        auto announce = [&] {
            tmem_wait_st();
            tc_fence_before();
            pg_mbar_arrive_warp(a_full + 8 * (as ^ 1), lane);
        };
        for (int u = blockIdx.x; ok && u < total; u += gridDim.x)
            for (int s = s_first(u), end = s_end(u); ok && s < end; s++) {
                ok = wait(r_full + 8 * rs, rp);
                for (int h = 0; ok && h < 2; h++) {
                    const uint32_t src = src0 + rs * C::RAW;
                    uint4 w[4];                                 // Q4_0: word t of four blocks; Q8_0: bytes 8 t .. of two
                    auto read = [&](int g) {
#pragma unroll
                        for (int t = 0; t < 4; t++) w[t] = pg_lds128(src + (uint32_t)(((g * 4 + t) ^ sw) * 16));
                    };
                    read(TYPE == PG_GGUF_Q4_0 ? h : 2 * h);
                    if (stored) announce();
                    if (!(ok = wait(a_empty + 8 * as, ap))) break;
                    tc_fence_after();
#pragma unroll
                    for (int p = 0; p < 2; p++) {               // blocks 2 p and 2 p + 1
                        if (TYPE != PG_GGUF_Q4_0 && p == 1) read(2 * h + 1);
                        uint32_t v[32];
#pragma unroll
                        for (int t = 0; t < 4; t++)
#pragma unroll
                            for (int b = 0; b < 2; b++) {
                                uint32_t f[4];
                                if constexpr (TYPE == PG_GGUF_Q4_0)
                                    gguf_nibbles_f16(p ? (b ? w[t].w : w[t].z) : (b ? w[t].y : w[t].x), f);
                                else
                                    gguf_bytes_f16(b ? w[t].z : w[t].x, b ? w[t].w : w[t].y, f);
#pragma unroll
                                for (int e = 0; e < 4; e++) v[16 * b + 4 * t + e] = f[e];
                            }
                        tmem_st32(dst0 + as * 64 + p * 32, v);
                    }
                    stored = true;
                    if (h == 1) pg_mbar_arrive_warp(r_empty + 8 * rs, lane);
                    as ^= 1;
                    if (as == 0) ap ^= 1;
                }
                if (++rs == C::RST) {
                    rs = 0;
                    rp ^= 1;
                }
            }
        if (ok && stored) announce();
    } else {
        // ---------------------------------------------------------------- sums and outputs: lane = row of W.  With 64 rows of x, two of a quarter's
        // four warps take a group of accumulators, half of the rows each, the other two the next one; above, all four take every group
        const int q = warp & 3, e = (warp - C::EW0) >> 2, row = q * 32 + lane;
        const int part = C::SETS == 2 ? e & 1 : e, set = C::SETS == 2 ? e >> 1 : 0;
        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + part * C::PART;
        const uint32_t scales = r_at + (uint32_t)(row >> 4) * C::FILL + 16 * C::SEG + (uint32_t)(row & 15) * 16;
        const uint32_t meet = c_at + (uint32_t)(part * C::PART * GT_N + row) * 4;
        asm volatile("griddepcontrol.wait;" ::: "memory");     // y may still be read by the predecessor
        uint32_t rs = 0, ts = set, tp = 0, cp = 0;
        for (int u = blockIdx.x; ok && u < total; u += gridDim.x) {
            const int tile = u / sp;
            float sum[C::PART];
#pragma unroll
            for (int j = 0; j < C::PART; j++) sum[j] = 0.0f;
            for (int s = s_first(u), end = s_end(u); ok && s < end; s++) {
#pragma unroll
                for (int g = 0; g < 8 / C::GB; g++) {
                    if (C::SETS == 2 && (g & 1) != set) continue;
                    if (!(ok = wait(t_full + 8 * ts, tp))) break;
                    tc_fence_after();
                    // (the slice's scales are there too: the products' quants came with them)
                    const uint32_t sc = scales + rs * C::RAW + g * C::GB * 2;
                    float d[C::GB];
#pragma unroll
                    for (int b = 0; b < C::GB; b++) {
                        uint16_t bits;
                        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(bits) : "r"(sc + b * 2));
                        d[b] = __half2float(__ushort_as_half(bits));
                    }
                    constexpr int P = C::PART <= 32 ? C::PART : 16;   // columns at a time
#pragma unroll
                    for (int b = 0; b < C::GB; b++)
#pragma unroll
                        for (int c = 0; c < C::PART; c += P) {
                            constexpr int LAST = C::PART % P ? C::PART % P : P;
                            const bool last = c + P >= C::PART;
                            uint32_t v[P];
                            if (last)
                                gt_ask<LAST>(taddr + (ts * C::GB + b) * MT + c, v);
                            else
                                gt_ask<P>(taddr + (ts * C::GB + b) * MT + c, v);
                            tmem_wait_ld();
                            if (last && b == C::GB - 1) {
                                tc_fence_before();
                                pg_mbar_arrive_warp(t_empty + 8 * ts, lane);
                                if (g >= 8 / C::GB - C::SETS) pg_mbar_arrive_warp(r_empty + 8 * rs, lane);   // (this warp's last group of the slice)
                            }
#pragma unroll
                            for (int j = 0; j < P; j++)
                                if (!last || j < LAST) sum[c + j] = fmaf(d[b], __uint_as_float(v[j]), sum[c + j]);
                        }
                    ts += C::SETS;
                    if (ts >= C::NBUF) {
                        ts -= C::NBUF;
                        tp ^= 1;
                    }
                }
                if (++rs == C::RST) rs = 0;
            }
            if (!ok) break;
            if constexpr (C::SETS == 2) {
                // the sets' sums meet in the first one
                if (set == 1) {
                    if (!(ok = wait(c_free + 8 * q, cp + 1))) break;
#pragma unroll
                    for (int j = 0; j < C::PART; j++) asm volatile("st.shared.f32 [%0], %1;" ::"r"(meet + j * GT_N * 4), "f"(sum[j]) : "memory");
                    pg_mbar_arrive_warp(c_full + 8 * q, lane);
                    cp ^= 1;
                    continue;
                }
                if (!(ok = wait(c_full + 8 * q, cp))) break;
#pragma unroll
                for (int j = 0; j < C::PART; j++) {
                    float f;
                    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(f) : "r"(meet + j * GT_N * 4));
                    sum[j] += f;
                }
                pg_mbar_arrive_warp(c_free + 8 * q, lane);
                cp ^= 1;
            }
            if (sp > 1) {
                float *slab = kp.slabs + ((int64_t)u * MT + part * C::PART) * GT_N + row;
#pragma unroll
                for (int j = 0; j < C::PART; j++) __stcg(slab + j * GT_N, sum[j]);
                unsigned int *ticket = kp.tickets + tile * 16 + part * 4 + q;
                __threadfence();
                __syncwarp();
                const unsigned int before = __shfl_sync(0xffffffffu, lane == 0 ? atomicAdd(ticket, 1u) : 0u, 0);
                if (before != (unsigned)(sp - 1)) continue;
                __threadfence();
                if (lane == 0) *ticket = 0;
                slab = kp.slabs + ((int64_t)tile * sp * MT + part * C::PART) * GT_N + row;
#pragma unroll
                for (int j = 0; j < C::PART; j++) sum[j] = __ldcg(slab + j * GT_N);
                for (int p = 1; p < sp; p++) {
                    slab += MT * GT_N;
#pragma unroll
                    for (int j = 0; j < C::PART; j++) sum[j] += __ldcg(slab + j * GT_N);
                }
            }
            const int64_t n = (int64_t)(tile / tiles_m) * GT_N + row;
            const int m0 = (tile % tiles_m) * MT + part * C::PART;
            if (n < N) {
                float *dst = y + (int64_t)m0 * N + n;
#pragma unroll
                for (int j = 0; j < C::PART; j++)
                    if (m0 + j < M) dst[j * N] = sum[j] * __ldcg(us + m0 + j);
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// ---------------------------------------------------------------- host side ----
int64_t gt_row_bytes(int64_t k) { return 4 * k + 4; }    // two planes and 2^-s

template <int TYPE, int MT>
int32_t gt_launch(pg_ctx *ctx, const pg_gguf_weight *w, const void *planes, const float *us, int64_t m, float *y, GtParts kp)
{
    using C = GtCfg<TYPE, MT>;
    CUtensorMap tx;
    const cuuint64_t dims[3] = {(cuuint64_t)w->k, (cuuint64_t)m, 2}, strides[2] = {(cuuint64_t)w->k * 2, (cuuint64_t)(w->k * m) * 2};
    const cuuint32_t box[3] = {64, MT, 2};
    const int32_t rc = pg_encode_bf16(&tx, planes, 3, dims, strides, box);   // (f16: the copies only move it)
    if (rc != PG_OK) return rc;
    auto kern = gguf_tc_kernel<TYPE, MT>;
    static std::atomic<uint64_t> smem_set{0};
    PG_CUDA(pg_max_smem_once(kern, (int)C::SMEM, ctx->device, smem_set));
    const int64_t units = ((m + MT - 1) / MT) * ((w->n + GT_N - 1) / GT_N) * kp.parts;
    kp.tickets = reinterpret_cast<unsigned int *>(ctx->splitk);
    kp.slabs = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(ctx->splitk) + GT_TICKET_BYTES);
    return launch_pdl(ctx, kern, dim3((unsigned)std::min<int64_t>(units, ctx->sm_count)), dim3(C::THREADS), C::SMEM, tx, (const uint8_t *)w->d_qs, w->n,
                      (int)(w->k / 256), (int)m, us, y, kp, ctx->d_status, ctx->wait_limit_ns);
}

template <int TYPE, int MT>
int32_t gw_launch(pg_ctx *ctx, const pg_gguf_weight *w, const void *planes, const float *us, int64_t m, float *y, GtParts kp)
{
    using C = GwCfg<TYPE, MT>;
    CUtensorMap tx, tw;
    // x: 64 k of the rows of both planes, a stage's blocks of 64 k behind each other
    const cuuint64_t xd[4] = {64, (cuuint64_t)m, 2, (cuuint64_t)w->k / 64}, xs[3] = {(cuuint64_t)w->k * 2, (cuuint64_t)(w->k * m) * 2, 128};
    const cuuint32_t xb[4] = {64, MT, 2, C::BK64};
    int32_t rc = pg_encode_bf16(&tx, planes, 4, xd, xs, xb);   // (f16: the copies only move it)
    // W: the fills of a slice of eight tiles of 16 rows
    const cuuint64_t nslices = (cuuint64_t)w->k / 256, tiles = (cuuint64_t)(w->n + 15) / 16;
    const cuuint64_t wd[4] = {64, C::FILL / 256, nslices, tiles}, ws[3] = {256, C::FILL, nslices * C::FILL};
    const cuuint32_t wb[4] = {64, C::FILL / 256, 1, 8};
    if (rc == PG_OK) rc = pg_encode_map(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT32, w->d_qs, 4, wd, ws, wb, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (rc != PG_OK) return rc;
    auto kern = gguf_tc_wide_kernel<TYPE, MT>;
    static std::atomic<uint64_t> smem_set{0};
    PG_CUDA(pg_max_smem_once(kern, (int)C::SMEM, ctx->device, smem_set));
    const int64_t units = ((m + MT - 1) / MT) * ((w->n + GT_N - 1) / GT_N) * kp.parts;
    kp.tickets = reinterpret_cast<unsigned int *>(ctx->splitk);
    kp.slabs = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(ctx->splitk) + GT_TICKET_BYTES);
    return launch_pdl(ctx, kern, dim3((unsigned)std::min<int64_t>(units, ctx->sm_count)), dim3(C::THREADS), C::SMEM, tx, tw, w->n, (int)nslices, (int)m, us,
                      y, kp, ctx->d_status, ctx->wait_limit_ns);
}

// rows of slabs that a context keeps for every product
int64_t gt_slab_rows(const pg_ctx *ctx) { return (int64_t)ctx->sm_count * 3 * 64; }

// Rows per tile and parts of K, by the shape alone (a portion of a call has those of the whole call): the fewest cycles by count --
// slices of the busiest CTA and what a tile costs at its end, more where slabs meet.  Measured, N 14336, K 4096: a block of 32 k takes 350 / 430
// cycles with 16 / 32 rows, 440 / 575 / 685 with 64 / 128 / 160; N 4096, K 4096, four parts of K: what the parts cost is 10000 / 14000 / 20000 cycles
// with 64 / 128 / 160 rows.
GtParts gt_plan(const pg_ctx *ctx, const pg_gguf_weight *w, int64_t m, int *mt)
{
    const int64_t nslices = w->k / 256, tiles_n = (w->n + GT_N - 1) / GT_N;
    static const int sizes[] = {16, 32, 64, 128, 160};
    double best = 0;
    *mt = 16;
    GtParts kp = {1, (int)nslices, nullptr, nullptr};
    for (int cand : sizes) {
        if (cand < 64 && cand < m) continue;
        if (cand > 16 && cand / 2 >= m) break;
        const int64_t tiles = tiles_n * ((m + cand - 1) / cand);
        for (int64_t parts = 1; parts <= std::min<int64_t>(16, nslices); parts++) {
            const int64_t slices = (nslices + parts - 1) / parts;
            if ((nslices + slices - 1) / slices != parts) continue;
            if (parts > 1 && (tiles * parts * cand > gt_slab_rows(ctx) || tiles * 16 * (int64_t)sizeof(int) > (int64_t)GT_TICKET_BYTES)) break;
            const int64_t rounds = (tiles * parts + ctx->sm_count - 1) / ctx->sm_count;
            const double block = cand < 64 ? 280.0 + cand * 4.0 : 300.0 + cand * 2.3;
            const double meet = parts == 1 ? 0.0 : cand < 64 ? 2500.0 + cand * parts * 4.0 : 4000.0 + cand * parts * 25.0;
            const double cost = rounds * (slices * 8.0 * block + 1500.0 + cand * 8.0 + meet);
            if (best == 0 || cost < best) {
                best = cost;
                *mt = cand;
                kp.parts = (int)parts;
                kp.slices = (int)slices;
            }
        }
    }
    return kp;
}

template <int TYPE>
int32_t gt_run(pg_ctx *ctx, const pg_gguf_weight *w, const void *planes, const float *us, int64_t m, float *y, int mt, const GtParts &kp)
{
    if (mt == 160) return gw_launch<TYPE, 160>(ctx, w, planes, us, m, y, kp);
    if (mt == 128) return gw_launch<TYPE, 128>(ctx, w, planes, us, m, y, kp);
    if (mt == 64) return gw_launch<TYPE, 64>(ctx, w, planes, us, m, y, kp);
    if (mt == 32) return gt_launch<TYPE, 32>(ctx, w, planes, us, m, y, kp);
    return gt_launch<TYPE, 16>(ctx, w, planes, us, m, y, kp);
}

}  // namespace

// From nine rows on.  For fewer only what csrc/pg_gguf_few.cu leaves -- one and two rows of large layers, K beyond 65536, parts of K without a
// workspace (a recording) -- and of that what the streaming form walks in four chunks of K and more (it has room for 16384 elements of x in
// all), or three on narrow layers.  Q4_0, us, streaming / this: K 14336, N 4096 at 3 / 5 / 8 rows 28.1 / 41.0 / 48.8 against 24.2 / 24.7 / 25.5; K 6144,
// N 4096 at 5 rows 17.3 / 15.1; K 8192, N 8192 at 5 / 8 rows 28.3 / 32.9 against 25.6 / 26.6, N 28672 62.0 / 66.3 against 81.5 / 82.6.  (One and two rows
// of K 32768 and 65536, N 4096, are slower here: two rows 39.3 / 79.2 against 48.1 / 87.1; their error is a quarter where channels stand out.)
bool pgk_matmul_gguf_tc_supports(const pg_ctx *ctx, const pg_gguf_weight *w, int64_t m)
{
    if (!(w->tiled && m >= 1 && m < (1 << 24) && w->n >= 1 && w->n < (1ll << 30))) return false;
    if (m > 8) return true;
    const int64_t rows = m > 4 ? 8 : m > 2 ? 4 : m, chunks = (w->k * rows + 16383) / 16384;
    const bool narrow = w->n <= 32ll * ctx->sm_count;
    return chunks >= 4 || (narrow && chunks == 3);
}

int32_t pgk_gguf_tc_reserve(pg_ctx *ctx, int64_t k)
{
    const int32_t rc = pg_scratch_reserve(ctx, (size_t)(GT_ROWS * gt_row_bytes(k)));
    if (rc != PG_OK) return rc;
    return pg_splitk_reserve(ctx, GT_TICKET_BYTES + (size_t)(gt_slab_rows(ctx) * GT_N) * sizeof(float));
}

int32_t pgk_matmul_gguf_tc(pg_ctx *ctx, const float *d_x, int64_t m, const pg_gguf_weight *w, float *d_y)
{
    // Rows in portions whose planes stay below GT_PLANES; while a graph is recorded the workspace cannot grow, and what there is (an
    // upload reserves some in its context) takes them.  Where there is none to be had, the streaming form does without.
    int mt;
    const GtParts kp = gt_plan(ctx, w, m, &mt);
    const int64_t row_bytes = gt_row_bytes(w->k);
    int64_t portion = std::min(m, std::max<int64_t>(GT_ROWS, GT_PLANES / row_bytes / mt * mt));
    if (ctx->capturing) {
        const int64_t fit = (int64_t)(ctx->scratch_bytes / (size_t)row_bytes), step = fit >= mt ? mt : 16;
        if (fit < portion) portion = fit / step * step;
        if (portion == 0 || (kp.parts > 1 && ctx->splitk_bytes < GT_TICKET_BYTES + (size_t)(gt_slab_rows(ctx) * GT_N) * sizeof(float)))
            return pgk_matmul_gguf_stream(ctx, d_x, m, w, d_y);
    } else if (pg_scratch_reserve(ctx, (size_t)(portion * row_bytes)) != PG_OK || pgk_gguf_tc_reserve(ctx, w->k) != PG_OK) {
        return pgk_matmul_gguf_stream(ctx, d_x, m, w, d_y);
    }
    for (int64_t r0 = 0; r0 < m; r0 += portion) {
        const int64_t rows = std::min(portion, m - r0);
        uint4 *planes = reinterpret_cast<uint4 *>(ctx->scratch);
        float *us = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(ctx->scratch) + rows * w->k * 4);
        // (few rows: several CTAs each, which all look for the largest element)
        const dim3 grid((unsigned)rows, (unsigned)std::max<int64_t>(1, std::min<int64_t>(w->k / 2048, 2 * ctx->sm_count / rows)));
        int32_t rc = w->type == PG_GGUF_Q4_0
                         ? launch_pdl(ctx, gguf_planes_kernel<true>, grid, dim3(256), 0, d_x, (int)r0, (int)rows, (int)w->k, planes, us)
                         : launch_pdl(ctx, gguf_planes_kernel<false>, grid, dim3(256), 0, d_x, (int)r0, (int)rows, (int)w->k, planes, us);
        if (rc != PG_OK) return rc;
        rc = w->type == PG_GGUF_Q4_0 ? gt_run<PG_GGUF_Q4_0>(ctx, w, planes, us, rows, d_y + r0 * w->n, mt, kp)
                                     : gt_run<PG_GGUF_Q8_0>(ctx, w, planes, us, rows, d_y + r0 * w->n, mt, kp);
        if (rc != PG_OK) return rc;
    }
    return PG_OK;
}
