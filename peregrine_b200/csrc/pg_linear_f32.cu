// y = a W^T in f32 accuracy on the 5th-generation tensor cores: bf16 weights as they are, f32 activations as three bf16 pieces.
//
//   * a = a1 + a2 + a3 with each piece the next eight significant bits (cut off, not rounded, and none zero): exact, and so is every product
//     with a bf16 weight.  `linear_split_kernel` writes the pieces as three planes (routed rows in the order of the route).
//   * D[n][m] = W (128 rows) x A^T (MT rows of a, all three planes): weights are the M side of the instruction, so that a lane of
//     the epilogue owns a column of y and 32 lanes store 128 contiguous bytes of a row.
//   * the sums: tcgen05's f32 accumulator cuts off what falls below its last bit, always towards zero, and a chain over a whole K
//     would add that up.  An accumulator therefore only lives for one block of 64 k (smallest pieces first); four warps, eight from
//     64 rows on, add the blocks in registers, rounded, while the next block's products run in the other accumulator.  A warp's chain per block
//     -- barrier, some 100 cycles for every 32 columns of TMEM, back to the products -- is what four warps could not hide at 128 rows (1413
//     cycles a block).  Two warps issue the products, a block each in turn, so that one's waits and commits lie beside the other's products.
//   * K has parts, whose number follows from the matrix alone (f32_parts): each part is summed up by itself, and the parts are added in
//     their order.  With few tiles they are spread over CTAs and meet in slabs, with tickets, as in linear_tc_kernel; else a CTA goes
//     through them one after the other and keeps the sum so far in TMEM.  So a row's outputs are the same whatever rows are beside it,
//     however a call is divided, and whatever workspace there is.
//
// From 64 rows on a pair of CTAs shares a tile's rows of a: each brings half of the planes and 128 rows of W of its own, which four more warps
// put into TMEM, where the products of all three planes take them from.  With W in shared memory one CTA's block of 64 k brought 64 KB and its
// products read 96 KB: 1250 cycles at 128 bytes each for 768 of products, 1318 measured; now 40 KB come in and some 64 KB are read.
//
// What bounds it: from about 64 rows the products and what is left of the ways through shared memory (1170 cycles a block); the stream of W
// below.  us, N 28672, K 4096, 33 / 64 / 128 / 333 / 777 rows: 84 / 88 / 107 / 238 / 520 with one CTA and four warps of sums, 60 / 61 / 82 / 204 / 442 now; N 4096,
// K 14336: 41 / 42 / 58 / 145 / 285 -> 36 / 37 / 53 / 128 / 250.
// Every mbarrier wait is bounded (pg_async.cuh).
#include <algorithm>

#include "pg_async.cuh"
#include "pg_lm.cuh"
#include "pg_tcgen05.cuh"

namespace {

constexpr int FN = 128;                // columns of y (rows of W) per tile
constexpr int FK = 64;                 // elements of K per stage = one 128-byte swizzle span
constexpr int F_ROWS = 128;            // rows for which a call finds room also while a graph is recorded
constexpr int64_t F_PLANES = 100 << 20, F_SLABS = 64 << 20;   // most bytes of planes (they stay in L2; longer calls go in portions), of slabs

template <int MT>
struct FCfg {
    static constexpr int STAGE_W = FN * FK * 2;
    static constexpr int CG = MT >= 64 ? 2 : 1;            // CTAs that share a tile's rows of a, each with 128 columns of y of its own
    static constexpr int PLANE = MT / CG * FK * 2;         // a CTA's part of a plane
    static constexpr int STAGE = STAGE_W + 3 * PLANE;
    static constexpr int ROOM = 232448 - (1024 + 512);
    static constexpr int STAGES = ROOM / STAGE > 10 ? 10 : ROOM / STAGE;
    static constexpr int ACC = MT < 32 ? 32 : MT;          // TMEM columns of an accumulator
    static constexpr int COLS = 4 * ACC;                   // two accumulators, the sum so far, and up to a power of two
    static constexpr int MW = 2;                           // warps that issue products, a block of K in turn
    static constexpr int EW = MT >= 64 ? 2 : 1;            // warps of the epilogue per TMEM quarter
    static constexpr int PART = MT / EW;                   // rows of a per such warp
    // From 64 rows on the weights go from shared memory to TMEM (32 columns a block, two such buffers), and the products take them from there:
    // three products read each piece of W, which is more than shared memory gives.
    static constexpr bool TA = CG == 2;
    static constexpr int A_COL = 3 * ACC;
    static constexpr int EW0 = TA ? 8 : 4;                 // first warp of the epilogue; copies, products, a warp without work, W to TMEM
    static constexpr int THREADS = (EW0 + 4 * EW) * 32;
    static constexpr size_t SMEM = (size_t)STAGES * STAGE + 1024 + 512;
};

struct FParts {
    int parts, blocks;       // K in `parts` parts of `blocks` 64-element blocks
    int runs, run;           // a unit takes `run` parts that follow each other; `runs` units make a tile
    float *slabs;            // [tile][part][MT][128]
    unsigned int *tickets;   // one per (tile, warp of the epilogue), zero between calls
};

// ---- the three planes of rows row0 .. of a: planes [3][rows][K] --------------------------------------------------------
// rt.row_pair: row r takes token row_pair[r] / top (by token), or row r.  Rows without a pair, and those behind the route's blocks, are left
// out: nobody reads what comes of them, and rows do not touch each other.  (157 tokens, eight of 64 experts each, 1256 pairs in some 8000 rows:
// K 2048 by token 41 -> 31 us, K 1024 by row 23 -> 17, a prompt of four layers 2266 -> 2211.)
__global__ void __launch_bounds__(256)
    linear_split_kernel(const float *__restrict__ a, int64_t lda, int row0, int rows, int K, const PgRouted rt, uint2 *__restrict__ planes)
{
    pg_pdl_begin();
    const int quads = K / 4;
    const int limit = rt.blocks ? min(rows, __ldcg(rt.blocks) * PG_ROUTE_BLOCK - row0) : rows;
    const int64_t plane = (int64_t)rows * quads;
    for (int r = blockIdx.y; r < limit; r += gridDim.y) {
        int64_t src = row0 + r;
        if (rt.blocks) {
            const int pair = __ldcg(rt.row_pair + row0 + r);
            if (pair < 0) continue;
            if (rt.by_token) src = pair / rt.top;
        }
        for (int c = blockIdx.x * 256 + threadIdx.x; c < quads; c += gridDim.x * 256) {
            const float4 v = __ldcg(reinterpret_cast<const float4 *>(a + src * lda) + c);
            const float x[4] = {v.x, v.y, v.z, v.w};
            uint32_t p[3][4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t bits = __float_as_uint(x[i]);
                const bool finite = (bits & 0x7f800000u) != 0x7f800000u;
                p[0][i] = finite || (bits & 0x007fffffu) == 0 ? bits & 0xffff0000u : bits | 0x00400000u;   // (a NaN stays one)
                // no piece of a number is zero, since an infinite weight times one would be NaN: one with nothing left gives up its last bit
                if (finite && x[i] == __uint_as_float(p[0][i]) && x[i] != 0.0f) p[0][i] -= 0x10000u;
                const float r1 = finite ? x[i] - __uint_as_float(p[0][i]) : 0.0f;
                p[1][i] = __float_as_uint(r1) & 0xffff0000u;
                if (r1 == __uint_as_float(p[1][i]) && r1 != 0.0f) p[1][i] -= 0x10000u;
                p[2][i] = __float_as_uint(r1 - __uint_as_float(p[1][i]));
            }
#pragma unroll
            for (int l = 0; l < 3; l++)
                planes[l * plane + (int64_t)r * quads + c] = make_uint2(__byte_perm(p[l][0], p[l][1], 0x7632), __byte_perm(p[l][2], p[l][3], 0x7632));
        }
    }
}

// 32 columns of this lane's TMEM row
__device__ __forceinline__ void f32_keep(uint32_t taddr, const uint32_t (&v)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, "
        "%22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]),
        "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]),
        "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

template <int MT, int ACT>
__global__ void __launch_bounds__(FCfg<MT>::THREADS, 1)
    linear_f32_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a, int M, int N, int K, float limit,
                      float *__restrict__ y, int64_t ldy, const PgRouted rt, int block0, const FParts kp, int32_t *status, unsigned long long limit_ns)
{
    using C = FCfg<MT>;
    constexpr int STAGES = C::STAGES, CG = C::CG;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = pg_smem(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_raw + (base - raw_addr) + (size_t)STAGES * C::STAGE);
    const uint32_t bar_full = pg_smem(bars);
    const uint32_t bar_empty = bar_full + 8 * STAGES;
    const uint32_t bar_tfull = bar_empty + 8 * STAGES;
    const uint32_t bar_tempty = bar_tfull + 16;
    const uint32_t bar_a = bar_tempty + 16, bar_afree = bar_a + 16, bar_w = bar_afree + 16;   // TMEM's buffers of W; this CTA's own tiles of W
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 3 * STAGES + 8);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = CG == 2 ? (int)pg_cluster_rank() : 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            pg_mbar_init(bar_full + 8 * s, 1);
            pg_mbar_init(bar_empty + 8 * s, 1);
            pg_mbar_init(bar_w + 8 * s, 1);
        }
        for (int i = 0; i < 2; i++) {
            pg_mbar_init(bar_tfull + 8 * i, 1);
            pg_mbar_init(bar_tempty + 8 * i, 4 * C::EW * CG);   // one arrival per epilogue warp
            pg_mbar_init(bar_a + 8 * i, 4 * CG);
            pg_mbar_init(bar_afree + 8 * i, 1);
        }
        *abort_flag = 0;
        pg_mbar_fence();
    }
    __syncwarp();
    if (warp == 1) tmem_alloc<CG>(pg_smem(tmem_slot), C::COLS);
    tc_fence_before();
    pg_group_sync<CG>();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const bool routed = rt.blocks != nullptr;
    if (routed) asm volatile("griddepcontrol.wait;" ::: "memory");   // the list of tiles comes from the preceding kernels
    constexpr int PER_BLOCK = PG_ROUTE_BLOCK / MT < 1 ? 1 : PG_ROUTE_BLOCK / MT;
    const int tiles_m = routed ? max(0, min(__ldcg(rt.blocks) - block0, M / PG_ROUTE_BLOCK)) * PER_BLOCK : (M + MT - 1) / MT;
    const int tiles_n = (N + CG * FN - 1) / (CG * FN), unit0 = blockIdx.x / CG, units = gridDim.x / CG;
    const int sp = kp.runs, total = tiles_m * tiles_n * sp;    // unit u: run u % sp of tile u / sp
    const int kblocks = K / FK, per = kp.run * kp.blocks;
    auto k_first = [&](int u) { return (u % sp) * per; };
    auto k_end = [&](int u) { return min(kblocks, (u % sp + 1) * per); };

    if (warp == 0) {
        // ---------------------------------------------------------------- producer
        if (lane == 0) {
            uint32_t stage = 0, phase = 0;
            bool ok = true;
            const uint32_t full_l = pg_leader<CG>(bar_full);
            // a tile of W, and what the stage's barrier counts: where W goes on to TMEM, W has a barrier of its own in each CTA
            auto ask_w = [&](int stage, int kb, int row) {
                if (C::TA) {
                    pg_mbar_expect(bar_w + 8 * stage, C::STAGE_W);
                    tma_load_2d(base + stage * C::STAGE, &tmap_w, bar_w + 8 * stage, kb * FK, row);
                    if (rank == 0) pg_mbar_expect(bar_full + 8 * stage, CG * 3 * C::PLANE);
                } else {
                    pg_mbar_expect(bar_full + 8 * stage, C::STAGE);
                    tma_load_2d(base + stage * C::STAGE, &tmap_w, bar_full + 8 * stage, kb * FK, row);
                }
            };
            // without a route the weight tiles of the first stages are requested before the predecessor has finished
            int early = 0;
            if (!routed) {
                if (unit0 < total) {
                    const int n0 = (unit0 / sp / tiles_m * CG + rank) * FN, first = k_first(unit0);
                    early = min(k_end(unit0) - first, STAGES);
                    for (int i = 0; i < early; i++) ask_w(i, first + i, n0);
                }
                asm volatile("griddepcontrol.wait;" ::: "memory");
            }
            for (int u = unit0; ok && u < total; u += units) {
                const int tile = u / sp;
                const int m0 = (tile % tiles_m) * MT, n0 = (tile / tiles_m * CG + rank) * FN;
                const int w0 = routed ? __ldcg(rt.block_expert + block0 + m0 / PG_ROUTE_BLOCK) * N + n0 : n0;
                for (int kb = k_first(u), end = k_end(u); kb < end; kb++) {
                    if (!(ok = pg_mbar_wait(bar_empty + 8 * stage, phase ^ 1, abort_flag, status, limit_ns))) break;
                    const uint32_t at = base + stage * C::STAGE;
                    if (early > 0)
                        early--;                            // announced and half filled above
                    else
                        ask_w(stage, kb, w0);
                    tma_load_3d_to<CG>(at + C::STAGE_W, &tmap_a, full_l + 8 * stage, kb * FK, m0 + rank * (MT / CG), 0);   // all three planes
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            if (!ok) {
                // give copies that are still in flight a bounded time to land before the CTA exits
                const unsigned long long t0 = pg_globaltimer_ns();
                while (pg_globaltimer_ns() - t0 < 2000000ull) {
                }
            }
        }
    } else if (warp < 4) {
        // ---------------------------------------------------------------- MMA issuers (the whole warp; one lane's products count): each has
        // every other block of K and one of the accumulators.  (An accumulator is waited for before a stage: the epilogue gives it back
        // in the order of the blocks, so that no stage is waited for whose use before last is still to be filled.)
        if (warp <= C::MW && rank == 0) {
            const uint32_t on = pg_elect();
            constexpr uint32_t idesc = make_idesc(CG * FN, MT);
            uint32_t count = 0;
            bool ok = true;
            for (int u = unit0; ok && u < total; u += units) {
                for (int kb = k_first(u), end = k_end(u); kb < end; kb++, count++) {
                    const uint32_t acc = count & 1, stage = count % STAGES;
                    if ((int)acc != warp - 1) continue;
                    ok = pg_mbar_wait_warp(bar_tempty + 8 * acc, (count / 2 & 1) ^ 1, abort_flag, status, limit_ns);
                    if (!ok || !(ok = pg_mbar_wait_warp(bar_full + 8 * stage, count / STAGES & 1, abort_flag, status, limit_ns))) break;
                    if (C::TA && !(ok = pg_mbar_wait_warp(bar_a + 8 * acc, count / 2 & 1, abort_flag, status, limit_ns))) break;
                    tc_fence_after();
                    const uint32_t at = base + stage * C::STAGE, d_tmem = tmem_base + acc * C::ACC;
                    const uint64_t dw = make_smem_desc(at), da = make_smem_desc(at + C::STAGE_W);
#pragma unroll
                    for (int l = 2; l >= 0; l--)
#pragma unroll
                        for (int j = 0; j < FK / 16; j++) {
                            const uint64_t dp = da + (uint64_t)(l * (C::PLANE >> 4) + j * 2);
                            if (C::TA)
                                umma_f16_ta_of<CG>(d_tmem, tmem_base + C::A_COL + acc * 32 + j * 8, dp, idesc, l != 2 || j != 0 ? 1u : 0u, on);
                            else
                                umma_f16(d_tmem, dw + (uint64_t)(j * 2), dp, idesc, l != 2 || j != 0 ? 1u : 0u, on);
                        }
                    if (C::TA) umma_commit_to<CG>(bar_afree + 8 * acc, on);
                    umma_commit_to<CG>(bar_empty + 8 * stage, on);     // stage reusable once these products have read it
                    umma_commit_to<CG>(bar_tfull + 8 * acc, on);
                }
            }
        }
    } else if (warp < C::EW0) {
        // ---------------------------------------------------------------- W to TMEM: lane = row of W
        const int row = (warp & 3) * 32 + lane;
        const uint32_t dst = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + C::A_COL, a_l = pg_leader<CG>(bar_a);
        uint32_t count = 0;
        bool ok = true;
        for (int u = unit0; ok && u < total; u += units) {
            for (int kb = k_first(u), end = k_end(u); kb < end; kb++, count++) {
                const uint32_t buf = count & 1, stage = count % STAGES, src = base + stage * C::STAGE + (uint32_t)row * 128;
                if (!(ok = pg_mbar_wait_warp(bar_w + 8 * stage, count / STAGES & 1, abort_flag, status, limit_ns))) break;
                uint32_t v[32];
#pragma unroll
                for (int p = 0; p < 8; p++) {
                    const uint4 w = pg_lds128(src + (uint32_t)((p ^ (row & 7)) * 16));
                    v[4 * p] = w.x, v[4 * p + 1] = w.y, v[4 * p + 2] = w.z, v[4 * p + 3] = w.w;
                }
                if (!(ok = pg_mbar_wait_warp(bar_afree + 8 * buf, (count / 2 & 1) ^ 1, abort_flag, status, limit_ns))) break;
                tc_fence_after();
                tmem_st32(dst + buf * 32, v);
                tmem_wait_st();
                tc_fence_before();
                pg_arrive_leader_warp<CG>(a_l + 8 * buf, lane);
            }
        }
    } else {
        // ---------------------------------------------------------------- sums and outputs: lane = column of y
        const int q = warp & 3, half = (warp - C::EW0) >> 2;     // TMEM lane quarter this warp may read, its rows of a
        if (!routed) asm volatile("griddepcontrol.wait;" ::: "memory");   // y may still be read by the predecessor
        const int rows = routed ? tiles_m * MT : M;
        const uint32_t tempty_l = pg_leader<CG>(bar_tempty);
        uint32_t acc = 0, acc_phase = 0;
        bool ok = true;
        for (int u = unit0; ok && u < total; u += units) {
            const int tile = u / sp;
            const int m0 = (tile % tiles_m) * MT + half * C::PART, n0 = (tile / tiles_m * CG + rank) * FN, mine_at = tile * CG + rank;
            const uint32_t lanes = tmem_base + ((uint32_t)(q * 32) << 16), so_far = lanes + 2 * C::ACC + half * C::PART;
            float sum[C::PART] = {};
            int part = (u % sp) * kp.run, next = k_first(u) + kp.blocks;   // the part under way, and the block behind it
            for (int kb = k_first(u), end = k_end(u); kb < end; kb++) {
                if (!(ok = pg_mbar_wait_warp(bar_tfull + 8 * acc, acc_phase, abort_flag, status, limit_ns))) break;
                tc_fence_after();
                const uint32_t taddr = lanes + acc * C::ACC + half * C::PART;
#pragma unroll
                for (int c = 0; c < C::ACC / C::EW; c += 32) {
                    uint32_t v[32];
                    tmem_ld32(taddr + c, v);
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (c + j < C::PART) sum[c + j] += __uint_as_float(v[j]);
                }
                tc_fence_before();
                pg_arrive_leader_warp<CG>(tempty_l + 8 * acc, lane);
                if (++acc == 2) {
                    acc = 0;
                    acc_phase ^= 1;
                }
                if (kp.parts > 1 && (kb + 1 == next || kb + 1 == end)) {
                    // the end of a part: to its slab, or onto the sum of those in front of it
                    if (sp > 1) {
                        float *slab = kp.slabs + (((int64_t)mine_at * kp.parts + part) * MT + half * C::PART) * FN + q * 32 + lane;
#pragma unroll
                        for (int j = 0; j < C::PART; j++) __stcg(slab + j * FN, sum[j]);
                    } else {
                        if (part > 0) {
#pragma unroll
                            for (int c = 0; c < C::ACC / C::EW; c += 32) {
                                uint32_t v[32];
                                tmem_ld32(so_far + c, v);
#pragma unroll
                                for (int j = 0; j < 32; j++)
                                    if (c + j < C::PART) sum[c + j] = __uint_as_float(v[j]) + sum[c + j];
                            }
                        }
                        if (kb + 1 < end) {
#pragma unroll
                            for (int c = 0; c < C::ACC / C::EW; c += 32) {
                                uint32_t v[32];
#pragma unroll
                                for (int j = 0; j < 32; j++) v[j] = c + j < C::PART ? __float_as_uint(sum[c + j]) : 0u;
                                f32_keep(so_far + c, v);
                            }
                        }
                    }
                    if (kb + 1 < end) {
#pragma unroll
                        for (int j = 0; j < C::PART; j++) sum[j] = 0.0f;
                    }
                    part++;
                    next += kp.blocks;
                }
            }
            if (!ok) break;
            const int n = n0 + q * 32 + lane;
            bool mine = true;
            if (sp > 1) {
                unsigned int *ticket = kp.tickets + (mine_at * C::EW + half) * 4 + q;
                __threadfence();
                __syncwarp();
                const unsigned int before = __shfl_sync(0xffffffffu, lane == 0 ? atomicAdd(ticket, 1u) : 0u, 0);
                mine = before == (unsigned)(sp - 1);
                if (mine) {
                    // the last part of these columns to finish adds all parts up, in their order
                    __threadfence();
                    if (lane == 0) *ticket = 0;
                    const float *slab = kp.slabs + ((int64_t)mine_at * kp.parts * MT + half * C::PART) * FN + q * 32 + lane;
#pragma unroll
                    for (int j = 0; j < C::PART; j++) sum[j] = __ldcg(slab + j * FN);
                    for (int p = 1; p < kp.parts; p++) {
                        slab += MT * FN;
#pragma unroll
                        for (int j = 0; j < C::PART; j++) sum[j] += __ldcg(slab + j * FN);
                    }
                }
            }
            if (!mine) continue;
            if (ACT == PG_ACT_NONE) {
                if (n < N) {
                    float *dst = y + (int64_t)m0 * ldy + n;
#pragma unroll
                    for (int j = 0; j < C::PART; j++)
                        if (m0 + j < rows) dst[j * ldy] = sum[j];
                }
            } else {
                // columns [8 gates | 8 ups] twice per warp; N is a multiple of 16
                float *dst = y + (int64_t)m0 * ldy + (n0 + q * 32) / 2 + (lane >> 4) * 8 + (lane & 7);
#pragma unroll
                for (int j = 0; j < C::PART; j++) {
                    const float u2 = __shfl_down_sync(0xffffffffu, sum[j], 8);
                    if (!(lane & 8) && n < N && m0 + j < rows) dst[j * ldy] = pg_glu<ACT>(sum[j], u2, limit);
                }
            }
        }
    }

    // (neither CTA of a pair may leave while the other can still touch its shared memory, barriers or TMEM)
    __syncwarp();
    tc_fence_before();
    pg_group_sync<CG>();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc<CG>(tmem_base, C::COLS);
    }
}

// ---------------------------------------------------------------- host side ----
template <int MT, int ACT>
int32_t launch(pg_ctx *ctx, const pg_linear *lin, const bf16 *planes, int64_t m, float limit, float *y, int64_t ldy, const PgRouted &rt, int block0, FParts kp)
{
    using C = FCfg<MT>;
    CUtensorMap tw, ta;
    const cuuint64_t wd[2] = {(cuuint64_t)lin->k, (cuuint64_t)(lin->experts * lin->n)}, ws[1] = {(cuuint64_t)lin->k * 2};
    const cuuint32_t wb[2] = {FK, FN};
    int32_t rc = pg_encode_bf16(&tw, lin->w, 2, wd, ws, wb);
    if (rc != PG_OK) return rc;
    const cuuint64_t ad[3] = {(cuuint64_t)lin->k, (cuuint64_t)m, 3}, as[2] = {(cuuint64_t)lin->k * 2, (cuuint64_t)(lin->k * m) * 2};
    const cuuint32_t ab[3] = {FK, MT / C::CG, 3};
    rc = pg_encode_bf16(&ta, planes, 3, ad, as, ab);
    if (rc != PG_OK) return rc;
    auto kern = linear_f32_kernel<MT, ACT>;
    static std::atomic<uint64_t> smem_set{0};
    PG_CUDA(pg_max_smem_once(kern, (int)C::SMEM, ctx->device, smem_set));
    const int64_t units = ((m + MT - 1) / MT) * ((lin->n + C::CG * FN - 1) / (C::CG * FN)) * kp.runs;
    kp.tickets = reinterpret_cast<unsigned int *>(ctx->splitk);
    kp.slabs = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(ctx->splitk) + PG_LM_TICKET_BYTES);
    return launch_pdl_cluster(ctx, kern, dim3((unsigned)(std::min<int64_t>(units, ctx->sm_count / C::CG) * C::CG)), dim3(C::THREADS), C::SMEM, C::CG, tw, ta, (int)m,
                              (int)lin->n, (int)lin->k, limit, y, ldy, rt, block0, kp, ctx->d_status, ctx->wait_limit_ns);
}

// Cycles by count: blocks of the busiest CTA (695 / 1004 / 1413 cycles with 16 / 64 / 128 rows and one CTA to a tile; pairs take 0.8 of that), and what a tile
// costs at its end, much more where parts meet.  K = N = 4096, four parts one after the other / two by two / all apart, one CTA to a tile: 128 rows 50 / 42 / 32 us,
// 333 rows 54 / 73 / 77, 1000 rows 97 / 140 / 179.
double f32_cost(int64_t rounds, int64_t blocks, int rows, int64_t parts, bool slabs)
{
    const double block = 320.0 + (FN + 3.0 * rows) * FK * 2 / 60.0;
    return rounds * (blocks * block + 2500.0 + rows * 8.0 + (slabs ? 3000.0 + rows * (100.0 + parts * 12.0) : (parts - 1) * rows * 4.0));
}

// The parts of K: what is best for one tile of 16 rows, where dividing K counts most, but no more than eight (N 512, 333 / 1000 rows: 30 / 40 us,
// with sixteen 34 / 46).  They do not follow the number of rows, so that the order of a row's sums does not either.
void f32_parts(const pg_ctx *ctx, const pg_linear *lin, FParts *kp)
{
    const int64_t kblocks = lin->k / FK, tiles = (lin->n + FN - 1) / FN;
    double best = 0;
    for (int64_t parts = 1; parts <= std::max<int64_t>(1, std::min<int64_t>(8, kblocks / 4)); parts++) {
        const int64_t blocks = (kblocks + parts - 1) / parts;
        if ((kblocks + blocks - 1) / blocks != parts || tiles * 8 * (int64_t)sizeof(int) > (int64_t)PG_LM_TICKET_BYTES) continue;
        const double cost = f32_cost((tiles * parts + ctx->sm_count - 1) / ctx->sm_count, blocks, 16, parts, parts > 1);
        if (best == 0 || cost < best) {
            best = cost;
            kp->parts = (int)parts;
            kp->blocks = (int)blocks;
        }
    }
}

template <int ACT>
int32_t dispatch(pg_ctx *ctx, const pg_linear *lin, const bf16 *planes, int64_t m, float limit, float *y, int64_t ldy, const PgRouted &rt, int block0)
{
    const int64_t kblocks = lin->k / FK, tiles_n = (lin->n + FN - 1) / FN;
    const bool routed = rt.blocks != nullptr;
    int mt = routed ? 128 : 16;
    while (mt < 128 && mt < m) mt *= 2;
    FParts kp = {1, (int)kblocks, 1, 1, nullptr, nullptr};
    if (!routed) {
        // rows per tile, and how many parts a CTA takes; slabs for parts of their own as far as there is room, which may grow except
        // while a graph is recorded
        f32_parts(ctx, lin, &kp);
        const int64_t slab = FN * (int64_t)sizeof(float);
        const int64_t room = ctx->capturing ? (int64_t)ctx->splitk_bytes - (int64_t)PG_LM_TICKET_BYTES : F_SLABS;
        const int full = mt;
        int64_t need = 0;
        double best = 0;
        for (int cand = full; cand >= std::min(full, 64); cand /= 2) {
            const int64_t cg = cand >= 64 ? 2 : 1, tiles = (tiles_n + cg - 1) / cg * cg * ((m + cand - 1) / cand);   // (pairs have two each)
            for (int64_t run = kp.parts; run >= 1; run--) {
                const int64_t runs = (kp.parts + run - 1) / run;
                if (runs > 1 && (tiles * kp.parts * cand * slab > room || tiles * 8 * (int64_t)sizeof(int) > (int64_t)PG_LM_TICKET_BYTES)) break;
                const double cost = f32_cost((tiles * runs + ctx->sm_count - 1) / ctx->sm_count, run * kp.blocks, cand, kp.parts, runs > 1);
                if (best == 0 || cost < best) {
                    best = cost;
                    mt = cand;
                    kp.run = (int)run;
                    kp.runs = (int)runs;
                    need = runs > 1 ? tiles * kp.parts * cand * slab : 0;
                }
            }
        }
        if (need > 0 && !ctx->capturing) {
            const int32_t rc = pg_splitk_reserve(ctx, PG_LM_TICKET_BYTES + (size_t)need);
            if (rc != PG_OK) return rc;
        }
    }
    if (mt == 128) return launch<128, ACT>(ctx, lin, planes, m, limit, y, ldy, rt, block0, kp);
    if (mt == 64) return launch<64, ACT>(ctx, lin, planes, m, limit, y, ldy, rt, block0, kp);
    if (mt == 32) return launch<32, ACT>(ctx, lin, planes, m, limit, y, ldy, rt, block0, kp);
    return launch<16, ACT>(ctx, lin, planes, m, limit, y, ldy, rt, block0, kp);
}

}  // namespace

int32_t pgk_linear_f32(pg_ctx *ctx, const pg_linear *lin, const float *a, int64_t lda, int64_t m, int act, float limit, void *y, int y_dtype, int64_t ldy,
                       const PgRouted *routed)
{
    PG_REQUIRE(y_dtype == PG_F32, "linear: an f32 step has f32 outputs");
    PG_REQUIRE((lin->n + 63) / 64 <= 65535, "linear: too many output columns for the f32 form");
    PG_REQUIRE(m < (1ll << 31) - 256 && lin->experts * lin->n < (1ll << 31) - 256, "linear: too many rows");
    const PgRouted none = {};
    const PgRouted &rt = routed ? *routed : none;
    // Rows in portions whose planes stay below F_PLANES: the same outputs as all at once.  While a graph is recorded, what there is of
    // the workspace takes them, and at least F_ROWS at a time
    const int64_t row_bytes = lin->k * 3 * (int64_t)sizeof(bf16);
    int64_t portion = std::min(m, std::max<int64_t>(F_ROWS, F_PLANES / row_bytes / F_ROWS * F_ROWS));
    if ((size_t)(portion * row_bytes) > ctx->scratch_bytes) {
        if (ctx->capturing) portion = std::min(portion, std::max<int64_t>(F_ROWS, (int64_t)(ctx->scratch_bytes / (size_t)row_bytes) / F_ROWS * F_ROWS));
        const int32_t rc = pg_scratch_reserve_recording(ctx, (size_t)(portion * row_bytes));
        if (rc != PG_OK) return rc;
    }
    bf16 *planes = reinterpret_cast<bf16 *>(ctx->scratch);
    for (int64_t r0 = 0; r0 < m; r0 += portion) {
        const int64_t rows = std::min(portion, m - r0);
        const dim3 grid((unsigned)((lin->k / 4 + 255) / 256), (unsigned)std::min<int64_t>(rows, 8192));
        int32_t rc = launch_pdl(ctx, linear_split_kernel, grid, dim3(256), 0, a, lda, (int)r0, (int)rows, (int)lin->k, rt, reinterpret_cast<uint2 *>(planes));
        if (rc != PG_OK) return rc;
        float *out = (float *)y + r0 * ldy;
        const int block0 = (int)(r0 / PG_ROUTE_BLOCK);
        rc = act == PG_ACT_NONE             ? dispatch<PG_ACT_NONE>(ctx, lin, planes, rows, limit, out, ldy, rt, block0)
             : act == PG_ACT_GELU_TANH_GLU ? dispatch<PG_ACT_GELU_TANH_GLU>(ctx, lin, planes, rows, limit, out, ldy, rt, block0)
                                            : dispatch<PG_ACT_CLAMPED_SWISH_GLU>(ctx, lin, planes, rows, limit, out, ldy, rt, block0);
        if (rc != PG_OK) return rc;
    }
    return PG_OK;
}
