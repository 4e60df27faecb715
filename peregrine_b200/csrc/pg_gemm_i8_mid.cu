// W8A8 product for batches between decoding and prompts (up to 128 rows, layers of up to one 128-column tile per SM), on the
// 5th-generation tensor cores: the integer GEMM of src/quant.rs:154-166 with its two-scale epilogue, bit for bit.
//
// Weights are the M side of the instruction: D[128 columns of y][rows of x] s32 in TMEM, rows of x rounded up to 16.  K is divided over
// the CTAs of a cluster, which work on one tile and meet in distributed shared memory: every CTA copies its sums into its own
// shared memory, and after one cluster barrier each adds all parts for its share of the rows, applies the scales and stores 512
// contiguous bytes per warp.
//
// What bounds it: the copies into shared memory -- per 128 k a CTA takes 16 KB of weights and as much as 16 KB of x from L2 -- and, on
// short K, the launch.  Dividing K needs no second pass through L2: with slabs in global memory and the last part adding them up (the
// form in pg_gemm_tcgen05.cu, which wider layers keep), K 14336, N 4096 spent 10 of 24 us in that.
//
// Every mbarrier wait is bounded (pg_async.cuh); a CTA that gives up still goes through both cluster barriers.
#include <algorithm>

#include "pg_async.cuh"
#include "pg_internal.cuh"
#include "pg_launch.cuh"
#include "pg_tcgen05.cuh"

namespace {

constexpr int MD_N = 128;                     // columns of y per tile
constexpr int MD_K = 128;                     // bytes of K per stage: one swizzle span
constexpr int MD_THREADS = 192, MD_WARPS = MD_THREADS / 32;
constexpr int MD_ROOM = 232448 - 1024 - 512;
constexpr int MD_MAX_PARTS = 8;
constexpr int MD_TWO_FROM = 20;            // k-blocks a part with two threads for the copies

// rows of x per tile
__host__ __device__ inline int md_rows(int M) { return (M + 15) & ~15; }
__host__ __device__ inline int md_stage(int rows) { return (MD_N + rows) * MD_K; }
__host__ __device__ inline int md_stages(int rows) { return MD_ROOM / md_stage(rows) < 12 ? MD_ROOM / md_stage(rows) : 12; }

__device__ __forceinline__ int4 md_peer_load(uint32_t local, uint32_t cta)
{
    int4 v;
    asm volatile(
        "{\n\t.reg .b32 a;\n\t"
        "mapa.shared::cluster.u32 a, %4, %5;\n\t"
        "ld.shared::cluster.v4.s32 {%0, %1, %2, %3}, [a];\n\t}"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "r"(local), "r"(cta)
        : "memory");
    return v;
}

// gives copies that are still in flight a bounded time to land before a CTA that gives up exits
__device__ __forceinline__ void md_settle()
{
    const unsigned long long t0 = pg_globaltimer_ns();
    while (pg_globaltimer_ns() - t0 < 2000000ull) {
    }
}

// TWO: a copy costs the thread that asks for it 230 cycles, so in a long part of K x has a thread of its own.  It starts later than one thread
// for both does, which a short part does not make up for; the line lies between the 16 and the 28 k-blocks measured.  us, one thread / two:
//   32 k-blocks a part (K 4096, N 14336), 12 / 17 / 40 rows   14.4 / 14.7 / 16.0          13.4 / 13.5 / 14.7
//   28 (K 14336, N 4096), 12 / 17 / 40 / 100 rows             16.1 / 16.7 / 18.7 / 20.0   15.3 / 15.8 / 17.3 / 19.3
//   16 (K 4096, N 6144), 12 / 17 / 40 / 100 rows               8.9 /  9.3 /  9.8 / 12.2    9.4 /  9.6 /  9.9 / 12.1
//    8 (K 4096, N 4096), 17 / 40 / 64 rows                     7.8 /  8.4 /  9.0           8.3 /  8.8 /  9.3
template <bool TWO>
__global__ void __launch_bounds__(MD_THREADS, 1)
    gemm_i8_mid_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const float *__restrict__ a_scales,
                       const float *__restrict__ w_scales, int M, int N, int K, int parts, float *__restrict__ y, int32_t *__restrict__ acc_out,
                       int32_t *status, unsigned long long limit_ns)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = pg_smem(smem_raw), base = (raw + 1023u) & ~1023u;
    const int rows = md_rows(M), stage_bytes = md_stage(rows), stages = md_stages(rows);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_raw + (base - raw) + stages * stage_bytes);
    const uint32_t bar_full = pg_smem(bars), bar_empty = bar_full + 8 * stages, bar_done = bar_empty + 8 * stages;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * stages + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t cols = rows <= 32 ? 32 : rows <= 64 ? 64 : 128;
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) {
            pg_mbar_init(bar_full + 8 * s, 1);
            pg_mbar_init(bar_empty + 8 * s, 1);
        }
        pg_mbar_init(bar_done, 1);
        *abort_flag = 0;
        pg_mbar_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(pg_smem(tmem_slot)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int part = blockIdx.x % parts, n0 = (blockIdx.x / parts) * MD_N;
    const int kblocks = (K + MD_K - 1) / MD_K, per = (kblocks + parts - 1) / parts;
    const int kb0 = min(kblocks, part * per), kb1 = min(kblocks, kb0 + per);   // (never empty: the host sees to it)

    bool ok = true;
    if (warp == 0 && !TWO) {
        if (lane == 0) {
            const int early = min(kb1 - kb0, stages);           // weights do not depend on the preceding kernel
            for (int i = 0; i < early; i++) {
                pg_mbar_expect(bar_full + 8 * i, (uint32_t)stage_bytes);
                tma_load_2d(base + i * stage_bytes, &tmap_w, bar_full + 8 * i, (kb0 + i) * MD_K, n0);
            }
            asm volatile("griddepcontrol.wait;" ::: "memory");
            int stage = 0, phase = 0;
            for (int kb = kb0; kb < kb1; kb++) {
                const uint32_t at = base + stage * stage_bytes;
                if (kb - kb0 >= early) {
                    if (!(ok = pg_mbar_wait(bar_empty + 8 * stage, phase ^ 1, abort_flag, status, limit_ns))) break;
                    pg_mbar_expect(bar_full + 8 * stage, (uint32_t)stage_bytes);
                    tma_load_2d(at, &tmap_w, bar_full + 8 * stage, kb * MD_K, n0);
                }
                tma_load_2d(at + MD_N * MD_K, &tmap_x, bar_full + 8 * stage, kb * MD_K, 0);
                if (++stage == stages) {
                    stage = 0;
                    phase ^= 1;
                }
            }
            if (!ok) md_settle();
        }
    } else if (TWO && (warp == 0 || warp == 2) && lane == 0) {
        // a thread for the weights, and one for x, which announces a stage's bytes (its warp has nothing else to do until all sums are there)
        if (warp == 2) asm volatile("griddepcontrol.wait;" ::: "memory");
        int stage = 0, phase = 1;
        for (int kb = kb0; kb < kb1; kb++) {
            const uint32_t at = base + stage * stage_bytes;
            if (!(ok = pg_mbar_wait(bar_empty + 8 * stage, phase, abort_flag, status, limit_ns))) break;
            if (warp == 0) {
                tma_load_2d(at, &tmap_w, bar_full + 8 * stage, kb * MD_K, n0);
            } else {
                pg_mbar_expect(bar_full + 8 * stage, (uint32_t)stage_bytes);
                tma_load_2d(at + MD_N * MD_K, &tmap_x, bar_full + 8 * stage, kb * MD_K, 0);
            }
            if (++stage == stages) {
                stage = 0;
                phase ^= 1;
            }
        }
        if (!ok) md_settle();
    }
    if (TWO) __syncwarp();
    if (warp == 1) {
        const uint32_t on = pg_elect();
        // kind::i8: D = s32 (2 at bit 4), A and B signed 8-bit (1 at bits 7 and 10), both K-major
        const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(rows >> 3) << 17) | ((uint32_t)(MD_N >> 4) << 24);
        int stage = 0, phase = 0;
        for (int kb = kb0; kb < kb1; kb++) {
            ok = __all_sync(0xffffffffu, pg_mbar_wait(bar_full + 8 * stage, phase, abort_flag, status, limit_ns));
            if (!ok) break;
            tc_fence_after();
            const uint32_t at = base + stage * stage_bytes;
            const uint64_t dw = make_smem_desc(at), dx = make_smem_desc(at + MD_N * MD_K);
#pragma unroll
            for (int j = 0; j < MD_K / 32; j++) umma_i8(tmem, dw + (uint64_t)(j * 2), dx + (uint64_t)(j * 2), idesc, kb != kb0 || j != 0 ? 1u : 0u, on);
            umma_commit(bar_empty + 8 * stage, on);
            if (++stage == stages) {
                stage = 0;
                phase ^= 1;
            }
        }
        if (ok) umma_commit(bar_done, on);
    } else if (warp > 1) {
        // lane = column of y: its sums go to [row][128] in the ring, which nothing else uses any more
        ok = __all_sync(0xffffffffu, (!TWO || ok) && pg_mbar_wait(bar_done, 0, abort_flag, status, limit_ns));
        if (ok) {
            tc_fence_after();
            const int q = warp & 3;
            const uint32_t dst = base + (uint32_t)(q * 32 + lane) * 4;
#pragma unroll 1
            for (int c = 0; c < rows; c += 32) {
                uint32_t v[32];
                tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + c, v);
#pragma unroll
                for (int j = 0; j < 32; j++)
                    if (c + j < M) asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + (uint32_t)(c + j) * (MD_N * 4)), "r"(v[j]) : "memory");
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    cl_sync();                                                  // all parts' sums are in place
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");        // the scales come from the preceding kernel; y may still be read by it
    {
        const int share = (M + parts - 1) / parts, m0 = part * share, m1 = min(M, m0 + share);
        const int n = n0 + lane * 4;
        const bool vec = (N & 3) == 0 && (((uintptr_t)y | (uintptr_t)acc_out) & 15) == 0;
        float ws[4];
#pragma unroll
        for (int i = 0; i < 4; i++) ws[i] = n + i < N && y ? __ldg(w_scales + n + i) : 0.0f;
        constexpr int R = 4;                                    // rows per warp and round: their loads are in flight together
        for (int mb = m0 + warp; mb < m1; mb += MD_WARPS * R) {
            int4 sum[R];
            float as[R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int m = min(mb + r * MD_WARPS, m1 - 1);
                as[r] = y ? __ldcg(a_scales + m) : 0.0f;
                sum[r] = md_peer_load(base + (uint32_t)m * (MD_N * 4) + lane * 16, 0);
            }
            for (int p = 1; p < parts; p++)
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const int4 v = md_peer_load(base + (uint32_t)min(mb + r * MD_WARPS, m1 - 1) * (MD_N * 4) + lane * 16, (uint32_t)p);
                    sum[r].x += v.x, sum[r].y += v.y, sum[r].z += v.z, sum[r].w += v.w;
                }
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int m = mb + r * MD_WARPS;
                if (m >= m1) break;
                const int64_t off = (int64_t)m * N + n;
                const int s[4] = {sum[r].x, sum[r].y, sum[r].z, sum[r].w};
                float o[4];
#pragma unroll
                for (int i = 0; i < 4; i++) o[i] = __fmul_rn(__fmul_rn(__int2float_rn(s[i]), as[r]), ws[i]);
                if (vec && n < N) {
                    if (acc_out) *reinterpret_cast<int4 *>(acc_out + off) = sum[r];
                    if (y) *reinterpret_cast<float4 *>(y + off) = make_float4(o[0], o[1], o[2], o[3]);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        if (n + i >= N) break;
                        if (acc_out) acc_out[off + i] = s[i];
                        if (y) y[off + i] = o[i];
                    }
                }
            }
        }
    }
    cl_sync();                                                  // a CTA's sums stay until its peers have read them
}

int32_t md_encode(CUtensorMap *map, const void *ptr, int64_t rows, int64_t k, int box_rows)
{
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)k};
    const cuuint32_t box[2] = {MD_K, (cuuint32_t)box_rows};
    return pg_encode_map(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, ptr, 2, dims, strides, box);
}

// clusters of `parts` CTAs that fit the device at once, with as much shared memory as there is
int32_t md_clusters(pg_ctx *ctx, int parts, int *fit)
{
    static std::atomic<int> known[64][MD_MAX_PARTS + 1];
    std::atomic<int> &k = known[ctx->device & 63][parts];
    int v = k.load(std::memory_order_relaxed);
    if (v == 0) {
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)parts;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)parts);
        cfg.blockDim = dim3(MD_THREADS);
        cfg.dynamicSmemBytes = MD_ROOM + 1024 + 512;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        PG_CUDA(cudaOccupancyMaxActiveClusters(&n, gemm_i8_mid_kernel<false>, &cfg));
        v = n + 1;
        k.store(v, std::memory_order_relaxed);
    }
    *fit = v - 1;
    return PG_OK;
}

}  // namespace

bool pgk_gemm_i8_mid_supports(pg_ctx *ctx, int64_t m, int64_t k, int64_t n)
{
    // (where every tile keeps its whole K, the epilogue's way through shared memory costs more than the other kernel's from some number of
    // rows on.  With quantiser, this / the other, us: K 4096, N 14336, 96 / 112 / 128 rows 16.2 / 17.5 / 18.7 against 18.2 / 18.5 / 18.7; K 2048,
    // N 16384 13.5 / 14.5 / 15.7 against 13.5 / 14.1 / 14.2.  The line is that of one thread for the copies on either side; on long K it would
    // lie behind 128 rows now: K 8192, N 12288, 100 rows 26.2 / 39.1)
    const int64_t tiles = (n + MD_N - 1) / MD_N;
    return m >= 1 && m <= 128 && n >= 1 && k >= 16 && k % 16 == 0 && k < (1ll << 31) && tiles <= ctx->sm_count && (m <= 96 || 2 * tiles <= ctx->sm_count);
}

int32_t pgk_gemm_i8_mid(pg_ctx *ctx, const int8_t *d_a, const float *d_as, int64_t m, int64_t k, const pg_qtensor *w, float *d_y, int32_t *d_acc)
{
    static std::atomic<uint64_t> smem_set{0}, smem_set_two{0};
    PG_CUDA(pg_max_smem_once(gemm_i8_mid_kernel<false>, MD_ROOM + 1024 + 512, ctx->device, smem_set));
    PG_CUDA(pg_max_smem_once(gemm_i8_mid_kernel<true>, MD_ROOM + 1024 + 512, ctx->device, smem_set_two));
    const int64_t n = w->cols, tiles = (n + MD_N - 1) / MD_N, kblocks = (k + MD_K - 1) / MD_K;
    // parts of K: as many as still have all their clusters on the GPU at once and at least four k-blocks each
    int parts = 1;
    for (int p = 2; p <= MD_MAX_PARTS && tiles * p <= ctx->sm_count && kblocks >= 4 * p; p++) {
        const int64_t per = (kblocks + p - 1) / p;
        if ((kblocks + per - 1) / per != p) continue;
        int fit = 0;
        const int32_t rc = md_clusters(ctx, p, &fit);
        if (rc != PG_OK) return rc;
        if (tiles <= fit) parts = p;
    }
    CUtensorMap tw, tx;
    const int rows = md_rows((int)m);
    int32_t rc = md_encode(&tw, w->d_data_i8_t, n, k, MD_N);
    if (rc == PG_OK) rc = md_encode(&tx, d_a, m, k, rows);
    if (rc != PG_OK) return rc;
    auto kern = (kblocks + parts - 1) / parts > MD_TWO_FROM ? gemm_i8_mid_kernel<true> : gemm_i8_mid_kernel<false>;
    return launch_pdl_cluster(ctx, kern, dim3((unsigned)(tiles * parts)), dim3(MD_THREADS), (size_t)md_stages(rows) * md_stage(rows) + 1024 + 512, parts,
                              tw, tx, d_as, (const float *)w->d_scales, (int)m, (int)n, (int)k, parts, d_y, d_acc, ctx->d_status, ctx->wait_limit_ns);
}
