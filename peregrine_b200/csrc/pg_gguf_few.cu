// Dequantising product y = x . dequant(W)^T for GGUF Q4_0 / Q8_0 weights and up to eight rows of x: one pass over the block stream, as
// csrc/pg_gguf_stream.cu makes it (which also describes the layout), with the arithmetic of csrc/pg_gguf_tc.cu on warp-level products.
//
//   * A warp has one slice of K (256 elements) for as long as the kernel runs.  Its part of x stays in registers as fragments: x * 2^s = h1 + h2,
//     two f16 numbers (s per row and slice: the slice's largest element lies in [2^14, 2^15)), 22 significant bits and more than 2^-39 of the
//     slice's largest element.  A row whose slice holds a NaN or an infinity gives NaN.
//   * The quants become f16 exactly.  A block is four m16n8k16 products (16 rows of W x 8 rows of x; two planes x two steps of 16 k, the smaller
//     plane first) into sums of its own, which the block's f16 scale then takes to the tile's f32 sums: sum += d * block, rounded once.
//   * A tile is 16 rows of W; `kw` warps, a slice each, share it, and 16 / kw such groups a CTA.  A warp streams its slices of its tiles through a
//     private ring, one bulk copy of 2304 / 4352 bytes each.  The parts of a tile meet in shared memory, added two by two in their order; the
//     warps take turns at that.
//   * K of more than 16 slices, and of fewer where gf_plan has it so: sp CTAs take the same tiles and write raw sums to slabs; the last of them to finish (a ticket per group)
//     adds them in their order and writes the outputs.  Nobody waits for anybody.
//
// Why beside the streaming form: that one takes three int8 products per block and joins their digits in integer arithmetic, and its digit
// planes of eight rows hold 2048 elements of K, after which it starts anew; here x stays in registers, whatever K is.  With one and two rows it
// makes one product per block, and is ahead.  What bounds this: the conversions of the quants, the same for one row as for eight.
//
// Every mbarrier wait is bounded; a warp that gave up goes on through the remaining barriers without computing.
#include <algorithm>

#include "pg_async.cuh"
#include "pg_gguf_f16.cuh"
#include "pg_internal.cuh"
#include "pg_launch.cuh"

namespace {

constexpr int GF_WARPS = 16, GF_THREADS = GF_WARPS * 32;
constexpr size_t GF_TICKET_BYTES = 64 * 1024;     // as in the other kernels that divide K: tickets, zero between calls, then slabs

template <int TYPE>
struct GfCfg {
    static constexpr int SEG = TYPE == PG_GGUF_Q4_0 ? 128 : 256;   // quant bytes per row and slice
    static constexpr int FILL = 16 * SEG + 256;
    static constexpr int SLOTS = TYPE == PG_GGUF_Q4_0 ? 5 : 3;
    static constexpr int RING = GF_WARPS * SLOTS * FILL;
    static constexpr int MEET = 2 * GF_WARPS * 512;                // [tile parity][warp][lane] four sums
    static constexpr int SMEM = RING + MEET + GF_WARPS * SLOTS * 8 + 16;
    static_assert(SMEM <= 227 * 1024, "shared memory");
};

// D = A (16 rows of W x 16 k) x B (16 k x 8 rows of x) + C
__device__ __forceinline__ void gf_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, const float (&c)[4])
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
// the eight nibbles of a word, minus 8, in the order of gguf_nibbles_f16: the upper nibble of a byte is 16 times as much of the last bits of 1024,
// which one multiply-add takes back exactly
__device__ __forceinline__ void gf_nibbles(uint32_t w, uint32_t (&h)[4])
{
    const __half2 sixteenth = __half2half2(__ushort_as_half(0x2c00)), less = __half2half2(__ushort_as_half(0xd480));   // 1 / 16, -72
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const uint32_t b = i ? w >> 8 : w;
        h[2 * i] = gguf_sub_f16((b & 0x000f000fu) | 0x64006400u, 0x64086408u);
        const uint32_t up = (b & 0x00f000f0u) | 0x64006400u;
        const __half2 r = __hfma2(*reinterpret_cast<const __half2 *>(&up), sixteenth, less);
        h[2 * i + 1] = *reinterpret_cast<const uint32_t *>(&r);
    }
}

template <int TYPE>
__global__ void __launch_bounds__(GF_THREADS, 1)
    gguf_few_kernel(const float *__restrict__ x, int M, const uint8_t *__restrict__ qs, int64_t N, int nslices, int kw, int sp, float *__restrict__ y,
                    float4 *slabs, unsigned int *tickets, int32_t *status, unsigned long long limit_ns)
{
    using C = GfCfg<TYPE>;
    extern __shared__ __align__(128) unsigned char smem[];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    float4 *meet = reinterpret_cast<float4 *>(smem + C::RING);
    const uint32_t bars = pg_smem(smem + C::RING + C::MEET), my_bar = bars + (uint32_t)warp * (C::SLOTS * 8);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + C::RING + C::MEET + GF_WARPS * C::SLOTS * 8);
    const uint32_t ring = pg_smem(smem) + (uint32_t)warp * (C::SLOTS * C::FILL);
    if (threadIdx.x == 0) {
        for (int i = 0; i < GF_WARPS * C::SLOTS; i++) pg_mbar_init(bars + 8 * i, 1);
        *abort_flag = 0;
        pg_mbar_fence();
    }
    __syncthreads();

    const int my_part = (int)blockIdx.x % sp, unit = (int)blockIdx.x / sp, units = (int)gridDim.x / sp;
    const int groups = GF_WARPS / kw, group = warp / kw, kp = warp - group * kw;
    const int slice = my_part * kw + kp;
    const bool has = group < groups && slice < nslices;    // (the last part of K may be shorter)
    const int64_t tiles = (N + 15) >> 4, per = (tiles + (int64_t)units * groups - 1) / ((int64_t)units * groups);
    const int64_t first = ((int64_t)unit * groups + group) * per;
    const int mine = group < groups ? (int)max((int64_t)0, min(per, tiles - first)) : 0;
    const uint8_t *src = qs + (first * nslices + slice) * (int64_t)C::FILL;
    auto issue = [&](int j, int slot) {
        if (lane == 0) {
            pg_mbar_expect(my_bar + 8 * slot, C::FILL);
            pg_bulk_load(ring + slot * C::FILL, src + (int64_t)j * nslices * C::FILL, C::FILL, my_bar + 8 * slot);
        }
    };
    for (int j = 0; j < C::SLOTS; j++)
        if (has && j < mine) issue(j, j);

    // x comes from the preceding kernel.  This lane: row g, eight elements of every block of the slice
    asm volatile("griddepcontrol.wait;" ::: "memory");
    uint4 h1[8], h2[8];
    float us;
    {
        float v[8][8];
        float top = 0.0f, poison = 0.0f;
        const float4 *xr = reinterpret_cast<const float4 *>(x + ((int64_t)g * nslices + slice) * 256 + t * 8);
#pragma unroll
        for (int b = 0; b < 8; b++) {
            float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
            if (has && g < M) {
                lo = pg_ld_fresh(xr + b * 8);
                hi = pg_ld_fresh(xr + b * 8 + 1);
            }
            v[b][0] = lo.x, v[b][1] = lo.y, v[b][2] = lo.z, v[b][3] = lo.w, v[b][4] = hi.x, v[b][5] = hi.y, v[b][6] = hi.z, v[b][7] = hi.w;
        }
#pragma unroll
        for (int b = 0; b < 8; b++)
#pragma unroll
            for (int i = 0; i < 8; i++) {
                top = fmaxf(top, fabsf(v[b][i]));
                poison += v[b][i] - v[b][i];               // 0, or NaN
            }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            poison += __shfl_xor_sync(0xffffffffu, poison, o);
        }
        const bool fine = poison == 0.0f;
        const int e = fine ? gguf_exponent(top) : 0;
        const float sc = scalbnf(1.0f, 14 - e);
        us = fine ? scalbnf(1.0f, e - 14) : NAN;
#pragma unroll
        for (int b = 0; b < 8; b++) gguf_split8<TYPE == PG_GGUF_Q4_0>(v[b], sc, h1[b], h2[b]);
    }
    // sums of this lane: rows g (0, 1) and g + 8 (2, 3) of the tile, rows 2 t and 2 t + 1 of x
    const float us0 = __shfl_sync(0xffffffffu, us, 8 * t), us1 = __shfl_sync(0xffffffffu, us, 8 * t + 4);
    auto store = [&](int64_t tile, const float4 &s) {
        const float r[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int64_t n = tile * 16 + g + (i >> 1) * 8;
            const int m = 2 * t + (i & 1);
            if (n < N && m < M) y[(int64_t)m * N + n] = r[i];
        }
    };

    bool ok = true;
    int slot = 0, turn = 0;
    uint32_t phase = 0;
    for (int j = 0; j < mine; j++) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        if (has) {
            ok = ok && pg_mbar_wait_warp(my_bar + 8 * slot, phase, abort_flag, status, limit_ns);
            if (ok) {
                const uint32_t at = ring + slot * C::FILL, lo_at = at + (uint32_t)g * C::SEG, hi_at = lo_at + 8 * C::SEG;
                const uint4 s0 = pg_lds128(at + 16 * C::SEG + g * 16), s1 = pg_lds128(at + 16 * C::SEG + (g + 8) * 16);
                const uint32_t sw0[4] = {s0.x, s0.y, s0.z, s0.w}, sw1[4] = {s1.x, s1.y, s1.z, s1.w};
                constexpr int BPL = TYPE == PG_GGUF_Q4_0 ? 4 : 2;  // blocks per 128-bit load of a row
#pragma unroll
                for (int q = 0; q < 8 / BPL; q++) {
                    const uint32_t piece = (uint32_t)((t ^ (g >> 1)) * 16 + ((q * 4) ^ ((g & 1) << 2)) * 16);
                    const uint4 qa = pg_lds128(lo_at + piece), qb = pg_lds128(hi_at + piece);
                    const uint32_t wa[4] = {qa.x, qa.y, qa.z, qa.w}, wb[4] = {qb.x, qb.y, qb.z, qb.w};
#pragma unroll
                    for (int i = 0; i < BPL; i++) {
                        const int b = q * BPL + i;
                        uint32_t a[4], c[4];
                        if constexpr (TYPE == PG_GGUF_Q4_0) {
                            gf_nibbles(wa[i], a);
                            gf_nibbles(wb[i], c);
                        } else {
                            gguf_bytes_f16(wa[2 * i], wa[2 * i + 1], a);
                            gguf_bytes_f16(wb[2 * i], wb[2 * i + 1], c);
                        }
                        const float zero[4] = {0.f, 0.f, 0.f, 0.f};
                        float p[4];
                        gf_mma(p, a[0], c[0], a[1], c[1], h2[b].x, h2[b].y, zero);
                        gf_mma(p, a[2], c[2], a[3], c[3], h2[b].z, h2[b].w, p);
                        gf_mma(p, a[0], c[0], a[1], c[1], h1[b].x, h1[b].y, p);
                        gf_mma(p, a[2], c[2], a[3], c[3], h1[b].z, h1[b].w, p);
                        const __half2 d0 = *reinterpret_cast<const __half2 *>(&sw0[b >> 1]), d1 = *reinterpret_cast<const __half2 *>(&sw1[b >> 1]);
                        const float f0 = b & 1 ? __high2float(d0) : __low2float(d0), f1 = b & 1 ? __high2float(d1) : __low2float(d1);
                        acc[0] = fmaf(f0, p[0], acc[0]);
                        acc[1] = fmaf(f0, p[1], acc[1]);
                        acc[2] = fmaf(f1, p[2], acc[2]);
                        acc[3] = fmaf(f1, p[3], acc[3]);
                    }
                }
                __syncwarp();                              // every lane has read the slot
                if (j + C::SLOTS < mine) issue(j + C::SLOTS, slot);
                acc[0] *= us0;
                acc[1] *= us1;
                acc[2] *= us0;
                acc[3] *= us1;
                if (++slot == C::SLOTS) {
                    slot = 0;
                    phase ^= 1;
                }
            }
        }
        float4 sum = make_float4(acc[0], acc[1], acc[2], acc[3]);
        if (kw > 1) {
            float4 *cells = meet + ((j & 1) * GF_WARPS + group * kw) * 32 + lane;
            cells[kp * 32] = sum;
            asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(kw * 32) : "memory");
            // (the warps add up in turn; the other buffer is written before the next barrier, this one again behind it)
            const bool my_turn = turn == kp;
            if (++turn == kw) turn = 0;
            if (!my_turn) continue;
            // (two by two: half the roundings on the way.  N 14336, K 4096: error 1.16e-7 -> 1.06e-7, and 18.6 -> 18.2 us of Q4_0, 19.0 -> 18.4 of Q8_0
            // with eight rows, since the loop needs no registers of its own)
            sum = make_float4(0.f, 0.f, 0.f, 0.f);
            int p = kw & 1;
            if (p) sum = cells[0];
#pragma unroll 2
            for (; p < kw; p += 2) {
                const float4 v = cells[p * 32], u = cells[p * 32 + 32];
                sum.x += v.x + u.x;
                sum.y += v.y + u.y;
                sum.z += v.z + u.z;
                sum.w += v.w + u.w;
            }
        }
        if (sp > 1)
            __stcg(slabs + ((int64_t)my_part * tiles + first + j) * 32 + lane, sum);
        else
            store(first + j, sum);
    }
    if (sp > 1) {
        __shared__ int last_in;
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            last_in = atomicAdd(tickets + unit, 1u) == (unsigned)(sp - 1);
            if (last_in) tickets[unit] = 0;
        }
        __syncthreads();
        if (last_in) {
            __threadfence();
            const int64_t t0 = (int64_t)unit * groups * per, t1 = min(tiles, t0 + (int64_t)groups * per);
            for (int64_t tile = t0 + warp; tile < t1; tile += GF_WARPS) {
                float4 sum = __ldcg(slabs + tile * 32 + lane);
                for (int p = 1; p < sp; p++) {
                    const float4 v = __ldcg(slabs + ((int64_t)p * tiles + tile) * 32 + lane);
                    sum.x += v.x;
                    sum.y += v.y;
                    sum.z += v.z;
                    sum.w += v.w;
                }
                store(tile, sum);
            }
        }
    }
    if (!ok) {
        // copies that are still in flight get a bounded time to land before the shared memory goes
        const unsigned long long t0 = pg_globaltimer_ns();
        while (pg_globaltimer_ns() - t0 < 2000000ull) {
        }
    }
}

// CTAs that share K, and warps that share a tile, by 10 ns: a round of tiles takes longer the more warps convert at once; slabs cost a fixed part and
// what the last CTA of a group does at the end, sixteen tiles at a time, sp parts of each.  (By rounds alone, slabs as three of them, K 5632 went to
// eleven CTAs of two warps: Q4_0, N 16000 / 28672 / 49152 30.9 / 50.6 / 82.5 us, with three of eight 26.8 / 42.0 / 66.0; K 2304, N 49152 38.0 against
// 31.6, K 4352, N 28672 37.5 against 35.6.)
void gf_plan(const pg_ctx *ctx, const pg_gguf_weight *w, int *sp, int *kw)
{
    const int64_t nslices = w->k / 256, tiles = (w->n + 15) / 16;
    int64_t best = 0;
    for (int64_t parts = (nslices + GF_WARPS - 1) / GF_WARPS; parts <= std::min<int64_t>(nslices, 16); parts++) {
        const int64_t each = (nslices + parts - 1) / parts, groups = GF_WARPS / each, slots = ctx->sm_count / parts * groups;
        if ((parts - 1) * each >= nslices) continue;
        int64_t cost = (tiles + slots - 1) / slots * (80 + 7 * groups * each);
        if (parts > 1) {
            const int64_t units = std::min<int64_t>(ctx->sm_count / parts, (tiles + groups - 1) / groups), mine = (tiles + units - 1) / units;
            cost += 250 + (mine + GF_WARPS - 1) / GF_WARPS * 14 * parts;
        }
        if (best == 0 || cost < best) {
            best = cost;
            *sp = (int)parts;
            *kw = (int)each;
        }
    }
}

template <int TYPE>
int32_t gf_launch(pg_ctx *ctx, const float *d_x, int M, const pg_gguf_weight *w, float *d_y, int sp, int kw)
{
    using C = GfCfg<TYPE>;
    auto kern = gguf_few_kernel<TYPE>;
    static std::atomic<uint64_t> smem_set{0};
    PG_CUDA(pg_max_smem_once(kern, C::SMEM, ctx->device, smem_set));
    const int64_t tiles = (w->n + 15) / 16, groups = GF_WARPS / kw;
    const int64_t units = std::min<int64_t>(ctx->sm_count / sp, (tiles + groups - 1) / groups);
    return launch_pdl(ctx, kern, dim3((unsigned)(units * sp)), dim3(GF_THREADS), (size_t)C::SMEM, d_x, M, (const uint8_t *)w->d_qs, w->n, (int)(w->k / 256), kw,
                      sp, d_y, reinterpret_cast<float4 *>(reinterpret_cast<unsigned char *>(ctx->splitk) + GF_TICKET_BYTES),
                      reinterpret_cast<unsigned int *>(ctx->splitk), ctx->d_status, ctx->wait_limit_ns);
}

}  // namespace

// Where the streaming form walks K in more than one chunk (it holds 16384 elements of x in all, rows rounded up to 1, 2, 4 or 8), and with four
// rows on narrow layers.  One and two rows only up to 2^25 elements of W: a second chunk costs them less there than the conversions do here.
// With few chunks the streaming form catches up on very wide layers, where its starts weigh least: the line lies between the 49152 columns
// at which they are level or this is ahead, and 65536.  us, streaming form or tensor cores with TMEM (whichever was taken) / this (2 to 3 % more than
// since the parts of a tile are added two by two):
//   Q4_0     K 4096, N 14336: 4 rows 15.6 / 17.6, 5 18.8 / 18.0, 8 21.4 / 18.5   N 28672: 5 rows 29.9 / 29.9, 8 32.1 / 30.1
//            N 43008: 5 rows 44.0 / 40.7, 8 46.8 / 41.6   N 65536: 5 rows 55.0 / 57.9, 8 57.6 / 58.3   N 128256: 5 rows 97.9 / 105.0, 8 100.8 / 107.9
//            K 4096, N 4096: 3 rows 7.4 / 7.4, 4 8.2 / 7.7, 5 11.1 / 7.9, 8 12.1 / 8.4   N 1024: 4 rows 6.2 / 4.9, 8 9.8 / 5.7
//            K 6144, N 32768: 3 rows 45.7 / 46.5, 8 53.8 / 48.1   N 65536: 3 rows 74.2 / 84.5, 8 85.3 / 86.5
//            K 8192, N 28672: 3 rows 54.2 / 53.9, 8 66.3 / 55.4   N 65536: 3 rows 94.9 / 110.1, 8 112.1 / 111.1 (four chunks)
//            K 14336, N 4096: 2 rows 17.9 / 19.7, 3 24.2 / 19.7, 8 25.5 / 20.7   K 9984, N 2490: 2 rows 13.6 / 11.0, 8 16.8 / 12.0
//            K 16640: N 1024, 1 row 12.3 / 8.7, N 4096, 1 row 17.1 / 21.2   K 32768: N 1024, 1 row 17.9 / 13.4, N 4096, 1 row 26.4 / 35.1
//            K 2048, N 12288: 4 rows 9.6 / 9.6, 8 10.3 / 10.4   N 128256: 8 rows 50.6 / 57.7   K 8192, N 8192: 2 rows 13.3 / 20.2, 3 20.9 / 20.4
//   Q8_0     K 4096, N 14336: 4 rows 16.6 / 18.2, 5 19.5 / 18.2, 8 21.0 / 19.0   N 65536: 5 rows 56.8 / 54.8   N 128256: 5 rows 102.2 / 99.3
//            K 8192, N 65536: 3 rows 96.1 / 103.6, 8 113.9 / 105.0   K 14336, N 4096: 2 rows 19.0 / 19.5, 8 26.2 / 20.7
// (Below the line some shapes of Q4_0 are up to 1.1 times as slow here, three rows at K 4352, N 28672 most, 31.0 / 33.8; their error is a third of
// the streaming form's, a tenth where channels stand out.)
bool pgk_matmul_gguf_few_supports(const pg_ctx *ctx, const pg_gguf_weight *w, int64_t m)
{
    if (!(w->tiled && m >= 1 && m <= 8 && w->k <= 256 * GF_WARPS * 16)) return false;
    const int64_t rows = m > 4 ? 8 : m > 2 ? 4 : m, chunks = (w->k * rows + 16383) / 16384;
    if (chunks < 2) return m == 4 && w->n <= 32ll * ctx->sm_count;
    if (m <= 2) return w->n * w->k <= 1ll << 25;
    return w->n <= 57344 || chunks >= (rows == 8 ? 4 : 3) || (rows == 8 && w->type == PG_GGUF_Q8_0);
}

// *taken = false: no workspace for the parts of K to be had (while a graph is recorded, or out of memory); nothing has been launched
int32_t pgk_matmul_gguf_few(pg_ctx *ctx, const float *d_x, int64_t m, const pg_gguf_weight *w, float *d_y, bool *taken)
{
    int sp = 1, kw = 1;
    gf_plan(ctx, w, &sp, &kw);
    *taken = true;
    if (sp > 1) {
        const size_t need = GF_TICKET_BYTES + (size_t)sp * (size_t)((w->n + 15) / 16) * 512;
        if (need > ctx->splitk_bytes && (ctx->capturing || pg_splitk_reserve(ctx, need) != PG_OK)) {
            *taken = false;
            return PG_OK;
        }
    }
    return w->type == PG_GGUF_Q4_0 ? gf_launch<PG_GGUF_Q4_0>(ctx, d_x, (int)m, w, d_y, sp, kw) : gf_launch<PG_GGUF_Q8_0>(ctx, d_x, (int)m, w, d_y, sp, kw);
}
