// The delta rule of long portions, 64 tokens at a time, with its products on the tensor cores.
//
// With the decays g of a chunk's tokens, c_a = g_0 .. g_a, r_ab = g_{b+1} .. g_a and the state S that the chunk finds:
//   (I + A) U = beta V - (beta c K) S,  A_ab = beta_a r_ab (k_a . k_b) for b < a
//   O = c (Q S) + P U,                  P_ab = r_ab (q_a . k_b) for b <= a
//   S <- c_63 S + K~^T U,               K~_b = r_63,b k_b
// What does not depend on S is made for all chunks at once: W = (I + A)^-1 (beta c K) and U0 = (I + A)^-1 (beta V)
// (delta_chunk_kernel, which has the convolution and the unit norms in it).  The chain that is left, U = U0 - W S and the two
// lines above, is three tcgen05 products per chunk (delta_chain_kernel, a CTA per head and 32 columns of the state, which stays in
// registers).
//
// Precision: that of delta_scan_kernel's f32.  A product's operands are pairs of f16 numbers, h + l: 23 significant bits, and all 24 of
// three in four f32 numbers.  All four products of the parts are taken.  W, Q, K~, P, A and the inverses have rows of norm at most one
// (keys are unit vectors and every step is a contraction), so a fixed scale of 2^14 keeps their bits; values, S and U are scaled by a
// power of two that follows from the largest element.  The tensor core cuts off what falls below an accumulator's last bit, so an
// accumulator takes the small products first or alone, and of the large ones two steps of sixteen; sums of accumulators are rounded,
// in registers.  What needs no product stays in f32: the diagonals of the inverses, and a token's own key in P.
// Against 64 bits, from the same inputs, these kernels / delta_scan_kernel, 130 to 4000 tokens: outputs 1.59e-7 ... 1.61e-7 / 1.57e-7 ...
// 1.65e-7, states 1.7e-7 / 2.0e-7 ... 2.2e-7; where little is forgotten 3.3e-7 / 4.3e-6 at 4000 tokens; where a few tokens are all that
// is kept 1.45e-7 / 1.39e-7, states 1.5e-7 / 1.3e-7.
//
// What is not finite stays with its token and those behind it: from the first token of a chunk with such a value, key or gate on,
// U is zero in the products, O is NaN, and so is the state behind the chunk.
#include <cuda_fp16.h>

#include <algorithm>

#include "pg_async.cuh"
#include "pg_delta.cuh"
#include "pg_tcgen05.cuh"

namespace {

constexpr int CT = DELTA_CHUNK, CD = 128;      // tokens of a chunk; width of a key and of a value
constexpr float OPERAND = 16384.0f, OPERAND_INV = 1.0f / 16384.0f;

// Images of operand tiles as the products read them: rows of 64 f16 elements, 128-byte swizzle, 64 rows = 8 KB.
// Per (chunk, head): W [part][half of d] | K~ [part][half of d] | P [part] | U0 [64][128] f32 | coefficients
// Per (chunk, key head): Q [part][half of d]
constexpr int TILE = 8192, W_AT = 0, KT_AT = 4 * TILE, P_AT = 8 * TILE, U0_AT = 10 * TILE, COEF_AT = U0_AT + CT * CD * 4;
constexpr int HEAD_BYTES = COEF_AT + 640, GROUP_BYTES = 4 * TILE;
constexpr int COEF_OWN = CT, COEF_LAST = 2 * CT, COEF_MAX = COEF_LAST + 1, COEF_BAD = COEF_LAST + 2;   // c [64], q_a . k_a [64], c_63, largest |U0|, first token that is not finite

// The chunks of the sequence at row0 are numbered from here on; none has another's number, since a sequence has at least DELTA_LONG tokens.
constexpr int ROWS_PER_CHUNK = 43;
__host__ __device__ constexpr int64_t first_chunk(int64_t row0) { return row0 / ROWS_PER_CHUNK; }
constexpr bool chunks_find_room()
{
    for (int T = DELTA_LONG; T < DELTA_LONG + 64 * ROWS_PER_CHUNK; T++)
        if (T / ROWS_PER_CHUNK < (T + CT - 1) / CT) return false;
    return true;
}
static_assert(chunks_find_room(), "two sequences would share a chunk");
__device__ __forceinline__ unsigned char *head_data(const DeltaShape &s, const DeltaWork &w, int64_t chunk, int h)
{
    return w.chunks + chunk * ((int64_t)s.H * HEAD_BYTES + (int64_t)s.G * GROUP_BYTES) + (int64_t)h * HEAD_BYTES;
}
__device__ __forceinline__ unsigned char *group_data(const DeltaShape &s, const DeltaWork &w, int64_t chunk, int g)
{
    return w.chunks + chunk * ((int64_t)s.H * HEAD_BYTES + (int64_t)s.G * GROUP_BYTES) + (int64_t)s.H * HEAD_BYTES + (int64_t)g * GROUP_BYTES;
}

// (a, b) = h + l
__device__ __forceinline__ void split2(float a, float b, uint32_t &h, uint32_t &l)
{
    const __half2 hi = __floats2half2_rn(a, b);
    const float2 f = __half22float2(hi);
    const __half2 lo = __floats2half2_rn(a - f.x, b - f.y);
    h = *reinterpret_cast<const uint32_t *>(&hi);
    l = *reinterpret_cast<const uint32_t *>(&lo);
}
__device__ __forceinline__ float2 join2(uint32_t h, uint32_t l)
{
    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&h)), b = __half22float2(*reinterpret_cast<const __half2 *>(&l));
    return make_float2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// (ah + al) times sixteen columns: the products of the two high parts, and the others
__device__ __forceinline__ void mma_pair(float (&d)[2][4], float (&e)[2][4], const uint32_t (&ah)[4], const uint32_t (&al)[4], const uint32_t (&bh)[4],
                                         const uint32_t (&bl)[4])
{
#pragma unroll
    for (int n = 0; n < 2; n++) {
        mma_f16(e[n], al, bl[2 * n], bl[2 * n + 1]);
        mma_f16(e[n], al, bh[2 * n], bh[2 * n + 1]);
        mma_f16(e[n], ah, bl[2 * n], bl[2 * n + 1]);
        mma_f16(d[n], ah, bh[2 * n], bh[2 * n + 1]);
    }
}
__device__ __forceinline__ void stsm4_t(uint32_t addr, const uint32_t (&r)[4])
{
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
__device__ __forceinline__ uint32_t bits(float x) { return __float_as_uint(x) & 0x7fffffffu; }   // |x|; NaN is the largest
__device__ __forceinline__ uint32_t warp_max(uint32_t v) { return __reduce_max_sync(0xffffffffu, v); }
constexpr uint32_t NOT_FINITE = 0x7f800000u;
// a power of two that brings a bound into [2^to, 2^(to + 1)), and its inverse (both normal numbers; no bound is so large that the
// lower limit counts)
__device__ __forceinline__ float2 scale_of(float bound, int to)
{
    const int e = min(100, max(-126, 127 + to - (int)(bits(bound) >> 23)));
    return make_float2(__uint_as_float((uint32_t)(127 + e) << 23), __uint_as_float((uint32_t)(127 - e) << 23));
}

// ---- what does not depend on the state: grid (G, chunks of the longest sequence, seqs), 512 threads ---------------------
// (I + A)^-1 goes by blocks of sixteen rows: X_J = T_J (rhs_J - sum over I < J of A_JI X_I), T_J the inverse of the diagonal
// block.  The blocks are mma.sync products of transposed tiles, X^T [sixteen columns][64 rows]: the sums of one are the left operand
// of the next without leaving the warp's registers.  The last chunks come first, so that the chain finds the first ones in L2.
//
// Bound by instructions: 59000 cycles a CTA at 4096 tokens, 20000 of them the convolution, 15000 the substitution.  4096 tokens of 32
// heads (430 MB in and out): 227 us, 212 with all products of a sum in one accumulator.  Then, with f32 multiply-adds over columns in place
// of the tiles 290, with all 64 rows of two columns in a thread's registers, unrolled, 448 (code that runs once is waited for).
constexpr int V_PITCH = 132, DIAG_PITCH = 20, T_PITCH = 48;
struct ChunkSmem {
    unsigned char k[4 * TILE];
    union {
        unsigned char q[4 * TILE], w0[4 * TILE];      // W of the first head, when the queries are done with
    };
    unsigned char w1[4 * TILE];
    unsigned char a[2][2 * TILE];                     // [head][part] A below its diagonal blocks
    float v[2][CT][V_PITCH];                          // values, then U0
    float diag[2][4][16][DIAG_PITCH];                 // diagonal blocks of A
    unsigned char t[2][4][2][16 * T_PITCH];           // their inverses [head][block][part][row][16]
    float l_hi[2][CT], l_lo[2][CT], beta[2][CT], c[2][CT], last[2][CT];   // sums of log g in two parts; r_63,b
    uint32_t top_v[2], largest[2];                    // largest |v|, |U0|
    int bad[2], bad_k;                                // first token that is not finite: of a head, of the keys
};

// z / (1 + e^-z), the quotient with a step of Newton's behind it (the exponent ends where the denominator's inverse does)
__device__ __forceinline__ float silu(float z)
{
    const float d = 1.0f + expf(fminf(-z, 87.0f)), r = __fdividef(1.0f, d), y = z * r;
    return fmaf(fmaf(-d, y, z), r, y);
}
// inputs of the convolution of four channels and tokens t .. t + 7
template <int TAPS>
__device__ __forceinline__ void load_inputs(const DeltaShape &s, const float *row0, int64_t ldp, const float *ring, int pos0, int t, int T, int c, float4 (&x)[TAPS + 7])
{
#pragma unroll
    for (int j = 0; j < TAPS + 7; j++) {
        const int at = t + j - (TAPS - 1);
        x[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (at >= 0) {
            if (at < T) x[j] = __ldcg(reinterpret_cast<const float4 *>(row0 + (int64_t)at * ldp + c));
        } else if (pos0 + at >= 0) {
            x[j] = __ldcg(reinterpret_cast<const float4 *>(ring + (int64_t)((pos0 + at) % TAPS) * s.C + c));
        }
    }
}

template <int TAPS>
__global__ void __launch_bounds__(512, 1)
    delta_chunk_kernel(const DeltaShape s, const pg_batch bt, const float *__restrict__ proj, int64_t ldp, const float *__restrict__ ring, const DeltaWork w)
{
    extern __shared__ __align__(1024) unsigned char chunk_smem[];
    ChunkSmem &sm = *reinterpret_cast<ChunkSmem *>(chunk_smem);
    pg_pdl_begin();
    const int seq = blockIdx.z, g = blockIdx.x, nth = gridDim.y - 1 - blockIdx.y, row0 = __ldcg(bt.d_seq_row0 + seq), T = __ldcg(bt.d_seq_row0 + seq + 1) - row0;
    const int t0 = nth * CT;
    if (T < DELTA_LONG || t0 >= T) return;
    const int rep = s.H / s.G, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int pos0 = __ldcg(bt.d_pos + row0);
    const float *first = proj + (int64_t)row0 * ldp;                  // the sequence's rows
    const float *rg = ring + (int64_t)__ldcg(bt.d_seq_slot + seq) * s.taps * s.C;
    const int64_t chunk = first_chunk(row0) + nth;
    const uint32_t k_at = pg_smem(sm.k), q_at = pg_smem(sm.q);
    if (tid == 0) sm.bad_k = CT;

    // gates of a head: two tokens a lane; log decays are added up in 64 bits
    float in_a[2], in_b[2];                                           // (asked for well before they are used)
    auto load_gates = [&](int h) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int a = lane * 2 + i;
            const float *tail = first + (int64_t)(t0 + a) * ldp + s.C + (int64_t)s.H * s.V;
            in_a[i] = t0 + a < T ? __ldcg(tail + s.H + h) : 0.0f;
            in_b[i] = t0 + a < T ? __ldcg(tail + h) : 0.0f;
        }
    };
    auto gates = [&](int x, int h) {
        const float al = __ldg(s.a_log + h), db = __ldg(s.dt_bias + h);
        double v[2];
        float be[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const bool in = t0 + lane * 2 + i < T;
            const float ld = in ? log_decay(in_a[i], al, db) : 0.0f;
            v[i] = (double)(ld < -1e4f ? -1e4f : ld);              // (its exponential is 0 either way; differences stay numbers)
            be[i] = in ? __fdiv_rn(1.0f, 1.0f + expf(-in_b[i])) : 0.0f;
        }
        double sum = v[0] + v[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += up;
        }
        const double all = __shfl_sync(0xffffffffu, sum, 31);
        double l = __shfl_up_sync(0xffffffffu, sum, 1);              // of the tokens in front of this lane's two
        if (lane == 0) l = 0.0;
        float *coef = reinterpret_cast<float *>(head_data(s, w, chunk, h) + COEF_AT);
        auto decay = [](double l) {                                   // e^l; the rest of l is below 2^-24 of it
            const float hi = (float)l;
            return expf(hi) * (1.0f + (float)(l - (double)hi));
        };
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int a = lane * 2 + i;
            l += v[i];
            sm.l_hi[x][a] = (float)l;
            sm.l_lo[x][a] = (float)(l - (double)(float)l);
            sm.beta[x][a] = be[i];
            const float c = decay(l);
            sm.c[x][a] = coef[a] = c;
            sm.last[x][a] = decay(all - l);
            if (!(bits(c) < NOT_FINITE && bits(be[i]) < NOT_FINITE)) atomicMin(&sm.bad[x], a);
        }
        if (lane == 0) coef[COEF_LAST] = decay(all);
    };
    // Convolution, eight tokens a warp and four channels a lane: queries (warps 0 .. 7) and keys, then the values of two heads.
    auto convolve = [&](int i, int h0) {
        const int a0 = (warp & 7) * 8, c = (i == 0 ? g : i == 1 ? s.G + g : 2 * s.G + h0 + i - 2) * CD + lane * 4;
        float4 x[TAPS + 7], wt[TAPS], y[8];
        load_inputs<TAPS>(s, first, ldp, rg, pos0, t0 + a0, T, c, x);
#pragma unroll
        for (int j = 0; j < TAPS; j++) wt[j] = __ldg(reinterpret_cast<const float4 *>(s.conv + (int64_t)j * s.C + c));
        uint32_t top = 0;
#pragma unroll
        for (int a = 0; a < 8; a++) {
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < TAPS; j++) {
                acc.x = fmaf(wt[j].x, x[a + j].x, acc.x), acc.y = fmaf(wt[j].y, x[a + j].y, acc.y);
                acc.z = fmaf(wt[j].z, x[a + j].z, acc.z), acc.w = fmaf(wt[j].w, x[a + j].w, acc.w);
            }
            const bool in = t0 + a0 + a < T;
            y[a] = in ? make_float4(silu(acc.x), silu(acc.y), silu(acc.z), silu(acc.w)) : make_float4(0.f, 0.f, 0.f, 0.f);
            const uint32_t m = max(max(bits(y[a].x), bits(y[a].y)), max(bits(y[a].z), bits(y[a].w)));
            if (i > 0 && m >= NOT_FINITE)
                atomicMin(i == 1 ? &sm.bad_k : &sm.bad[i - 2], a0 + a);
            else
                top = max(top, m);
        }
        if (i < 2) {
            // sums of squares: halved among the lanes until lane l has the one of token l >> 2, whose norm it then works out
            float ss[8];
#pragma unroll
            for (int a = 0; a < 8; a++) ss[a] = y[a].x * y[a].x + y[a].y * y[a].y + y[a].z * y[a].z + y[a].w * y[a].w;
#pragma unroll
            for (int n = 4; n > 0; n >>= 1)
#pragma unroll
                for (int a = 0; a < n; a++) {
                    const bool up = (lane & (n * 4)) != 0;
                    const float give = up ? ss[a] : ss[a + n], keep = up ? ss[a + n] : ss[a];
                    ss[a] = keep + __shfl_xor_sync(0xffffffffu, give, n * 4);
                }
            ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], 1);
            ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], 2);
            const float mine = __fdiv_rn(i == 0 ? s.qscale : 1.0f, sqrtf(ss[0] + s.unit_eps)) * OPERAND;
            unsigned char *img = (i == 0 ? sm.q : sm.k) + (lane >= 16 ? TILE : 0) + (lane & 1) * 8;
#pragma unroll
            for (int a = 0; a < 8; a++) {
                const float inv = __shfl_sync(0xffffffffu, mine, a * 4);
                uint2 h, l;
                split2(y[a].x * inv, y[a].y * inv, h.x, l.x);
                split2(y[a].z * inv, y[a].w * inv, h.y, l.y);
                const int at = (a0 + a) * 128 + ((((lane & 15) >> 1) ^ a) << 4);
                *reinterpret_cast<uint2 *>(img + at) = h;
                *reinterpret_cast<uint2 *>(img + 2 * TILE + at) = l;
            }
        } else {
#pragma unroll
            for (int a = 0; a < 8; a++) *reinterpret_cast<float4 *>(&sm.v[i - 2][a0 + a][lane * 4]) = y[a];
            top = warp_max(top);
            if (lane == 0) atomicMax(&sm.top_v[i - 2], top);
        }
    };
    // products of the pairs: warps 0 .. 7 k_a . k_b, 8 .. 15 q_a . k_b; sixteen rows and every other block of sixteen columns
    // up to the diagonal a warp
    const int slab = (warp >> 1) & 3, odd = warp & 1;
    float dots[2][2][4] = {};
    auto products = [&]() {
        float low[2][2][4] = {}, two[2][2][4];
        const uint32_t rows_at = warp < 8 ? k_at : q_at;
        const int ra = slab * 16 + (lane & 15), rb = odd * 16 + (lane & 7) + (lane >> 4) * 8;
#pragma unroll 4
        for (int kk = 0; kk < CD / 16; kk++) {
            const uint32_t half = (kk >> 2) * TILE;
            const int ca = (kk & 3) * 2 + (lane >> 4), cb = (kk & 3) * 2 + ((lane >> 3) & 1);
            uint32_t ah[4], al[4];
            const uint32_t at = rows_at + half + ra * 128 + ((ca ^ (ra & 7)) << 4);
            pg_ldsm4(ah, at);
            pg_ldsm4(al, at + 2 * TILE);
#pragma unroll
            for (int j = 0; j < 2; j++) {
                if (2 * j + odd > slab) break;
                const int r = j * 32 + rb;
                uint32_t bh[4], bl[4];
                const uint32_t bat = k_at + half + r * 128 + ((cb ^ (r & 7)) << 4);
                pg_ldsm4(bh, bat);
                pg_ldsm4(bl, bat + 2 * TILE);
                if (!(kk & 1)) {
#pragma unroll
                    for (int n = 0; n < 2; n++)
#pragma unroll
                        for (int i = 0; i < 4; i++) two[j][n][i] = 0.0f;
                }
                mma_pair(two[j], low[j], ah, al, bh, bl);
                if (kk & 1) {
#pragma unroll
                    for (int n = 0; n < 2; n++)
#pragma unroll
                        for (int i = 0; i < 4; i++) dots[j][n][i] += two[j][n][i];
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int i = 0; i < 4; i++) dots[j][n][i] += low[j][n][i];
    };

#pragma unroll 1
    for (int h0 = g * rep; h0 < (g + 1) * rep; h0 += 2) {
        const int heads = min(2, (g + 1) * rep - h0);
        const bool keys = h0 == g * rep;                              // the first heads come with the queries and keys
        if (tid < 2) sm.bad[tid] = CT, sm.top_v[tid] = sm.largest[tid] = 0;
        __syncthreads();
        const int gate = (warp & 7) == 1 ? warp >> 3 : 2;             // warps 1 and 9 have no products of pairs: gates meanwhile
        if (gate < heads) load_gates(h0 + gate);
#pragma unroll 1
        for (int i = (keys ? 0 : 2) + (warp >> 3); i < 2 + heads; i += 2) convolve(i, h0);
        __syncthreads();
        if (keys) {
            uint4 *dst = reinterpret_cast<uint4 *>(group_data(s, w, chunk, g));
#pragma unroll
            for (int i = 0; i < GROUP_BYTES / 16 / 512; i++) dst[i * 512 + tid] = reinterpret_cast<const uint4 *>(sm.q)[i * 512 + tid];
            products();
        }
        if (gate < heads) gates(gate, h0 + gate);
        __syncthreads();
        const int bad = min(sm.bad[warp >> 3], sm.bad_k);             // (of the head whose substitution this warp does, which may lower it)
        // A (warps 0 .. 7; its diagonal blocks apart, in f32) and P
        for (int x = 0; x < heads; x++) {
            unsigned char *out = warp < 8 ? sm.a[x] : head_data(s, w, chunk, h0 + x) + P_AT;
            float *own = reinterpret_cast<float *>(head_data(s, w, chunk, h0 + x) + COEF_AT) + COEF_OWN;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int a = slab * 16 + (lane >> 2) + i * 8;
                const float ha = sm.l_hi[x][a], la = sm.l_lo[x][a], f = warp < 8 ? sm.beta[x][a] * OPERAND_INV : OPERAND_INV;
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const int block = 2 * j + odd;
                    if (warp < 8 && block > slab) continue;
#pragma unroll
                    for (int n = 0; n < 2; n++) {
                        const int b = block * 16 + n * 8 + (lane & 3) * 2;
                        float e0 = 0.0f, e1 = 0.0f;
                        if (block <= slab) {
                            const float2 hb = *reinterpret_cast<const float2 *>(&sm.l_hi[x][b]), lb = *reinterpret_cast<const float2 *>(&sm.l_lo[x][b]);
                            e0 = f * dots[j][n][2 * i] * expf((ha - hb.x) + (la - lb.x));
                            e1 = f * dots[j][n][2 * i + 1] * expf((ha - hb.y) + (la - lb.y));
                        }
                        if (warp < 8 && block == slab) {
                            *reinterpret_cast<float2 *>(&sm.diag[x][slab][a & 15][b & 15]) =
                                make_float2(b < a ? e0 * OPERAND_INV : 0.0f, b + 1 < a ? e1 * OPERAND_INV : 0.0f);
                        } else {
                            // (a token's own key is added in f32)
                            if (warp >= 8 && (b == a || b + 1 == a)) own[a] = (b == a ? e0 : e1) * OPERAND_INV;
                            uint32_t h, l;
                            split2(b < a ? e0 : 0.0f, b + 1 < a ? e1 : 0.0f, h, l);
                            unsigned char *p = out + a * 128 + (((b >> 3) ^ (a & 7)) << 4) + (b & 7) * 2;
                            *reinterpret_cast<uint32_t *>(p) = h;
                            *reinterpret_cast<uint32_t *>(p + TILE) = l;
                        }
                    }
                }
            }
        }
        __syncthreads();
        if (warp < 8) {
            // inverses of the diagonal blocks, a column a lane
            const int x = warp >> 2, J = warp & 3, c = lane & 15;
            if (x < heads) {
                float v[16];
#pragma unroll
                for (int a = 0; a < 16; a++) {
                    float sum = a == c ? 1.0f : 0.0f;
#pragma unroll
                    for (int q = 0; q < (a + 3) / 4; q++) {
                        const float4 r = *reinterpret_cast<const float4 *>(&sm.diag[x][J][a][q * 4]);
                        const float e[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
                        for (int b = 0; b < 4; b++)
                            if (q * 4 + b < a) sum = fmaf(-e[b], v[q * 4 + b], sum);
                    }
                    v[a] = sum;
                }
                if (lane < 16) {
#pragma unroll
                    for (int a = 0; a < 16; a++) {
                        const float e = a == c ? 0.0f : v[a] * OPERAND;              // (the diagonal is added in f32)
                        const __half h = __float2half_rn(e), l = __float2half_rn(e - __half2float(h));
                        *reinterpret_cast<__half *>(&sm.t[x][J][0][a * T_PITCH + c * 2]) = h;
                        *reinterpret_cast<__half *>(&sm.t[x][J][1][a * T_PITCH + c * 2]) = l;
                    }
                }
            }
        } else {
            // K~
#pragma unroll 1
            for (int x = 0; x < heads; x++) {
                unsigned char *out = head_data(s, w, chunk, h0 + x) + KT_AT;
#pragma unroll 2
                for (int i = tid - 256; i < 2 * TILE / 16; i += 256) {
                    const float r = sm.last[x][(i >> 3) & 63];
                    const uint4 kh = *reinterpret_cast<const uint4 *>(sm.k + i * 16), kl = *reinterpret_cast<const uint4 *>(sm.k + 2 * TILE + i * 16);
                    const uint32_t ph[4] = {kh.x, kh.y, kh.z, kh.w}, pl[4] = {kl.x, kl.y, kl.z, kl.w};
                    uint32_t oh[4], ol[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const float2 v = join2(ph[e], pl[e]);
                        split2(v.x * r, v.y * r, oh[e], ol[e]);
                    }
                    *reinterpret_cast<uint4 *>(out + i * 16) = make_uint4(oh[0], oh[1], oh[2], oh[3]);
                    *reinterpret_cast<uint4 *>(out + 2 * TILE + i * 16) = make_uint4(ol[0], ol[1], ol[2], ol[3]);
                }
            }
        }
        __syncthreads();
        // X^T of two heads, eight warps each: four have W, 32 columns a warp, four U0
        const int x = warp >> 3;
        if (x < heads) {
            const bool of_v = (warp & 4) != 0;
            const int d0 = (warp & 3) * 32;
            // (|u_a| <= 65 max |v|, and so are the sums in front of T: a state is at most the sum of the values behind it)
            const float2 scale = of_v ? scale_of(__uint_as_float(sm.top_v[x]), 7) : make_float2(1.0f, 1.0f);
            unsigned char *img = x == 0 ? sm.w0 : sm.w1;
            const uint32_t a_at = pg_smem(sm.a[x]), w_at = pg_smem(img);
            const int rn = (lane & 7) + (lane >> 4) * 8, cn = (lane >> 3) & 1;      // rows and chunks of ldmatrix: plain; transposed alike
            uint32_t top = 0;
            int worst = CT;
            // (loops are not unrolled: code that runs once is waited for)
#pragma unroll 1
            for (int d = d0; d < d0 + 32; d += 16) {
                uint32_t xh[3][4], xl[3][4];                                         // [block of rows] left operands
#pragma unroll 1
                for (int J = 0; J < 4; J++) {
                    const int r = J * 16 + rn;
                    float acc[2][4] = {}, low[2][4] = {};
#pragma unroll
                    for (int I = 0; I < 3; I++) {
                        if (I >= J) break;
                        uint32_t bh[4], bl[4];
                        const uint32_t at = a_at + r * 128 + (((2 * I + cn) ^ (r & 7)) << 4);
                        pg_ldsm4(bh, at);
                        pg_ldsm4(bl, at + TILE);
                        float one[2][4] = {};
                        mma_pair(one, low, xh[I], xl[I], bh, bl);
#pragma unroll
                        for (int n = 0; n < 2; n++)
#pragma unroll
                            for (int i = 0; i < 4; i++) acc[n][i] += one[n][i];
                    }
#pragma unroll
                    for (int n = 0; n < 2; n++)
#pragma unroll
                        for (int i = 0; i < 4; i++) acc[n][i] += low[n][i], low[n][i] = 0.0f;
                    uint32_t th[4], tl[4];
                    pg_ldsm4(th, pg_smem(sm.t[x][J][0]) + rn * T_PITCH + cn * 16);
                    pg_ldsm4(tl, pg_smem(sm.t[x][J][1]) + rn * T_PITCH + cn * 16);
                    const uint32_t tile_at = (d >> 6) * TILE + r * 128 + (((((d & 63) >> 3) + cn) ^ (r & 7)) << 4);
                    const int a0 = J * 16 + (lane & 3) * 2, col = d + (lane >> 2);  // of this lane: columns col and col + 8, rows a0, + 1, + 8, + 9
                    float2 z[2][2];
                    if (of_v) {
#pragma unroll
                        for (int n = 0; n < 2; n++)
#pragma unroll
                            for (int i = 0; i < 2; i++) z[n][i] = make_float2(sm.v[x][a0 + 8 * n][col + 8 * i], sm.v[x][a0 + 8 * n + 1][col + 8 * i]);
                    } else {
                        uint32_t kh[4], kl[4];
                        pg_ldsm4_t(kh, k_at + tile_at);
                        pg_ldsm4_t(kl, k_at + 2 * TILE + tile_at);
#pragma unroll
                        for (int n = 0; n < 2; n++)
#pragma unroll
                            for (int i = 0; i < 2; i++) z[n][i] = join2(kh[2 * n + i], kl[2 * n + i]);
                    }
                    // right side minus the sums
                    uint32_t yh[4], yl[4];
#pragma unroll
                    for (int n = 0; n < 2; n++) {
                        const int a = a0 + 8 * n;
                        const float2 be = *reinterpret_cast<const float2 *>(&sm.beta[x][a]);
                        const float2 c = of_v ? make_float2(scale.x, scale.x) : *reinterpret_cast<const float2 *>(&sm.c[x][a]);
                        const float f0 = be.x * c.x, f1 = be.y * c.y;
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            const float y0 = fmaf(f0, z[n][i].x, -OPERAND_INV * acc[n][2 * i]), y1 = fmaf(f1, z[n][i].y, -OPERAND_INV * acc[n][2 * i + 1]);
                            z[n][i] = make_float2(a < bad ? y0 : 0.0f, a + 1 < bad ? y1 : 0.0f);
                            split2(z[n][i].x, z[n][i].y, yh[2 * n + i], yl[2 * n + i]);
                        }
                    }
                    float o[2][4] = {};
                    mma_pair(o, low, yh, yl, th, tl);
                    uint32_t nh[4], nl[4];
#pragma unroll
                    for (int n = 0; n < 2; n++)
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            z[n][i].x = fmaf(o[n][2 * i] + low[n][2 * i], OPERAND_INV, z[n][i].x), z[n][i].y = fmaf(o[n][2 * i + 1] + low[n][2 * i + 1], OPERAND_INV, z[n][i].y);
                            split2(z[n][i].x, z[n][i].y, nh[2 * n + i], nl[2 * n + i]);
                        }
#pragma unroll
                    for (int I = 0; I < 3; I++)
                        if (I == J) {
#pragma unroll
                            for (int e = 0; e < 4; e++) xh[I][e] = nh[e], xl[I][e] = nl[e];
                        }
                    if (of_v) {
#pragma unroll
                        for (int n = 0; n < 2; n++)
#pragma unroll
                            for (int i = 0; i < 2; i++) {
                                const int a = a0 + 8 * n;
                                const float u[2] = {z[n][i].x * scale.y, z[n][i].y * scale.y};
#pragma unroll
                                for (int e = 0; e < 2; e++) {
                                    sm.v[x][a + e][col + 8 * i] = u[e];
                                    const bool fine = bits(u[e]) < NOT_FINITE;
                                    top = a + e < bad && fine ? max(top, bits(u[e])) : top;
                                    worst = a + e < bad && !fine ? min(worst, a + e) : worst;
                                }
                            }
                    } else {
                        stsm4_t(w_at + tile_at, nh);
                        stsm4_t(w_at + 2 * TILE + tile_at, nl);
                    }
                }
            }
            __syncwarp();
            unsigned char *out = head_data(s, w, chunk, h0 + x);
            if (of_v) {
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const int a = i * 4 + (lane >> 3), col = d0 + (lane & 7) * 4;
                    *reinterpret_cast<float4 *>(out + U0_AT + (a * CD + col) * 4) = *reinterpret_cast<const float4 *>(&sm.v[x][a][col]);
                }
                top = warp_max(top);
                if (lane == 0) atomicMax(&sm.largest[x], top);
                if (worst < CT) atomicMin(&sm.bad[x], worst);
            } else {
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const int a = (i & 7) * 8 + (lane >> 2);
                    const int at = (i >> 3) * 2 * TILE + (d0 >> 6) * TILE + a * 128 + (((((d0 & 63) >> 3) + (lane & 3)) ^ (a & 7)) << 4);
                    *reinterpret_cast<uint4 *>(out + W_AT + at) = *reinterpret_cast<const uint4 *>(img + at);
                }
            }
        }
        __syncthreads();
        if (tid < heads) {
            float *coef = reinterpret_cast<float *>(head_data(s, w, chunk, h0 + tid) + COEF_AT);
            coef[COEF_MAX] = __uint_as_float(sm.largest[tid]);
            coef[COEF_BAD] = __int_as_float(min(sm.bad[tid], sm.bad_k));
        }
        __syncthreads();
    }
}

// ---- the chain: grid (4, H, seqs); warps 0 .. 15 hold the state, warp 16 issues products, warp 17 copies ---------------
// A chunk is a chain of two products and what turns the sums of one into operands of the next; the third, and the writing of
// O, run beside it.  Operands come through a ring of 16 KB slots, seven a chunk, as soon as a slot is free, and are asked for in L2
// some chunks ahead (the four CTAs of a head share that).
//
// Bound by that chain: 4600 cycles a chunk, 1200 of them the first product, whose operands are 96 KB of shared memory.  4096 tokens of
// 32 heads 167 us; 145 with one accumulator a product (192 with two fixed buffers and eight warps); delta_scan_kernel, four tokens at a
// time, 820.
constexpr int CHAIN_WARPS = 16, CHAIN_THREADS = (CHAIN_WARPS + 2) * 32, COLS = 32, PART = 8;
constexpr int SLOT = 2 * TILE, SLOTS = 12, PER_CHUNK = 7, AHEAD = 3;
constexpr int S_SM = 0, U_SM = 2 * TILE, RING_SM = 3 * TILE, OWN_SM = RING_SM + SLOTS * SLOT, BARS_SM = OWN_SM + CT * COLS * 4;
constexpr int CHAIN_SMEM = BARS_SM + 256 + 1024;
// TMEM columns: four accumulators of [W; Q] S, two of K~^T U, two of P U, each [32 with the high part | 32 with the low part]
constexpr int ACC = 2 * COLS, WS_ACC = 0, KU_ACC = 4 * ACC, PU_ACC = 6 * ACC;

__device__ __forceinline__ void tmem_ld8_async(uint32_t taddr, uint32_t (&v)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}
// eight columns of a row of an operand tile [row][32 h | 32 l]
__device__ __forceinline__ void put_row(uint32_t tile, int row, int part, const float (&v)[PART], float scale)
{
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; i++) split2(v[2 * i] * scale, v[2 * i + 1] * scale, h[i], l[i]);
    const uint32_t at = tile + row * 128;
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at + ((part ^ (row & 7)) << 4)), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3]) : "memory");
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at + (((4 + part) ^ (row & 7)) << 4)), "r"(l[0]), "r"(l[1]), "r"(l[2]), "r"(l[3]) : "memory");
}
__device__ __forceinline__ uint32_t max4(uint4 v) { return max(max(v.x, v.y), max(v.z, v.w)); }
__device__ __forceinline__ void bulk_prefetch(const void *p, uint32_t bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

__global__ void __launch_bounds__(CHAIN_THREADS, 1)
    delta_chain_kernel(const DeltaShape s, const pg_batch bt, const DeltaWork w, float *state, int32_t *status, unsigned long long limit_ns)
{
    extern __shared__ uint8_t chain_raw[];
    __shared__ volatile int abort_flag;
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(16) uint32_t top_s[2][CHAIN_WARPS], top_u[2][CHAIN_WARPS / 2];
    pg_pdl_begin();
    const int seq = gridDim.z - 1 - blockIdx.z, h = blockIdx.y, g = h / (s.H / s.G), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = __ldcg(bt.d_seq_row0 + seq), T = __ldcg(bt.d_seq_row0 + seq + 1) - row0;
    if (T < DELTA_LONG) return;
    const uint32_t raw = pg_smem(chain_raw), base = (raw + 1023u) & ~1023u, full = base + BARS_SM, empty = full + 8 * SLOTS, bar_s = empty + 8 * SLOTS,
                   bar_u = bar_s + 8, bar_d1 = bar_s + 16, bar_d2 = bar_s + 24, bar_d3 = bar_s + 32;
    if (threadIdx.x == 0) {
        for (int i = 0; i < SLOTS; i++) {
            pg_mbar_init(full + 8 * i, 1);
            pg_mbar_init(empty + 8 * i, 1);
        }
        pg_mbar_init(bar_s, CHAIN_WARPS);
        pg_mbar_init(bar_u, CHAIN_WARPS);
        pg_mbar_init(bar_d1, 1);
        pg_mbar_init(bar_d2, 1);
        pg_mbar_init(bar_d3, 1);
        abort_flag = 0;
        pg_mbar_fence();
    }
    if (warp == CHAIN_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(pg_smem(&tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const int64_t chunk0 = first_chunk(row0);
    const int chunks = (T + CT - 1) / CT;
    const int64_t step = (int64_t)s.H * HEAD_BYTES + (int64_t)s.G * GROUP_BYTES;      // from chunk to chunk
    const unsigned char *mine = head_data(s, w, chunk0, h);

    if (warp == CHAIN_WARPS + 1) {
        if (lane == 0) {
            const unsigned char *hd = mine, *gd = group_data(s, w, chunk0, g);
            auto ask = [&](int i) {
                if (i >= chunks) return;
                bulk_prefetch(mine + i * step + blockIdx.x * (HEAD_BYTES / 4), HEAD_BYTES / 4);
                if (h % (s.H / s.G) == 0) bulk_prefetch(group_data(s, w, chunk0 + i, g) + blockIdx.x * (GROUP_BYTES / 4), GROUP_BYTES / 4);
            };
            for (int i = 1; i < AHEAD; i++) ask(i);
            bool ok = true;
            int slot = 0, phase = 0;
            for (int i = 0; ok && i < chunks; i++, hd += step, gd += step) {
                ask(i + AHEAD);
                for (int j = 0; j < PER_CHUNK; j++) {
                    const uint32_t bar = full + 8 * slot, at = base + RING_SM + slot * SLOT;
                    if (!(ok = pg_mbar_wait(empty + 8 * slot, phase ^ 1, &abort_flag, status, limit_ns))) break;
                    pg_mbar_expect(bar, SLOT);
                    // (the low parts come first)
                    if (j < 4) {                          // 64 rows of W, 64 of Q
                        pg_bulk_load(at, hd + W_AT + (j ^ 2) * TILE, TILE, bar);
                        pg_bulk_load(at + TILE, gd + (j ^ 2) * TILE, TILE, bar);
                    } else {                              // K~, its other part, P
                        pg_bulk_load(at, hd + KT_AT + (j < 6 ? (j ^ 1) - 4 : 2) * SLOT, SLOT, bar);
                    }
                    if (++slot == SLOTS) {
                        slot = 0;
                        phase ^= 1;
                    }
                }
            }
            if (!ok) {
                // give copies that are still in flight a bounded time to land before the CTA exits
                const unsigned long long at = pg_globaltimer_ns();
                while (pg_globaltimer_ns() - at < 2000000ull) {
                }
            }
        }
    } else if (warp == CHAIN_WARPS) {
        const uint32_t on = pg_elect();
        auto wait = [&](uint32_t bar, uint32_t parity) {
            const bool ok = (bool)__all_sync(0xffffffffu, pg_mbar_wait(bar, parity, &abort_flag, status, limit_ns));
            tc_fence_after();
            return ok;
        };
        // f16 operands: bits 7 and 10 are zero
        constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(2 * COLS >> 3) << 17) | (128u >> 4 << 24) | IDESC_B_MN_MAJOR;
        const uint64_t desc_s = make_smem_desc_mn(base + S_SM, TILE), desc_u = make_smem_desc_mn(base + U_SM, TILE);
        int slot = 0, phase = 0;
        auto next = [&]() {
            umma_commit(empty + 8 * slot, on);
            if (++slot == SLOTS) {
                slot = 0;
                phase ^= 1;
            }
        };
        bool ok = true;
        for (int i = 0; ok && i < chunks; i++) {
            if (!(ok = wait(bar_s, i & 1))) break;
#pragma unroll
            for (int t = 0; t < 4; t++) {
                if (!(ok = wait(full + 8 * slot, phase))) break;
                const uint64_t desc = make_smem_desc(base + RING_SM + slot * SLOT);
#pragma unroll
                for (int j = 0; j < 4; j++) 
                    umma_f16(tmem + WS_ACC + (t < 2 ? 0 : ((t & 1) * 2 + (j >> 1)) * ACC), desc + (uint64_t)(j * 2), desc_s + (uint64_t)(((t & 1) * 4 + j) * (2048 >> 4)), idesc,
                             (t | j) == 0 || (t == 3 && !(j & 1)) || (t == 2 && j == 2) ? 0u : 1u, on);
                if (t == 3) umma_commit(bar_d1, on);
                next();
            }
            if (!ok || !(ok = wait(bar_u, i & 1))) break;
#pragma unroll
            for (int t = 0; t < 2; t++) {
                if (!(ok = wait(full + 8 * slot, phase))) break;
                const uint64_t desc = make_smem_desc_mn(base + RING_SM + slot * SLOT, TILE);
#pragma unroll
                for (int j = 0; j < 4; j++)
                    umma_f16(tmem + KU_ACC + (t & (j >> 1)) * ACC, desc + (uint64_t)(j * (2048 >> 4)), desc_u + (uint64_t)(j * (2048 >> 4)), idesc | IDESC_A_MN_MAJOR,
                             (t | j) == 0 || (t == 1 && j == 2) ? 0u : 1u, on);
                if (t == 1) umma_commit(bar_d2, on);
                next();
            }
            if (!ok || !(ok = wait(full + 8 * slot, phase))) break;
            // the products of P are rows 64 .. 127 of the instruction, where the read-outs lie; rows 0 .. 63 are what lies in front
            const uint64_t desc = make_smem_desc(base + RING_SM + slot * SLOT - TILE);
#pragma unroll
            for (int t = 1; t >= 0; t--)
#pragma unroll
                for (int j = 0; j < 4; j++)
                    umma_f16(tmem + PU_ACC + (t == 0 ? (j >> 1) * ACC : 0), desc + (uint64_t)(t * (TILE >> 4) + j * 2), desc_u + (uint64_t)(j * (2048 >> 4)), idesc,
                             (t == 1 && j == 0) || (t == 0 && j == 2) ? 0u : 1u, on);
            umma_commit(bar_d3, on);
            next();
        }
    } else {
        const int q = warp & 3, part = warp >> 2, d = q * 32 + lane, a = d & 63;      // row of the state; row of the chunk
        const int col = blockIdx.x * COLS + part * PART;
        const bool outputs = q >= 2;                                                    // rows of Q, else of W
        const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16) + part * PART;
        auto wait = [&](uint32_t bar, uint32_t parity) { return (bool)__all_sync(0xffffffffu, pg_mbar_wait(bar, parity, &abort_flag, status, limit_ns)); };
        auto sums = [&](uint32_t at, float (&v)[PART]) {  // two accumulators: products with the high parts, and with the low ones
            uint32_t x[PART], y[PART], z[PART], t[PART];
            tmem_ld8_async(at, x);
            tmem_ld8_async(at + ACC, z);
            tmem_ld8_async(at + COLS, y);
            tmem_ld8_async(at + ACC + COLS, t);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < PART; j++) v[j] = (__uint_as_float(x[j]) + __uint_as_float(z[j])) + (__uint_as_float(y[j]) + __uint_as_float(t[j]));
        };
        auto largest_of = [&](const uint32_t (&v)[CHAIN_WARPS]) {
            const uint4 *p = reinterpret_cast<const uint4 *>(v);
            return __uint_as_float(max(max(max4(p[0]), max4(p[1])), max(max4(p[2]), max4(p[3]))));
        };
        float *st = state + (((int64_t)__ldcg(bt.d_seq_slot + seq) * s.H + h) * CD + d) * s.vs + col;
        float S[PART] = {};
        if (__ldcg(bt.d_pos + row0) > 0) {
#pragma unroll
            for (int j = 0; j < PART / 4; j++) {
                const float4 v = __ldcg(reinterpret_cast<const float4 *>(st) + j);
                S[4 * j] = v.x, S[4 * j + 1] = v.y, S[4 * j + 2] = v.z, S[4 * j + 3] = v.w;
            }
        }
        uint32_t top = 0;
#pragma unroll
        for (int j = 0; j < PART; j++) top = max(top, bits(S[j]));
        top = warp_max(top);
        if (lane == 0) top_s[0][warp] = top;
        asm volatile("bar.sync 1, %0;" ::"n"(CHAIN_WARPS * 32) : "memory");
        float2 scale_s = scale_of(largest_of(top_s[0]), 14);
        put_row(base + S_SM, d, part, S, scale_s.x);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) pg_mbar_arrive(bar_s);
        const unsigned char *next_chunk = mine;
        float u0[PART], n_c = 0.0f, n_own = 0.0f, n_last = 0.0f, n_max = 0.0f;
        float4 *mine_f32 = reinterpret_cast<float4 *>(chain_raw + (base - raw) + OWN_SM) + ((q & 1) * 4 + part) * 64 + lane;   // U of this lane's token
        int n_bad = CT;
        auto load_next = [&]() {                          // what the next chunk needs besides operands
            const float *coef = reinterpret_cast<const float *>(next_chunk + COEF_AT);
            if (outputs) {
                n_c = __ldcg(coef + a);
                n_own = __ldcg(coef + COEF_OWN + a);
            } else {
                const float4 *src = reinterpret_cast<const float4 *>(next_chunk + U0_AT) + (a * CD + col) / 4;
#pragma unroll
                for (int j = 0; j < PART / 4; j++) {
                    const float4 v = __ldcg(src + j);
                    u0[4 * j] = v.x, u0[4 * j + 1] = v.y, u0[4 * j + 2] = v.z, u0[4 * j + 3] = v.w;
                }
            }
            n_last = __ldcg(coef + COEF_LAST);
            n_max = __ldcg(coef + COEF_MAX);
            n_bad = __float_as_int(__ldcg(coef + COEF_BAD));
            next_chunk += step;
        };
        load_next();
        bool ok = true;
        for (int i = 0; i < chunks; i++) {
            const float c = n_c, own = n_own, last = n_last, u0_max = n_max;
            const int bad = n_bad;
            if (!(ok = wait(bar_s, i & 1))) break;
            const float largest = largest_of(top_s[i & 1]);
            // |U| <= |U0| + |w| |S column|, and a column of S has 128 elements
            const float2 scale_u = scale_of(u0_max + 12.0f * largest, 14);
            if (outputs) {                                // the sums of the read-outs in front may go
                tc_fence_before();
                if (lane == 0) pg_mbar_arrive(bar_u);
            }
            if (!(ok = wait(bar_d1, i & 1))) break;
            tc_fence_after();
            float o[PART];
            {
                float more[PART];
                sums(lanes + WS_ACC, o);
                sums(lanes + WS_ACC + 2 * ACC, more);
#pragma unroll
                for (int j = 0; j < PART; j++) o[j] += more[j];
            }
            if (!outputs) {
                const float inv = scale_s.y * OPERAND_INV;
                uint32_t most = 0;
#pragma unroll
                for (int j = 0; j < PART; j++) {
                    o[j] = a < bad ? fmaf(-inv, o[j], u0[j]) : 0.0f;
                    most = max(most, bits(o[j]));
                }
                put_row(base + U_SM, a, part, o, scale_u.x);
#pragma unroll
                for (int j = 0; j < PART / 4; j++) mine_f32[j * 32] = make_float4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
                most = warp_max(most);
                if (lane == 0) top_u[i & 1][q * 4 + part] = most;
                tc_fence_before();
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) pg_mbar_arrive(bar_u);
            } else {
                const float f = c * scale_s.y * OPERAND_INV;
#pragma unroll
                for (int j = 0; j < PART; j++) o[j] *= f;
            }
            if (i + 1 < chunks) load_next();
            if (!(ok = wait(bar_u, i & 1))) break;
            {
                const uint4 *p = reinterpret_cast<const uint4 *>(top_u[i & 1]);
                scale_s = scale_of(fmaf(64.5f, __uint_as_float(max(max4(p[0]), max4(p[1]))), largest), 14);
            }
            if (outputs) {
#pragma unroll
                for (int j = 0; j < PART / 4; j++) {
                    const float4 u = mine_f32[j * 32];
                    o[4 * j] = fmaf(own, u.x, o[4 * j]), o[4 * j + 1] = fmaf(own, u.y, o[4 * j + 1]);
                    o[4 * j + 2] = fmaf(own, u.z, o[4 * j + 2]), o[4 * j + 3] = fmaf(own, u.w, o[4 * j + 3]);
                }
            }
            const float inv_u = scale_u.y * OPERAND_INV;
            if (!(ok = wait(bar_d2, i & 1))) break;
            tc_fence_after();
            {
                float v[PART];
                sums(lanes + KU_ACC, v);
                top = 0;
#pragma unroll
                for (int j = 0; j < PART; j++) {
                    S[j] = fmaf(last, S[j], v[j] * inv_u);
                    if (bad < CT) S[j] = __uint_as_float(0x7fc00000u);
                    top = max(top, bits(S[j]));
                }
            }
            if (i + 1 < chunks) {
                put_row(base + S_SM, d, part, S, scale_s.x);
                top = warp_max(top);
                if (lane == 0) top_s[(i + 1) & 1][warp] = top;
                tc_fence_before();
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) pg_mbar_arrive(bar_s);
            }
            if (outputs) {
                if (!(ok = wait(bar_d3, i & 1))) break;
                tc_fence_after();
                float v[PART];
                sums(lanes + PU_ACC, v);
                if (i * CT + a < T) {
                    float4 *dst = reinterpret_cast<float4 *>(w.o + ((int64_t)(row0 + i * CT + a) * s.H + h) * CD + col);
#pragma unroll
                    for (int j = 0; j < PART; j++) {
                        o[j] = fmaf(inv_u, v[j], o[j]);
                        if (a >= bad) o[j] = __uint_as_float(0x7fc00000u);
                    }
#pragma unroll
                    for (int j = 0; j < PART / 4; j++) dst[j] = make_float4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
                }
            }
        }
        if (ok) {
#pragma unroll
            for (int j = 0; j < PART / 4; j++) reinterpret_cast<float4 *>(st)[j] = make_float4(S[4 * j], S[4 * j + 1], S[4 * j + 2], S[4 * j + 3]);
        }
        tc_fence_before();
    }
    __syncwarp();
    __syncthreads();
    if (warp == CHAIN_WARPS) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

template <int TAPS>
int32_t run_chunks(pg_ctx *ctx, const DeltaShape &s, const pg_batch *bt, const float *proj, int64_t ldp, const float *ring, const DeltaWork &w)
{
    static std::atomic<uint64_t> set{0};
    PG_CUDA(pg_max_smem_once(delta_chunk_kernel<TAPS>, (int)sizeof(ChunkSmem), ctx->device, set));
    return launch_pdl(ctx, delta_chunk_kernel<TAPS>, dim3((unsigned)s.G, (unsigned)((bt->max_len + CT - 1) / CT), (unsigned)bt->seqs), dim3(512),
                      sizeof(ChunkSmem), s, *bt, proj, ldp, ring, w);
}

}  // namespace

// Heads of 128 x 128 with short convolutions (a thread keeps their inputs in registers) whose rows start on 16-byte boundaries.
bool pgk_delta_chunk_supports(const DeltaShape &s, const float *proj, int64_t ldp, const float *ring, const float *state)
{
    return s.D == CD && s.V == CD && s.taps >= 2 && s.taps <= 4 && ldp % 4 == 0 &&
           (((uintptr_t)proj | (uintptr_t)ring | (uintptr_t)state | (uintptr_t)s.conv) & 15) == 0;
}

int64_t pgk_delta_chunk_floats(int64_t kv_heads, int64_t heads, int64_t dim, int64_t vdim, int64_t taps, int64_t max_rows)
{
    if (dim != CD || vdim != CD || taps < 2 || taps > 4 || max_rows < DELTA_LONG) return 0;
    return (first_chunk(max_rows) + 1) * ((heads * HEAD_BYTES + kv_heads * GROUP_BYTES) / 4) + 256;
}

int32_t pgk_delta_chunk(pg_ctx *ctx, const DeltaShape &s, const pg_batch *bt, const float *proj, int64_t ldp, const float *ring, const DeltaWork &w,
                        float *state)
{
    const int32_t rc = s.taps == 2   ? run_chunks<2>(ctx, s, bt, proj, ldp, ring, w)
                       : s.taps == 3 ? run_chunks<3>(ctx, s, bt, proj, ldp, ring, w)
                                     : run_chunks<4>(ctx, s, bt, proj, ldp, ring, w);
    if (rc != PG_OK) return rc;
    static std::atomic<uint64_t> set{0};
    PG_CUDA(pg_max_smem_once(delta_chain_kernel, CHAIN_SMEM, ctx->device, set));
    return launch_pdl(ctx, delta_chain_kernel, dim3(CD / COLS, (unsigned)s.H, (unsigned)bt->seqs), dim3(CHAIN_THREADS), (size_t)CHAIN_SMEM, s, *bt, w, state,
                      ctx->d_status, ctx->wait_limit_ns);
}
