// What the kernels of the delta rule share: the layer's sizes and parameters, the convolution, the workspace.
#pragma once

#include "pg_lm.cuh"

struct DeltaShape {
    int H, G, D, V, taps, C;        // C: convolution channels 2 G D + H V
    int vs;                         // state row stride
    float eps, unit_eps, qscale;
    const float *conv, *a_log, *dt_bias, *norm;
};

__device__ __forceinline__ float softplus(float x) { return x > 20.0f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float log_decay(float a, float a_log, float dt_bias) { return -expf(a_log) * softplus(a + dt_bias); }

// one channel of the convolution at position pos; row: this token's input row, t: tokens of the same sequence and step
// in front of it; older inputs come from the ring
__device__ __forceinline__ float conv_at(const DeltaShape &s, const float *row, int64_t ldp, const float *ring, int c, int t, int pos)
{
    float acc = 0.0f;
    for (int j = 0; j < s.taps; j++) {
        const int back = s.taps - 1 - j;                  // tokens back
        float x = 0.0f;
        if (back <= t)
            x = __ldcg(row - (int64_t)back * ldp + c);
        else if (back <= pos)
            x = __ldcg(ring + (int64_t)((pos - back) % s.taps) * s.C + c);
        acc = fmaf(__ldg(s.conv + (int64_t)j * s.C + c), x, acc);
    }
    return pg_silu(acc);
}

// rows q [G D] | k [G D] | v [H V] | o [H V] per token, coefficients of blocks of four tokens (pg_delta.cu), and what
// pg_delta_chunk.cu makes of chunks of 64
struct DeltaWork {
    float *q, *k, *v, *o, *coef;
    unsigned char *chunks;
};

// pg_delta_chunk.cu: sequences of at least DELTA_LONG tokens of a step, o for their rows and their states.  From there on the chunks are
// the faster form: 64 / 100 / 128 / 192 tokens of 32 heads 48 / 51 / 51 / 54 us against 48 / 56 / 64 / 78 by blocks of four, of 16 heads 43 / 44 / 45 / 48
// against 35 / 42 / 50 / 62; sixty sequences of 65 tokens 843 against 724, eight of 64 tokens 98 against 116.  Below that a chunk that is
// hardly filled takes as much workspace as a full one, and the outputs' error is 1 to 2 % above that of blocks of four.
constexpr int DELTA_CHUNK = 64, DELTA_LONG = 128;
bool pgk_delta_chunk_supports(const DeltaShape &s, const float *proj, int64_t ldp, const float *ring, const float *state);
int64_t pgk_delta_chunk_floats(int64_t kv_heads, int64_t heads, int64_t dim, int64_t vdim, int64_t taps, int64_t max_rows);
int32_t pgk_delta_chunk(pg_ctx *ctx, const DeltaShape &s, const pg_batch *bt, const float *proj, int64_t ldp, const float *ring, const DeltaWork &w,
                        float *state);
