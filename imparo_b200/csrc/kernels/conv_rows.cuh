// A short causal convolution on every channel of 32-bit rows, for ragged batches (channel_conv.cu, mamba2.cu): a thread owns
// four neighbouring channels of R consecutive rows of the batch and slides along them, so that an input row is read 1 + (TAPS -
// 1) / R times instead of TAPS times, 16 bytes at a time and all of a thread's rows in flight together.
#pragma once
#include "common.cuh"

namespace imparo {

struct ConvRows {
    const float* in; size_t stride; int col0, channels;         // input rows, the convolved stretch's first column
    const float* w;                                             // [channels, TAPS], the last tap on the row itself
    const float* in_bias; const float* out_bias;                // added to every input of this launch / to the sum; or null
    const float* state;                                         // [slots, TAPS - 1, channels], oldest first
    const int* item_row_start; const int* item_of_token; const int* item_slot;
    int n_slots, n_tok;
    float* out; size_t out_stride;
    int silu;
    int kernel;                                                 // the number a bad slot is reported under
    int* status;
};

// What the vector form needs; a caller with anything else keeps a thread per (row, channel).
static inline bool conv_rows_take(const ConvRows& p, int taps) {
    return taps >= 2 && taps <= 4 && p.channels % 4 == 0 && p.col0 % 4 == 0 && p.stride % 4 == 0 && p.out_stride % 4 == 0 &&
           (((uintptr_t)p.in | (uintptr_t)p.w | (uintptr_t)p.state | (uintptr_t)p.out | (uintptr_t)p.in_bias | (uintptr_t)p.out_bias) & 15) == 0;
}

// Rows per thread: four once that still leaves every SM 512 threads, else one.
static inline int conv_rows_per_thread(int n_tok, int channels) { return (long long)n_tok * (channels / 4) >= 4LL * 148 * 512 ? 4 : 1; }

// c: first of the thread's four channels, t0: its first row.  Waits for the previous kernel after its weights are loaded.
template <int TAPS, int R>
__device__ __forceinline__ void conv_rows(const ConvRows& p, int c, int t0) {
    constexpr int H = TAPS - 1;
    const bool on = c < p.channels && t0 < p.n_tok;
    float wt[4 * TAPS];
    float4 ib = make_float4(0.f, 0.f, 0.f, 0.f), ob = ib;
    if (on) {
#pragma unroll
        for (int i = 0; i < TAPS; ++i) {
            const float4 f = __ldg(reinterpret_cast<const float4*>(p.w + (size_t)c * TAPS) + i);
            wt[4 * i] = f.x; wt[4 * i + 1] = f.y; wt[4 * i + 2] = f.z; wt[4 * i + 3] = f.w;
        }
        if (p.in_bias) ib = *reinterpret_cast<const float4*>(p.in_bias + c);
        if (p.out_bias) ob = *reinterpret_cast<const float4*>(p.out_bias + c);
    }
    // whose rows these are: from the batch description, so before the wait, and for all rows at once
    int slot_r[R], j_r[R];
    if (on) {
        int item_r[R];
#pragma unroll
        for (int r = 0; r < R; ++r) item_r[r] = p.item_of_token[min(t0 + r, p.n_tok - 1)];
#pragma unroll
        for (int r = 0; r < R; ++r) { j_r[r] = t0 + r - p.item_row_start[item_r[r]]; slot_r[r] = p.item_slot[item_r[r]]; }
    }
    pdl_wait();
    if (!on) return;
    float4 u[H + R];
#pragma unroll
    for (int e = 0; e < H + R; ++e) {
        const int t = t0 - H + e;
        u[e] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t >= 0 && t < p.n_tok) {
            const float4 f = *reinterpret_cast<const float4*>(p.in + (size_t)t * p.stride + p.col0 + c);
            u[e] = make_float4(f.x + ib.x, f.y + ib.y, f.z + ib.z, f.w + ib.w);
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int t = t0 + r;
        if (t >= p.n_tok) break;
        const int j = j_r[r], slot = slot_r[r];
        if (slot < 0 || slot >= p.n_slots) {
            if (c == 0) report(p.status, IMPARO_ST_SLOT_RANGE, p.kernel, t, slot);
            continue;
        }
        float4 acc = ob;
#pragma unroll
        for (int k = 0; k < TAPS; ++k) {
            float4 v = u[r + k];
            if (j < H - k)                                       // before the portion: the slot's rows
                v = *reinterpret_cast<const float4*>(p.state + ((size_t)slot * H + j + k) * p.channels + c);
            acc.x += wt[k] * v.x;
            acc.y += wt[TAPS + k] * v.y;
            acc.z += wt[2 * TAPS + k] * v.z;
            acc.w += wt[3 * TAPS + k] * v.w;
        }
        if (p.silu) acc = make_float4(silu(acc.x), silu(acc.y), silu(acc.z), silu(acc.w));
        *reinterpret_cast<float4*>(p.out + (size_t)t * p.out_stride + c) = acc;
    }
}

}  // namespace imparo
