// Gated causal depthwise convolution with per-request rolling state, for a ragged batch.
//
// Formula (zeraix/imparo, imparo-cpu/src/ops.rs:109-167; imparo-cuda/native/lfm2_ops.cuh:48-97):
//   rows of bcx are [b | c | x];  v[t] = b[t]*x[t];  seq = state ++ v  (state = the taps-1
//   raw v before this portion, oldest first, zeros for a fresh request);
//   sum[t] = sum_k w[ch,k] * seq[t+k]  (tap 0 meets the oldest value);  y[t] = c[t]*sum[t];
//   state' = the last taps-1 values of seq (partly the old state when the portion is
//   shorter than taps-1).  A bias, which the reference does not have, is added to sum
//   before the gate.
//
// One launch does output and state.  A thread owns (token, channel) — or, for prompt portions, 16 bytes
// of channels of one or several tokens.  Tokens at least taps-1 into their portion need only bcx.
// The thread of a portion's FIRST token also computes the outputs of the next taps-2 tokens and
// then writes the new state; it reads the whole old state into registers first, and no other
// thread touches that state, so the update in place is race-free.  The input may also be the
// split partials of the product before (summed here), see ConvIn.
#include "common.cuh"

namespace imparo {

constexpr int MAX_TAPS = 16;

// The input rows [b | c | x]: a stored tensor of T, or the partial results of a product that was
// cut along K (float [parts][tokens][3 * width]).  Partials are summed in split order and rounded
// to T, which is what the product's own fold would have stored.
// MODE 0: a tensor; 1: at most four partials (straight-line code, so that the loads of the
// several values a thread needs are all in flight together); 2: any number of partials.
template <typename T, int MODE>
struct ConvIn {
    const T* rows;
    const float* part;
    int parts;
    size_t part_stride;
    __device__ __forceinline__ float at(size_t idx) const {
        if (MODE == 0) return to_f32(rows[idx]);
        float acc = 0.f;
        if (MODE == 1) {
            float v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = u < parts ? __ldcg(part + (size_t)u * part_stride + idx) : 0.f;
#pragma unroll
            for (int u = 0; u < 4; ++u) if (u < parts) acc += v[u];
        } else {
            for (int s0 = 0; s0 < parts; s0 += 8) {
                float v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = s0 + u < parts ? __ldcg(part + (size_t)(s0 + u) * part_stride + idx) : 0.f;
#pragma unroll
                for (int u = 0; u < 8; ++u) if (s0 + u < parts) acc += v[u];
            }
        }
        return to_f32(from_f32<T>(acc));
    }
};

// The thread of a portion's first token, for one channel: outputs of the first min(n, taps-1)
// tokens from the old state, then the new state.  wk: this channel's taps (loaded by the caller,
// before it waited for the previous kernel).  Everything the outputs need is requested in one
// batch of loads: a decode token costs one round trip to memory after the wait.
template <typename T, int MODE>
__device__ __forceinline__ void conv_portion_head(const ConvIn<T, MODE>& bcx, const float* wk, float b0,
                                                  float* __restrict__ state, int slot,
                                                  T* __restrict__ y, int item, int start, int n, int ch,
                                                  int width, int taps, int n_slots, int* status) {
    const int hist = taps - 1;
    const size_t stride = (size_t)3 * width;
    if (slot < 0 || slot >= n_slots) {
        if (ch == 0) report(status, IMPARO_ST_SLOT_RANGE, 4, item, slot);
        return;
    }
    float* st = state + (size_t)slot * hist * width + ch;
    // seq[e], e in [0, hist + m): the old state then the first m values of this portion
    float seq[2 * MAX_TAPS], gate[MAX_TAPS];
    const int m = min(n, hist);
#pragma unroll
    for (int e = 0; e < MAX_TAPS; ++e) if (e < hist) seq[e] = st[(size_t)e * width];
#pragma unroll
    for (int e = 0; e < MAX_TAPS; ++e) {
        if (e < m) {
            const size_t r = (size_t)(start + e) * stride;
            seq[hist + e] = bcx.at(r + ch) * bcx.at(r + 2 * (size_t)width + ch);
            gate[e] = bcx.at(r + width + ch);
        }
    }
    for (int e = 0; e < m; ++e) {
        float acc = 0.f;
        for (int k = 0; k < taps; ++k) acc += wk[k] * seq[e + k];
        acc += b0;
        y[(size_t)(start + e) * width + ch] = from_f32<T>(gate[e] * acc);
    }
    // new state slot s = seq_full[n + s]
    for (int s = 0; s < hist; ++s) {
        const int e = n + s;
        float v;
        if (e < hist + m) {
            v = seq[e];
        } else {
            const size_t r = (size_t)(start + e - hist) * stride;
            v = bcx.at(r + ch) * bcx.at(r + 2 * (size_t)width + ch);
        }
        st[(size_t)s * width] = v;
    }
}

// The batch description (which request a token belongs to, where its portion starts, its state
// slot) comes from the host before the step and the taps are weights: both are read before the
// wait on the previous kernel, so that after it only activations and state remain to be fetched.
template <typename T, int MODE>
__global__ void gated_conv_kernel(const ConvIn<T, MODE> bcx, const float* __restrict__ w,
                                  const float* __restrict__ bias, float* __restrict__ state,
                                  const int* __restrict__ item_row_start, const int* __restrict__ item_of_token,
                                  const int* __restrict__ item_slot, T* __restrict__ y,
                                  int n_tok, int width, int taps, int n_slots, int* status) {
    pdl_trigger();
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)n_tok * width) return;
    const int t = (int)(idx / width), ch = (int)(idx % width);
    const int item = item_of_token[t];
    const int start = item_row_start[item];
    const int n = item_row_start[item + 1] - start;
    const int rel = t - start;
    const int hist = taps - 1;
    if (rel > 0 && rel < hist) return;           // written by the thread of the portion's first token
    const int slot = rel == 0 ? item_slot[item] : 0;
    const size_t stride = (size_t)3 * width;
    float wk[MAX_TAPS];
#pragma unroll
    for (int k = 0; k < MAX_TAPS; ++k) wk[k] = k < taps ? w[(size_t)ch * taps + k] : 0.f;
    const float b0 = bias ? bias[ch] : 0.f;
    pdl_wait();

    if (rel >= hist) {
        float v[MAX_TAPS];
#pragma unroll
        for (int k = 0; k < MAX_TAPS; ++k) {
            if (k < taps) {
                const size_t r = (size_t)(t - hist + k) * stride;
                v[k] = bcx.at(r + ch) * bcx.at(r + 2 * (size_t)width + ch);
            }
        }
        const float gate = bcx.at((size_t)t * stride + width + ch);
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < MAX_TAPS; ++k) if (k < taps) acc += wk[k] * v[k];
        acc += b0;
        y[(size_t)t * width + ch] = from_f32<T>(gate * acc);
        return;
    }
    if (n == 1 && slot >= 0 && slot < n_slots) {
        // a decode token: everything in registers, one batch of loads
        float* st = state + (size_t)slot * hist * width + ch;
        float sv[MAX_TAPS];
#pragma unroll
        for (int e = 0; e < MAX_TAPS - 1; ++e) sv[e] = e < hist ? st[(size_t)e * width] : 0.f;
        const size_t r = (size_t)t * stride;
        const float bx = bcx.at(r + ch) * bcx.at(r + 2 * (size_t)width + ch);
        const float gate = bcx.at(r + width + ch);
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < MAX_TAPS; ++k) {
            if (k < hist) acc += wk[k] * sv[k];
            else if (k == hist) acc += wk[k] * bx;
        }
        acc += b0;
        y[(size_t)t * width + ch] = from_f32<T>(gate * acc);
#pragma unroll
        for (int e = 0; e < MAX_TAPS - 1; ++e)
            if (e < hist) st[(size_t)e * width] = (e + 1 < hist) ? sv[e + 1] : bx;
        return;
    }
    conv_portion_head<T, MODE>(bcx, wk, b0, state, slot, y, item, start, n, ch, width, taps, n_slots, status);
}

// 16 bytes of channels at a time, for prompt-sized batches and two to four taps: a thread owns V consecutive channels (8
// bfloat16, 4 float) of R consecutive tokens of the batch and slides along them, all its rows in flight together.  Same sums in
// the same order as gated_conv_kernel.  The thread that has a portion's first token makes the outputs of the portion's first
// taps-1 tokens and the new state for its V channels in two batches of loads (channel by channel through conv_portion_head they
// were eight to sixteen dependent trips to memory, most of a short prompt's 9 us).  131 tokens of 2,048 channels (B200): 9.1 ->
// 4.1 us; 2,048 tokens: 14.2 -> 13.8 us; float, 1,000 tokens of 1,024 channels: 28.5 -> 5.2 us.
template <typename T> struct Wide;
template <> struct Wide<__nv_bfloat16> {
    static constexpr int V = 8;
    uint4 q;
    __device__ __forceinline__ void get(float (&f)[8]) const {
        const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
        for (int i = 0; i < 4; ++i) { const float2 v = __bfloat1622float2(p[i]); f[2 * i] = v.x; f[2 * i + 1] = v.y; }
    }
    __device__ __forceinline__ void set(const float (&f)[8]) {
        __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    }
};
template <> struct Wide<float> {
    static constexpr int V = 4;
    float4 q;
    __device__ __forceinline__ void get(float (&f)[4]) const { f[0] = q.x; f[1] = q.y; f[2] = q.z; f[3] = q.w; }
    __device__ __forceinline__ void set(const float (&f)[4]) { q = make_float4(f[0], f[1], f[2], f[3]); }
};

template <typename T, int TAPS, int R>
__global__ void __launch_bounds__(256)
gated_conv_rows_kernel(const T* __restrict__ bcx, const float* __restrict__ w, const float* __restrict__ bias,
                       float* __restrict__ state, const int* __restrict__ item_row_start, const int* __restrict__ item_of_token,
                       const int* __restrict__ item_slot, T* __restrict__ y, int n_tok, int width, int n_slots, int* status) {
    constexpr int V = Wide<T>::V, H = TAPS - 1;
    using W = Wide<T>;
    pdl_trigger();
    const int per_row = width / V;
    const size_t idx = (size_t)blockIdx.x * 256 + threadIdx.x;
    const int t0 = (int)(idx / per_row) * R, ch = (int)(idx % per_row) * V;
    if (t0 >= n_tok) return;
    // the thread's tap weights: w[(ch + i) * taps + k], V * TAPS consecutive floats
    float wv[V * TAPS], b0[V];
    const float4* wp = reinterpret_cast<const float4*>(w + (size_t)ch * TAPS);
#pragma unroll
    for (int e = 0; e < V * TAPS / 4; ++e) {
        const float4 f = __ldg(wp + e);
        wv[4 * e] = f.x; wv[4 * e + 1] = f.y; wv[4 * e + 2] = f.z; wv[4 * e + 3] = f.w;
    }
#pragma unroll
    for (int i = 0; i < V; ++i) b0[i] = bias ? bias[ch + i] : 0.f;
    const size_t stride = (size_t)3 * width;
    auto put = [&](int t, const W& gate, const float (&v)[TAPS][V]) {
        float c[V], o[V];
        gate.get(c);
#pragma unroll
        for (int i = 0; i < V; ++i) {
            float acc = 0.f;
#pragma unroll
            for (int k = 0; k < TAPS; ++k) acc += wv[i * TAPS + k] * v[k][i];
            o[i] = c[i] * (acc + b0[i]);
        }
        W out;
        out.set(o);
        *reinterpret_cast<W*>(y + (size_t)t * width + ch) = out;
    };
    auto product = [&](const W& b, const W& x, float (&v)[V]) {
        float bf[V], xf[V];
        b.get(bf); x.get(xf);
#pragma unroll
        for (int i = 0; i < V; ++i) v[i] = bf[i] * xf[i];
    };
    auto at = [&](int t, int part) { return *reinterpret_cast<const W*>(bcx + (size_t)t * stride + (size_t)part * width + ch); };
    // whose rows these are: from the batch description, so before the wait, and for all rows at once
    int item_r[R], start_r[R];
#pragma unroll
    for (int r = 0; r < R; ++r) item_r[r] = item_of_token[min(t0 + r, n_tok - 1)];
#pragma unroll
    for (int r = 0; r < R; ++r) start_r[r] = item_row_start[item_r[r]];
    pdl_wait();
    W b[H + R], x[H + R], c[R];
#pragma unroll
    for (int e = 0; e < H + R; ++e) {
        const int t = t0 - H + e;
        if (t >= 0 && t < n_tok) { b[e] = at(t, 0); x[e] = at(t, 2); if (e >= H) c[e - H] = at(t, 1); }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int t = t0 + r;
        if (t >= n_tok) break;
        const int item = item_r[r], start = start_r[r];
        const int rel = t - start;
        if (rel >= H) {
            float v[TAPS][V];
#pragma unroll
            for (int k = 0; k < TAPS; ++k) product(b[r + k], x[r + k], v[k]);
            put(t, c[r], v);
            continue;
        }
        if (rel > 0) continue;                       // by the thread that has the portion's first token
        const int n = item_row_start[item + 1] - start, slot = item_slot[item], m = min(n, H);
        if (slot < 0 || slot >= n_slots) {
            if (ch == 0) report(status, IMPARO_ST_SLOT_RANGE, 4, item, slot);
            continue;
        }
        // seq: the old state, then the portion's first rows; last: the rows the new state ends with
        float* st = state + (size_t)slot * H * width + ch;
        float seq[2 * H][V], last[H][V];
        W hb[H], hx[H], hc[H], lb[H], lx[H];
#pragma unroll
        for (int e = 0; e < H; ++e) {
#pragma unroll
            for (int i = 0; i < V; i += 4) {
                const float4 f = *reinterpret_cast<const float4*>(st + (size_t)e * width + i);
                seq[e][i] = f.x; seq[e][i + 1] = f.y; seq[e][i + 2] = f.z; seq[e][i + 3] = f.w;
            }
            if (e < m) { hb[e] = at(start + e, 0); hx[e] = at(start + e, 2); hc[e] = at(start + e, 1); }
            const int from = n - H + e;              // the new state's entry e is this row of the portion, or an old entry
            if (from >= 0) { lb[e] = at(start + from, 0); lx[e] = at(start + from, 2); }
        }
#pragma unroll
        for (int e = 0; e < H; ++e) {
            if (e < m) product(hb[e], hx[e], seq[H + e]);
            const int from = n - H + e;
            if (from >= 0) product(lb[e], lx[e], last[e]);
            else {
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    last[e][i] = 0.f;
#pragma unroll
                    for (int o = 0; o < H; ++o) if (o == H + from) last[e][i] = seq[o][i];
                }
            }
        }
#pragma unroll
        for (int e = 0; e < H; ++e) {
            if (e < m) {
                float v[TAPS][V];
#pragma unroll
                for (int k = 0; k < TAPS; ++k)
#pragma unroll
                    for (int i = 0; i < V; ++i) v[k][i] = seq[e + k][i];
                put(start + e, hc[e], v);
            }
        }
#pragma unroll
        for (int e = 0; e < H; ++e)
#pragma unroll
            for (int i = 0; i < V; i += 4)
                *reinterpret_cast<float4*>(st + (size_t)e * width + i) = make_float4(last[e][i], last[e][i + 1], last[e][i + 2], last[e][i + 3]);
    }
}

// bfloat16 with a width that is a multiple of 8 and any number of taps, for prompt-sized batches: a thread owns eight
// consecutive channels of one token and moves 16 bytes at a time.  Same sums in the same order as gated_conv_kernel; the thread
// of a portion's first token walks its eight channels through conv_portion_head.
__global__ void gated_conv_bf16x8_kernel(const __nv_bfloat16* __restrict__ bcx, const float* __restrict__ w,
                                         const float* __restrict__ bias, float* __restrict__ state,
                                         const int* __restrict__ item_row_start, const int* __restrict__ item_of_token,
                                         const int* __restrict__ item_slot, __nv_bfloat16* __restrict__ y,
                                         int n_tok, int width, int taps, int n_slots, int* status) {
    pdl_trigger();
    const int per_row = width >> 3;
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)n_tok * per_row) return;
    const int t = (int)(idx / per_row), ch = (int)(idx % per_row) << 3;
    const int hist = taps - 1;
    const int item = item_of_token[t];
    const int start = item_row_start[item];
    const int rel = t - start;
    pdl_wait();
    if (rel < hist) {
        if (rel != 0) return;
        const int n = item_row_start[item + 1] - start;
        const int slot = item_slot[item];
        for (int i = 0; i < 8; ++i) {
            float wk[MAX_TAPS];
            for (int k = 0; k < taps; ++k) wk[k] = w[(size_t)(ch + i) * taps + k];
            conv_portion_head<__nv_bfloat16, 0>(ConvIn<__nv_bfloat16, 0>{bcx, nullptr, 0, 0}, wk, bias ? bias[ch + i] : 0.f, state, slot, y, item, start, n,
                                             ch + i, width, taps, n_slots, status);
        }
        return;
    }
    const size_t stride = (size_t)3 * width;
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
    const uint4 c = *reinterpret_cast<const uint4*>(bcx + (size_t)t * stride + width + ch);
    for (int k = 0; k < taps; ++k) {
        const __nv_bfloat16* r = bcx + (size_t)(t - hist + k) * stride;
        const uint4 b = *reinterpret_cast<const uint4*>(r + ch);
        const uint4 x = *reinterpret_cast<const uint4*>(r + 2 * (size_t)width + ch);
        const __nv_bfloat162* bp = reinterpret_cast<const __nv_bfloat162*>(&b);
        const __nv_bfloat162* xp = reinterpret_cast<const __nv_bfloat162*>(&x);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 bf = __bfloat1622float2(bp[i]), xf = __bfloat1622float2(xp[i]);
            acc[2 * i] += w[(size_t)(ch + 2 * i) * taps + k] * (bf.x * xf.x);
            acc[2 * i + 1] += w[(size_t)(ch + 2 * i + 1) * taps + k] * (bf.y * xf.y);
        }
    }
    if (bias) {
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += bias[ch + i];
    }
    const __nv_bfloat162* cp = reinterpret_cast<const __nv_bfloat162*>(&c);
    uint4 out;
    __nv_bfloat162* op = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 cf = __bfloat1622float2(cp[i]);
        op[i] = __floats2bfloat162_rn(cf.x * acc[2 * i], cf.y * acc[2 * i + 1]);
    }
    *reinterpret_cast<uint4*>(y + (size_t)t * width + ch) = out;
}

}  // namespace imparo

using namespace imparo;

// bcx: [n_tok, 3 * width] of the dtype; or, when parts > 0, float partial results
// [parts][n_tok][3 * width] (split s at bcx + s * part_stride floats) of a product cut along K,
// which this kernel sums (the dtype then names the output and the rounding of the sum).
extern "C" int imparo_gated_conv(const void* bcx, int dtype, const float* w, const float* bias, float* state,
                                 const int* item_row_start, const int* item_of_token, const int* item_slot,
                                 void* y, int n_tok, int width, int taps, int n_slots, int parts, long long part_stride,
                                 int* status, cudaStream_t stream) {
    if (n_tok <= 0) return 0;
    if (taps < 2 || taps > MAX_TAPS) return -6;
    if (parts < 0 || (parts > 0 && part_stride < (long long)n_tok * 3 * width)) return -2;
    const size_t n = (size_t)n_tok * width;
    const int threads = 256;
    const unsigned blocks = (unsigned)((n + threads - 1) / threads);
    const float* part = parts > 0 ? (const float*)bcx : nullptr;
    const int mode = parts == 0 ? 0 : (parts <= 4 ? 1 : 2);
#define IMPARO_CONV(T_, M_) do { \
        ConvIn<T_, M_> in{(const T_*)bcx, part, parts, (size_t)part_stride}; \
        launch(gated_conv_kernel<T_, M_>, dim3(blocks), dim3(threads), 0, stream, in, w, bias, state, item_row_start, \
               item_of_token, item_slot, (T_*)y, n_tok, width, taps, n_slots, status); } while (0)
    // prompt-sized batches, 16 bytes of channels at a time
    const int v = dtype == IMPARO_DT_BF16 ? 8 : 4;
    const bool wide = parts == 0 && n_tok >= 64 && width % v == 0 && (((uintptr_t)bcx | (uintptr_t)y) & 15) == 0;
    if (wide && taps <= 4 && (((uintptr_t)w | (uintptr_t)state) & 15) == 0) {
        // four tokens per thread once that still leaves every SM 512 threads
        const size_t all = (size_t)n_tok * (width / v);
        const int r = all >= (size_t)4 * 148 * 512 ? 4 : 1;
        const dim3 grid((unsigned)(((size_t)((n_tok + r - 1) / r) * (width / v) + 255) / 256));
#define IMPARO_CONVR(T_, TAPS_, R_) launch(gated_conv_rows_kernel<T_, TAPS_, R_>, grid, dim3(256), 0, stream, (const T_*)bcx, w, bias, state, \
        item_row_start, item_of_token, item_slot, (T_*)y, n_tok, width, n_slots, status)
#define IMPARO_CONVT(T_, TAPS_) do { if (r == 4) IMPARO_CONVR(T_, TAPS_, 4); else IMPARO_CONVR(T_, TAPS_, 1); } while (0)
#define IMPARO_CONVW(T_) do { if (taps == 2) IMPARO_CONVT(T_, 2); else if (taps == 3) IMPARO_CONVT(T_, 3); else IMPARO_CONVT(T_, 4); } while (0)
        if (dtype == IMPARO_DT_F32) IMPARO_CONVW(float);
        else if (dtype == IMPARO_DT_BF16) IMPARO_CONVW(__nv_bfloat16);
        else return -1;
#undef IMPARO_CONVW
#undef IMPARO_CONVT
#undef IMPARO_CONVR
        IMPARO_CHECK_LAUNCH();
        return 0;
    }
    if (dtype == IMPARO_DT_F32) {
        if (mode == 0) IMPARO_CONV(float, 0); else if (mode == 1) IMPARO_CONV(float, 1); else IMPARO_CONV(float, 2);
    } else if (dtype == IMPARO_DT_BF16) {
        if (wide) {
            const size_t n8 = (size_t)n_tok * (width >> 3);
            launch(gated_conv_bf16x8_kernel, dim3((unsigned)((n8 + threads - 1) / threads)), dim3(threads), 0, stream, (const __nv_bfloat16*)bcx,
                   w, bias, state, item_row_start, item_of_token, item_slot, (__nv_bfloat16*)y, n_tok, width, taps, n_slots, status);
        } else if (mode == 0) IMPARO_CONV(__nv_bfloat16, 0);
        else if (mode == 1) IMPARO_CONV(__nv_bfloat16, 1);
        else IMPARO_CONV(__nv_bfloat16, 2);
#undef IMPARO_CONV
    } else return -1;
    IMPARO_CHECK_LAUNCH();
    return 0;
}
