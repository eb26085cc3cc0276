// The matrix memory with exponential gates (mlstm.cu) for long portions as products: chunks of 64 rows side by side.
//
// With m_t = max(f_t + m_(t-1), a_t), keep_t = exp(f_t + m_(t-1) - m_t), put_t = exp(a_t - m_t), c_i = keep_first .. keep_i and
// p_ij = keep_(j+1) .. keep_i inside a chunk (every factor at most one) the recurrence unrolls to
//     P_ij  = (q_i . k_j) p_ij put_j   (j <= i),   S_i^T q_i = c_i S_in^T q_i + sum_j P_ij v_j,   n_i . q_i = c_i n_in . q_i + sum_j P_ij
//     S_out = c_end S_in + sum_t (p_end,t put_t k_t) v_t^T,   n_out alike
// Two launches around the scan over the chunks in mlstm.cu:
//  (1) local: per (chunk, head, 64 value columns): the chunk's own S, n, maximum (from an empty state) and sum of f.
//  (2) out:   per (chunk, head): the matrix P once, then per 64 value columns one product with dim + 64 terms per entry.
// Everything is 32-bit; maxima are walked row by row, and a weight between two rows is the product of the rows' factors between
// them, as the row walk would have it (never the exponential of a difference of long sums).
//
// Bound by the latency of the products' own operations and of their reads of shared memory at 7 to 8 warps per SM (the output launch
// issues in 31% of the cycles, its 32-bit units work in 17%).  In mlstm.cu a chunk's CTA
// walks its rows one after the other with a state column per lane: with 8 heads of 64 keys and 128
// values and 2,048 rows 37 + 9 + 81 us (local, scan, out), here 15 + 9 + 28 (B200).  Against 64 bits the states are as exact as the row
// walk's, the outputs in the median too (2e-7; a row whose n . q nearly cancels is off by more either way).
#include "mlstm_chunk.cuh"
#include "chunk_products.cuh"

namespace imparo {
namespace mx {

using namespace chunks;             // (a block has VB value columns and THREADS threads)
constexpr int C = MLSTM_PRODUCTS_CHUNK;

__device__ __forceinline__ float log_sigmoid(float z) { return fminf(z, 0.f) - log1pf(expf(-fabsf(z))); }

// Gates of the chunk's rows: as[r] log input gate, fs[r] log forget gate (one thread per row; rows beyond n are not written)
__device__ __forceinline__ void gates(const MlstmProducts& p, int first, int n, int h, float* as, float* fs) {
    const int r = threadIdx.x;
    if (r < n) {
        const float* row = p.proj + (size_t)(first + r) * p.stride;
        as[r] = p.cap * tanhf((row[p.i_off + h] + p.i_bias[h]) / p.cap);
        fs[r] = log_sigmoid(p.cap * tanhf((row[p.f_off + h] + p.f_bias[h]) / p.cap));
    }
}
// ms[r]: the running maximum from m on (one thread; the others wait at the caller's barrier)
__device__ __forceinline__ void maxima(float m, int n, const float* as, const float* fs, float* ms) {
    for (int r = 0; r < n; ++r) {
        m = fmaxf(fs[r] + m, as[r]);
        ms[r] = m;
    }
}
// as -> put, fs -> keep (rows beyond n: put 0, keep 1), one thread per row
__device__ __forceinline__ void factors(float m, int n, float* as, float* fs, const float* ms) {
    const int r = threadIdx.x;
    if (r < C) {
        const float before = r == 0 ? m : ms[r - 1 < n ? r - 1 : 0];
        const float put = r < n ? expf(as[r] - ms[r]) : 0.f, keep = r < n ? expf(fs[r] + before - ms[r]) : 1.f;
        as[r] = put;
        fs[r] = keep;
    }
}

// ---- (1) -------------------------------------------------------------------------------------------------------------
template <int NM> struct LocalSmem { static constexpr size_t FLOATS = (size_t)C * NM + C * VB + 3 * C; };

template <int NM>
__global__ void __launch_bounds__(THREADS)
mlstm_local_kernel(const MlstmProducts p) {
    extern __shared__ __align__(16) float sm[];
    float* ks = sm;                                        // [C][NM]
    float* xs = ks + C * NM;                               // [C][VB]
    float* as = xs + C * VB;                               // [C]   log input gate, put, then put p_end
    float* fs = as + C;                                    // [C]   log forget gate, then keep
    float* ms = fs + C;                                    // [C]
    pdl_trigger();
    const int chunk = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * VB, tid = threadIdx.x;
    int item, first;
    const int n = chunk_rows<C>(p, chunk, item, first);
    pdl_wait();
    if (n == 0) return;
    const float* rows = p.proj + (size_t)first * p.stride;
    const int cols = min(VB, p.vdim - v0);
    for (int e = tid; e < C * (NM / 4); e += THREADS) {
        const int r = e / (NM / 4), d = (e % (NM / 4)) * 4;
        if (r < n && d < p.dim) cp16(ks + r * NM + d, rows + (size_t)r * p.stride + p.k_off + h * p.dim + d);
        else *reinterpret_cast<float4*>(ks + r * NM + d) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    fetch_rows<C>(xs, rows + p.v_off + (size_t)h * p.vdim + v0, p.stride, n, cols);
    cp_commit();
    gates(p, first, n, h, as, fs);
    __syncthreads();
    float total = 0.f;
    if (tid == 0) {
        for (int r = 0; r < n; ++r) total += fs[r];
        maxima(-INFINITY, n, as, fs, ms);                  // an empty state has no maximum
    }
    __syncthreads();
    factors(-INFINITY, n, as, fs, ms);                     // (keep of the first row: exp(-inf) = 0, and nothing to keep)
    __syncthreads();
    float w = 0.f;
    if (tid < C) {
        w = as[tid];
        for (int i = n - 1; i > tid; --i) w *= fs[i];
    }
    __syncthreads();
    if (tid < C) as[tid] = w;
    cp_wait_all();
    __syncthreads();
    for (int e = tid; e < C * (VB / 4); e += THREADS) {    // the rows' weights
        float4* q = reinterpret_cast<float4*>(xs) + e;
        const float u = as[e / (VB / 4)];
        if (e / (VB / 4) < n) *q = make_float4(q->x * u, q->y * u, q->z * u, q->w * u);
    }
    const size_t ch = (size_t)chunk * p.heads + h;
    const int vb0 = v0 / 32, vb1 = min(p.vblocks, vb0 + VB / 32);
    for (int d = tid; d < p.dim; d += THREADS) {
        float s = 0.f;
        for (int r = 0; r < n; ++r) s = fmaf(as[r], ks[r * NM + d], s);
        for (int vb = vb0; vb < vb1; ++vb) p.chunk_n[(ch * p.vblocks + vb) * p.dim + d] = s;
    }
    if (tid == 0)
        for (int vb = vb0; vb < vb1; ++vb) {
            float* mb = p.chunk_mb + (ch * p.vblocks + vb) * 3;
            mb[0] = ms[n - 1]; mb[1] = total; mb[2] = 0.f;
        }
    __syncthreads();
    const int nq = (tid >> 4) * 8, vq = (tid & 15) * 4;
    float* out = p.chunk_S + ch * p.dim * p.vdim + v0;
#pragma unroll
    for (int nb = 0; nb < NM; nb += 64) {
        if (nb >= p.dim) break;
        float2 acc[8][2] = {};
        product<NM>(acc, ks, nb + nq, xs, vq, n);
        if (vq < cols) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (nb + nq + i < p.dim)
                    *reinterpret_cast<float4*>(out + (size_t)(nb + nq + i) * p.vdim + vq) = make_float4(acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y);
        }
    }
}

// ---- (2) -------------------------------------------------------------------------------------------------------------
template <int NM>
struct OutSmem {
    static constexpr size_t KM = NM * C > C * C ? NM * C : C * C;                 // k by channel, later P
    static constexpr size_t FLOATS = (size_t)NM * C + KM + C * C + (NM + C) * VB + NM + 6 * C;
};

template <int NM>
__global__ void __launch_bounds__(THREADS)
mlstm_out_kernel(const MlstmProducts p) {
    extern __shared__ __align__(16) float sm[];
    float* qt = sm;                                        // [NM][C]   q, channel by channel
    float* kt = qt + NM * C;                               // [NM][C]   k alike; then P, column by column
    float* gt = kt + OutSmem<NM>::KM;                      // [C j][C i]  k_j . q_i
    float* right = gt + C * C;                             // [NM + C][VB]  S_in, then v
    float* ns = right + (NM + C) * VB;                     // [NM]      n_in
    float* as = ns + NM;                                   // [C]       log input gate, then put
    float* fs = as + C;                                    // [C]       log forget gate, then keep
    float* ms = fs + C;                                    // [C]
    float* sums = ms + C;                                  // [2][C]    the two halves of a row's sum of P
    float* den = sums + 2 * C;                             // [C]
    pdl_trigger();
    const int chunk = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    int item, first;
    const int n = chunk_rows<C>(p, chunk, item, first);
    pdl_wait();
    if (n == 0) return;
    const float* rows = p.proj + (size_t)first * p.stride;
    const size_t ch = (size_t)chunk * p.heads + h;
    auto fetch = [&](int v0) {
        const int cols = min(VB, p.vdim - v0);
        const float* from = p.chunk_S + ch * p.dim * p.vdim + v0;
        for (int e = tid; e < NM * (VB / 4); e += THREADS) {
            const int k = e / (VB / 4), v = (e % (VB / 4)) * 4;
            if (k < p.dim && v < cols) cp16(right + k * VB + v, from + (size_t)k * p.vdim + v);
            else *reinterpret_cast<float4*>(right + k * VB + v) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        fetch_rows<C>(right + NM * VB, rows + p.v_off + (size_t)h * p.vdim + v0, p.stride, n, cols);
        cp_commit();
    };
    fetch(0);
    for (int e = tid; e < C * (NM / 4); e += THREADS) {    // a lane a row: its four channels go to four rows of the transposed tile
        const int r = e % C, s = (e / C) * 4;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f), k = q;
        if (r < n && s < p.dim) {
            const float* row = rows + (size_t)r * p.stride + h * p.dim + s;
            q = *reinterpret_cast<const float4*>(row + p.q_off);
            k = *reinterpret_cast<const float4*>(row + p.k_off);
        }
        qt[s * C + r] = q.x; qt[(s + 1) * C + r] = q.y; qt[(s + 2) * C + r] = q.z; qt[(s + 3) * C + r] = q.w;
        kt[s * C + r] = k.x; kt[(s + 1) * C + r] = k.y; kt[(s + 2) * C + r] = k.z; kt[(s + 3) * C + r] = k.w;
    }
    for (int d = tid; d < NM; d += THREADS) ns[d] = d < p.dim ? p.chunk_n[ch * p.vblocks * p.dim + d] : 0.f;
    const float m_in = p.chunk_mb[ch * p.vblocks * 3 + 2];
    gates(p, first, n, h, as, fs);
    __syncthreads();
    const int lq = (tid >> 4) * 8, rq = (tid & 15) * 4;
    const bool busy = (lq & ~15) < n;                      // the warp's 16 rows: a short chunk's products are its own warps' only
    if (tid == THREADS - 1) maxima(m_in, n, as, fs, ms);
    {
        float2 acc[8][2] = {};                             // rows j, columns i
        if (busy) product<C>(acc, kt, lq, qt, rq, NM);
        __syncthreads();                                   // kt is written over from here on; ms is whole
#pragma unroll
        for (int j = 0; j < 8; ++j)
            *reinterpret_cast<float4*>(gt + (lq + j) * C + rq) = make_float4(acc[j][0].x, acc[j][0].y, acc[j][1].x, acc[j][1].y);
    }
    factors(m_in, n, as, fs, ms);
    __syncthreads();
    {
        const int i = tid & (C - 1), half = tid >> 6, j_lo = half * 32, j_hi = j_lo + 31;
        float sum = 0.f;
        if (i < n) {
            // row i, columns j of one half, from the diagonal down: the weight grows by one row at a time
            float w = 1.f;
            for (int r = i; r > j_hi; --r) w *= fs[r];
#pragma unroll 1
            for (int j8 = j_hi; j8 >= j_lo; j8 -= 8) {
                float eight = 0.f;                         // (a row's sum by eights: n . q cancels, and its error is the output's)
#pragma unroll
                for (int j = j8; j > j8 - 8; --j) {
                    const float v = j <= i ? gt[j * C + i] * (w * as[j]) : 0.f;
                    kt[j * C + i] = v;
                    eight += v;
                    if (j <= i) w *= fs[j];
                }
                sum += eight;
            }
        }
        sums[half * C + i] = sum;
    }
    __syncthreads();
    if (tid < n) {
        float c = 1.f, nq = 0.f;
        for (int r = 0; r <= tid; ++r) c *= fs[r];
#pragma unroll 1
        for (int d8 = 0; d8 < NM; d8 += 8) {
            float eight = 0.f;
#pragma unroll
            for (int d = d8; d < d8 + 8; ++d) eight = fmaf(ns[d], qt[d * C + tid], eight);
            nq += eight;
        }
        nq = fmaf(c, nq, sums[tid] + sums[C + tid]) * p.q_scale;
        den[tid] = fmaxf(fabsf(nq), expf(-ms[tid])) + 1e-6f;
    }
    if (tid < p.vblocks && first + n == p.item_row_start[item + 1]) {
        const int slot = p.item_slot[item];
        if (slot >= 0 && slot < p.n_slots)
            for (int vb = tid; vb < p.vblocks; vb += THREADS) p.state_m[((size_t)slot * p.heads + h) * p.vblocks + vb] = ms[n - 1];
    }
    float c0 = 1.f;
    for (int r = 0; r < lq; ++r) c0 *= fs[r];
    for (int v0 = 0; v0 < p.vdim; v0 += VB) {
        if (v0 > 0) {
            __syncthreads();                               // the last block's operands have been read
            fetch(v0);
        }
        cp_wait_all();
        __syncthreads();                                   // (the first time also: P and den are whole)
        const float* v = right + NM * VB;
        float2 acc[8][2] = {}, inside[8][2] = {};
        if (busy) {
            product<C>(acc, qt, lq, right, rq, NM);
            product<C, true>(inside, kt, lq, v, rq, lq + 8);
        }
        const int cols = min(VB, p.vdim - v0);
        float* out = p.out + (size_t)first * p.heads * p.vdim + (size_t)h * p.vdim + v0 + rq;
        float c = c0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            c *= fs[lq + i];
            if (lq + i < n && rq < cols) {
                const float d = den[lq + i];
                *reinterpret_cast<float4*>(out + (size_t)(lq + i) * p.heads * p.vdim) =
                    make_float4(fmaf(c, acc[i][0].x, inside[i][0].x) * p.q_scale / d, fmaf(c, acc[i][0].y, inside[i][0].y) * p.q_scale / d,
                                fmaf(c, acc[i][1].x, inside[i][1].x) * p.q_scale / d, fmaf(c, acc[i][1].y, inside[i][1].y) * p.q_scale / d);
            }
        }
    }
}

template <int NM>
static int configure() {
    static bool configured = false;
    if (configured) return 0;
    cudaError_t e = cudaFuncSetAttribute(mlstm_local_kernel<NM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(LocalSmem<NM>::FLOATS * 4));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(mlstm_out_kernel<NM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(OutSmem<NM>::FLOATS * 4));
    configured = e == cudaSuccess;
    return (int)e;
}
template <int NM>
static int run(const MlstmProducts& p, int max_chunks, bool out, cudaStream_t stream) {
    const int rc = configure<NM>();
    if (rc) return rc;
    if (out) launch(mlstm_out_kernel<NM>, dim3(max_chunks, p.heads), dim3(THREADS), OutSmem<NM>::FLOATS * 4, stream, p);
    else launch(mlstm_local_kernel<NM>, dim3(max_chunks, p.heads, (p.vdim + VB - 1) / VB), dim3(THREADS), LocalSmem<NM>::FLOATS * 4, stream, p);
    IMPARO_CHECK_LAUNCH();
    return 0;
}

}  // namespace mx

bool mlstm_products_take(const MlstmProducts& p) {
    return p.dim >= 4 && p.dim <= 128 && p.dim % 4 == 0 && p.vdim >= 4 && p.vdim % 4 == 0 && p.stride % 4 == 0 && p.q_off % 4 == 0 &&
           p.k_off % 4 == 0 && p.v_off % 4 == 0 && (p.vdim + mx::VB - 1) / mx::VB <= 65535 &&
           (((uintptr_t)p.proj | (uintptr_t)p.chunk_S | (uintptr_t)p.out) & 15) == 0;
}
int mlstm_products_local(const MlstmProducts& p, int max_chunks, cudaStream_t stream) {
    return p.dim <= 64 ? mx::run<64>(p, max_chunks, false, stream) : mx::run<128>(p, max_chunks, false, stream);
}
int mlstm_products_out(const MlstmProducts& p, int max_chunks, cudaStream_t stream) {
    return p.dim <= 64 ? mx::run<64>(p, max_chunks, true, stream) : mx::run<128>(p, max_chunks, true, stream);
}

}  // namespace imparo
