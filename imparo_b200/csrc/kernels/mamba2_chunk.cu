// The selective state-space recurrence (mamba2.cu) for long portions as products: chunks of 64 rows side by side.
//
// With e_t = exp(a dt_t) of a head (a = -exp(A_log)), c_i = e_first .. e_i and p_ij = e_(j+1) .. e_i inside a chunk, the recurrence
// S <- e_t S + dt_t B_t x_t^T;  y_t = S^T C_t + D x_t  unrolls to
//     y_i   = c_i S_in^T C_i + sum_(j<=i) (C_i . B_j) p_ij dt_j x_j + D x_i
//     S_out = c_end S_in + sum_t (p_end,t dt_t B_t) x_t^T
// and C_i . B_j is one matrix for all heads of a group.  Three launches:
//  (1) state: per (chunk, HG heads of a group, 64 value columns): every chunk's own sum, and the logarithm of c_end.
//  (2) scan:  per (request, head) over its chunks: the state each chunk starts from; the slot's new state.
//  (3) out:   per (chunk, HG heads of a group, 64 value columns): the group's matrix once, then per head one product with 64 +
//             state terms per entry.
// Everything is 32-bit; a decay between two rows is the product of the rows' decays between them.
//
// Two launches walk the rows in mamba2.cu (a state column per thread, 3 operations per row and state entry): with 32 heads of 64
// values, state size 64 and 1,999 rows 47 + 20 + 68 us (state, scan, out), here 18 + 7 + 42 (B200; bound by the latency of the
// products' reads at 8 warps per SM).  Error against 64 bits 1.4e-7 and 1.7e-7.  Which portions come here: parts/mamba2.py and
// mamba2_products_pay in kernels/ops.py.
#include "chunk_products.cuh"

namespace imparo {
namespace mc {

using namespace chunks;             // (a CTA has VB value columns and THREADS threads)
constexpr int C = 64;               // rows per chunk

struct Rows {
    const float* xbc; const float* dt; const float* A_log; const float* D;
    const int* item_row_start; const int* item_slot;
    int n_items, n_slots, heads, vdim, N, groups;
};

// ---- (1) -------------------------------------------------------------------------------------------------------------
template <int NM, int HG>
struct StateSmem { static constexpr size_t FLOATS = (size_t)C * NM + 2 * C * VB + 2 * HG * C; };

template <int NM, int HG>
__global__ void __launch_bounds__(THREADS)
state_kernel(const Rows p, float* __restrict__ chunk_state, float* __restrict__ chunk_decay) {
    extern __shared__ __align__(16) float sm[];
    float* bs = sm;                                        // [C][NM]
    float* xs = bs + C * NM;                               // [2][C][VB]
    float* es = xs + 2 * C * VB;                           // [HG][C]   a dt
    float* ws = es + HG * C;                               // [HG][C]   p_end dt
    pdl_trigger();
    const int h0 = blockIdx.x * HG, chunk = blockIdx.y, v0 = blockIdx.z * VB, tid = threadIdx.x;
    int item, first;
    const int n = chunk_rows<C>(p, chunk, item, first);
    const int inner = p.heads * p.vdim, g = h0 / (p.heads / p.groups);
    const size_t channels = (size_t)inner + 2 * p.groups * p.N;
    pdl_wait();
    if (n == 0) return;
    const float* rows = p.xbc + (size_t)first * channels;
    const int cols = min(VB, p.vdim - v0);
    for (int e = tid; e < C * (NM / 4); e += THREADS) {
        const int r = e / (NM / 4), s = (e % (NM / 4)) * 4;
        if (r < n && s < p.N) cp16(bs + r * NM + s, rows + (size_t)r * channels + inner + g * p.N + s);
        else *reinterpret_cast<float4*>(bs + r * NM + s) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    fetch_rows<C>(xs, rows + (size_t)h0 * p.vdim + v0, channels, n, cols);
    cp_commit();
    for (int e = tid; e < HG * C; e += THREADS) {
        const int hh = e / C, r = e % C;
        const float step = r < n ? p.dt[(size_t)(first + r) * p.heads + h0 + hh] : 0.f;
        es[e] = r < n ? -expf(p.A_log[h0 + hh]) * step : 0.f;           // (not -infinity times zero beyond the rows)
        ws[e] = step;
    }
    __syncthreads();
    if (blockIdx.z == 0 && tid < HG) {
        float total = 0.f;
        for (int r = 0; r < n; ++r) total += es[tid * C + r];
        chunk_decay[(size_t)chunk * p.heads + h0 + tid] = total;
    }
    __syncthreads();
    for (int e = tid; e < HG * C; e += THREADS) es[e] = expf(es[e]);
    __syncthreads();
    for (int e = tid; e < HG * C; e += THREADS) {
        const int hh = e / C, r = e % C;
        float w = ws[e];
        for (int i = n - 1; i > r; --i) w *= es[hh * C + i];
        ws[e] = w;
    }
    const int nq = (tid >> 4) * 8, vq = (tid & 15) * 4;
    for (int hh = 0; hh < HG; ++hh) {
        if (hh + 1 < HG) fetch_rows<C>(xs + ((hh + 1) & 1) * C * VB, rows + (size_t)(h0 + hh + 1) * p.vdim + v0, channels, n, cols);
        cp_commit();
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        float* x = xs + (hh & 1) * C * VB;
        for (int e = tid; e < C * (VB / 4); e += THREADS) {           // the rows' weights
            float4* q = reinterpret_cast<float4*>(x) + e;
            const float w = ws[hh * C + e / (VB / 4)];
            *q = make_float4(q->x * w, q->y * w, q->z * w, q->w * w);
        }
        __syncthreads();
        float* out = chunk_state + (((size_t)chunk * p.heads + h0 + hh) * p.N) * p.vdim + v0;
#pragma unroll
        for (int nb = 0; nb < NM; nb += 64) {
            float2 acc[8][2] = {};
            product<NM>(acc, bs, nb + nq, x, vq, n);
            if (vq < cols) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (nb + nq + i < p.N)
                        *reinterpret_cast<float4*>(out + (size_t)(nb + nq + i) * p.vdim + vq) = make_float4(acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y);
            }
        }
        __syncthreads();                                              // x is filled again by the head after the next
    }
}

// ---- (2) -------------------------------------------------------------------------------------------------------------
// per request and head: chunk_state[c] becomes the state BEFORE chunk c; the slot gets the state after the last chunk.  A thread
// owns four entries; eight chunks' loads in flight.
__global__ void __launch_bounds__(128)
scan_kernel(const Rows p, float* __restrict__ chunk_state, const float* __restrict__ chunk_decay, float* __restrict__ state, int* status) {
    pdl_trigger();
    const int h = blockIdx.x, item = blockIdx.y;
    const int slot = p.item_slot[item];
    int c0 = 0;
    for (int i = 0; i < item; ++i) c0 += (p.item_row_start[i + 1] - p.item_row_start[i] + C - 1) / C;
    const int n_chunks = (p.item_row_start[item + 1] - p.item_row_start[item] + C - 1) / C;
    pdl_wait();
    if (slot < 0 || slot >= p.n_slots) {
        if (threadIdx.x == 0 && h == 0 && blockIdx.z == 0) report(status, IMPARO_ST_SLOT_RANGE, 63, item, slot);
        return;
    }
    const int per = p.N * p.vdim / 4, e = blockIdx.z * 128 + threadIdx.x;
    if (e >= per) return;
    float4* sp = reinterpret_cast<float4*>(state + ((size_t)slot * p.heads + h) * per * 4) + e;
    float4* cs = reinterpret_cast<float4*>(chunk_state + ((size_t)c0 * p.heads + h) * per * 4) + e;
    const float* cd = chunk_decay + (size_t)c0 * p.heads + h;
    const size_t step = (size_t)p.heads * per;
    float4 S = *sp;
    for (int c = 0; c < n_chunks; c += 8) {
        float4 own[8];
        float dec[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (c + u < n_chunks) {
                own[u] = cs[(size_t)(c + u) * step];
                dec[u] = expf(cd[(size_t)(c + u) * p.heads]);
            }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (c + u < n_chunks) {
                cs[(size_t)(c + u) * step] = S;
                S = make_float4(fmaf(dec[u], S.x, own[u].x), fmaf(dec[u], S.y, own[u].y), fmaf(dec[u], S.z, own[u].z), fmaf(dec[u], S.w, own[u].w));
            }
        }
    }
    *sp = S;
}

// ---- (3) -------------------------------------------------------------------------------------------------------------
template <int NM, int HG>
struct OutSmem {
    static constexpr size_t BM = NM * C > C * C ? NM * C : C * C;                 // B by column, later a head's matrix
    static constexpr size_t FLOATS = (size_t)NM * C + BM + C * C + (NM + C) * VB + 2 * HG * C;
};

template <int NM, int HG>
__global__ void __launch_bounds__(THREADS)
out_kernel(const Rows p, const float* __restrict__ chunk_state, float* __restrict__ y) {
    extern __shared__ __align__(16) float sm[];
    float* ct = sm;                                        // [NM][C]   C, state entry by state entry
    float* bt = ct + NM * C;                               // [NM][C]   B alike; then the head's matrix, column by column
    float* gt = bt + OutSmem<NM, HG>::BM;                  // [C j][C i]  C_i . B_j
    float* right = gt + C * C;                             // [NM + C][VB]  S_in, then x (one head's: two CTAs fit on an SM)
    float* es = right + (NM + C) * VB;                 // [HG][C]   e
    float* ds = es + HG * C;                               // [HG][C]   dt
    pdl_trigger();
    const int h0 = blockIdx.x * HG, chunk = blockIdx.y, v0 = blockIdx.z * VB, tid = threadIdx.x;
    int item, first;
    const int n = chunk_rows<C>(p, chunk, item, first);
    const int inner = p.heads * p.vdim, g = h0 / (p.heads / p.groups);
    const size_t channels = (size_t)inner + 2 * p.groups * p.N;
    pdl_wait();
    if (n == 0) return;
    const int slot = p.item_slot[item];
    if (slot < 0 || slot >= p.n_slots) return;             // (2) has recorded it
    const float* rows = p.xbc + (size_t)first * channels;
    const int cols = min(VB, p.vdim - v0);
    auto fetch = [&](int hh) {
        float* s = right;
        const float* from = chunk_state + (((size_t)chunk * p.heads + h0 + hh) * p.N) * p.vdim + v0;
        for (int e = tid; e < NM * (VB / 4); e += THREADS) {
            const int k = e / (VB / 4), v = (e % (VB / 4)) * 4;
            if (k < p.N && v < cols) cp16(s + k * VB + v, from + (size_t)k * p.vdim + v);
            else *reinterpret_cast<float4*>(s + k * VB + v) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        fetch_rows<C>(s + NM * VB, rows + (size_t)(h0 + hh) * p.vdim + v0, channels, n, cols);
    };
    for (int e = tid; e < C * (NM / 4); e += THREADS) {    // a lane a row: its four entries go to four rows of the transposed tile
        const int r = e % C, s = (e / C) * 4;
        float4 b = make_float4(0.f, 0.f, 0.f, 0.f), c = b;
        if (r < n && s < p.N) {
            const float* row = rows + (size_t)r * channels + inner + g * p.N + s;
            b = *reinterpret_cast<const float4*>(row);
            c = *reinterpret_cast<const float4*>(row + p.groups * p.N);
        }
        bt[s * C + r] = b.x; bt[(s + 1) * C + r] = b.y; bt[(s + 2) * C + r] = b.z; bt[(s + 3) * C + r] = b.w;
        ct[s * C + r] = c.x; ct[(s + 1) * C + r] = c.y; ct[(s + 2) * C + r] = c.z; ct[(s + 3) * C + r] = c.w;
    }
    for (int e = tid; e < HG * C; e += THREADS) {
        const int hh = e / C, r = e % C;
        const float step = r < n ? p.dt[(size_t)(first + r) * p.heads + h0 + hh] : 0.f;
        ds[e] = step;
        es[e] = r < n ? expf(-expf(p.A_log[h0 + hh]) * step) : 1.f;
    }
    __syncthreads();
    const int lq = (tid >> 4) * 8, rq = (tid & 15) * 4;
    const bool busy = (lq & ~15) < n;                      // the warp's 16 rows: a short chunk's products are its own warps' only
    {
        float2 acc[8][2] = {};                             // rows j, columns i
        if (busy) product<C>(acc, bt, lq, ct, rq, NM);
        __syncthreads();                                   // bt is written over from here on
#pragma unroll
        for (int j = 0; j < 8; ++j)
            *reinterpret_cast<float4*>(gt + (lq + j) * C + rq) = make_float4(acc[j][0].x, acc[j][0].y, acc[j][1].x, acc[j][1].y);
    }
    for (int hh = 0; hh < HG; ++hh) {
        fetch(hh);
        cp_commit();
        __syncthreads();                                   // gt is whole
        const int i = tid & (C - 1), j_lo = (tid >> 6) * 32, j_hi = j_lo + 31;
        if (i < n) {
            // row i, columns j of one half, from the diagonal down: the decay grows by one row at a time
            const float* e = es + hh * C;
            const float* d = ds + hh * C;
            float w = 1.f;
            for (int r = i; r > j_hi; --r) w *= e[r];
#pragma unroll 8
            for (int j = j_hi; j >= j_lo; --j) {
                bt[j * C + i] = j <= i ? gt[j * C + i] * (w * d[j]) : 0.f;
                if (j <= i) w *= e[j];
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const float* s = right;
        const float* x = s + NM * VB;
        float2 acc[8][2] = {}, inside[8][2] = {};
        if (busy) {
            product<C>(acc, ct, lq, s, rq, NM);
            product<C, true>(inside, bt, lq, x, rq, lq + 8);
        }
        const float skip = p.D[h0 + hh];
        float c = 1.f;
        for (int r = 0; r < lq; ++r) c *= es[hh * C + r];
        float* out = y + (size_t)first * inner + (size_t)(h0 + hh) * p.vdim + v0 + rq;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            c *= es[hh * C + lq + i];
            if (lq + i < n && rq < cols) {
                const float4 xv = *reinterpret_cast<const float4*>(x + (lq + i) * VB + rq);
                *reinterpret_cast<float4*>(out + (size_t)(lq + i) * inner) =
                    make_float4(fmaf(c, acc[i][0].x, inside[i][0].x) + skip * xv.x, fmaf(c, acc[i][0].y, inside[i][0].y) + skip * xv.y,
                                fmaf(c, acc[i][1].x, inside[i][1].x) + skip * xv.z, fmaf(c, acc[i][1].y, inside[i][1].y) + skip * xv.w);
            }
        }
        __syncthreads();                                   // this head's operands are filled again
    }
}

// HS, HG: heads per CTA of (1) and of (3)
template <int NM, int HS, int HG>
static int run(const Rows& p, int max_chunks, float* chunk_state, float* chunk_decay, float* state, float* y, int* status, cudaStream_t stream) {
    constexpr size_t s1 = StateSmem<NM, HS>::FLOATS * 4, s3 = OutSmem<NM, HG>::FLOATS * 4;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(state_kernel<NM, HS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s1);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(out_kernel<NM, HG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s3);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const dim3 grid(p.heads / HG, max_chunks, (p.vdim + VB - 1) / VB);
    const dim3 sgrid(p.heads / HS, max_chunks, (p.vdim + VB - 1) / VB);
    launch(state_kernel<NM, HS>, sgrid, dim3(THREADS), s1, stream, p, chunk_state, chunk_decay);
    IMPARO_CHECK_LAUNCH();
    launch(scan_kernel, dim3(p.heads, p.n_items, (p.N * p.vdim / 4 + 127) / 128), dim3(128), 0, stream, p, chunk_state,
           (const float*)chunk_decay, state, status);
    IMPARO_CHECK_LAUNCH();
    launch(out_kernel<NM, HG>, grid, dim3(THREADS), s3, stream, p, (const float*)chunk_state, y);
    IMPARO_CHECK_LAUNCH();
    return 0;
}

template <int NM>
static int run_hg(const Rows& p, int max_chunks, float* chunk_state, float* chunk_decay, float* state, float* y, int* status, cudaStream_t stream) {
    // heads per CTA: as many as share B and C while every SM still has a CTA (one head: the group's matrix is made per head);
    // the sums of (1) share only B and are quicker in smaller CTAs
    const long long ctas = (long long)p.heads * max_chunks * ((p.vdim + VB - 1) / VB);
    const int per_group = p.heads / p.groups;
    if (per_group % 4 == 0 && ctas >= 4 * 148) return run<NM, 2, 4>(p, max_chunks, chunk_state, chunk_decay, state, y, status, stream);
    if (per_group % 2 == 0 && ctas >= 2 * 148) return run<NM, 2, 2>(p, max_chunks, chunk_state, chunk_decay, state, y, status, stream);
    return run<NM, 1, 1>(p, max_chunks, chunk_state, chunk_decay, state, y, status, stream);
}

}  // namespace mc
}  // namespace imparo

using namespace imparo;

// Whether imparo_mamba2_products takes these sizes: state and value sizes multiples of 4, state size up to 128.
extern "C" int imparo_mamba2_products_take(int heads, int vdim, int N, int groups) {
    return heads >= 1 && groups >= 1 && heads % groups == 0 && vdim >= 4 && vdim % 4 == 0 && N >= 4 && N % 4 == 0 && N <= 128;
}

// As imparo_mamba2_scan; chunk_state float32 [max_chunks, heads, N, vdim], chunk_decay float32 [max_chunks, heads], max_chunks >=
// n_tok / 64 + n_items.  -25: sizes or alignments it does not take.  Three launches.
extern "C" int imparo_mamba2_products(const float* xbc, const float* dt, const float* A_log, const float* D, float* state,
                                      const int* item_row_start, const int* item_slot, int n_items, int n_slots, float* y, int heads,
                                      int vdim, int N, int groups, int max_chunks, float* chunk_state, float* chunk_decay, int* status,
                                      cudaStream_t stream) {
    if (n_items <= 0 || max_chunks <= 0) return 0;
    if (!imparo_mamba2_products_take(heads, vdim, N, groups) || n_items > 65535 || max_chunks > 65535) return -25;
    if (((uintptr_t)xbc | (uintptr_t)state | (uintptr_t)y | (uintptr_t)chunk_state) & 15) return -25;
    const mc::Rows p{xbc, dt, A_log, D, item_row_start, item_slot, n_items, n_slots, heads, vdim, N, groups};
    return N <= 64 ? mc::run_hg<64>(p, max_chunks, chunk_state, chunk_decay, state, y, status, stream)
                   : mc::run_hg<128>(p, max_chunks, chunk_state, chunk_decay, state, y, status, stream);
}
