// The gated delta rule (delta_rule.cu) for long portions: chunks of 64 rows side by side.
//
// With c_i = product of the decays g of a chunk's rows up to i (per key channel) and p_ij = product of those of the rows
// after j up to i, the recurrence  S <- g S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q  unrolls inside a chunk to
//     u_i + beta_i sum_(j<i) [ sum_d k_i k_j p_ij ] u_j  =  beta_i (v_i - (k_i c_i)^T S_in)
//     o_i  =  (q_i c_i)^T S_in + sum_(j<=i) [ sum_d q_i k_j p_ij ] u_j
//     S_out = c_end S_in + sum_j (k_j p_end,j) u_j^T
// and the left side, a unit lower triangular system with the same matrix for every right side, is solved once for beta v and
// once for beta k c:  u = W_v - W_k S_in.  Three launches:
//  (1) local: per (chunk, head), from the rows alone: the two matrices of bracketed sums, W_v and W_k, and k p_end, q c.
//  (2) scan:  per (request, head, 8 value columns), chunk after chunk: u, the state the chunk starts from, the next one.
//  (3) out:   per (chunk, head, 64 value columns): o as one product with 64 + dim terms per entry.
// Everything is 32-bit, and every decay between two rows is the product of the decays between them, multiplied up row by
// row (never a quotient, nor the exponential of a difference of long sums): a decay of zero needs no care, and the error is
// the row walk's (tests compare both with 64 bits).
//
// B200, 8 heads of key size 64 and value size 128, 2,048 rows: 421 us for the row walk, 141 us for the three launches (local 43,
// scan 82, out 16); error against 64 bits 1.1e-7 and 1.4e-7.  Which portions come here: parts/delta_rule.py.
//
// A request's rows are cut into chunks from its portion's first row on, so the cut depends on the portion alone.
#include "chunk_products.cuh"

namespace imparo {
namespace dc {

using chunks::chunk_rows;
using chunks::cp16;

constexpr int C = 64;               // rows per chunk
constexpr int PC = C + 4;           // row of a staged matrix with 64 columns: four floats more, so that eight lanes' 16-byte
                                    // reads of eight rows fall into different banks
constexpr int VB = 8;               // value columns of a CTA of (2) ...
constexpr int VP = 12;              // ... and their row in shared memory (the same reason)

struct Rows {
    const float* qkv; size_t stride; int q_off, k_off, v_off;
    const float* g;                 // decays [tokens, heads * dim]
    const float* beta;              // [tokens, heads]
    const int* item_row_start; const int* item_slot;
    int n_items, n_slots, heads, kv_heads, dim, vdim;
};

// What (1) leaves per (chunk, head), in floats
struct Layout {
    size_t wk, kend, qc, pt, cend, u, s_in, total;
    __host__ __device__ Layout(int dim, int vdim) {
        wk = 0;                                         // [dim][C]     W_k, channel by channel
        kend = wk + (size_t)dim * C;                    // [C][dim]     k p_end
        qc = kend + (size_t)C * dim;                    // [dim][C]     q c, channel by channel
        pt = qc + (size_t)dim * C;                      // [C j][C i]   the output's matrix, column by column
        cend = pt + (size_t)C * C;                      // [dim]
        u = cend + dim;                                 // [C][vdim]    W_v, then u
        s_in = u + (size_t)C * vdim;                    // [dim][vdim]
        total = s_in + (size_t)dim * vdim;
    }
};

// ---- (1) -------------------------------------------------------------------------------------------------------------
// Bound by the issue of 32-bit arithmetic and the latency of its reads of shared memory: 3 operations per pair of rows and
// channel for the two matrices (eight lanes share a column j of them, each with an eighth of the channels and its running
// products in registers, walking down the rows i; a warp has four columns from the left and then as many from the right, so
// that all warps walk 68 rows), 2,016 per column for the solve (a thread per column, in place in shared memory, in blocks of
// 16 rows).
template <int DM>
struct LocalSmem {
    static constexpr int PD = DM + 4;
    static constexpr size_t KQ = 2 * C * PD > C * 128 ? 2 * C * PD : C * 128;    // k and q, later W_v of 128 columns
    static constexpr size_t FLOATS = KQ + C * PD + 2 * C * (C + 4) + C;
};

template <int DM>
__global__ void __launch_bounds__(256)
delta_local_kernel(const Rows p, float* __restrict__ scratch) {
    constexpr int PD = DM + 4, PA = C + 4, W4 = DM / 32;
    extern __shared__ __align__(16) float sm[];
    float* ks = sm;                                       // [C][PD]
    float* qs = sm + C * PD;                              // [C][PD]
    float* xs = sm;                                       // [C][128], over k and q
    float* gs = sm + LocalSmem<DM>::KQ;                   // [C][PD]   decays, then k c, then W_k
    float* as = gs + C * PD;                              // [C][PA]   beta_i sum_d k_i k_j p_ij
    float* ps = as + C * PA;                              // [C j][PA]  sum_d q_i k_j p_ij, column by column
    float* bs = ps + C * PA;                              // [C]
    pdl_trigger();
    const int chunk = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    int item, first;
    const int n = chunk_rows<C>(p, chunk, item, first);
    pdl_wait();
    if (n == 0) return;
    const int dim = p.dim, vdim = p.vdim, kvh = h / (p.heads / p.kv_heads);
    const Layout at(dim, vdim);
    float* out = scratch + ((size_t)chunk * p.heads + h) * at.total;
    // everything requested at once; zeros for k and q, ones for g beyond the chunk's rows and the head's channels
    for (int e = tid; e < C * (DM / 4); e += 256) {
        const int r = e / (DM / 4), d = (e % (DM / 4)) * 4;
        const int to = r * PD + d;
        if (r < n && d < dim) {
            const float* row = p.qkv + (size_t)(first + r) * p.stride + (size_t)kvh * dim + d;
            cp16(ks + to, row + p.k_off);
            cp16(qs + to, row + p.q_off);
            cp16(gs + to, p.g + ((size_t)(first + r) * p.heads + h) * dim + d);
        } else {
            *reinterpret_cast<float4*>(ks + to) = make_float4(0.f, 0.f, 0.f, 0.f);
            *reinterpret_cast<float4*>(qs + to) = make_float4(0.f, 0.f, 0.f, 0.f);
            *reinterpret_cast<float4*>(gs + to) = make_float4(1.f, 1.f, 1.f, 1.f);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (tid < C) bs[tid] = tid < n ? p.beta[(size_t)(first + tid) * p.heads + h] : 0.f;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    {
        // this lane's column of four, and its channels: groups of four, `part`, part + 8, ... (the lanes' reads side by side)
        const int warp = tid >> 5, jl = (tid >> 3) & 3, part = tid & 7;
#pragma unroll 1
        for (int side = 0; side < 2; ++side) {
            const int j0 = side == 0 ? 4 * warp : C - 4 - 4 * warp, j = j0 + jl;
            float2 w[W4][2];
#pragma unroll
            for (int x = 0; x < W4; ++x) w[x][0] = w[x][1] = make_float2(0.f, 0.f);
            auto row = [&](int i, bool start) {
                float2 a = make_float2(0.f, 0.f), b = a;
#pragma unroll
                for (int x = 0; x < W4; ++x) {
                    const int d = (x * 8 + part) * 4;
                    const float4 k = *reinterpret_cast<const float4*>(ks + i * PD + d);
                    const float4 q = *reinterpret_cast<const float4*>(qs + i * PD + d);
                    const float4 g = *reinterpret_cast<const float4*>(gs + i * PD + d);
                    const float2 k0 = make_float2(k.x, k.y), k1 = make_float2(k.z, k.w);
                    w[x][0] = start ? k0 : __fmul2_rn(w[x][0], make_float2(g.x, g.y));
                    w[x][1] = start ? k1 : __fmul2_rn(w[x][1], make_float2(g.z, g.w));
                    a = __ffma2_rn(k0, w[x][0], a); a = __ffma2_rn(k1, w[x][1], a);
                    b = __ffma2_rn(make_float2(q.x, q.y), w[x][0], b); b = __ffma2_rn(make_float2(q.z, q.w), w[x][1], b);
                }
                float sa = a.x + a.y, sb = b.x + b.y;
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) {
                    sa += __shfl_xor_sync(0xffffffffu, sa, o);
                    sb += __shfl_xor_sync(0xffffffffu, sb, o);
                }
                if (part == 0) as[i * PA + j] = i > j ? bs[i] * sa : 0.f;
                if (part == 1) ps[j * PA + i] = i >= j ? sb : 0.f;
            };
            for (int i = part; i < j0; i += 8) ps[j * PA + i] = 0.f;
            for (int i = j0; i < j0 + 4; ++i) row(i, i == j);
#pragma unroll 2
            for (int i = j0 + 4; i < C; ++i) row(i, false);
        }
    }
    __syncthreads();
    for (int e = tid; e < C * (C / 4); e += 256) {
        const int j = e / (C / 4), i = (e % (C / 4)) * 4;
        *reinterpret_cast<float4*>(out + at.pt + (size_t)j * C + i) = *reinterpret_cast<const float4*>(ps + j * PA + i);
    }
    // q c and k p_end; then k c in place of the decays
    for (int task = tid; task < 2 * dim; task += 256) {
        const bool is_q = task < dim;
        const int d = is_q ? task : task - dim;
        float c = 1.f;
        if (is_q) {
            float* dst = out + at.qc + (size_t)d * C;
#pragma unroll 2
            for (int i = 0; i < C; i += 4) {
                float v[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) { c *= gs[(i + r) * PD + d]; v[r] = qs[(i + r) * PD + d] * c; }
                *reinterpret_cast<float4*>(dst + i) = make_float4(v[0], v[1], v[2], v[3]);
            }
            out[at.cend + d] = c;
        } else {
            float* dst = out + at.kend + d;
#pragma unroll 8
            for (int i = C - 1; i >= 0; --i) { dst[(size_t)i * dim] = ks[i * PD + d] * c; c *= gs[i * PD + d]; }
        }
    }
    __syncthreads();
    for (int d = tid; d < DM; d += 256) {
        float c = 1.f;
#pragma unroll 8
        for (int i = 0; i < C; ++i) { c *= gs[i * PD + d]; gs[i * PD + d] = ks[i * PD + d] * c; }
    }
    __syncthreads();
    // the solves: threads 0-127 W_v, 128 columns at a time, threads 128-255 W_k
    auto solve = [&](float* x, int ld) {
#pragma unroll 1
        for (int b = 0; b < C; b += 16) {
            float acc[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[i] = 0.f;
#pragma unroll 1
            for (int j = 0; j < b; j += 4) {
                const float x0 = x[j * ld], x1 = x[(j + 1) * ld], x2 = x[(j + 2) * ld], x3 = x[(j + 3) * ld];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float4 a = *reinterpret_cast<const float4*>(as + (b + i) * PA + j);
                    acc[i] = fmaf(-a.x, x0, acc[i]); acc[i] = fmaf(-a.y, x1, acc[i]);
                    acc[i] = fmaf(-a.z, x2, acc[i]); acc[i] = fmaf(-a.w, x3, acc[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[i] = fmaf(bs[b + i], x[(b + i) * ld], acc[i]);
            // inside the block a finished row is taken out of all rows below it at once
#pragma unroll
            for (int jq = 0; jq < 16; jq += 4) {
                float4 a[16];
#pragma unroll
                for (int i = jq + 1; i < 16; ++i) a[i] = *reinterpret_cast<const float4*>(as + (b + i) * PA + b + jq);
#pragma unroll
                for (int i = jq + 1; i < 16; ++i) acc[i] = fmaf(-a[i].x, acc[jq], acc[i]);
#pragma unroll
                for (int i = jq + 2; i < 16; ++i) acc[i] = fmaf(-a[i].y, acc[jq + 1], acc[i]);
#pragma unroll
                for (int i = jq + 3; i < 16; ++i) acc[i] = fmaf(-a[i].z, acc[jq + 2], acc[i]);
#pragma unroll
                for (int i = jq + 4; i < 16; ++i) acc[i] = fmaf(-a[i].w, acc[jq + 3], acc[i]);
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) x[(b + i) * ld] = acc[i];
        }
    };
    for (int v0 = 0; v0 < vdim; v0 += 128) {
        if (tid < 128) {
            const int v = v0 + tid;
            if (v < vdim) {
                const float* src = p.qkv + (size_t)first * p.stride + p.v_off + (size_t)h * vdim + v;
#pragma unroll 32
                for (int i = 0; i < C; ++i) xs[i * 128 + tid] = i < n ? src[(size_t)i * p.stride] : 0.f;
                solve(xs + tid, 128);
                float* dst = out + at.u + v;
#pragma unroll 8
                for (int i = 0; i < C; ++i) dst[(size_t)i * vdim] = xs[i * 128 + tid];
            }
        } else if (v0 == 0 && tid - 128 < dim) {
            const int d = tid - 128;
            solve(gs + d, PD);
            float* dst = out + at.wk + (size_t)d * C;
#pragma unroll 4
            for (int i = 0; i < C; i += 4)
                *reinterpret_cast<float4*>(dst + i) = make_float4(gs[i * PD + d], gs[(i + 1) * PD + d], gs[(i + 2) * PD + d], gs[(i + 3) * PD + d]);
        }
    }
}

// ---- (2) -------------------------------------------------------------------------------------------------------------
// acc: 4 rows x 4 columns of sums of which each of the eight lanes that differ in their three low bits holds a share;
// afterwards a lane holds two neighbours of a row of them: row and first column returned as 4 * row + column.  Always added in
// the same order.
__device__ __forceinline__ int share_rows(const float2 (&acc)[4][2], int lane, float2& mine) {
    const bool b0 = lane & 1, b1 = lane & 2, b2 = lane & 4;
    float2 two[2][2], one[2];
    auto swap = [](float2 v, int o) { return make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o)); };
    auto plus = [](float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); };
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int v = 0; v < 2; ++v) two[r][v] = plus(b0 ? acc[r + 2][v] : acc[r][v], swap(b0 ? acc[r][v] : acc[r + 2][v], 1));
#pragma unroll
    for (int v = 0; v < 2; ++v) one[v] = plus(b1 ? two[1][v] : two[0][v], swap(b1 ? two[0][v] : two[1][v], 2));
    mine = plus(b2 ? one[1] : one[0], swap(b2 ? one[0] : one[1], 4));
    return 4 * ((b0 ? 2 : 0) + (b1 ? 1 : 0)) + (b2 ? 2 : 0);
}

// acc += a (four rows) times b (four columns)
__device__ __forceinline__ void patch(float2 (&acc)[4][2], const float4& a, const float4& b) {
    const float2 b0 = make_float2(b.x, b.y), b1 = make_float2(b.z, b.w);
    const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 a2 = make_float2(av[i], av[i]);
        acc[i][0] = __ffma2_rn(a2, b0, acc[i][0]);
        acc[i][1] = __ffma2_rn(a2, b1, acc[i][1]);
    }
}

template <int DM>
struct ScanSmem {
    static constexpr int PK = DM + 4;
    static constexpr size_t STAGE = (size_t)DM * PC + C * PK + C * VB + DM;       // W_k, k p_end, W_v, c_end of a chunk
    static constexpr size_t FLOATS = 2 * STAGE + (DM + C) * VP;
};

// Bound by its chain: per chunk two products of 64 x dim x 8 that follow one another, each on 256 threads (a thread a patch
// of 4 x 4 with an eighth of the terms, so that two 16-byte reads of shared memory feed 16 operations), with the next chunk's
// matrices copied meanwhile.  Eight value columns: with 8 heads and 128 values 128 CTAs (16 columns, 64 CTAs: 95 us for
// 2,048 rows where eight took 72, both with two-way bank conflicts that are gone since).
template <int DM>
__global__ void __launch_bounds__(256)
delta_scan_chunks_kernel(const Rows p, float* __restrict__ scratch, float* __restrict__ state, int* status) {
    constexpr int PK = ScanSmem<DM>::PK;
    constexpr size_t STAGE = ScanSmem<DM>::STAGE;
    extern __shared__ __align__(16) float sm[];
    float* Ss = sm + 2 * STAGE;                            // [DM][VP]
    float* us = Ss + DM * VP;                              // [C][VP]
    pdl_trigger();
    const int h = blockIdx.y, item = blockIdx.z, v0 = blockIdx.x * VB, tid = threadIdx.x, lane = tid & 31;
    const int slot = p.item_slot[item];
    int chunk0 = 0;
    for (int i = 0; i < item; ++i) chunk0 += (p.item_row_start[i + 1] - p.item_row_start[i] + C - 1) / C;
    const int n_chunks = (p.item_row_start[item + 1] - p.item_row_start[item] + C - 1) / C;
    pdl_wait();
    if (slot < 0 || slot >= p.n_slots) {
        if (tid == 0 && blockIdx.x == 0) report(status, IMPARO_ST_SLOT_RANGE, 73, item, slot);
        return;
    }
    const int dim = p.dim, vdim = p.vdim;
    const Layout at(dim, vdim);
    float* Sg = state + (((size_t)slot * p.heads + h) * dim) * vdim + v0;
    const size_t step = (size_t)p.heads * at.total;
    float* mine = scratch + ((size_t)chunk0 * p.heads + h) * at.total;
    // what no copy writes (channels from dim on, columns from vdim on) stays zero
    for (size_t e = tid; e < ScanSmem<DM>::FLOATS; e += 256) sm[e] = 0.f;
    __syncthreads();
    for (int e = tid; e < dim * (VB / 4); e += 256) {
        const int d = e / (VB / 4), v = (e % (VB / 4)) * 4;
        if (v0 + v < vdim) *reinterpret_cast<float4*>(Ss + d * VP + v) = *reinterpret_cast<const float4*>(Sg + (size_t)d * vdim + v);
    }
    auto fetch = [&](int c) {
        if (c < n_chunks) {
            const float* src = mine + (size_t)c * step;
            float* wk = sm + (c & 1) * STAGE;
            float* ke = wk + DM * PC;
            float* wv = ke + C * PK;
            float* ce = wv + C * VB;
            for (int e = tid; e < dim * (C / 4); e += 256) cp16(wk + (e / (C / 4)) * PC + (e % (C / 4)) * 4, src + at.wk + (size_t)e * 4);
            const int d4 = dim / 4;
            for (int e = tid; e < C * d4; e += 256) cp16(ke + (e / d4) * PK + (e % d4) * 4, src + at.kend + (size_t)e * 4);
            for (int e = tid; e < C * (VB / 4); e += 256) {
                const int i = e / (VB / 4), v = (e % (VB / 4)) * 4;
                if (v0 + v < vdim) cp16(wv + i * VB + v, src + at.u + (size_t)i * vdim + v0 + v);
            }
            for (int e = tid; e < d4; e += 256) cp16(ce + e * 4, src + at.cend + e * 4);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0);
    const int part = tid & 7, vq = ((tid >> 3) & 1) * 4, rq = (tid >> 4) * 4;      // terms part, part + 8, ...; columns; rows
    for (int c = 0; c < n_chunks; ++c) {
        fetch(c + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const float* wk = sm + (c & 1) * STAGE;
        const float* ke = wk + DM * PC;
        const float* wv = ke + C * PK;
        const float* ce = wv + C * VB;
        float* own = mine + (size_t)c * step;
        {
            float2 acc[4][2] = {}, sum;
#pragma unroll
            for (int k = 0; k < DM; k += 8)
                patch(acc, *reinterpret_cast<const float4*>(wk + (k + part) * PC + rq), *reinterpret_cast<const float4*>(Ss + (k + part) * VP + vq));
            const int e = share_rows(acc, lane, sum), r = rq + (e >> 2), v = vq + (e & 3);
            const float2 w = *reinterpret_cast<const float2*>(wv + r * VB + v);
            const float2 u = make_float2(w.x - sum.x, w.y - sum.y);
            *reinterpret_cast<float2*>(us + r * VP + v) = u;
            if (v0 + v < vdim) *reinterpret_cast<float2*>(own + at.u + (size_t)r * vdim + v0 + v) = u;
        }
        __syncthreads();
        // (every thread reads and writes its own entries of the state here)
#pragma unroll
        for (int dq = 0; dq < DM; dq += 64) {
            float2 acc[4][2] = {}, sum;
#pragma unroll
            for (int i = 0; i < C; i += 8)
                patch(acc, *reinterpret_cast<const float4*>(ke + (i + part) * PK + dq + rq), *reinterpret_cast<const float4*>(us + (i + part) * VP + vq));
            const int e = share_rows(acc, lane, sum), d = dq + rq + (e >> 2), v = vq + (e & 3);
            float2 s = *reinterpret_cast<const float2*>(Ss + d * VP + v);
            const float keep = ce[d];
            if (d < dim && v0 + v < vdim) *reinterpret_cast<float2*>(own + at.s_in + (size_t)d * vdim + v0 + v) = s;
            s = make_float2(fmaf(keep, s.x, sum.x), fmaf(keep, s.y, sum.y));
            *reinterpret_cast<float2*>(Ss + d * VP + v) = s;
        }
        __syncthreads();
    }
    for (int e = tid; e < dim * (VB / 4); e += 256) {
        const int d = e / (VB / 4), v = (e % (VB / 4)) * 4;
        if (v0 + v < vdim) *reinterpret_cast<float4*>(Sg + (size_t)d * vdim + v) = *reinterpret_cast<const float4*>(Ss + d * VP + v);
    }
}

// ---- (3) -------------------------------------------------------------------------------------------------------------
// A CTA owns 64 rows x 64 value columns, a thread a patch of 8 x 4: three 16-byte reads of shared memory per 32 operations.
template <int DM>
__global__ void __launch_bounds__(128)
delta_out_kernel(const Rows p, const float* __restrict__ scratch, float* __restrict__ o) {
    extern __shared__ __align__(16) float sm[];
    float* left = sm;                                      // [DM + C][C]   q c, then the output's matrix, column by column
    float* right = sm + (DM + C) * C;                      // [DM + C][64]  S_in, then u
    pdl_trigger();
    const int chunk = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * 64, tid = threadIdx.x;
    int item, first;
    const int n = chunk_rows<C>(p, chunk, item, first);
    pdl_wait();
    if (n == 0) return;
    const int slot = p.item_slot[item];
    if (slot < 0 || slot >= p.n_slots) return;             // (2) has recorded it
    const int dim = p.dim, vdim = p.vdim;
    const Layout at(dim, vdim);
    const float* own = scratch + ((size_t)chunk * p.heads + h) * at.total;
    for (int e = tid; e < dim * (C / 4); e += 128) cp16(left + e * 4, own + at.qc + (size_t)e * 4);
    for (int e = tid; e < C * (C / 4); e += 128) cp16(left + dim * C + e * 4, own + at.pt + (size_t)e * 4);
    for (int e = tid; e < (dim + C) * 16; e += 128) {
        const int k = e / 16, v = (e % 16) * 4;
        const float* src = k < dim ? own + at.s_in + (size_t)k * vdim : own + at.u + (size_t)(k - dim) * vdim;
        if (v0 + v < vdim) cp16(right + k * 64 + v, src + v0 + v);
        else *reinterpret_cast<float4*>(right + k * 64 + v) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int rq = (tid >> 4) * 8, vq = (tid & 15) * 4;
    float2 acc[8][2] = {}, inner[8][2] = {};                // from the starting state; from the chunk's own rows
    auto terms = [&](float2 (&t)[8][2], int from, int to) {
#pragma unroll 4
        for (int k = from; k < to; ++k) {
            const float4 a = *reinterpret_cast<const float4*>(left + k * C + rq), a1 = *reinterpret_cast<const float4*>(left + k * C + rq + 4);
            const float4 b = *reinterpret_cast<const float4*>(right + k * 64 + vq);
            const float2 b0 = make_float2(b.x, b.y), b1 = make_float2(b.z, b.w);
            const float av[8] = {a.x, a.y, a.z, a.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float2 a2 = make_float2(av[i], av[i]);
                t[i][0] = __ffma2_rn(a2, b0, t[i][0]);
                t[i][1] = __ffma2_rn(a2, b1, t[i][1]);
            }
        }
    };
    terms(acc, 0, dim);
    // rows of u before the thread's first, then its own, each row with the ones up to itself: a term beyond a row is left out and
    // not multiplied by zero, so that a row that is not finite reaches no earlier one
    terms(inner, dim, dim + rq);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const float4 a = *reinterpret_cast<const float4*>(left + (dim + rq + u) * C + rq), a1 = *reinterpret_cast<const float4*>(left + (dim + rq + u) * C + rq + 4);
        const float4 b = *reinterpret_cast<const float4*>(right + (dim + rq + u) * 64 + vq);
        const float2 b0 = make_float2(b.x, b.y), b1 = make_float2(b.z, b.w);
        const float av[8] = {a.x, a.y, a.z, a.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
        for (int i = u; i < 8; ++i) {
            const float2 a2 = make_float2(av[i], av[i]);
            inner[i][0] = __ffma2_rn(a2, b0, inner[i][0]);
            inner[i][1] = __ffma2_rn(a2, b1, inner[i][1]);
        }
    }
    if (v0 + vq >= vdim) return;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if (rq + i < n)
            *reinterpret_cast<float4*>(o + ((size_t)(first + rq + i) * p.heads + h) * vdim + v0 + vq) =
                make_float4(acc[i][0].x + inner[i][0].x, acc[i][0].y + inner[i][0].y, acc[i][1].x + inner[i][1].x, acc[i][1].y + inner[i][1].y);
}

template <int DM>
static int run(const Rows& p, int max_chunks, float* scratch, float* state, float* out, int* status, cudaStream_t stream) {
    constexpr size_t s1 = LocalSmem<DM>::FLOATS * 4, s2 = ScanSmem<DM>::FLOATS * 4, s3 = (size_t)(DM + C) * (C + 64) * 4;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(delta_local_kernel<DM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s1);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_scan_chunks_kernel<DM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s2);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_out_kernel<DM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s3);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    launch(delta_local_kernel<DM>, dim3(max_chunks, p.heads), dim3(256), s1, stream, p, scratch);
    IMPARO_CHECK_LAUNCH();
    launch(delta_scan_chunks_kernel<DM>, dim3((p.vdim + VB - 1) / VB, p.heads, p.n_items), dim3(256), s2, stream, p, scratch, state, status);
    IMPARO_CHECK_LAUNCH();
    launch(delta_out_kernel<DM>, dim3(max_chunks, p.heads, (p.vdim + 63) / 64), dim3(128), s3, stream, p, (const float*)scratch, out);
    IMPARO_CHECK_LAUNCH();
    return 0;
}

}  // namespace dc
}  // namespace imparo

using namespace imparo;

// Floats of scratch per chunk of 64 rows (0: sizes the chunks do not take: a key size that is no multiple of 4 or above 128, a
// value size that is no multiple of 4).
extern "C" long long imparo_delta_chunk_floats(int heads, int dim, int vdim) {
    if (heads < 1 || dim < 4 || dim > 128 || dim % 4 || vdim < 4 || vdim % 4) return 0;
    return (long long)heads * (long long)dc::Layout(dim, vdim).total;
}

// As imparo_delta_scan; max_chunks: at least the chunks of all requests (tokens / 64 + requests), scratch: max_chunks times
// imparo_delta_chunk_floats, 16-byte aligned.  -25: sizes, offsets or alignments it does not take.
extern "C" int imparo_delta_chunked(const float* qkv, long long qkv_stride, int q_off, int k_off, int v_off, const float* g,
                                    const float* beta, float* state, const int* item_row_start, const int* item_slot, int n_slots,
                                    int n_items, int max_chunks, float* scratch, float* out, int heads, int kv_heads, int dim,
                                    int vdim, int* status, cudaStream_t stream) {
    if (n_items <= 0 || max_chunks <= 0) return 0;
    if (heads < 1 || kv_heads < 1 || heads % kv_heads) return -2;
    if (imparo_delta_chunk_floats(heads, dim, vdim) == 0 || q_off % 4 || k_off % 4 || qkv_stride % 4) return -25;
    if (((uintptr_t)qkv | (uintptr_t)g | (uintptr_t)state | (uintptr_t)scratch | (uintptr_t)out) & 15) return -25;
    if (heads > 65535 || n_items > 65535) return -25;
    const dc::Rows p{qkv, (size_t)qkv_stride, q_off, k_off, v_off, g, beta, item_row_start, item_slot, n_items, n_slots, heads, kv_heads, dim, vdim};
    return dim <= 64 ? dc::run<64>(p, max_chunks, scratch, state, out, status, stream)
                     : dc::run<128>(p, max_chunks, scratch, state, out, status, stream);
}
