// Causal attention of prompt portions over the paged cache in 32-bit: tiles of 64 queries of one head against tiles of 64 keys.
//
// The split-key kernel (attention_split.cu) reads every key for every query: 1,000 tokens in three portions of 16 heads of 64 took
// 241 us with its combine.  Here a key is read once per 64 queries and both products run on patches of 8 x 4 in registers, so it is
// bound by the issue of 32-bit operations and, for few tiles, by the longest portion's last tile, whose CTA walks all of the
// request's keys: 94 us (B200; a warp per scheduler and CTA, so mostly latency).  Few rows over many keys are the split-key kernel's
// therefore (kernels/ops.py, attention_f32_tiles_pay).  Scores, softmax (expf, running maximum per row) and sums are 32-bit; keys are
// added tile by tile in order.
#include "common.cuh"
#include <type_traits>

namespace imparo {
namespace af {

constexpr int TQ = 64, TK = 64, THREADS = 128;

struct Params {
    const float* q; const float* k; const float* v; float* out;
    const int* item_row_start; const int* item_start_pos; const int* table;
    int n_items, max_blocks, page_size, n_pages, window, nh, nkv, hd;
    float scale;
    int* status;
};

// HM: head size, padded (64 or 128; channels from hd on are zero).  A thread owns rows lq .. lq + 7 and, of the scores, keys rq ..
// rq + 3, of the output columns rq .. rq + 3 (and + 64); the 16 lanes of a half warp share their rows.
template <int HM>
__global__ void __launch_bounds__(THREADS)
attn_prefill_f32_kernel(const Params p) {
    extern __shared__ __align__(16) float sm[];
    float* qt = sm;                          // [HM][TQ]
    float* kt = qt + HM * TQ;                // [HM][TK]
    float* vs = kt + HM * TK;                // [TK][HM]
    float* pt = vs + TK * HM;                // [TK][TQ]  probabilities by key; groups of four rows at a place that depends on the key
    __shared__ int cache_row[TK];
    pdl_trigger();
    const int tid = threadIdx.x, h = blockIdx.y, kvh = h / (p.nh / p.nkv);
    // tiles of all portions, the last ones (of the last portion) first: the longest walk of a portion starts early
    int total = 0;
    for (int i = 0; i < p.n_items; ++i) total += (p.item_row_start[i + 1] - p.item_row_start[i] + TQ - 1) / TQ;
    int g = total - 1 - (int)blockIdx.x, item = 0;
    if (g < 0) return;
    for (;; ++item) {
        const int tiles = (p.item_row_start[item + 1] - p.item_row_start[item] + TQ - 1) / TQ;
        if (g < tiles) break;
        g -= tiles;
    }
    const int row0 = p.item_row_start[item] + g * TQ, n = min(TQ, p.item_row_start[item + 1] - row0);
    const int pos0 = p.item_start_pos[item] + g * TQ;
    const int* tab = p.table + (size_t)item * p.max_blocks;
    pdl_wait();
    const size_t qw = (size_t)p.nh * p.hd, kw = (size_t)p.nkv * p.hd;
    for (int e = tid; e < TQ * (HM / 4); e += THREADS) {           // a lane a row: its four channels go to four rows of the transposed tile
        const int r = e % TQ, d = (e / TQ) * 4;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < n && d < p.hd) x = *reinterpret_cast<const float4*>(p.q + (size_t)(row0 + r) * qw + (size_t)h * p.hd + d);
        qt[d * TQ + r] = x.x; qt[(d + 1) * TQ + r] = x.y; qt[(d + 2) * TQ + r] = x.z; qt[(d + 3) * TQ + r] = x.w;
    }
    const int lq = (tid >> 4) * 8, rq = (tid & 15) * 4;
    constexpr int CB = HM / 64;
    float2 o[CB][8][2] = {};
    float m[8], l[8];
    int lo[8];                                                     // first key of each row
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        m[i] = -INFINITY; l[i] = 0.f;
        lo[i] = first_key(pos0 + lq + i, p.window, 0);
    }
    const int first = first_key(pos0, p.window, 0), last = pos0 + n;          // keys [first, last)
    for (int key0 = first; key0 < last; key0 += TK) {
        const int nk = min(TK, last - key0);
        __syncthreads();                                           // the tile before is no longer read
        if (tid < TK) {
            int row = -1;
            if (tid < nk) {
                const int block = (key0 + tid) / p.page_size;
                const int page = block < p.max_blocks ? tab[block] : -1;
                if (page < 0 || page >= p.n_pages) report(p.status, IMPARO_ST_PAGE_RANGE, 96, item, page);
                else row = page * p.page_size + (key0 + tid) % p.page_size;
            }
            cache_row[tid] = row;
        }
        __syncthreads();
        // values straight into place; keys through registers (a lane a key), eight 16-byte loads in flight
#pragma unroll 8
        for (int e = tid; e < TK * (HM / 4); e += THREADS) {
            const int r = e / (HM / 4), d = (e % (HM / 4)) * 4, row = cache_row[r];
            if (row >= 0 && d < p.hd)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(vs + r * HM + d)),
                             "l"(p.v + (size_t)row * kw + (size_t)kvh * p.hd + d) : "memory");
            else *reinterpret_cast<float4*>(vs + r * HM + d) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        {
            const int r = tid % TK, row = cache_row[r];
            const float* src = p.k + (size_t)(row >= 0 ? row : 0) * kw + (size_t)kvh * p.hd;
#pragma unroll
            for (int e0 = 0; e0 < HM / 4; e0 += 16) {              // (128 threads: two channel groups of four per step)
                float4 x[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int d = (e0 + 2 * u + tid / TK) * 4;
                    x[u] = (row >= 0 && d < p.hd) ? *reinterpret_cast<const float4*>(src + d) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int d = (e0 + 2 * u + tid / TK) * 4;
                    kt[d * TK + r] = x[u].x; kt[(d + 1) * TK + r] = x[u].y; kt[(d + 2) * TK + r] = x[u].z; kt[(d + 3) * TK + r] = x[u].w;
                }
            }
        }
        __syncthreads();
        float2 s[8][2] = {};
#pragma unroll 4
        for (int d = 0; d < HM; ++d) {
            const float4 a = *reinterpret_cast<const float4*>(qt + d * TQ + lq), b = *reinterpret_cast<const float4*>(qt + d * TQ + lq + 4);
            const float4 c = *reinterpret_cast<const float4*>(kt + d * TK + rq);
            const float2 c01 = make_float2(c.x, c.y), c23 = make_float2(c.z, c.w);
            const float av[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float2 a2 = make_float2(av[i], av[i]);
                s[i][0] = __ffma2_rn(a2, c01, s[i][0]);
                s[i][1] = __ffma2_rn(a2, c23, s[i][1]);
            }
        }
        float alpha[8];
        float pr[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int pos = pos0 + lq + i;
            const float sv[4] = {s[i][0].x, s[i][0].y, s[i][1].x, s[i][1].y};
            float top = -INFINITY;
            bool seen[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int key = key0 + rq + c;
                seen[c] = key <= pos && key >= lo[i] && cache_row[rq + c] >= 0;
                pr[i][c] = sv[c] * p.scale;
                if (seen[c]) top = fmaxf(top, pr[i][c]);
            }
#pragma unroll
            for (int w = 1; w < 16; w <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, w));
            const float m_new = fmaxf(m[i], top);
            alpha[i] = m_new == -INFINITY ? 1.f : expf(m[i] - m_new);         // (no key seen yet: nothing to scale)
            float sum = 0.f;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                pr[i][c] = seen[c] && m_new != -INFINITY ? expf(pr[i][c] - m_new) : 0.f;
                sum += pr[i][c];
            }
            l[i] = l[i] * alpha[i] + sum;
            m[i] = m_new;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int key = rq + c, turn = (key >> 2) & 15;
            float* row = pt + key * TQ;
            *reinterpret_cast<float4*>(row + (((lq >> 2) ^ turn) << 2)) = make_float4(pr[0][c], pr[1][c], pr[2][c], pr[3][c]);
            *reinterpret_cast<float4*>(row + ((((lq >> 2) + 1) ^ turn) << 2)) = make_float4(pr[4][c], pr[5][c], pr[6][c], pr[7][c]);
        }
#pragma unroll
        for (int b = 0; b < CB; ++b)
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int w = 0; w < 2; ++w) o[b][i][w] = __fmul2_rn(o[b][i][w], make_float2(alpha[i], alpha[i]));
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        // the tile's keys that all 16 rows of the warp see, [all0, all1), and before and after them those that some see: what a row
        // does not see is left out and not multiplied by zero, so that a key's row that is not finite reaches no other query
        const int w0 = pos0 + (lq & ~15);                              // position of the warp's first row
        const int seen0 = max(0, first_key(w0, p.window, 0) - key0), seen1 = min(nk, w0 + 16 - key0);
        const int all0 = min(max(seen0, first_key(w0 + 15, p.window, 0) - key0), seen1), all1 = max(all0, min(w0 + 1 - key0, seen1));
        auto add = [&](int k, auto masked) {
            const int turn = (k >> 2) & 15;
            const float4 a = *reinterpret_cast<const float4*>(pt + k * TQ + (((lq >> 2) ^ turn) << 2));
            const float4 b = *reinterpret_cast<const float4*>(pt + k * TQ + ((((lq >> 2) + 1) ^ turn) << 2));
            const float av[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int cb = 0; cb < CB; ++cb) {
                const float4 c = *reinterpret_cast<const float4*>(vs + k * HM + 64 * cb + rq);
                const float2 c01 = make_float2(c.x, c.y), c23 = make_float2(c.z, c.w);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (decltype(masked)::value && (key0 + k > pos0 + lq + i || key0 + k < lo[i])) continue;
                    const float2 a2 = make_float2(av[i], av[i]);
                    o[cb][i][0] = __ffma2_rn(a2, c01, o[cb][i][0]);
                    o[cb][i][1] = __ffma2_rn(a2, c23, o[cb][i][1]);
                }
            }
        };
        // (a loop of its own for whole tiles: 8,000 keys at head size 128 1,483 us with it and 1,663 us without; at 64 1,233 and 961)
        if (HM == 128 && all0 == 0 && all1 == TK) {
#pragma unroll 4
            for (int k = 0; k < TK; ++k) add(k, std::false_type{});
        } else {
#pragma unroll 1
            for (int k = seen0; k < all0; ++k) add(k, std::true_type{});
#pragma unroll 4
            for (int k = all0; k < all1; ++k) add(k, std::false_type{});
#pragma unroll 1
            for (int k = all1; k < seen1; ++k) add(k, std::true_type{});
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float sum = l[i];
#pragma unroll
        for (int w = 1; w < 16; w <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
        const float inv = sum > 0.f ? sum : 1.f;
        if (lq + i < n) {
#pragma unroll
            for (int cb = 0; cb < CB; ++cb) {
                const int d = 64 * cb + rq;
                if (d < p.hd)
                    *reinterpret_cast<float4*>(p.out + (size_t)(row0 + lq + i) * qw + (size_t)h * p.hd + d) =
                        make_float4(o[cb][i][0].x / inv, o[cb][i][0].y / inv, o[cb][i][1].x / inv, o[cb][i][1].y / inv);
            }
        }
    }
}

template <int HM>
static int run(const Params& p, int tiles, cudaStream_t stream) {
    constexpr size_t smem = (size_t)(HM * TQ + HM * TK + TK * HM + TK * TQ) * 4;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(attn_prefill_f32_kernel<HM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    launch(attn_prefill_f32_kernel<HM>, dim3(tiles, p.nh), dim3(THREADS), smem, stream, p);
    IMPARO_CHECK_LAUNCH();
    return 0;
}

}  // namespace af
}  // namespace imparo

using namespace imparo;

// q, out: float32 [n_tok, nh * hd]; caches float32 [n_pages, page_size, nkv * hd]; the portions' rows are those from
// item_row_start[0] on.  -25: a head size that is no multiple of 4 or above 128, addresses that are no multiples of 16 bytes.
extern "C" int imparo_attention_prefill_f32(const float* q, const float* k_cache, const float* v_cache, const int* item_row_start,
                                            const int* item_start_pos, int n_items, const int* table, int max_blocks, int page_size,
                                            int n_pages, int window, float scale, float* out, int n_tok, int nh, int nkv, int hd,
                                            int* status, cudaStream_t stream) {
    if (n_tok <= 0 || n_items <= 0) return 0;
    if (nkv < 1 || nh % nkv) return -5;
    if (hd < 4 || hd > 128 || hd % 4 || nh > 65535 || (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out) & 15)) return -25;
    const af::Params p{q, k_cache, v_cache, out, item_row_start, item_start_pos, table, n_items, max_blocks, page_size, n_pages, window, nh, nkv, hd,
                       scale, status};
    if ((long long)n_tok / af::TQ + n_items > 0x7fffffff) return -2;
    const int tiles = n_tok / af::TQ + n_items;                    // at least the portions' tiles
    return hd <= 64 ? af::run<64>(p, tiles, stream) : af::run<128>(p, tiles, stream);
}
