// bfloat16 products of at most eight rows (a decode step of few requests):
//     out[T, N] (+)= f(X)[T, K] * W[N, K]^T,   T <= 8, 32-bit accumulation
// with what used to be kernels of their own at both ends: the RMS norm of the 32-bit stream on the way in, and the gate, the
// add into the stream or the gated short convolution of one-token rows on the way out.
//
// What bounds it: W streams from HBM once, and a step is a chain of some hundred such products, so what the kernels cost beside
// their bytes counts as much.  So K stays whole inside a CTA (no split partials to fold by a later kernel, no cluster), every SM
// gets the same number of output features to within one (F / 148, any number: no tile of 128 rows that leaves SMs idle), and
// all weights that the ring holds (64 KB) are requested before the wait on the kernel ahead.
//
// A ninth warp copies W into a ring of stages, two tiles of 8 rows by 512 k each: W is seen as [k / 64][row][64 k], so that one tensor
// copy brings a tile of any first row, 8 KB, in 128-byte lines swizzled by row.  The eight others share a stage's k: a warp owns two
// groups of 32.  Sixteen rows of W are the M of mma.sync.m16n8k16 and the T tokens its N; k is permuted inside a group of 32 the
// same way for both operands (lane c of a row holds k = 8c .. 8c+7), so a 16-byte load is two fragments.  The tokens of a stretch of
// 2,048 k stay in registers.  At the end the eight warps' sums meet in shared memory and are added in warp order.
// (The tensor cores run at a few percent of their rate here, so tcgen05 would gain nothing: eight tokens fill a sixteenth of its
// smallest tile, and its accumulator would have to come back through tensor memory.  W by untiled copies of 1 KB, or by 16-byte
// cp.async of every thread, streamed at 3.4 TB/s with as many bytes in flight, this way at 5.5.)
//
// B200, one token / eight: gate+up 16,384 x 2,048 with its norm 13.9 / 14.9 us (the weight streamer and the norm kernel 13.4 + 3 / 13.9 +
// 3.3), 2,048 x 8,192 7.8 / 8.7, 2,048 x 2,048 2.5 / 3.1.  Whole decode steps, before / after: 350M one row 456 / 362 us, eight rows
// 505 / 439; 1.2B one row 722 / 647, four rows 783 / 703, eight rows 770 / 771: there every SM's reading of the whole input costs what
// was saved, and most of that step's products go elsewhere (FEW_ROWS_STREAM and _rows_pay in kernels/ops.py).
//
// Every wait on an mbarrier is bounded: when one runs out the kernel records IMPARO_ST_WAIT_LIMIT in the status word, stops waiting,
// lets its copies land (again with a limit) and returns.
#include "tcgen05.cuh"

namespace imparo {
namespace nr {

using tc::mbar_init;
using tc::mbar_expect_tx;
using tc::BK;
using tc::smem_u32;

constexpr int WARPS = 8, THREADS = 32 * WARPS;  // the multiplying warps; one more copies
constexpr int MAX_T = 8;
constexpr int GROUPS = 8;                       // groups of 32 k that a warp takes of one stretch
constexpr int STRETCH = WARPS * GROUPS * 32;    // 2,048 k
constexpr int BATCH = 2;                        // groups that a warp takes of one stage
constexpr int SPAN = WARPS * BATCH * 32;        // k of a stage: 512
constexpr int TILE_BYTES = 8 * SPAN * 2;        // [8 blocks of 64 k][8 rows][128 bytes]
constexpr int STAGE_BYTES = 2 * TILE_BYTES;
constexpr int STAGES = 4;                       // 64 KB: with what else a CTA needs, the next kernel's CTA fits beside this one
constexpr int RING_BYTES = STAGES * STAGE_BYTES;
constexpr int ALIGN_SLACK = 1024;               // tiles lie on 1,024 bytes
constexpr int RED_STRIDE = 10;                  // floats per row of the warps' sums (8 tokens; even, and few bank conflicts)
constexpr int MAX_TILES = 8;                    // most pairs of 8-row tiles of a CTA: 128 rows of W
constexpr int CONV_TAPS = 4;                    // most taps of the fused convolution

enum Input { IN_BF16 = 0, IN_NORM = 1 };
enum Output { OUT_BF16 = 0, OUT_F32 = 1, OUT_ADD = 2, OUT_GATED = 3, OUT_CONV = 4 };

struct Params {
    const void* x;              // IN_BF16: bfloat16 [T, ldx]; IN_NORM: the float32 stream [T, ldx]
    const float* nw;            // IN_NORM: the norm's weight [K]
    float eps;
    const __nv_bfloat16* w;     // [parts * F, K], part p's rows from p * F on (parts: 1; OUT_GATED 2; OUT_CONV 3)
    void* out;                  // [T, ldo]
    int T, F, K, ldx, ldo;
    int max_nd;                 // the most pairs of 8-row tiles of a CTA
    int act;                    // OUT_GATED: gated_act's kind, its limit and the two products' biases ([2F], or null)
    float limit;
    const float* bias;
    // OUT_CONV: rows b, c, x of the product -> y = c * (taps over b * x and the state), state moved on by one
    const float* taps;          // [F, n_taps]
    const float* conv_bias;     // [F] or null
    float* state;               // [slots, n_taps - 1, F]
    const int* item_of_token;
    const int* item_slot;
    int n_taps, n_slots;
    int* status;
};

// false when the wait ran out: two seconds of the device's clock
__device__ __noinline__ bool wait_long(uint64_t* bar, uint32_t parity) {
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    do {
        if (tc::mbar_wait(bar, parity, 16)) return true;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    } while (t - t0 < 2000000000ULL);
    return false;
}
__device__ __forceinline__ bool wait_for(uint64_t* bar, uint32_t parity) { return tc::mbar_wait(bar, parity, 1) || wait_long(bar, parity); }
// all multiplying warps, and not the copying one
__device__ __forceinline__ void workers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); }

// a tile: 8 rows from `row` on, 512 k from block `kb` of 64 on (rows and blocks beyond the matrix: zeros)
__device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int row, int kb) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(dst), "l"(map), "r"(smem_u32(bar)), "r"(0), "r"(row), "r"(kb) : "memory");
}
__device__ __forceinline__ uint4 lds16(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float rounded(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

template <int OUT> struct Parts { static constexpr int value = OUT == OUT_GATED ? 2 : OUT == OUT_CONV ? 3 : 1; };

// shared memory: the ring; then the warps' sums ([warp][row][RED_STRIDE], nd pairs of tiles), and in the same place before them, with
// IN_NORM, the normed tokens and the norm's weight
__host__ __device__ constexpr size_t red_bytes(int nd) { return (size_t)WARPS * nd * 16 * RED_STRIDE * 4; }
// bytes of a normed token's row: the banks again
__host__ __device__ constexpr int tok_pitch(int K) { return (K * 2 + 127) / 128 * 128 + 64; }
__host__ __device__ constexpr size_t norm_bytes(int T, int K) { return (size_t)T * tok_pitch(K) + (size_t)K * 4; }

// The loops over stretches, pairs of tiles and stages are not unrolled, and a pair's sums go to shared memory when its stretch ends:
// a CTA runs every stage once, and with all of them as straight code (30 KB for 110 rows) eight rows through the norm cost
// 5 us more, for the fetching of instructions.
template <int IN, int OUT>
__device__ __forceinline__ void rows_product(const CUtensorMap& map_w, const Params& p) {
    constexpr int P = Parts<OUT>::value;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[STAGES], empty[STAGES];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, c = lane & 3;                   // row of a tile and token; which 16 bytes of a group
    const int f0 = (int)((long long)p.F * blockIdx.x / gridDim.x), f1 = (int)((long long)p.F * (blockIdx.x + 1) / gridDim.x);
    const int nf = f1 - f0;
    const int tiles = P * ((nf + 7) >> 3);                   // 8-row tiles: the parts of features f0 .. f0+7, then of the next eight
    const int nd = (tiles + 1) >> 1;                         // pairs of them: the 16 rows of a stage
    const int n_stretch = (p.K + STRETCH - 1) / STRETCH;
    float* red = reinterpret_cast<float*>(smem + RING_BYTES);
    uint8_t* toks = smem + RING_BYTES;
    const int pitch = tok_pitch(p.K);
    float* nws = reinterpret_cast<float*>(toks + p.T * pitch);

    pdl_trigger();
    if (tid == 0) {
#pragma unroll
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == WARPS) {
        // ---- the copies, stage after stage in the order they are multiplied.  W is written by no kernel: nothing here waits for the
        // kernel ahead ----
        int i = 0;
        bool ok = lane == 0;
#pragma unroll 1
        for (int s = 0; s < n_stretch && ok; ++s) {
            const int k_end = min(p.K, (s + 1) * STRETCH);
#pragma unroll 1
            for (int d = 0; d < nd && ok; ++d) {
                const int t0 = 2 * d, t1 = 2 * d + 1;
                const int row0 = (t0 % P) * p.F + f0 + (t0 / P) * 8, row1 = (t1 % P) * p.F + f0 + (t1 / P) * 8;
                const bool two = t1 < tiles;
#pragma unroll 1
                for (int k0 = s * STRETCH; k0 < k_end; k0 += SPAN, ++i) {
                    const int st = i % STAGES;
                    if (i >= STAGES && !wait_for(&empty[st], ((i / STAGES) - 1) & 1)) { ok = false; break; }
                    mbar_expect_tx(&full[st], two ? STAGE_BYTES : TILE_BYTES);
                    const uint32_t dst = smem_u32(smem) + st * STAGE_BYTES;
                    load_tile(dst, &map_w, &full[st], row0, k0 / BK);
                    if (two) load_tile(dst + TILE_BYTES, &map_w, &full[st], row1, k0 / BK);
                }
            }
        }
        if (lane == 0) {
            if (!ok) report(p.status, IMPARO_ST_WAIT_LIMIT, 50, blockIdx.x, i);
            // the last copies land before the warp leaves, also where the multiplying warps gave up on them
            for (int u = max(0, i - STAGES); u < i; ++u) wait_for(&full[u % STAGES], (u / STAGES) & 1);
        }
        __syncwarp();
        pdl_wait();                                          // (the chain's order: no kernel is complete before the one ahead)
        return;
    }

    if (IN == IN_NORM) {
#pragma unroll 1
        for (int i = tid * 4; i < p.K; i += THREADS * 4) *reinterpret_cast<float4*>(nws + i) = __ldg(reinterpret_cast<const float4*>(p.nw + i));
    }
    // what the end needs and no kernel writes
    const int items = nf * p.T;
    const int t_own = tid / nf, f_own = tid - t_own * nf;    // (the first of this thread's results)
    float tap[CONV_TAPS], cbias = 0.f;
    int slot = -1;
    if (OUT == OUT_CONV && tid < items) {
#pragma unroll
        for (int k = 0; k < CONV_TAPS; ++k) tap[k] = k < p.n_taps ? __ldg(p.taps + (size_t)(f0 + f_own) * p.n_taps + k) : 0.f;
        if (p.conv_bias) cbias = __ldg(p.conv_bias + f0 + f_own);
        slot = p.item_slot[p.item_of_token[t_own]];
    }
    pdl_wait();

    float state[CONV_TAPS - 1], old = 0.f;
    if (OUT == OUT_ADD && tid < items) old = __ldcg(reinterpret_cast<const float*>(p.out) + (size_t)t_own * p.ldo + f0 + f_own);
    if (OUT == OUT_CONV && tid < items && slot >= 0 && slot < p.n_slots) {
#pragma unroll
        for (int e = 0; e < CONV_TAPS - 1; ++e)
            state[e] = e < p.n_taps - 1 ? __ldcg(p.state + ((size_t)slot * (p.n_taps - 1) + e) * p.F + f0 + f_own) : 0.f;
    }
    if (IN == IN_NORM) {
        // a warp a token: its row in registers, normed into shared memory
        workers_sync();                                      // the norm's weight is there
        if (warp < p.T) {
            const float4* xr = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.x) + (size_t)warp * p.ldx) + lane;
            constexpr int NV = STRETCH / 128;
            float4 v[NV];
#pragma unroll
            for (int j = 0; j < NV; ++j) v[j] = (j * 32 + lane) * 4 < p.K ? __ldcg(xr + j * 32) : make_float4(0.f, 0.f, 0.f, 0.f);
            float ss = 0.f;
#pragma unroll
            for (int j = 0; j < NV; ++j) ss += v[j].x * v[j].x + v[j].y * v[j].y + v[j].z * v[j].z + v[j].w * v[j].w;
            ss = warp_sum(ss);
            const float scale = 1.0f / sqrtf(ss / (float)p.K + p.eps);
            uint8_t* row = toks + warp * pitch;
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                const int k = (j * 32 + lane) * 4;
                if (k < p.K) {
                    const float4 w = *reinterpret_cast<const float4*>(nws + k);
                    *reinterpret_cast<uint2*>(row + k * 2) = make_uint2(pack2(v[j].x * scale * w.x, v[j].y * scale * w.y),
                                                                        pack2(v[j].z * scale * w.z, v[j].w * scale * w.w));
                }
            }
        }
        workers_sync();
    }

    // ---- multiply: lane (g, c) holds token g's k = 8c .. 8c+7 of every group ----
    // this lane's 16 bytes of a stage's first group (the second is four blocks of 64 k on): two lanes of a quarter share a bank
    const uint32_t mine = smem_u32(smem) + (warp >> 1) * 1024 + g * 128 + ((((warp & 1) * 4 + c) ^ g) << 4);
    float* sums = red + ((size_t)warp * p.max_nd * 16 + g) * RED_STRIDE + 2 * c;
    int i = 0;
    bool ok = true;
#pragma unroll 1
    for (int s = 0; s < n_stretch && ok; ++s) {
        uint4 tok[GROUPS];
#pragma unroll
        for (int j = 0; j < GROUPS; ++j) {
            const int k = s * STRETCH + (j * WARPS + warp) * 32 + c * 8;
            tok[j] = make_uint4(0u, 0u, 0u, 0u);
            if (g < p.T && k < p.K) {
                if (IN == IN_NORM) tok[j] = *reinterpret_cast<const uint4*>(toks + g * pitch + k * 2);
                else tok[j] = __ldcg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.x) + (size_t)g * p.ldx + k));
            }
        }
        if (IN == IN_NORM) workers_sync();                   // the sums may be written over the tokens
#pragma unroll 1
        for (int d = 0; d < nd && ok; ++d) {
            float acc[4] = {0.f, 0.f, 0.f, 0.f}, more[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int b = 0; b < GROUPS / BATCH; ++b) {
                const int k = s * STRETCH + b * SPAN;
                if (k >= p.K) break;
                const int st = i % STAGES;
                ok = __all_sync(0xffffffffu, wait_for(&full[st], (i / STAGES) & 1));
                if (!ok) break;
                ++i;
                uint4 a[BATCH][2];
#pragma unroll
                for (int u = 0; u < BATCH; ++u) {
                    const uint32_t at = mine + st * STAGE_BYTES + u * 4096;
                    a[u][0] = lds16(at);
                    a[u][1] = lds16(at + TILE_BYTES);        // (a pair's second tile that does not exist: rows nobody reads)
                }
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty[st])) : "memory");
#pragma unroll
                for (int u = 0; u < BATCH; ++u) {
                    const uint4 x = tok[b * BATCH + u];
                    mma16816(u & 1 ? more : acc, a[u][0].x, a[u][1].x, a[u][0].y, a[u][1].y, x.x, x.y);
                    mma16816(u & 1 ? more : acc, a[u][0].z, a[u][1].z, a[u][0].w, a[u][1].w, x.z, x.w);
                }
            }
            // rows g and g + 8 of the pair, tokens 2c and 2c + 1 (this lane's own place)
            float2* r0 = reinterpret_cast<float2*>(sums + (size_t)d * 16 * RED_STRIDE);
            float2* r1 = reinterpret_cast<float2*>(sums + ((size_t)d * 16 + 8) * RED_STRIDE);
            float2 u = make_float2(acc[0] + more[0], acc[1] + more[1]), v = make_float2(acc[2] + more[2], acc[3] + more[3]);
            if (s > 0) { u.x += r0->x; u.y += r0->y; v.x += r1->x; v.y += r1->y; }
            *r0 = u;
            *r1 = v;
        }
    }
    if (!ok && lane == 0) report(p.status, IMPARO_ST_WAIT_LIMIT, 51, blockIdx.x, i);
    workers_sync();

    auto sum_of = [&](int part, int f, int t) {              // feature f0 + f of a part, token t: the warps in order
        const float* r = red + (((size_t)(f >> 3) * P + part) * 8 + (f & 7)) * RED_STRIDE + t;
        float v = 0.f;
#pragma unroll
        for (int u = 0; u < WARPS; ++u) v += r[(size_t)u * p.max_nd * 16 * RED_STRIDE];
        return v;
    };
#pragma unroll 1
    for (int item = tid; item < items; item += THREADS) {
        const int t = item / nf, f = item - t * nf;
        const size_t o = (size_t)t * p.ldo + f0 + f;
        if (OUT == OUT_BF16) {
            reinterpret_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(sum_of(0, f, t));
        } else if (OUT == OUT_F32) {
            reinterpret_cast<float*>(p.out)[o] = sum_of(0, f, t);
        } else if (OUT == OUT_ADD) {
            if (item != tid) old = __ldcg(reinterpret_cast<const float*>(p.out) + o);
            reinterpret_cast<float*>(p.out)[o] = old + sum_of(0, f, t);
        } else if (OUT == OUT_GATED) {
            float a = sum_of(0, f, t), u = sum_of(1, f, t);
            if (p.bias) { a += __ldg(p.bias + f0 + f); u += __ldg(p.bias + p.F + f0 + f); }
            reinterpret_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(gated_act_bf16(p.act, p.limit, a, u));
        } else {                                             // OUT_CONV: one item per thread
            if (slot < 0 || slot >= p.n_slots) {
                if (f == 0) report(p.status, IMPARO_ST_SLOT_RANGE, 4, p.item_of_token[t], slot);
                continue;
            }
            // the product's rows rounded as the tensor between the two kernels was
            const float bx = rounded(sum_of(0, f, t)) * rounded(sum_of(2, f, t));
            const float gate = rounded(sum_of(1, f, t));
            const int hist = p.n_taps - 1;
            float y = 0.f;
#pragma unroll
            for (int k = 0; k < CONV_TAPS; ++k) {
                if (k < hist) y += tap[k] * state[k < CONV_TAPS - 1 ? k : 0];
                else if (k == hist) y += tap[k] * bx;
            }
            reinterpret_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(gate * (y + cbias));
            float* st = p.state + (size_t)slot * hist * p.F + f0 + f;
#pragma unroll
            for (int e = 0; e < CONV_TAPS - 1; ++e)
                if (e < hist) st[(size_t)e * p.F] = e + 1 < hist ? state[e + 1 < CONV_TAPS - 1 ? e + 1 : 0] : bx;
        }
    }
}

template <int IN, int OUT>
__global__ void __launch_bounds__(THREADS + 32, 2) rows_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ Params p) {
    rows_product<IN, OUT>(map_w, p);
}

}  // namespace nr

// (a name of its own in profiles and timelines)
template <int IN>
__global__ void __launch_bounds__(nr::THREADS + 32, 2)
gated_conv_product_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ nr::Params p) {
    nr::rows_product<IN, nr::OUT_CONV>(map_w, p);
}

namespace nr {

// Features a CTA takes, and how many CTAs: one per SM (a second wave would wait for the first), as long as its rows fit the
// accumulators; nothing otherwise.
static int plan(int parts, int T, int F, int sms, bool conv, int* tiles) {
    const int grid = F < sms ? F : sms;
    const int nf = (F + grid - 1) / grid;
    const int nd = (parts * ((nf + 7) / 8) + 1) / 2;
    if (nd > MAX_TILES || (conv && nf * T > THREADS)) return 0;
    *tiles = nd;
    return grid;
}

template <int IN, int OUT>
static int launch_rows(const CUtensorMap& mw, const Params& p, int grid, cudaStream_t stream, bool configure) {
    void (*kern)(CUtensorMap, Params);
    if constexpr (OUT == OUT_CONV) kern = gated_conv_product_kernel<IN>;
    else kern = rows_kernel<IN, OUT>;
    auto bytes = [](int nd, int T, int K) {
        const size_t sums = red_bytes(nd), norm = IN == IN_NORM ? norm_bytes(T, K) : 0;
        return ALIGN_SLACK + RING_BYTES + (sums > norm ? sums : norm);
    };
    static_assert(RING_BYTES + red_bytes(MAX_TILES) <= 113 * 1024 && RING_BYTES + norm_bytes(MAX_T, STRETCH) <= 113 * 1024, "two CTAs per SM");
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes(MAX_TILES, MAX_T, STRETCH)));
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    if (configure) return 0;
    launch(kern, dim3(grid), dim3(THREADS + 32), bytes(p.max_nd, p.T, p.K), stream, mw, p);
    IMPARO_CHECK_LAUNCH();
    return 0;
}
template <int IN>
static int launch_out(int out_kind, const CUtensorMap& mw, const Params& p, int grid, cudaStream_t stream, bool configure) {
    switch (out_kind) {
        case OUT_BF16: return launch_rows<IN, OUT_BF16>(mw, p, grid, stream, configure);
        case OUT_F32: return launch_rows<IN, OUT_F32>(mw, p, grid, stream, configure);
        case OUT_ADD: return launch_rows<IN, OUT_ADD>(mw, p, grid, stream, configure);
        case OUT_GATED: return launch_rows<IN, OUT_GATED>(mw, p, grid, stream, configure);
        case OUT_CONV: return launch_rows<IN, OUT_CONV>(mw, p, grid, stream, configure);
    }
    return -22;
}

static int sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 0;
    }
    return n;
}

// W [rows, K] as [K / 64][rows][64], boxes of 8 blocks by 8 rows
static int get_tiles_map(const void* w, uint64_t rows, uint64_t K, CUtensorMap* out) {
    std::lock_guard<std::mutex> lock(tc::g_mutex);
    if (!tc::g_encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
        if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn) return -20;
        tc::g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled>(fn);
    }
    const tc::MapKey key{w, rows, K, K, 8};
    auto it = tc::g_maps.find(key);
    if (it != tc::g_maps.end()) { *out = it->second; return 0; }
    if (tc::g_maps.size() > 4096) tc::g_maps.clear();
    CUtensorMap m;
    const cuuint64_t dims[3] = {(cuuint64_t)BK, rows, K / BK};
    const cuuint64_t strides[2] = {K * 2, BK * 2};
    const cuuint32_t box[3] = {(cuuint32_t)BK, 8, SPAN / BK};
    const cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = tc::g_encode(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(w), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return -21;
    tc::g_maps.emplace(key, m);
    *out = m;
    return 0;
}

static int run(int in_kind, int out_kind, Params& p, cudaStream_t stream) {
    if (p.T <= 0 || p.F <= 0) return 0;
    if (p.T > MAX_T) return -25;
    if (p.K % BK != 0) return -25;
    if (p.K <= 0 || (((uintptr_t)p.x | (uintptr_t)p.w) & 15)) return -23;
    if (in_kind == IN_NORM && (((uintptr_t)p.nw) & 15)) return -23;
    if (in_kind == IN_NORM ? (p.K > STRETCH || p.ldx % 4 != 0) : p.ldx % 8 != 0) return in_kind == IN_NORM && p.K > STRETCH ? -25 : -23;
    const int parts = out_kind == OUT_GATED ? 2 : out_kind == OUT_CONV ? 3 : 1;
    int nd = 0;
    const int sms = sm_count();
    if (sms <= 0) return -25;
    const int grid = plan(parts, p.T, p.F, sms, out_kind == OUT_CONV, &nd);
    if (grid == 0) return -25;
    p.max_nd = nd;
    CUtensorMap mw;
    const int rc = get_tiles_map(p.w, (uint64_t)parts * p.F, (uint64_t)p.K, &mw);
    if (rc) return rc;
    return in_kind == IN_NORM ? launch_out<IN_NORM>(out_kind, mw, p, grid, stream, false) : launch_out<IN_BF16>(out_kind, mw, p, grid, stream, false);
}

}  // namespace nr
}  // namespace imparo

using namespace imparo::nr;

// out = f(x) w^T for at most eight rows.  norm (float32 [K]) given: x is a float32 stream [T, K] with row stride ldx, and its RMS norm
// is what is multiplied; else x is bfloat16.  out_kind: 0 bfloat16, 1 float32, 2 added to float32, 3 gated (w [2F, K], act / limit /
// bias as in imparo_gemm_tc_gated).  -25: not a case for this kernel (nothing was launched).
extern "C" int imparo_gemm_rows(const void* x, int ldx, const float* norm, float eps, const void* w, void* out, int ldo, int T, int F,
                                int K, int out_kind, int act, float limit, const float* bias, int* status, cudaStream_t stream) {
    if (out_kind < 0 || out_kind > OUT_GATED || act < 0 || act > 2) return -22;
    Params p = {};
    p.x = x; p.ldx = ldx; p.nw = norm; p.eps = eps; p.w = reinterpret_cast<const __nv_bfloat16*>(w); p.out = out; p.ldo = ldo;
    p.T = T; p.F = F; p.K = K; p.act = act; p.limit = limit; p.bias = bias; p.status = status;
    return run(norm ? IN_NORM : IN_BF16, out_kind, p, stream);
}

// The input product of the gated short convolution and the convolution itself, for one-token rows: w [3F, K] (rows b, c, x),
// y [T, F] bfloat16; taps, bias, state as in imparo_gated_conv.  Every token is a request's only one.
extern "C" int imparo_gemm_rows_conv(const void* x, int ldx, const float* norm, float eps, const void* w, const float* taps,
                                     const float* conv_bias, float* state, const int* item_of_token, const int* item_slot, void* y,
                                     int T, int F, int K, int n_taps, int n_slots, int* status, cudaStream_t stream) {
    if (n_taps < 2 || n_taps > CONV_TAPS) return -25;
    Params p = {};
    p.x = x; p.ldx = ldx; p.nw = norm; p.eps = eps; p.w = reinterpret_cast<const __nv_bfloat16*>(w); p.out = y; p.ldo = F;
    p.T = T; p.F = F; p.K = K; p.taps = taps; p.conv_bias = conv_bias; p.state = state; p.item_of_token = item_of_token;
    p.item_slot = item_slot; p.n_taps = n_taps; p.n_slots = n_slots; p.status = status;
    return run(norm ? IN_NORM : IN_BF16, OUT_CONV, p, stream);
}

// Whether the kernel takes a product (its shape only): 1 or 0.
extern "C" int imparo_gemm_rows_takes(int T, int F, int K, int parts, int norm, int sms) {
    int nd = 0;
    return T >= 1 && T <= MAX_T && F >= 1 && K >= BK && K % BK == 0 && (!norm || K <= STRETCH) && plan(parts, T, F, sms, parts == 3, &nd) > 0;
}

// Every instantiation's shared-memory attribute, ahead of the first launch (refused while a stream is being captured).
extern "C" int imparo_gemm_rows_configure() {
    Params p = {};
    CUtensorMap m = {};
    if (sm_count() <= 0) return -25;
    for (int out = OUT_BF16; out <= OUT_CONV; ++out) {
        int rc = launch_out<IN_NORM>(out, m, p, 1, nullptr, true);
        if (!rc) rc = launch_out<IN_BF16>(out, m, p, 1, nullptr, true);
        if (rc) return rc;
    }
    return 0;
}
