// True 32-bit matrix product: out[M,N] (+)= A[M,K] * W[N,K]^T.
//
// This is the matrix product of the 32-bit path.  Layout follows the reference: W[n_out, n_in] row-major,
// y[t,o] = sum_i W[o,i]*x[t,i] (imparo-cpu/src/ops.rs:660,688-690).  A row's result depends neither on how many other
// rows the call carries nor on where in the call it stands.
//
//  (1) sgemm_split_kernel: rows of 16-byte groups.  Every 32-bit operand is cut into three bfloat16 pieces, h + m / 2^8 +
//      l / 2^16, that add up to it to its last bit (8 + 8 + 8 significant bits, each piece rounded to nearest, so the
//      remainders carry either sign; held at their own scales, the lower pieces keep all their bits however small the operand
//      is), and six of the nine products of pieces run on the tensor cores: what is left out is below 2^-26 of a product, a
//      quarter of a 32-bit rounding, or, where an operand is subnormal, below 2^-151 of the other operand, a quarter of half
//      its last place.  The large product of a stretch of 64 k (h times h) is summed by the tensor core into an accumulator
//      of its own, read back and added to the others' in registers with 32-bit rounding: the tensor core's accumulator
//      truncates, and over a whole K that adds up to more than the FFMA chain's error.  The small products, 2^-8 and 2^-16
//      of it, have an accumulator each over all of K, at their scales, so that what they add to a small result is not lost
//      below the smallest 32-bit number.  At the upper end a result that is not finite (an operand whose first piece
//      rounds to infinity, a sum that overflows) is computed again by the FFMA chain, which then says what it is.
//  (2) sgemm_nt_kernel: everything else, FFMA only, one accumulator per element summed over k = 0..K-1 in order.
#include "tcgen05.cuh"

namespace imparo {

// ---- (2) ----------------------------------------------------------------------------------------------------------
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

__global__ void __launch_bounds__(256)
sgemm_nt_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                int M, int N, int K, int lda, int ldc, int accumulate) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = tid % 16, ty = tid / 16;        // 16 x 16 threads, each 4 x 4 outputs
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        // each thread loads 4 elements of each tile: row = idx / BK, col = idx % BK
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int idx = tid + r * 256;
            const int row = idx / BK, col = idx % BK;
            const int gm = m0 + row, gn = n0 + row, gk = k0 + col;
            As[col][row] = (gm < M && gk < K) ? A[(size_t)gm * lda + gk] : 0.f;
            Ws[col][row] = (gn < N && gk < K) ? W[(size_t)gn * K + gk] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = Ws[kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * TM + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx * TN + j;
            if (gn >= N) continue;
            float* c = C + (size_t)gm * ldc + gn;
            *c = accumulate ? (*c + acc[i][j]) : acc[i][j];
        }
    }
}


// ---- (1) ----------------------------------------------------------------------------------------------------------
namespace sp {

using namespace imparo::tc;

constexpr int TM = 128;                                       // rows of A per tile (tensor-memory lanes)
constexpr int WORKERS = 16;                                   // warps that cut operands and read accumulators out
// ... one that issues the MMAs and, where the operands are cut beforehand, one that loads them
template <bool CUT> constexpr int threads() { return 32 * (WORKERS + (CUT ? 2 : 1)); }
template <int TN, bool CUT> constexpr int stages() { return CUT && TN == 64 ? 3 : 2; }

constexpr uint32_t A_PLANE = TM * 128;
template <int TN> constexpr uint32_t b_plane() { return TN * 128; }
template <int TN> constexpr uint32_t stage_bytes() { return 3 * (A_PLANE + b_plane<TN>()); }
template <int TN, bool CUT> constexpr size_t smem_bytes() { return 1024 + (size_t)stages<TN, CUT>() * stage_bytes<TN>() + 256; }
// Accumulators, TN columns each: [large, even stretches | small x 2^8 | small x 2^16 | large, odd stretches]
template <int TN> constexpr uint32_t tmem_cols() { return 4 * TN; }

struct Params {
    const float* a; const float* w; float* c;
    int M, N, K, lda, ldc, accumulate, kblocks;
    int* status;
};

// two neighbours cut into three bfloat16 pieces each (h + m / 2^8 + l / 2^16 is the operand, exactly), packed in pairs
__device__ __forceinline__ void cut(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l) {
    auto pack = [](float u, float v) { __nv_bfloat162 t = __floats2bfloat162_rn(u, v); return *reinterpret_cast<uint32_t*>(&t); };
    auto rest = [](float2 v, uint32_t piece) {       // (both steps are exact: the subtraction, and times a power of two)
        v = __ffma2_rn(make_float2(__uint_as_float(piece << 16), __uint_as_float(piece & 0xffff0000u)), make_float2(-1.f, -1.f), v);
        return __fmul2_rn(v, make_float2(256.f, 256.f));
    };
    float2 v = make_float2(x, y);
    h = pack(v.x, v.y);
    v = rest(v, h);
    m = pack(v.x, v.y);
    v = rest(v, m);
    l = pack(v.x, v.y);
}

template <int COLS>
__device__ __forceinline__ void tmem_add(uint32_t taddr, float (&acc)[COLS]) {
    float v[COLS / 16][16];
    tmem_ld_chunks<COLS / 16>(taddr, v);
#pragma unroll
    for (int j = 0; j < COLS; ++j) acc[j] += v[j >> 4][j & 15];
}

// one element by the FFMA chain: what a result that is not finite is
__device__ __noinline__ float whole_sum(const float* x, const float* w, int K) {
    float t = 0.f;
    for (int k = 0; k < K; ++k) t = fmaf(x[k], w[k], t);
    return t;
}

__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr), "r"(0u) : "memory");
}

// One CTA per tile of TM x TN outputs.  A stretch of 64 k is 3 planes of A (16 KB each) and 3 of W in shared memory, in the
// swizzled layout of a bfloat16 K-major operand; sixteen warps read the 32-bit operands (one stretch ahead, in registers), cut
// them and store the planes, the seventeenth issues the MMAs; before a stage is filled again the sixteen read the large
// accumulator of the stretch that had it (two alternate) and clear it.
// The planes of W lie one after the other, so that one MMA takes two of them as its N operand where the two accumulators are
// neighbours: (h x m, h x l) and (m x h, m x m) are one MMA each per 16 k into the two small accumulators, 16 per stretch
// instead of 24, and A's planes are read for four instead of six.  The order of the sums is the same for both widths.
// What bounds it: the workers' share of a stretch (loads, cutting, stores, reading out, one after the other in a warp), 3,000
// cycles at TN = 128 and 2,250 at TN = 64, which is what the large product alone takes (3,100 and 2,000).  Sixteen workers and
// not eight: the loop's straight code is half as long per warp, and eight waited for instructions more than for anything else.
// At TN = 64 one MMA could take all three planes (12 per stretch, 93 -> 86 us at K 4,608); the sums would not be those of the
// wide tile.
// FFMA kernel -> 24 MMAs -> this (B200, us): 1,000 x 9,216 x 1,024: 837 -> 139 -> 132 (143 TFLOP/s); 1,000 x 1,024 x 4,608:
// 920 -> 112 -> 93; 60 x 3,072 x 1,024: 77 -> 27.6 -> 23.6; 2,048 x 1,024 x 8,192: 230 -> 215 (the last two).  Error against
// 64 bits: 5.7e-7 -> 1.05e-7 -> 1.04e-7 (K 1,024), 1.2e-6 -> 1.8e-7 -> 1.7e-7 (K 4,608).
//
// CUT: the operands have been cut beforehand (cut_planes_kernel): map_a and map_w are their planes, three times M and three times N
// rows one below the other, and a loading warp brings a stretch's six tiles by TMA; the workers only read the accumulators out.  In
// the kernel alone every tile of W is cut once per 128 rows of A and every tile of A once per 64 or 128 columns, which with some
// hundred rows or more is most of the workers' time.  The sums are the same, bit for bit.  What bounds it then: shared memory, 160 KB of
// operands read and 96 KB written per stretch of a wide tile.  1,000 x 9,216 x 1,024 (B200, with the cutting): 131 -> 116 us; 1,000 x
// 1,024 x 4,608: 94 -> 82; 2,048 x 16,384 x 2,048: 900 -> 747.  Where it pays: _cut_pays in kernels/ops.py.
template <int TN, bool CUT>
__global__ void __launch_bounds__(threads<CUT>(), 1)
sgemm_split_kernel(const Params p, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w) {
    constexpr uint32_t B_PLANE = b_plane<TN>(), STAGE = stage_bytes<TN>();
    constexpr int STAGES = stages<TN, CUT>();
    constexpr int ROUND = WORKERS * 4;                        // rows of a stretch per round of the workers
    constexpr int COLS = TN * 4 / WORKERS;                    // accumulator columns of a worker thread
    constexpr int A_IT = TM / ROUND, B_IT = TN / ROUND;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE);      // [STAGES] the stage's planes are stored
    uint64_t* empty = full + STAGES;                                          // [STAGES] ... and read by its MMAs
    uint64_t* acc_empty = empty + STAGES;                                     // [2] a stretch's large products are in the workers' registers
    uint64_t* done = acc_empty + 2;                                           // [1] every MMA is complete
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * TM, n0 = blockIdx.y * TN;
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], CUT ? 1 : WORKERS); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) mbar_init(&acc_empty[b], WORKERS);
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == WORKERS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols<TN>()) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    pdl_trigger();                                            // (after the allocation: a follower's cannot come before it)

    if (warp == WORKERS) {
        if (lane == 0) {
            const uint32_t one = instr_desc(TM, TN), two = instr_desc(TM, 2 * TN);
            for (int kb = 0; kb < p.kblocks; ++kb) {
                const int s = kb % STAGES, b = kb & 1;
                // CUT: the workers arrive once more, when they have cleared all accumulators
                if ((CUT || kb >= 2) && !mbar_wait(&acc_empty[b], ((kb >> 1) - (CUT ? 0 : 1)) & 1)) {
                    report(p.status, IMPARO_ST_WAIT_LIMIT, 90, blockIdx.x, kb);
                    break;
                }
                if (!mbar_wait(&full[s], (kb / STAGES) & 1)) { report(p.status, IMPARO_ST_WAIT_LIMIT, 91, blockIdx.x, kb); break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t a0 = smem_desc(smem_u32(smem) + s * STAGE), b0 = smem_desc(smem_u32(smem) + s * STAGE + 3 * A_PLANE);
                // (every accumulator is zero before it is first used: the workers clear them)
                auto mma = [&](uint32_t d, int pa, int pb, int k, uint32_t idesc) {
                    umma(tmem + d, a0 + (uint64_t)((pa * A_PLANE + k * UMMA_K * 2) >> 4), b0 + (uint64_t)((pb * B_PLANE + k * UMMA_K * 2) >> 4), idesc, 1u);
                };
#pragma unroll
                for (int k = 0; k < 4; ++k) mma(b ? 3 * TN : 0, 0, 0, k, one);         // h x h
#pragma unroll
                for (int k = 0; k < 4; ++k) mma(TN, 0, 1, k, two);                     // h x m, h x l
#pragma unroll
                for (int k = 0; k < 4; ++k) mma(TN, 1, 0, k, two);                     // m x h, m x m
#pragma unroll
                for (int k = 0; k < 4; ++k) mma(2 * TN, 2, 0, k, one);                 // l x h
                umma_commit(&empty[s]);
            }
            // what has been issued must be complete before the CTA gives its memory back, also after a wait that ran out
            umma_commit(done);
            mbar_wait(done, 0);
        }
    } else if (CUT && warp == WORKERS + 1) {
        if (lane == 0) {
            pdl_wait();                                       // the planes were written by the kernel before
            int kb = 0;
            // (the first stretch's MMAs also wait for the workers to have cleared the accumulators: acc_empty, below)
            for (; kb < p.kblocks; ++kb) {
                const int s = kb % STAGES;
                if (kb >= STAGES && !mbar_wait(&empty[s], ((kb / STAGES) - 1) & 1)) {
                    report(p.status, IMPARO_ST_WAIT_LIMIT, 93, blockIdx.x, kb);
                    break;
                }
                uint8_t* base = smem + s * STAGE;
                mbar_expect_tx(&full[s], STAGE);
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    tma_load_2d(base + u * A_PLANE, &map_a, &full[s], kb * 64, u * p.M + m0);
                    tma_load_2d(base + 3 * A_PLANE + u * B_PLANE, &map_w, &full[s], kb * 64, u * p.N + n0);
                }
            }
            // the last copies land before the warp leaves, also where the MMAs gave up on them
            for (int u = max(0, kb - STAGES); u < kb; ++u) mbar_wait(&full[u % STAGES], (u / STAGES) & 1);
        }
    } else {
        // a thread's piece of a stretch: 8 neighbours of k (chunk `c`) of the rows r0, r0 + ROUND, ...
        const int r0 = tid >> 3, c = tid & 7;
        float4 ra[A_IT][2], rb[B_IT][2];                       // the stretch to be cut next
        auto load = [&](const float* base, int ld, int row, int rows, int kb, float4 (&v)[2]) {
            const int k = kb * 64 + c * 8;
            const float* src = base + (size_t)row * ld + k;
            const bool in = row < rows;
            v[0] = (in && k < p.K) ? __ldg(reinterpret_cast<const float4*>(src)) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[1] = (in && k + 4 < p.K) ? __ldg(reinterpret_cast<const float4*>(src + 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        auto load_a = [&](int kb, int i) { load(p.a, p.lda, m0 + r0 + ROUND * i, p.M, kb, ra[i]); };
        auto load_b = [&](int kb, int i) { load(p.w, p.K, n0 + r0 + ROUND * i, p.N, kb, rb[i]); };
        auto store = [&](uint8_t* base, uint32_t plane, int row, const float4 (&v)[2]) {
            uint4 h, m, l;
            cut(v[0].x, v[0].y, h.x, m.x, l.x);
            cut(v[0].z, v[0].w, h.y, m.y, l.y);
            cut(v[1].x, v[1].y, h.z, m.z, l.z);
            cut(v[1].z, v[1].w, h.w, m.w, l.w);
            uint8_t* at = base + row * 128 + ((c ^ (row & 7)) << 4);
            *reinterpret_cast<uint4*>(at) = h;
            *reinterpret_cast<uint4*>(at + plane) = m;
            *reinterpret_cast<uint4*>(at + 2 * plane) = l;
        };
        const int quad = warp & 3, part = warp >> 2;
        const uint32_t lanes = (uint32_t)(quad * 32) << 16;
        float acc[COLS];
#pragma unroll
        for (int j = 0; j < COLS; ++j) acc[j] = 0.f;
        bool ok = true;
        // the large products of stretch kb, whose MMAs are complete (`empty` of its stage: what says so)
        auto drain = [&](int kb) {
            const int b = kb & 1;
            if (!mbar_wait(&empty[kb % STAGES], (kb / STAGES) & 1)) { if (lane == 0) report(p.status, IMPARO_ST_WAIT_LIMIT, 92, blockIdx.x, kb); ok = false; }
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) return;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t at = tmem + lanes + (uint32_t)((b ? 3 * TN : 0) + part * COLS);
            tmem_add<COLS>(at, acc);
#pragma unroll
            for (int j = 0; j < COLS; j += 16) tmem_zero16(at + j);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[b])) : "memory");
        };
        if constexpr (!CUT) {
#pragma unroll
            for (int i = 0; i < B_IT; ++i) load_b(0, i);       // W is written by no kernel
            pdl_wait();
#pragma unroll
            for (int i = 0; i < A_IT; ++i) load_a(0, i);
        }
#pragma unroll
        for (int j = 0; j < (int)tmem_cols<TN>() / 4; j += 16) tmem_zero16(tmem + lanes + (uint32_t)(part * (tmem_cols<TN>() / 4) + j));
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");       // (the first stretch's arrival tells the MMAs)
        if constexpr (CUT) {
            __syncwarp();
            if (lane < 2) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[lane])) : "memory");
            pdl_wait();                                       // before any result is written, or added to what the kernel before wrote
            for (int kb = 0; kb < p.kblocks && ok; ++kb) drain(kb);
        }
        for (int kb = 0; !CUT && kb < p.kblocks && ok; ++kb) {
            const int s = kb % STAGES;
            if (kb >= STAGES) {                                // the stage is free, and its stretch's accumulator can be read
                drain(kb - STAGES);
                if (!ok) break;
            }
            uint8_t* base = smem + s * STAGE;
            // a piece's registers are asked to be filled again as soon as they are stored (beyond the last stretch the
            // loads are masked off)
#pragma unroll
            for (int i = 0; i < A_IT; ++i) {
                store(base, A_PLANE, r0 + ROUND * i, ra[i]);
                load_a(kb + 1, i);
            }
#pragma unroll
            for (int i = 0; i < B_IT; ++i) {
                store(base + 3 * A_PLANE, B_PLANE, r0 + ROUND * i, rb[i]);
                load_b(kb + 1, i);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");       // the planes are read by the async proxy
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full[s])) : "memory");
        }
        for (int kb = max(0, p.kblocks - STAGES); !CUT && kb < p.kblocks && ok; ++kb) drain(kb);
        if (ok && !mbar_wait(done, 0)) { if (lane == 0) report(p.status, IMPARO_ST_WAIT_LIMIT, 94, blockIdx.x, p.kblocks); ok = false; }
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t at = tmem + lanes + (uint32_t)(part * COLS);
            float small[COLS];                                 // (m m + h l + l h) / 2^8 + h m + m h, then / 2^8
#pragma unroll
            for (int j = 0; j < COLS; ++j) small[j] = 0.f;
            tmem_add<COLS>(at + 2 * TN, small);
#pragma unroll
            for (int j = 0; j < COLS; ++j) small[j] *= 0.00390625f;
            tmem_add<COLS>(at + TN, small);
#pragma unroll
            for (int j = 0; j < COLS; ++j) acc[j] = fmaf(small[j], 0.00390625f, acc[j]);
            const int row = m0 + quad * 32 + lane;
            if (row < p.M) {
                const int col0 = n0 + part * COLS;
                float* out = p.c + (size_t)row * p.ldc + col0;
                const bool vec = (p.ldc & 3) == 0 && (((uintptr_t)p.c) & 15) == 0;
#pragma unroll
                for (int j = 0; j < COLS; j += 4) {
                    float v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        v[e] = acc[j + e];
                        if (col0 + j + e < p.N && !isfinite(v[e]))
                            v[e] = whole_sum(p.a + (size_t)row * p.lda, p.w + (size_t)(col0 + j + e) * p.K, p.K);
                    }
                    if (vec && col0 + j + 4 <= p.N) {
                        float4* dst = reinterpret_cast<float4*>(out + j);
                        if (p.accumulate) {
                            const float4 old = *dst;
                            v[0] = old.x + v[0]; v[1] = old.y + v[1]; v[2] = old.z + v[2]; v[3] = old.w + v[3];
                        }
                        *dst = make_float4(v[0], v[1], v[2], v[3]);
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (col0 + j + e < p.N) out[j + e] = p.accumulate ? out[j + e] + v[e] : v[e];
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == WORKERS) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols<TN>()) : "memory");
    }
}

// The planes of a matrix of `rows` rows of K (row stride ld): [3][rows][Kp] bfloat16, Kp = K rounded up to 8, zeros beyond K.  A thread
// cuts eight neighbours.  Bound by memory: 4 bytes in, 6 out.  Both operands in one launch: the first a_rows rows are A's.
__global__ void __launch_bounds__(256)
cut_planes_kernel(const float* __restrict__ a, int lda, int a_rows, const float* __restrict__ w, int w_rows, int K, uint4* __restrict__ pa,
                  uint4* __restrict__ pw) {
    pdl_trigger();
    const int per_row = (K + 7) / 8;
    const long long idx = (long long)blockIdx.x * 256 + threadIdx.x;
    const long long r = idx / per_row;
    const int c = (int)(idx - r * per_row);
    const bool mine = r < (long long)a_rows + w_rows, of_a = r < a_rows;
    const float* src = of_a ? a + (size_t)r * lda + c * 8 : w + (size_t)(r - a_rows) * K + c * 8;
    float4 v0 = make_float4(0.f, 0.f, 0.f, 0.f), v1 = v0;
    auto load = [&]() {
        v0 = __ldg(reinterpret_cast<const float4*>(src));
        if (c * 8 + 4 < K) v1 = __ldg(reinterpret_cast<const float4*>(src) + 1);
    };
    if (mine && !of_a) load();                                // W is written by no kernel
    pdl_wait();
    if (!mine) return;
    if (of_a) load();
    uint4 h, m, l;
    cut(v0.x, v0.y, h.x, m.x, l.x);
    cut(v0.z, v0.w, h.y, m.y, l.y);
    cut(v1.x, v1.y, h.z, m.z, l.z);
    cut(v1.z, v1.w, h.w, m.w, l.w);
    uint4* dst = of_a ? pa + (size_t)r * per_row + c : pw + (size_t)(r - a_rows) * per_row + c;
    const size_t plane = (size_t)(of_a ? a_rows : w_rows) * per_row;
    dst[0] = h;
    dst[plane] = m;
    dst[2 * plane] = l;
}

template <int TN, bool CUT>
static int launch_split(const Params& p, const CUtensorMap& ma, const CUtensorMap& mw, cudaStream_t stream) {
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(sgemm_split_kernel<TN, CUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<TN, CUT>());
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    launch(sgemm_split_kernel<TN, CUT>, dim3((p.M + TM - 1) / TM, (p.N + TN - 1) / TN), dim3(threads<CUT>()), smem_bytes<TN, CUT>(), stream, p, ma, mw);
    IMPARO_CHECK_LAUNCH();
    return 0;
}

// tiles of 128 x 64 where tiles of 128 x 128 would leave more than half of the 148 SMs without one (1,000 x 1,024 x
// 4,608: 93 against 121 us); above that the wide tile is the faster one (500 x 3,072 x 1,024, 96 wide tiles: 34 against
// 49 us; 1,000 x 9,216 x 1,024: 132 against 194).  The sums are the same either way.
static bool narrow(int M, int N) { return (long long)((M + 127) / 128) * ((N + 127) / 128) * 2 <= 148; }

}  // namespace sp

}  // namespace imparo

// status: where a wait that ran out is recorded.
extern "C" int imparo_sgemm_nt(const float* A, const float* W, float* C, int M, int N, int K,
                               int lda, int ldc, int accumulate, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return -1;
    // rows of whole 16-byte groups: the tensor cores
    if (K % 4 == 0 && lda % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0 && (N + 63) / 64 <= 65535) {
        imparo::sp::Params p{A, W, C, M, N, K, lda, ldc, accumulate, (K + 63) / 64, status};
        const CUtensorMap none = {};
        return imparo::sp::narrow(M, N) ? imparo::sp::launch_split<64, false>(p, none, none, stream)
                                        : imparo::sp::launch_split<128, false>(p, none, none, stream);
    }
    dim3 grid((N + imparo::BN - 1) / imparo::BN, (M + imparo::BM - 1) / imparo::BM);
    if (grid.y > 65535) return -2;
    launch(imparo::sgemm_nt_kernel, grid, dim3(256), 0, stream, A, W, C, M, N, K, lda, ldc, accumulate);
    IMPARO_CHECK_LAUNCH();
    return 0;
}

// Scratch that imparo_sgemm_cut needs, in bytes; 0 where it does not take the product (rows of no 16-byte groups).
extern "C" long long imparo_sgemm_cut_bytes(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0 || K % 4 != 0 || (N + 63) / 64 > 65535) return 0;
    return 6LL * ((K + 7) / 8 * 8) * ((long long)M + N);
}

// imparo_sgemm_nt with the operands cut into their planes first, by a launch of its own, into scratch (16-byte aligned,
// imparo_sgemm_cut_bytes).  -25: not taken, nothing launched.
extern "C" int imparo_sgemm_cut(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldc, int accumulate,
                                void* scratch, int* status, cudaStream_t stream) {
    using namespace imparo;
    if (imparo_sgemm_cut_bytes(M, N, K) == 0 || lda % 4 != 0 || (((uintptr_t)A | (uintptr_t)W | (uintptr_t)scratch) & 15)) return -25;
    const uint64_t Kp = (uint64_t)(K + 7) / 8 * 8;
    uint16_t* pa = reinterpret_cast<uint16_t*>(scratch);
    uint16_t* pw = pa + 3 * (size_t)M * Kp;
    const long long threads = ((long long)M + N) * (long long)(Kp / 8), blocks = (threads + 255) / 256;
    if (blocks > 0x7fffffffLL) return -25;
    CUtensorMap ma, mw;
    const bool thin = sp::narrow(M, N);
    int rc = tc::get_map(pa, 3 * (uint64_t)M, Kp, Kp, 128u, &ma);
    if (!rc) rc = tc::get_map(pw, 3 * (uint64_t)N, Kp, Kp, thin ? 64u : 128u, &mw);
    if (rc) return rc;
    launch(sp::cut_planes_kernel, dim3((unsigned)blocks), dim3(256), 0, stream, A, lda, M, W, N, K, reinterpret_cast<uint4*>(pa),
           reinterpret_cast<uint4*>(pw));
    IMPARO_CHECK_LAUNCH();
    const sp::Params p{A, W, C, M, N, K, lda, ldc, accumulate, (K + 63) / 64, status};
    return thin ? sp::launch_split<64, true>(p, ma, mw, stream) : sp::launch_split<128, true>(p, ma, mw, stream);
}
