// The float32 product C[M,N] = A[M,K] * W[N,K]^T of large matrices on the fifth-generation tensor cores.
//
// Every float32 is the exact sum of three bfloat16 (8 bits of its mantissa each), and a product of two bfloat16 is exact in float32. Of
// the nine products of parts the six with a weight of 2^-16 and more are taken (the others are below 2^-22 of |a w|, of either sign).
// The tensor cores cut their sums off towards zero, so the products of the first parts run from zero over 64 terms at a time, and those
// sums are added up in registers by rounded additions; the five others, 2^-7 and less of the whole, stay in an accumulator of their
// own over a part of K. K is cut into parts of at most 1,024 terms (longer ones beyond 8), a CTA each, which meet in a cluster and are
// added up in order. K alone decides all this, so a row's bits do not depend on M, nor on the row's place in the batch.
//
// D = W A^T: 128 rows of W are the M side, up to 160 rows of A (tokens) the N side, so that a few tokens cost few columns and a step's
// weights are read once. W's parts go to tensor memory and not back to shared memory, whose reads would bound the products.
//
//   W warps (8)      cut W up: from the TMA ring (float32) into tensor memory, a lane a row, each warpgroup half of the 64 columns; and
//                    add the finished sums of 64 terms to their registers, each warpgroup half of the tokens
//   A warps (4 or 8) cut A up: from L2 through registers into swizzled shared memory; beyond 48 rows one warp brings the parts by TMA
//   one warp         TMA: 128 x 64 float32 of W a stage
//   one warp         tcgen05.mma, and the tensor memory
//
// An infinity and what is no number make a NaN here, also where the product itself has none: an element that comes out as NaN is
// computed again as the chains of gemm_f32.cu.
//
// 301 rows, us (gemm_f32.cu): 5120 x 3072 67 (227), 3072 x 3072 62 (143), 16384 x 3072 175 (668), 3072 x 8192 120 (363). Error against
// 64 bits 1.3e-7 of the result (3.6e-7; 5.8e-7 with K = 8192). Cutting A up in every CTA cost issue slots that the tensor cores waited
// for (81, 78, 217, 148 us), which is why more than 48 rows are cut once, by a kernel of its own. 2 rows: 25, 23, 63, 33 us
// (27, 19, 57, 37), 128256 x 3072 287 (320).
//
// Every wait on an mbarrier is bounded by a clock; a wait that runs out sets *status and the CTA winds down.
#include "tcgen05.cuh"

namespace stride {
namespace f32tc {

using namespace tc;

constexpr int kRows = 128, kBlockK = 64, kWThreads = 256, kPart = 1024;
constexpr int kBoxBytes = kRows * 128, kStageBytes = 2 * kBoxBytes;       // 32 float32 of 128 rows a box

__host__ __device__ __forceinline__ int parts_of(int K) {
    const int p = (K + kPart - 1) / kPart;
    return p > 8 ? 8 : p;
}

// Eight columns of 32 lanes.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
// Eight registers into eight columns; tmem_st_wait() before anybody reads them.
__device__ __forceinline__ void tmem_st8_issue(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Two float32 as three pairs of bfloat16 (the first number in the low half): x = first + second + third. The first is cut off (no
// conversion, and nothing finite becomes an infinity), the second rounded, which leaves a third of either sign: what the products that
// are left out add up to has no sign of its own.
__device__ __forceinline__ uint32_t high_halves(float lo, float hi) { return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632); }
__device__ __forceinline__ void cut2(float x, float y, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    p0 = high_halves(x, y);
    x -= __uint_as_float(__float_as_uint(x) & 0xFFFF0000u);
    y -= __uint_as_float(__float_as_uint(y) & 0xFFFF0000u);
    const __nv_bfloat162 second = __floats2bfloat162_rn(x, y);
    p1 = *reinterpret_cast<const uint32_t*>(&second);
    x -= __uint_as_float(p1 << 16);
    y -= __uint_as_float(p1 & 0xFFFF0000u);
    p2 = high_halves(x, y);
}

__device__ __forceinline__ float4 load_cluster_f4(const float* local, uint32_t rank) {
    uint32_t remote;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
    return v;
}

// One arrival for the whole warp.
__device__ __forceinline__ void warp_arrive(uint32_t bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}
__device__ __forceinline__ void named_barrier(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// One element as gemm_f32.cu has it: eight chains of fused multiply-adds, added up in order.
__device__ __forceinline__ float element(const float* __restrict__ a, const float* __restrict__ w, int K) {
    const int L = (K + 127) / 128 * 16;
    float total = 0.f;
    for (int p = 0; p < 8; ++p) {
        float chain = 0.f;
        for (int k = p * L; k < min(K, (p + 1) * L); ++k) chain = fmaf(__ldcg(a + k), w[k], chain);
        total = p ? total + chain : chain;
    }
    return total;
}

// A [M, K] into its three parts [3, M, K], four columns a thread.
__global__ void __launch_bounds__(256)
cut_rows_kernel(const float* __restrict__ A, int lda, int K, long long quads, size_t part, __nv_bfloat16* __restrict__ to, int a_vec) {
    pdl_trigger();
    pdl_wait();
    const int row_quads = K / 4;
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < quads; i += gridDim.x * 256LL) {
        const long long m = i / row_quads;
        const int k = static_cast<int>(i - m * row_quads) * 4;
        const float* const p = A + m * lda + k;
        const float4 x = a_vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
        uint2 x0, x1, x2;
        cut2(x.x, x.y, x0.x, x1.x, x2.x);
        cut2(x.z, x.w, x0.y, x1.y, x2.y);
        __nv_bfloat16* const o = to + m * K + k;
        *reinterpret_cast<uint2*>(o) = x0;
        *reinterpret_cast<uint2*>(o + part) = x1;
        *reinterpret_cast<uint2*>(o + 2 * part) = x2;
    }
}

template <int HALF>
struct Shape {
    static constexpr int TOKENS = 2 * HALF;                       // rows of A a CTA
    static constexpr int W_STAGES = 3;
    static constexpr int A_PART = TOKENS * 128, A_BYTES = 3 * A_PART;         // 64 bfloat16 a row; three parts
    static constexpr int RING = W_STAGES * kStageBytes + 2 * A_BYTES, OUT = TOKENS * kRows * 4;
    static constexpr int SMEM = (RING > OUT ? RING : OUT) + 1024;
    static constexpr int COLS = 2 * TOKENS + 192 <= 256 ? 256 : 512;            // two accumulators, two stages of W's parts
    static constexpr int CTAS = COLS == 256 ? 2 : 1;
    static constexpr bool READY = HALF >= 48;                     // A comes cut up (cut_rows_kernel)
    static constexpr int A_THREADS = READY ? 32 : HALF == 8 ? 128 : 256;
    static constexpr int THREADS = kWThreads + A_THREADS + 64;
};

template <int HALF>
__global__ void __launch_bounds__(Shape<HALF>::THREADS, Shape<HALF>::CTAS)
gemm_nt_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const float* __restrict__ A,
                      const float* __restrict__ W, float* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc, int blocks, int a_vec,
                      int* __restrict__ status) {
    using S = Shape<HALF>;
    constexpr int TOKENS = S::TOKENS, W_STAGES = S::W_STAGES, A_THREADS = S::A_THREADS, PIECES = S::READY ? 1 : TOKENS * 16 / A_THREADS;
    constexpr int CH = HALF % 16 == 0 ? 16 : 8;
    constexpr int TMA_WARP = (kWThreads + A_THREADS) / 32, MMA_WARP = TMA_WARP + 1;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* const smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* const a_s = smem + W_STAGES * kStageBytes;
    __shared__ __align__(8) uint64_t w_full[W_STAGES], w_empty[W_STAGES];
    __shared__ __align__(8) uint64_t cut[2], used[2], a_full[2], main_done, main_read, all_done;
    __shared__ uint32_t tmem_slot;

    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * TOKENS, n0 = blockIdx.y * kRows, part = blockIdx.z, parts = gridDim.z;
    const int k_blocks = (K + kBlockK - 1) / kBlockK, first = part * blocks, count = min(blocks, k_blocks - first);   // 64 columns each, one at least
    if (threadIdx.x == 0) {
        for (int s = 0; s < W_STAGES; ++s) {
            mbar_init(smem_u32(&w_full[s]), 1);
            mbar_init(smem_u32(&w_empty[s]), kWThreads / 32);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(smem_u32(&cut[s]), (kWThreads + (S::READY ? 0 : A_THREADS)) / 32);
            mbar_init(smem_u32(&used[s]), 1);
            mbar_init(smem_u32(&a_full[s]), 1);
        }
        mbar_init(smem_u32(&main_done), 1);
        mbar_init(smem_u32(&main_read), kWThreads / 32);
        mbar_init(smem_u32(&all_done), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) tmem_alloc(smem_u32(&tmem_slot), S::COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot, t_main = tmem, t_cross = tmem + TOKENS, t_w = tmem + 2 * TOKENS;      // + 96 a stage, 32 a part

    bool ok = true;
    if (warp < kWThreads / 32) {
        const int quad = warp & 3, half = warp >> 2, row = quad * 32 + lane;
        const uint32_t lanes = static_cast<uint32_t>(quad * 32) << 16;
        float acc[HALF];
#pragma unroll
        for (int i = 0; i < HALF; ++i) acc[i] = 0.f;
        auto add = [&](uint32_t from) {
#pragma unroll
            for (int j = 0; j < HALF; j += CH) {
                float v[CH];
                if constexpr (CH == 16) tmem_ld16(from + lanes + half * HALF + j, v);
                else tmem_ld8(from + lanes + half * HALF + j, v);
#pragma unroll
                for (int e = 0; e < CH; ++e) acc[j + e] += v[e];
            }
        };
        auto take = [&](int i) {            // the finished sums of block i
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&main_done), i & 1, status, 63));
            if (!ok) return;
            tc_fence_after();
            add(t_main);
            tc_fence_before();
            warp_arrive(smem_u32(&main_read));
        };
        for (int i = 0; i < count; ++i) {
            const int s = i & 1, ws = i % W_STAGES;
            ok = mbar_wait(smem_u32(&w_full[ws]), (i / W_STAGES) & 1, status, 63);
            ok = ok && (i < 2 || mbar_wait(smem_u32(&used[s]), ((i >> 1) & 1) ^ 1, status, 63));
            if (!(ok = __all_sync(0xffffffffu, ok))) break;
            tc_fence_after();
            const unsigned char* const w_from = smem + ws * kStageBytes + half * kBoxBytes + row * 128;
            const uint32_t to = t_w + lanes + s * 96 + half * 16;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t p0[8], p1[8], p2[8];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 x = *reinterpret_cast<const float4*>(w_from + (((4 * h + q) ^ (row & 7)) * 16));
                    cut2(x.x, x.y, p0[2 * q], p1[2 * q], p2[2 * q]);
                    cut2(x.z, x.w, p0[2 * q + 1], p1[2 * q + 1], p2[2 * q + 1]);
                }
                tmem_st8_issue(to + 8 * h, p0);
                tmem_st8_issue(to + 8 * h + 32, p1);
                tmem_st8_issue(to + 8 * h + 64, p2);
            }
            warp_arrive(smem_u32(&w_empty[ws]));
            tmem_st_wait();
            tc_fence_before();
            warp_arrive(smem_u32(&cut[s]));
            if (i > 0) take(i - 1);
            if (!ok) break;
        }
        if (ok) take(count - 1);
        if (ok) ok = mbar_wait(smem_u32(&all_done), 0, status, 63);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        if (ok) add(t_cross);
        tc_fence_before();
        float* const to = reinterpret_cast<float*>(smem) + half * HALF * kRows + row;
        named_barrier(1, kWThreads);        // the last tile of W has been read by all of these warps: the sums take the ring's place
#pragma unroll
        for (int j = 0; j < HALF; ++j) to[j * kRows] = acc[j];
    } else if (warp < TMA_WARP) {
        if constexpr (S::READY) {
            const bool issuer = elect_one();
            if (issuer) prefetch_map(&map_a);
            pdl_wait();
            int i = 0;
            for (; i < count; ++i) {
                const int s = i & 1;
                if (i >= 2) ok = mbar_wait(smem_u32(&used[s]), ((i >> 1) & 1) ^ 1, status, 61);
                if (!(ok = __all_sync(0xffffffffu, ok))) break;
                if (issuer) {
                    const uint32_t bar = smem_u32(&a_full[s]), to = smem_u32(a_s + s * S::A_BYTES);
                    mbar_expect_tx(bar, S::A_BYTES);
                    for (int p = 0; p < 3; ++p) tma_load_2d(to + p * S::A_PART, &map_a, bar, (first + i) * kBlockK, p * M + m0);
                }
                __syncwarp();
            }
            for (int j = i > 2 ? i - 2 : 0; j < i; ++j) mbar_wait(smem_u32(&a_full[j & 1]), (j >> 1) & 1, status, 61);
        } else {
            const int tid = threadIdx.x - kWThreads, c = (tid & 15) * 4;
            float4 next[PIECES];        // a piece: 4 columns of a token; 16 threads a row of 256 bytes
            auto ask = [&](int block) {
                const int k = (first + block) * kBlockK + c;
#pragma unroll
                for (int i = 0; i < PIECES; ++i) {
                    const int m = m0 + (tid >> 4) + i * (A_THREADS / 16);
                    next[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (m < M && k < K) {       // K is a multiple of 8: a piece lies inside or outside
                        const float* const p = A + static_cast<size_t>(m) * lda + k;
                        next[i] = a_vec ? __ldcg(reinterpret_cast<const float4*>(p)) : make_float4(__ldcg(p), __ldcg(p + 1), __ldcg(p + 2), __ldcg(p + 3));
                    }
                }
            };
            pdl_wait();
            ask(0);
            for (int i = 0; i < count; ++i) {
                const int s = i & 1;
                if (i >= 2) ok = mbar_wait(smem_u32(&used[s]), ((i >> 1) & 1) ^ 1, status, 63);
                if (!(ok = __all_sync(0xffffffffu, ok))) break;
                unsigned char* const a_to = a_s + s * S::A_BYTES;
#pragma unroll
                for (int p = 0; p < PIECES; ++p) {
                    const int r = (tid >> 4) + p * (A_THREADS / 16);
                    uint2 x0, x1, x2;
                    cut2(next[p].x, next[p].y, x0.x, x1.x, x2.x);
                    cut2(next[p].z, next[p].w, x0.y, x1.y, x2.y);
                    unsigned char* const to = a_to + r * 128 + (((tid & 15) >> 1) ^ (r & 7)) * 16 + (tid & 1) * 8;
                    *reinterpret_cast<uint2*>(to) = x0;
                    *reinterpret_cast<uint2*>(to + S::A_PART) = x1;
                    *reinterpret_cast<uint2*>(to + 2 * S::A_PART) = x2;
                }
                fence_proxy_async();
                warp_arrive(smem_u32(&cut[s]));
                if (i + 1 < count) ask(i + 1);
            }
        }
    } else if (warp == TMA_WARP) {
        // weights are written by no kernel: nothing here waits for the kernel before
        const bool issuer = elect_one();
        if (issuer) prefetch_map(&map_w);
        int i = 0;
        for (; i < count; ++i) {
            const int s = i % W_STAGES;
            if (i >= W_STAGES) ok = mbar_wait(smem_u32(&w_empty[s]), ((i / W_STAGES) & 1) ^ 1, status, 61);
            if (!(ok = __all_sync(0xffffffffu, ok))) break;
            if (issuer) {
                const uint32_t bar = smem_u32(&w_full[s]), to = smem_u32(smem + s * kStageBytes);
                mbar_expect_tx(bar, kStageBytes);
                tma_load_2d(to, &map_w, bar, (first + i) * kBlockK, n0);
                tma_load_2d(to + kBoxBytes, &map_w, bar, (first + i) * kBlockK + 32, n0);
            }
            __syncwarp();
        }
        // what is on its way lands before the CTA leaves, also when nobody reads it any more
        for (int j = i > W_STAGES ? i - W_STAGES : 0; j < i; ++j) mbar_wait(smem_u32(&w_full[j % W_STAGES]), (j / W_STAGES) & 1, status, 61);
    } else {
        const bool issuer = elect_one();
        const uint32_t idesc = instr_desc_bf16(kRows, min(TOKENS, (M - m0 + 15) / 16 * 16), false);
        for (int i = 0; i < count; ++i) {
            const int s = i & 1;
            ok = mbar_wait(smem_u32(&cut[s]), (i >> 1) & 1, status, 62);
            if (S::READY) ok = ok && mbar_wait(smem_u32(&a_full[s]), (i >> 1) & 1, status, 62);
            ok = ok && (i == 0 || mbar_wait(smem_u32(&main_read), (i - 1) & 1, status, 62));
            if (!(ok = __all_sync(0xffffffffu, ok))) break;
            tc_fence_after();
            const uint64_t a0 = smem_desc_sw128(smem_u32(a_s + s * S::A_BYTES));
            const uint64_t a1 = a0 + (S::A_PART >> 4), a2 = a0 + (2 * S::A_PART >> 4);
            const uint32_t w0 = t_w + s * 96, w1 = w0 + 32, w2 = w0 + 64;
            if (issuer) {
#pragma unroll
                for (int k = 0; k < 4; ++k) umma_bf16_tmem_a(t_main, w0 + 8 * k, a0 + 2 * k, idesc, k > 0 ? 1u : 0u);
                umma_commit(smem_u32(&main_done));
#pragma unroll
                for (int k = 0; k < 4; ++k) {       // the smallest first
                    umma_bf16_tmem_a(t_cross, w2 + 8 * k, a0 + 2 * k, idesc, i > 0 || k > 0 ? 1u : 0u);
                    umma_bf16_tmem_a(t_cross, w0 + 8 * k, a2 + 2 * k, idesc, 1u);
                    umma_bf16_tmem_a(t_cross, w1 + 8 * k, a1 + 2 * k, idesc, 1u);
                    umma_bf16_tmem_a(t_cross, w1 + 8 * k, a0 + 2 * k, idesc, 1u);
                    umma_bf16_tmem_a(t_cross, w0 + 8 * k, a1 + 2 * k, idesc, 1u);
                }
                umma_commit(smem_u32(&used[s]));
            }
            __syncwarp();
        }
        if (issuer) umma_commit(smem_u32(&all_done));
        __syncwarp();
        mbar_wait(smem_u32(&all_done), 0, status, 62);
    }
    float* const sums = reinterpret_cast<float*>(smem);     // [token][row of W]
    __syncthreads();
    if (warp == MMA_WARP) tmem_dealloc(tmem, S::COLS);
    cluster_arrive();
    cluster_wait();
    const int live = min(TOKENS, M - m0), share = (live + parts - 1) / parts;
    const bool wide = (ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
    for (int o = threadIdx.x; o < share * (kRows / 4); o += S::THREADS) {
        const int t = part * share + o / (kRows / 4), col = o % (kRows / 4) * 4, n = n0 + col;
        if (t >= live || n >= N) continue;
        float4 x = load_cluster_f4(sums + t * kRows + col, 0);
        for (int p = 1; p < parts; ++p) {
            const float4 y = load_cluster_f4(sums + t * kRows + col, p);
            x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
        }
        float e[4] = {x.x, x.y, x.z, x.w};
        float* const out = C + static_cast<size_t>(m0 + t) * ldc + n;
        if (isnan(x.x) || isnan(x.y) || isnan(x.z) || isnan(x.w)) {
#pragma unroll 1
            for (int i = 0; i < 4; ++i) {
                float y = i == 0 ? x.x : i == 1 ? x.y : i == 2 ? x.z : x.w;
                if (isnan(y) && n + i < N) y = element(A + static_cast<size_t>(m0 + t) * lda, W + static_cast<size_t>(n + i) * ldw, K);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (i == j) e[j] = y;
            }
        }
        if (wide && n + 3 < N) {
            *reinterpret_cast<float4*>(out) = make_float4(e[0], e[1], e[2], e[3]);
        } else {
            for (int i = 0; i < 4; ++i)
                if (n + i < N) out[i] = e[i];
        }
    }
    cluster_arrive();           // a CTA's shared memory stays until the others have read it
    cluster_wait();
}

// W [rows, cols] float32 in boxes of 128 rows x 32 columns, 128-byte swizzle; what lies outside reads as zero.
inline bool make_map_f32(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld) {
    EncodeFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 4};
    const cuuint32_t box[2] = {32, kRows}, elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct Args {
    const float *A, *W;
    float* C;
    int M, N, K, lda, ldw, ldc;
    __nv_bfloat16* parts;
    int* status;
};

template <int HALF>
int run(const Args& g, cudaStream_t stream) {
    using S = Shape<HALF>;
    const cudaError_t e = allow_shared<gemm_nt_f32_tc_kernel<HALF>>(S::SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    CUtensorMap map, map_a;
    if (!make_map_f32(&map, g.W, g.N, g.K, g.ldw)) return STRIDE_UNSUPPORTED;
    const int a_vec = (g.lda & 3) == 0 && (reinterpret_cast<uintptr_t>(g.A) & 15) == 0;
    if constexpr (S::READY) {
        // (a box that begins in one part's last rows ends in the next part's: columns of the product that nobody stores)
        if (!make_map(&map_a, g.parts, 3LL * g.M, g.K, g.K, S::TOKENS)) return STRIDE_UNSUPPORTED;
        const long long quads = static_cast<long long>(g.M) * (g.K / 4);
        const int grid = static_cast<int>(min((quads + 255) / 256, 148LL * 8));
        stride::launch(cut_rows_kernel, dim3(grid), dim3(256), 0, stream, g.A, g.lda, g.K, quads, static_cast<size_t>(g.M) * g.K, g.parts, a_vec);
    } else {
        map_a = map;
    }
    const int k_blocks = (g.K + kBlockK - 1) / kBlockK, blocks = (k_blocks + parts_of(g.K) - 1) / parts_of(g.K), parts = (k_blocks + blocks - 1) / blocks;
    // neighbouring CTAs share a tile of W: the second one finds it in L2
    const dim3 grid((g.M + S::TOKENS - 1) / S::TOKENS, (g.N + kRows - 1) / kRows, parts);
    const cudaError_t launched = stride::launch_clusters(gemm_nt_f32_tc_kernel<HALF>, grid, dim3(S::THREADS), S::SMEM, stream, parts, map, map_a, g.A,
                                                         g.W, g.C, g.M, g.N, g.K, g.lda, g.ldw, g.ldc, blocks, a_vec, g.status);
    return launched != cudaSuccess ? static_cast<int>(launched) : STRIDE_LAUNCH_STATUS();
}

}  // namespace f32tc
}  // namespace stride

extern "C" {

// Bytes of scratch for M rows of A: the parts of more rows than the product cuts up by itself.
long long stride_gemm_nt_f32_tc_scratch(int M, int K) { return M > 48 ? 6LL * M * K : 0; }

// Returns -2 for what it does not take, which depends on the matrix W alone.
int stride_gemm_nt_f32_tc(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, void* scratch,
                          long long scratch_bytes, int* status, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || lda < K || ldw < K || ldc < N || status == nullptr) return STRIDE_BAD_ARGUMENT;
    if (N < 512 || K < 512 || K % 8 || ldw % 4 || reinterpret_cast<uintptr_t>(W) % 16 || N > 65535 * 128) return STRIDE_UNSUPPORTED;
    if (M == 0) return 0;
    if (scratch_bytes < stride_gemm_nt_f32_tc_scratch(M, K) || reinterpret_cast<uintptr_t>(scratch) % 16) return STRIDE_BAD_ARGUMENT;
    const stride::f32tc::Args g{A, W, C, M, N, K, lda, ldw, ldc, static_cast<__nv_bfloat16*>(scratch), status};
    if (M <= 16) return stride::f32tc::run<8>(g, stream);
    if (M <= 48) return stride::f32tc::run<24>(g, stream);
    if (M <= 96) return stride::f32tc::run<48>(g, stream);
    return stride::f32tc::run<80>(g, stream);
}

}  // extern "C"
