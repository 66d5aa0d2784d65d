// The float32 product C[M,N] = A[M,K] * W[N,K]^T of large matrices on the fifth-generation tensor cores.
//
// A float32 is the sum of three bfloat16 (of 6, 8 and 8 bits of its mantissa and their signs; the splitting into bfloat16 is that of G. Henry,
// P. T. P. Tang and A. Heinecke, "Leveraging the bfloat16 artificial intelligence datatype for higher-precision computations", 2019), and a
// product of two bfloat16 is exact in float32. Eight of the nine products of parts are taken; third x third, 2^-30 of |a w|, is left out. The
// numbers are worked on times 2^40, so that the parts of small ones, subnormal ones too, are no subnormal bfloat16 (whose steps of 2^-133 would
// take their bits); numbers of 2^70 and sums of 2^48 and more become infinities on the way and are done again, see below.
//
// The tensor cores cut the terms of a sum off where they lie far below its largest, and every sum towards zero. So the products of first parts
// run from zero over 64 terms at a time, whose 12 bits then lose nothing unless they lie 2^6 and more apart (parts of 8 bits made sums of terms
// of one sign come out low, by 1.1e-7 to 1.5e-7), and those sums are added up in registers by rounded additions; the seven others, 2^-5 and
// less of the whole and, by the rounding of the parts, of either sign, stay in an accumulator of their own over a part of K. K is cut into up to
// eight parts, a CTA (or half a CTA's time) each, which meet in a cluster and are added up by twos and then in order. N and K alone decide all this, so a row's bits do not depend on
// M, nor on the row's place in the batch.
//
// D = W A^T: 128 rows of W are the M side, up to 160 rows of A (tokens) the N side, so that a few tokens cost few columns and a step's
// weights are read once. W's parts go to tensor memory and not back to shared memory, whose reads would bound the products.
//
//   W warps (8)      cut W up: from the TMA ring (float32) into tensor memory, a lane a row; and add the finished sums of 64 terms to their
//                    registers, each warpgroup half of the tokens. Up to 96 tokens the warpgroups take turns with W's blocks of 64 columns (a
//                    wait, a fence or an arrival costs a warp some 100 cycles, and so comes half as often), beyond both cut half of each
//   A warps (4 or 8) cut A up: from L2 through registers into swizzled shared memory; beyond 48 rows one warp brings the parts by TMA
//   one warp         TMA: 128 x 64 float32 of W a stage
//   one warp         tcgen05.mma, and the tensor memory
//
// What comes out as no finite number is computed again as the chains of gemm_f32.cu.
//
// us (gemm_f32.cu), one row: 5120 x 3072 15.0 (15.1), 3072 x 3072 11.0 (8.8), 16384 x 3072 35 (38), 3072 x 8192 24 (21), 128256 x 3072 249 (304); two rows
// 15.2 (17.1), 11.0 (9.8), 36 (42), 24 (24), 251 (296); 301 rows 76 (223), 60 (146), 190 (665), 129 (376). Bound by the waits, fences and arrivals between
// the warps where rows are few (some 0.75 us a block and CTA), by the products beyond (8 x 2 x 301 x 16384 x 3072 at 1.3 PFLOP/s). Six products of
// parts of 8 bits took 301 rows in 58, 55, 166 and 110 us, with the errors named above. Error against 64 bits of sum |a w|, K = 3072, rms: normal
// numbers 2.2e-9 (1.0e-8), of one sign 4.4e-8 (1.0e-7), one term 2.5e-8 (the same). One kind measured goes the other way: terms of one sign that lie very
// far apart (log-normal, sigma 3, in both operands) 2.8e-7 to 3.0e-7 whatever K (1.1e-7 at 512, 1.6e-7 at 1024, 4.1e-7 at 3072, 1.2e-6 at 8192).
//
// Every wait on an mbarrier is bounded by a clock; a wait that runs out sets *status and the CTA winds down.
#include "tcgen05.cuh"

namespace stride {
namespace f32tc {

using namespace tc;

constexpr int kRows = 128, kBlockK = 64, kWThreads = 256, kMaxParts = 8;
constexpr float kUp = 0x1p40f, kDown = 0x1p-80f;
constexpr int kBoxBytes = kRows * 128, kStageBytes = 2 * kBoxBytes;       // 32 float32 of 128 rows a box

// Parts of K, each with CTAs of its own: as many as make the shortest walk for up to 16 tokens, where two CTAs share an SM, some 256 run side by
// side (clusters do not fill a GPC to the last SM; of seven they fill it worst) and beginning and end cost a CTA about four blocks. N and K
// alone decide. One row, us, by parts: 3072 x 3072 1 38.9, 2 20.8, 4 12.6, 6 12.8, 8 11.0; 16384 x 3072 1 59, 2 35.4, 3 41.7, 8 46.6; 28672 x 4096 1 81, 2 90, 8
// 97. With many rows fewer parts would do (301 of 3072 x 3072 49 us in five, 60 in eight as four CTAs).
__host__ inline int parts_of(int N, int K) {
    const long long tiles = (N + kRows - 1) / kRows;
    const int blocks = (K + kBlockK - 1) / kBlockK;
    int best = 1;
    long long least = 0;
    for (int p = 1; p <= kMaxParts && p <= blocks; ++p) {
        const long long walk = (tiles * p + 255) / 256 * ((blocks + p - 1) / p + 4);
        if (p != 7 && (p == 1 || walk < least)) {
            best = p;
            least = walk;
        }
    }
    return best;
}

// Parts that a CTA of 48 and more tokens, one an SM, takes one after the other, 1 or 2: the shorter walk, where beginning, end and exchange cost a
// CTA about eight blocks and some 128 run side by side (148 in clusters of one or two). A row's bits are the same: two parts' sums are added up
// first either way. us (one part a CTA): 4096 x 4096 48 rows 24 (38), 301 76 (102); 3072 x 3072 19 (23), 60 (68); 5120 x 3072 24 (27), 75 (83); 4096 x 14336 67 (101),
// 231 (255). Of two parts in all 301 rows of 16384 x 3072 take 195 (188): left apart. 6144 x 4096, five parts, 48 rows: 65 in clusters of three, which do not
// all fit at once, 37 in five.
__host__ inline int parts_a_cta(int M, int N, int tokens, int parts, int blocks) {
    if (parts < 3) return 1;
    const long long tiles = static_cast<long long>((N + kRows - 1) / kRows) * ((M + tokens - 1) / tokens);
    auto walk = [&](int per) {
        const int ctas = (parts + per - 1) / per, room = ctas <= 2 ? 148 : 128;
        return (tiles * ctas + room - 1) / room * (per * blocks + 7 + per);
    };
    return walk(2) <= walk(1) ? 2 : 1;
}

// Eight columns of 32 lanes; tmem_ld_wait() before anybody uses them.
__device__ __forceinline__ void tmem_ld8_issue(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[8]) {      // (through r: nothing that uses it may come before)
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])
                 :
                 : "memory");
}
// Eight registers into eight columns; tmem_st_wait() before anybody reads them.
__device__ __forceinline__ void tmem_st8_issue(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Pairs of float32 in one instruction.
__device__ __forceinline__ uint64_t pair(float x, float y) { uint64_t p; asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(x), "f"(y)); return p; }
__device__ __forceinline__ void unpair(uint64_t p, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(p)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) { uint64_t d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(b), "l"(pair(-1.f, -1.f)), "l"(a));
    return d;
}

// Two float32, times kUp, as three pairs of bfloat16 (the first number in the low half): x = first + second + third. The first has 6 bits
// and is rounded (Veltkamp's splitting): a product of two firsts has 12, so 64 of them add up without a loss unless they lie far apart, and
// what the seven other products add up to has no sign of its own. The second is rounded to its 8 bits, the third is what is left (8 bits: 24 in all).
__device__ __forceinline__ void cut2(float x, float y, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    const uint64_t v = pair(x, y), all = mul2(v, pair(kUp, kUp)), far = mul2(v, pair(kUp * 262145.f, kUp * 262145.f));     // 2^18 + 1
    const uint64_t first = add2(far, sub2(all, far)), rest = sub2(all, first);
    unpair(first, x, y);
    p0 = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
    unpair(rest, x, y);
    const __nv_bfloat162 second = __floats2bfloat162_rn(x, y);
    p1 = *reinterpret_cast<const uint32_t*>(&second);
    unpair(sub2(rest, pair(__uint_as_float(p1 << 16), __uint_as_float(p1 & 0xFFFF0000u))), x, y);
    p2 = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
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
    static constexpr int MAINS = 3 * TOKENS + 192 <= 512 ? 2 : 1;                // accumulators of the first products
    static constexpr int COLS = (MAINS + 1) * TOKENS + 192 <= 256 ? 256 : 512;   // those, the others', two stages of W's parts
    static constexpr int CTAS = COLS == 256 ? 2 : 1;
    static constexpr bool TURNS = MAINS == 2;                     // the warpgroups take turns with W's blocks (else half of the columns each)
    static constexpr bool READY = HALF >= 48;                     // A comes cut up (cut_rows_kernel)
    static constexpr int A_THREADS = READY ? 32 : HALF == 8 ? 128 : 256;
    static constexpr int THREADS = kWThreads + A_THREADS + 64;
};

// PAIRS: a CTA has two parts of K, one after the other (see parts_a_cta). A kernel of its own: the first part's sums, kept meanwhile, cost the other 5 %.
template <int HALF, bool PAIRS>
__global__ void __launch_bounds__(Shape<HALF>::THREADS, Shape<HALF>::CTAS)
gemm_nt_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const float* __restrict__ A,
                      const float* __restrict__ W, float* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc, int blocks, int a_vec,
                      int* __restrict__ status) {
    using S = Shape<HALF>;
    constexpr int TOKENS = S::TOKENS, MAINS = S::MAINS, W_STAGES = S::W_STAGES, A_THREADS = S::A_THREADS, PIECES = S::READY ? 1 : TOKENS * 16 / A_THREADS;
    constexpr int W_WARPS = S::TURNS ? 4 : 8, STEP = S::TURNS ? 2 : 1;         // warps that cut a block up, blocks from one of theirs to the next
    constexpr int TMA_WARP = (kWThreads + A_THREADS) / 32, MMA_WARP = TMA_WARP + 1;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* const smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* const a_s = smem + W_STAGES * kStageBytes;
    __shared__ __align__(8) uint64_t w_full[W_STAGES], w_empty[W_STAGES];
    __shared__ __align__(8) uint64_t cut[2], used[2], a_full[2], main_done[S::MAINS], main_read[S::MAINS], all_done, cross_read;
    __shared__ uint32_t tmem_slot;

    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * TOKENS, n0 = blockIdx.y * kRows, part = blockIdx.z, parts = gridDim.z, span = PAIRS ? 2 * blocks : blocks;
    const int k_blocks = (K + kBlockK - 1) / kBlockK, first = part * span, count = min(span, k_blocks - first);     // 64 columns each, one at least
    const bool two = PAIRS && count > blocks;
    if (threadIdx.x == 0) {
        for (int s = 0; s < W_STAGES; ++s) {
            mbar_init(smem_u32(&w_full[s]), 1);
            mbar_init(smem_u32(&w_empty[s]), W_WARPS);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(smem_u32(&cut[s]), W_WARPS + (S::READY ? 0 : A_THREADS / 32));
            mbar_init(smem_u32(&used[s]), 1);
            mbar_init(smem_u32(&a_full[s]), 1);
        }
        for (int s = 0; s < MAINS; ++s) {
            mbar_init(smem_u32(&main_done[s]), 1);
            mbar_init(smem_u32(&main_read[s]), kWThreads / 32);
        }
        mbar_init(smem_u32(&all_done), 1);
        mbar_init(smem_u32(&cross_read), kWThreads / 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) tmem_alloc(smem_u32(&tmem_slot), S::COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot, t_main = tmem, t_cross = tmem + MAINS * TOKENS, t_w = t_cross + TOKENS;      // + 96 a stage, 32 a part

    bool ok = true;
    if (warp < kWThreads / 32) {
        const int quad = warp & 3, half = warp >> 2, row = quad * 32 + lane;
        const uint32_t lanes = static_cast<uint32_t>(quad * 32) << 16;
        float acc[HALF];
#pragma unroll
        for (int i = 0; i < HALF; ++i) acc[i] = 0.f;
        // sums of N accumulators, one after the other
        auto add = [&](auto... from) {
            constexpr int N = sizeof...(from);
            const uint32_t at[N] = {from...};
#pragma unroll
            for (int j = 0; j < HALF; j += 8) {
                uint32_t v[N][8];
#pragma unroll
                for (int n = 0; n < N; ++n) tmem_ld8_issue(at[n] + lanes + half * HALF + j, v[n]);
#pragma unroll
                for (int n = 0; n < N; ++n) tmem_ld_wait(v[n]);
#pragma unroll
                for (int n = 0; n < N; ++n)
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[j + e] += __uint_as_float(v[n][e]);
            }
        };
        auto wait_main = [&](int i) { return mbar_wait(smem_u32(&main_done[i % MAINS]), (i / MAINS) & 1, status, 63); };
        auto take = [&](int i) {            // the finished sums of block i
            if (!(ok = __all_sync(0xffffffffu, wait_main(i)))) return;
            tc_fence_after();
            add(t_main + i % MAINS * TOKENS);
            tc_fence_before();
            warp_arrive(smem_u32(&main_read[i % MAINS]));
        };
        [[maybe_unused]] auto take2 = [&](int i) {           // of two blocks at once
            if (!(ok = __all_sync(0xffffffffu, wait_main(i) && wait_main(i + 1)))) return;
            tc_fence_after();
            add(t_main + i % MAINS * TOKENS, t_main + (i + 1) % MAINS * TOKENS);
            tc_fence_before();
            __syncwarp();
            if (lane < 2) mbar_arrive(smem_u32(&main_read[lane]));
        };
        auto finish = [&](int phase) {      // a part's other products
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&all_done), phase, status, 63));
            if (!ok) return;
            tc_fence_after();
            add(t_cross);
            tc_fence_before();
        };
        float kept[PAIRS ? HALF : 1];    // the first part's sums
        int taken = 0;
        auto take_to = [&](int end) {
            if (S::TURNS && taken + 2 == end && !(two && (end == blocks || end == blocks + 1))) {
                take2(taken);
                taken = end;
            }
            for (; ok && taken < end; ++taken) {
                take(taken);
                if constexpr (PAIRS) {
                    if (!ok || !two || taken + 1 != blocks) continue;
                    finish(0);
                    warp_arrive(smem_u32(&cross_read));
#pragma unroll
                    for (int j = 0; j < HALF; ++j) {
                        kept[j] = acc[j];
                        acc[j] = 0.f;
                    }
                }
            }
        };
        for (int i = S::TURNS ? half : 0; i < count; i += STEP) {
            const int s = i & 1, ws = i % W_STAGES;
            // (in this order: a warpgroup that takes turns has not seen the phases of w_full that belong to the other's blocks, and a wait on a
            // phase passes while the one before it is not over; that block i - 2 has been used tells that all blocks up to it have come)
            ok = i < 2 || mbar_wait(smem_u32(&used[s]), ((i >> 1) & 1) ^ 1, status, 63);
            ok = ok && mbar_wait(smem_u32(&w_full[ws]), (i / W_STAGES) & 1, status, 63);
            if (!(ok = __all_sync(0xffffffffu, ok))) break;
            tc_fence_after();
            const unsigned char* const w_from = smem + ws * kStageBytes + row * 128;
            const uint32_t to = t_w + lanes + s * 96;
#pragma unroll 1
            for (int g = 0; g < 2 * STEP; ++g) {        // 16 columns
                const int h = S::TURNS ? g : 2 * half + g;
                uint32_t p0[8], p1[8], p2[8];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 x = *reinterpret_cast<const float4*>(w_from + (h >> 1) * kBoxBytes + (((4 * (h & 1) + q) ^ (row & 7)) * 16));
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
            take_to(i);
            if (!ok) break;
        }
        if (ok) take_to(count);
        if (ok) finish(two ? 1 : 0);
        if constexpr (PAIRS) {
            if (two) {
#pragma unroll
                for (int j = 0; j < HALF; ++j) acc[j] = kept[j] + acc[j];
            }
        }
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
                    if (m0 + r >= M && i >= 2) continue;        // both buffers hold zeros there
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
        int phase = 0;
        const uint32_t idesc = instr_desc_bf16(kRows, min(TOKENS, (M - m0 + 15) / 16 * 16), false);
        for (int i = 0; i < count; ++i) {
            const int s = i & 1;
            ok = mbar_wait(smem_u32(&cut[s]), (i >> 1) & 1, status, 62);
            if (S::READY) ok = ok && mbar_wait(smem_u32(&a_full[s]), (i >> 1) & 1, status, 62);
            ok = ok && (i < MAINS || mbar_wait(smem_u32(&main_read[i % MAINS]), (i / MAINS - 1) & 1, status, 62));
            if (two && i == blocks) ok = ok && mbar_wait(smem_u32(&cross_read), 0, status, 62);
            if (!(ok = __all_sync(0xffffffffu, ok))) break;
            tc_fence_after();
            const uint64_t a0 = smem_desc_sw128(smem_u32(a_s + s * S::A_BYTES));
            const uint64_t a1 = a0 + (S::A_PART >> 4), a2 = a0 + (2 * S::A_PART >> 4);
            const uint32_t w0 = t_w + s * 96, w1 = w0 + 32, w2 = w0 + 64;
            if (issuer) {
#pragma unroll
                for (int k = 0; k < 4; ++k) umma_bf16_tmem_a(t_main + i % MAINS * TOKENS, w0 + 8 * k, a0 + 2 * k, idesc, k > 0 ? 1u : 0u);
                umma_commit(smem_u32(&main_done[i % MAINS]));
#pragma unroll
                for (int k = 0; k < 4; ++k) {       // the smallest first
                    umma_bf16_tmem_a(t_cross, w2 + 8 * k, a1 + 2 * k, idesc, (i > 0 && !(two && i == blocks)) || k > 0 ? 1u : 0u);
                    umma_bf16_tmem_a(t_cross, w1 + 8 * k, a2 + 2 * k, idesc, 1u);
                    umma_bf16_tmem_a(t_cross, w2 + 8 * k, a0 + 2 * k, idesc, 1u);
                    umma_bf16_tmem_a(t_cross, w0 + 8 * k, a2 + 2 * k, idesc, 1u);
                    umma_bf16_tmem_a(t_cross, w1 + 8 * k, a1 + 2 * k, idesc, 1u);
                    umma_bf16_tmem_a(t_cross, w1 + 8 * k, a0 + 2 * k, idesc, 1u);
                    umma_bf16_tmem_a(t_cross, w0 + 8 * k, a1 + 2 * k, idesc, 1u);
                }
                umma_commit(smem_u32(&used[s]));
                if (two && i + 1 == blocks) umma_commit(smem_u32(&all_done));
            }
            __syncwarp();
            if (two && i + 1 == blocks) phase = 1;
        }
        if (issuer) umma_commit(smem_u32(&all_done));
        __syncwarp();
        mbar_wait(smem_u32(&all_done), phase, status, 62);
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
        float4 of[kMaxParts] = {};          // all on their way at once
#pragma unroll
        for (int p = 0; p < kMaxParts; ++p)
            if (p < parts) of[p] = load_cluster_f4(sums + t * kRows + col, p);
        // two parts' sums, and then those of the pairs in order
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int p = 0; p < kMaxParts; p += 2)
            if (p < parts) {
                const float4 a = of[p], b = of[p + 1];
                const bool with = p + 1 < parts;
                if (PAIRS) {                // of[p] is a pair's sum already
                    x.x += a.x; x.y += a.y; x.z += a.z; x.w += a.w;
                    if (with) { x.x += b.x; x.y += b.y; x.z += b.z; x.w += b.w; }
                } else if (with) {
                    x.x += a.x + b.x; x.y += a.y + b.y; x.z += a.z + b.z; x.w += a.w + b.w;
                } else {
                    x.x += a.x; x.y += a.y; x.z += a.z; x.w += a.w;
                }
            }
        float e[4] = {x.x * kDown, x.y * kDown, x.z * kDown, x.w * kDown};
        float* const out = C + static_cast<size_t>(m0 + t) * ldc + n;
        if (!(isfinite(x.x) && isfinite(x.y) && isfinite(x.z) && isfinite(x.w))) {
#pragma unroll 1
            for (int i = 0; i < 4; ++i) {
                float y = i == 0 ? x.x : i == 1 ? x.y : i == 2 ? x.z : x.w;
                if (isfinite(y) || n + i >= N) continue;
                y = element(A + static_cast<size_t>(m0 + t) * lda, W + static_cast<size_t>(n + i) * ldw, K);
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

template <int HALF, bool PAIRS>
cudaError_t launch_product(const Args& g, dim3 grid, const CUtensorMap& map, const CUtensorMap& map_a, int blocks, int a_vec, cudaStream_t stream) {
    using S = Shape<HALF>;
    const cudaError_t e = allow_shared<gemm_nt_f32_tc_kernel<HALF, PAIRS>>(S::SMEM);
    if (e != cudaSuccess) return e;
    return stride::launch_clusters(gemm_nt_f32_tc_kernel<HALF, PAIRS>, grid, dim3(S::THREADS), S::SMEM, stream, static_cast<int>(grid.z), map, map_a, g.A, g.W,
                                   g.C, g.M, g.N, g.K, g.lda, g.ldw, g.ldc, blocks, a_vec, g.status);
}

template <int HALF>
int run(const Args& g, cudaStream_t stream) {
    using S = Shape<HALF>;
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
    const int k_blocks = (g.K + kBlockK - 1) / kBlockK, wanted = parts_of(g.N, g.K), blocks = (k_blocks + wanted - 1) / wanted;
    const int parts = (k_blocks + blocks - 1) / blocks, per = S::CTAS == 1 ? parts_a_cta(g.M, g.N, S::TOKENS, parts, blocks) : 1;
    // neighbouring CTAs share a tile of W: the second one finds it in L2
    const dim3 grid((g.M + S::TOKENS - 1) / S::TOKENS, (g.N + kRows - 1) / kRows, (parts + per - 1) / per);
    cudaError_t launched;
    if constexpr (S::CTAS == 1)
        launched = per == 2 ? launch_product<HALF, true>(g, grid, map, map_a, blocks, a_vec, stream) : launch_product<HALF, false>(g, grid, map, map_a, blocks, a_vec, stream);
    else
        launched = launch_product<HALF, false>(g, grid, map, map_a, blocks, a_vec, stream);
    return launched != cudaSuccess ? static_cast<int>(launched) : STRIDE_LAUNCH_STATUS();
}

}  // namespace f32tc
}  // namespace stride

extern "C" {

// Scratch: 6 bytes a number of A beyond 48 rows, the parts of more rows than the product cuts up by itself. Returns -2 for what it does not take, which
// depends on the matrix W alone.
int stride_gemm_nt_f32_tc(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, void* scratch,
                          long long scratch_bytes, int* status, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || lda < K || ldw < K || ldc < N || status == nullptr) return STRIDE_BAD_ARGUMENT;
    if (N < 512 || K < 512 || K % 8 || ldw % 4 || reinterpret_cast<uintptr_t>(W) % 16 || N > 65535 * 128) return STRIDE_UNSUPPORTED;
    if (M == 0) return 0;
    if (scratch_bytes < (M > 48 ? 6LL * M * K : 0) || reinterpret_cast<uintptr_t>(scratch) % 16) return STRIDE_BAD_ARGUMENT;
    const stride::f32tc::Args g{A, W, C, M, N, K, lda, ldw, ldc, static_cast<__nv_bfloat16*>(scratch), status};
    if (M <= 16) return stride::f32tc::run<8>(g, stream);
    if (M <= 48) return stride::f32tc::run<24>(g, stream);
    if (M <= 96) return stride::f32tc::run<48>(g, stream);
    return stride::f32tc::run<80>(g, stream);
}

}  // extern "C"
