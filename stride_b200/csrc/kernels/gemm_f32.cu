// True float32 matrix product for the 32-bit path: C[M,N] = A[M,K] * W[N,K]^T, for the matrices that gemm_f32_tc.cu leaves here.
//
// Plain FMA on the CUDA cores, no tensor-core mode of reduced precision. The terms of an output are cut into 8 parts of
// 16 * ceil(K / 128) consecutive ones; a part is one chain of fused multiply-adds in the order of k, and the parts are added
// up in order. (8 short chains: the error against 64 bits is smaller than that of one long chain, and there is work for 8 threads
// or CTAs in an output.) K alone decides this, so a row's result does not depend on M, on the row's place in the batch or on which
// of the kernels below ran it: the 32-bit path is bitwise the same however the tokens are cut. Weights are stored [out, in]
// row-major as in the checkpoint (python/stride_worker/model.py:258-260).
#include "common.cuh"

namespace stride {
namespace f32 {

constexpr int PARTS = 8;
__host__ __device__ __forceinline__ int part_length(int K) { return (K + 127) / 128 * 16; }

__device__ __forceinline__ void cp16(float* dst, const float* src) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ------------------------------------------------------------------------------------------------ few rows: stream the weights
// Up to 16 rows of A. What bounds it is the read of W: a CTA owns 16 rows of W at a time and all of K, a thread one row and one part
// of K for every row of A; 32 columns of each part are a tile, tiles come through a ring by cp.async, and the ring goes straight on
// into the CTA's next 16 rows, so that it never empties between them. The rows of A come along tile by tile (from L2).
// 2 rows, K = 3072: 3072 rows of W 12 us, 16384 44 us (4.6 TB/s), 128256 296 us (5.3 TB/s); the 64 x 64 tile of one chain that was
// here before took 272, 384 and 1727 us. 16 rows: 25, 91 and 614 us (the reads of shared memory).
template <int MT, int STAGES>
__global__ void __launch_bounds__(128) gemm_nt_f32_stream_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                                                                 int M, int N, int K, int lda, int ldw, int ldc) {
    constexpr int BN = 16, BK = 32, LD = PARTS * BK + 4, PIECES = PARTS * BK / 4;
    extern __shared__ float4 smem4[];
    float* const ws = reinterpret_cast<float*>(smem4);              // [STAGES][BN][LD]
    float* const as = ws + STAGES * BN * LD;                        // [STAGES][MT][LD]
    float* const sums = as + STAGES * MT * LD;                      // [PARTS][MT][BN]
    pdl_trigger();
    const int tid = threadIdx.x, tiles = (N + BN - 1) / BN, L = part_length(K), ktiles = (L + BK - 1) / BK;
    const int mine = (tiles - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
    const int steps = mine * ktiles;
    // a thread's 16-byte pieces all lie in one column of the tile: (part, column) are the same for every step's row
    const int part_of = (tid % PIECES) / (BK / 4), c_of = (tid % PIECES) % (BK / 4) * 4, r_of = tid / PIECES;
    auto load = [&](float* to, const float* __restrict__ from, int ld, int rows, int limit, int k) {
        // past the last row, the part's end or the last column: zeros on both sides, which leave a chain as it is
        const bool live = k < L && part_of * L + k < K;
#pragma unroll
        for (int r = r_of; r < rows; r += 128 / PIECES) {
            float* const d = to + r * LD + part_of * BK + c_of;
            if (live && r < limit) cp16(d, from + static_cast<size_t>(r) * ld + part_of * L + k);
            else *reinterpret_cast<float4*>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    int w_step = 0, w_tile = blockIdx.x, w_kt = 0, a_step = 0, a_kt = 0;       // the next tiles to ask for
    auto load_w = [&] {
        load(ws + (w_step % STAGES) * BN * LD, W + static_cast<size_t>(w_tile) * BN * ldw, ldw, BN, N - w_tile * BN, w_kt * BK + c_of);
        ++w_step;
        if (++w_kt == ktiles) { w_kt = 0; w_tile += gridDim.x; }
    };
    auto load_a = [&] {
        load(as + (a_step % STAGES) * MT * LD, A, lda, MT, M, a_kt * BK + c_of);
        ++a_step;
        if (++a_kt == ktiles) a_kt = 0;
    };
    for (int s = 0; s < STAGES - 1; ++s)
        if (s < steps) load_w();            // weights are written by no kernel: their first tiles are asked for ahead of the wait
    pdl_wait();
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) load_a();
        cp_commit();
    }
    const int n = tid % BN, part = tid / BN;
    float acc[MT] = {};
    int tile = blockIdx.x, kt = 0;
    for (int step = 0; step < steps; ++step) {
        cp_wait<STAGES - 2>();
        __syncthreads();
        if (step + STAGES - 1 < steps) { load_w(); load_a(); }
        cp_commit();
        const float* const w = ws + (step % STAGES) * BN * LD + n * LD + part * BK;
        const float* const a = as + (step % STAGES) * MT * LD + part * BK;
#pragma unroll
        for (int c = 0; c < BK; c += 4) {
            const float4 x = *reinterpret_cast<const float4*>(w + c);
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                const float4 y = *reinterpret_cast<const float4*>(a + i * LD + c);
                acc[i] = fmaf(y.x, x.x, acc[i]);
                acc[i] = fmaf(y.y, x.y, acc[i]);
                acc[i] = fmaf(y.z, x.z, acc[i]);
                acc[i] = fmaf(y.w, x.w, acc[i]);
            }
        }
        if (++kt < ktiles) continue;
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            sums[(part * MT + i) * BN + n] = acc[i];
            acc[i] = 0.f;
        }
        __syncthreads();
        for (int o = tid; o < MT * BN; o += 128) {
            const int i = o / BN, col = tile * BN + o % BN;
            float total = sums[o];
#pragma unroll
            for (int p = 1; p < PARTS; ++p) total += sums[p * MT * BN + o];
            if (i < M && col < N) C[static_cast<size_t>(i) * ldc + col] = total;
        }
        kt = 0;
        tile += gridDim.x;
    }
    cp_wait<0>();
}

// ------------------------------------------------------------------------------------------------ more rows: register tiles
// BM x BN outputs a cluster of 8 CTAs, a part of K each: even a matrix of 3072 rows then has work for every SM. What bounds it
// is the FMA rate, and beside it the reads of shared memory: 8 x TN outputs a thread, two columns at a time by the packed FMA
// (each half rounds as a single FMA does), which leaves issue slots for the reads. Tiles of 16 columns go through registers into
// shared memory, transposed (k-major), twice buffered; a block of 8 rows is exchanged with its neighbour by k, so that the four
// threads that store the pieces of one row meet no bank twice. In the end the CTAs lay their sums into their shared memory, and
// each adds up an eighth of the rows over the cluster in the order of the parts. 301 rows: 38 to 46 TFLOP/s (16384 x 3072 in
// 664 us, 3072 x 8192 in 381 us); tiles of 64 x 128 with 16 columns a thread spill and reach 36.
__device__ __forceinline__ uint64_t both(float x) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float4 load_cluster_f4(const float* local, uint32_t rank) {
    uint32_t remote;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(local))), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
    return v;
}

// ALONE: up to 128 columns a part is one tile of 16, and where the outputs alone fill the device a cluster's exchange is most of the time:
// one CTA then takes all parts and adds them up as they come. 1,024 rows of 2048 x 64 11 us, 32 in clusters; 301 rows of 1000 x 33 5.6 and
// 8.0; with fewer tiles than 64 both are level (100 rows 5.4 us) and from 65 columns on the clusters win by the parts side by side.
// One tile of K has no parts to spread.
__device__ __forceinline__ void add2(uint64_t& total, uint64_t part) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(total) : "l"(part)); }

template <int BM, int BN, int TN, bool VEC, bool ALONE>
__global__ void __launch_bounds__(BM / 8 * (BN / TN)) gemm_nt_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W,
                                                                              float* __restrict__ C, int M, int N, int K, int lda, int ldw,
                                                                              int ldc) {
    constexpr int BK = 16, THREADS = BM / 8 * (BN / TN), WN = TN * 8, WARPS_N = BN / WN;      // a warp: 32 rows x WN columns
    constexpr int PA = BM * BK / 4 / THREADS, PW = BN * BK / 4 / THREADS, LDS = BN + 4;
    static_assert(PA * THREADS * 4 == BM * BK && PW * THREADS * 4 == BN * BK, "whole pieces a thread");
    constexpr int TILES = 2 * BK * (BM + BN), OUT = BM * LDS;
    __shared__ __align__(16) float smem[TILES > OUT ? TILES : OUT];
    float (*const As)[BK][BM] = reinterpret_cast<float (*)[BK][BM]>(smem);
    float (*const Ws)[BK][BN] = reinterpret_cast<float (*)[BK][BN]>(smem + 2 * BK * BM);
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int row = (warp / WARPS_N) * 32 + (lane >> 3) * 4, col = (warp % WARPS_N) * WN + (lane & 7) * 4;
    const int L = part_length(K), part = blockIdx.z, k_first = ALONE ? 0 : part * L, k_end = ALONE ? K : min(K, k_first + L);

    auto fetch = [&](const float* __restrict__ from, int ld, int r, int limit, int k) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < limit) {
            const float* p = from + static_cast<size_t>(r) * ld + k;
            if (VEC) {
                if (k < k_end) v = *reinterpret_cast<const float4*>(p);
            } else {
                if (k < k_end) v.x = p[0];
                if (k + 1 < k_end) v.y = p[1];
                if (k + 2 < k_end) v.z = p[2];
                if (k + 3 < k_end) v.w = p[3];
            }
        }
        return v;
    };
    float4 ra[PA], rw[PW];
    auto fetch_w = [&](int k0) {
#pragma unroll
        for (int p = 0; p < PW; ++p) rw[p] = fetch(W, ldw, n0 + (tid + p * THREADS) / 4, N, k0 + (tid & 3) * 4);
    };
    auto fetch_a = [&](int k0) {
#pragma unroll
        for (int p = 0; p < PA; ++p) ra[p] = fetch(A, lda, m0 + (tid + p * THREADS) / 4, M, k0 + (tid & 3) * 4);
    };
    auto put = [&](int b) {
        const int q = tid & 3;
#pragma unroll
        for (int p = 0; p < PA; ++p) {
            const int r = ((tid + p * THREADS) / 4) ^ (q * 8);
            As[b][q * 4][r] = ra[p].x; As[b][q * 4 + 1][r] = ra[p].y; As[b][q * 4 + 2][r] = ra[p].z; As[b][q * 4 + 3][r] = ra[p].w;
        }
#pragma unroll
        for (int p = 0; p < PW; ++p) {
            const int r = ((tid + p * THREADS) / 4) ^ (q * 8);
            Ws[b][q * 4][r] = rw[p].x; Ws[b][q * 4 + 1][r] = rw[p].y; Ws[b][q * 4 + 2][r] = rw[p].z; Ws[b][q * 4 + 3][r] = rw[p].w;
        }
    };

    uint64_t acc[8][TN / 2];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0;
    uint64_t total[ALONE ? 8 : 1][ALONE ? TN / 2 : 1];
    fetch_w(k_first);
    pdl_wait();
    fetch_a(k_first);
    put(0);
    __syncthreads();
    int b = 0;
    for (int k0 = k_first; k0 < k_end; k0 += BK) {
        const bool more = k0 + BK < k_end;
        if (more) { fetch_w(k0 + BK); fetch_a(k0 + BK); }
        // past the part's end both tiles hold zeros, which leave an accumulator's value as it is
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            const int x = (k >> 2) * 8;
            const float4 a0 = *reinterpret_cast<const float4*>(&As[b][k][row ^ x]);
            const float4 a1 = *reinterpret_cast<const float4*>(&As[b][k][(row + 16) ^ x]);
            const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            uint64_t w[TN / 2];
#pragma unroll
            for (int j = 0; j < TN / 4; ++j) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&Ws[b][k][(col + 32 * j) ^ x]);
                w[2 * j] = v.x;
                w[2 * j + 1] = v.y;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint64_t aa = both(a[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], aa, w[j]);
            }
        }
        if constexpr (ALONE) {  // the end of a part (a part without columns adds zero, which only makes -0 a 0)
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) {
                    if (k0 == 0) total[i][j] = acc[i][j];
                    else add2(total[i][j], acc[i][j]);
                    acc[i][j] = 0;
                }
        }
        if (more) {
            put(b ^ 1);         // last read one step ago, ahead of the barrier that ended it
            __syncthreads();
            b ^= 1;
        }
    }
    __syncthreads();
    if constexpr (ALONE) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < TN / 2; ++j) {
                acc[i][j] = total[i][j];
                if (K <= (PARTS - 1) * BK) add2(acc[i][j], 0);
            }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN / 4; ++j)
            *reinterpret_cast<ulonglong2*>(smem + (row + (i & 3) + (i >> 2) * 16) * LDS + col + 32 * j) = make_ulonglong2(acc[i][2 * j], acc[i][2 * j + 1]);
    if constexpr (ALONE) {
        __syncthreads();
    } else {
        cluster_arrive();
        cluster_wait();
    }
    const bool wide = (ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
    constexpr int ROWS = ALONE ? BM : BM / PARTS;
    for (int o = tid; o < ROWS * (BN / 4); o += THREADS) {
        const int r = (ALONE ? 0 : part * ROWS) + o / (BN / 4), c = o % (BN / 4) * 4, m = m0 + r, n = n0 + c;
        if (m >= M || n >= N) continue;
        float4 t;
        if constexpr (ALONE) {
            t = *reinterpret_cast<const float4*>(smem + r * LDS + c);
        } else {
            float4 v[PARTS];
#pragma unroll
            for (int p = 0; p < PARTS; ++p) v[p] = load_cluster_f4(smem + r * LDS + c, p);
            t = v[0];
#pragma unroll
            for (int p = 1; p < PARTS; ++p) { t.x += v[p].x; t.y += v[p].y; t.z += v[p].z; t.w += v[p].w; }
        }
        float* const out = C + static_cast<size_t>(m) * ldc + n;
        if (wide && n + 3 < N) {
            *reinterpret_cast<float4*>(out) = t;
        } else {
            const float e[4] = {t.x, t.y, t.z, t.w};
            for (int i = 0; i < 4; ++i)
                if (n + i < N) out[i] = e[i];
        }
    }
    if constexpr (!ALONE) {
        cluster_arrive();       // a CTA's shared memory stays until the others have read it
        cluster_wait();
    }
}

struct Args {
    const float *A, *W;
    float* C;
    int M, N, K, lda, ldw, ldc;
};

template <int MT, int STAGES>
int run_stream(const Args& g, cudaStream_t stream) {
    constexpr int bytes = (STAGES * (16 + MT) * (PARTS * 32 + 4) + PARTS * MT * 16) * 4, fit = 220 * 1024 / (bytes + 1024);
    const cudaError_t e = allow_shared<gemm_nt_f32_stream_kernel<MT, STAGES>>(bytes);
    if (e != cudaSuccess) return static_cast<int>(e);
    const int grid = min((g.N + 15) / 16, 148 * fit);
    stride::launch(gemm_nt_f32_stream_kernel<MT, STAGES>, dim3(grid), dim3(128), bytes, stream, g.A, g.W, g.C, g.M, g.N, g.K, g.lda, g.ldw, g.ldc);
    return STRIDE_LAUNCH_STATUS();
}

template <int BM, int BN, int TN>
int run_tile(const Args& g, bool vec, cudaStream_t stream) {
    const dim3 grid((g.N + BN - 1) / BN, (g.M + BM - 1) / BM, PARTS), block(BM / 8 * (BN / TN));
    if (grid.y > 65535) return STRIDE_UNSUPPORTED;
    if (g.K <= 16 || (g.K <= PARTS * 16 && static_cast<long long>(grid.x) * grid.y >= 64)) {
        const dim3 one(grid.x, grid.y);
        if (vec) stride::launch(gemm_nt_f32_tile_kernel<BM, BN, TN, true, true>, dim3(one), dim3(block), 0, stream, g.A, g.W, g.C, g.M, g.N, g.K, g.lda, g.ldw, g.ldc);
        else stride::launch(gemm_nt_f32_tile_kernel<BM, BN, TN, false, true>, dim3(one), dim3(block), 0, stream, g.A, g.W, g.C, g.M, g.N, g.K, g.lda, g.ldw, g.ldc);
        return STRIDE_LAUNCH_STATUS();
    }
    if (vec) stride::launch_clusters(gemm_nt_f32_tile_kernel<BM, BN, TN, true, false>, grid, block, 0, stream, PARTS, g.A, g.W, g.C, g.M, g.N, g.K, g.lda, g.ldw, g.ldc);
    else stride::launch_clusters(gemm_nt_f32_tile_kernel<BM, BN, TN, false, false>, grid, block, 0, stream, PARTS, g.A, g.W, g.C, g.M, g.N, g.K, g.lda, g.ldw, g.ldc);
    return STRIDE_LAUNCH_STATUS();
}

}  // namespace f32
}  // namespace stride

extern "C" int stride_gemm_nt_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                                  cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0 || lda < K || ldw < K || ldc < N) return STRIDE_BAD_ARGUMENT;
    if (M == 0) return 0;
    const stride::f32::Args g{A, W, C, M, N, K, lda, ldw, ldc};
    const bool vec = (K & 3) == 0 && (lda & 3) == 0 && (ldw & 3) == 0 && ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0;
    if (vec && (M <= 4 || (M <= 16 && K > 16))) {
        if (M == 1) return stride::f32::run_stream<1, 6>(g, stream);
        if (M == 2) return stride::f32::run_stream<2, 5>(g, stream);
        if (M <= 4) return stride::f32::run_stream<4, 5>(g, stream);
        if (M <= 8) return stride::f32::run_stream<8, 4>(g, stream);
        return stride::f32::run_stream<16, 3>(g, stream);
    }
    // (a row of W of one tile of K and 5 to 16 rows of A: tiles, 2.5 us for 16 rows of 2048 x 16, 3.5 streamed)
    // 3072 x 3072 in us, 32 x 64 (4 columns a thread) / 64 x 64 (4) / 64 x 64 (8): 20 rows 41 / 45 / 55, 48 rows 53 / 47 / 55,
    // 100 rows 79 / 68 / 62, 301 rows 172 / 146 / 148; 16384 x 3072: 102 / 148 / 148, 180 / 154 / 150, 348 / 296 / 277, 849 / 721 / 664
    if (M <= 32) return stride::f32::run_tile<32, 64, 4>(g, vec, stream);
    if (M <= 64) return stride::f32::run_tile<64, 64, 4>(g, vec, stream);
    return stride::f32::run_tile<64, 64, 8>(g, vec, stream);
}
