// Attention over a compressed cache: per token one latent vector c [rank] (RMS-normed) and one rotated key part
// k_r [rot] shared by all heads. Per head a the key is [W_uk_a c | k_r] and the value W_uv_a c, so with the query's
// plain part folded through W_uk (q~_a = W_uk_a^T q_a [rank]) the score of a key is
//   s = (q~_a . c + q_rot_a . k_r) * scale
// and the head's output W_uv_a (sum_j p_j c_j): every head reads the same [rank + rot] numbers per key and nothing
// but c and k_r is kept. (Portions of prompts may expand keys and values for the length of a pass instead:
// latent_gather here, attention_prefill_tc.cu.) Kernels:
//
//   latent_prepare    norms the latent (float32 statistics, plain weight), rotates the shared key part and the
//                     rotated part of every query head (pairs (2i, 2i+1), angle from a float32 table), writes the
//                     latent and the key part into their pages and the rotated queries beside the folded ones;
//   head_gemm         the per-head products with W_uk (folding) and W_uv (unfolding, with an optional sigmoid gate
//                     per (token, head) in its epilogue): float32 FMA with a fixed k order for float32 operands,
//                     tensor-core tiles (mma_tile.cuh) for bfloat16;
//   latent_attention  the exact kernel: one warp per (token, head), keys walked in groups of 32 aligned to
//                     position 0 with an online softmax, so a token's result does not depend on how the step was
//                     cut; float32 arithmetic in both storage types. (The bfloat16 kernel on the tensor cores is
//                     latent_attention_tc.cu.)
#include "common.cuh"
#include "mma_tile.cuh"

namespace stride {

// ------------------------------------------------------------------------------------------------ prepare
// q: [tokens, ldq], head a at column a * (dim + rot), plain part first (a column block of proj, or a buffer of its own
// when the queries come through a latent); proj: [tokens, ld] with the latent projection (rank + rot columns) at
// kv_off, or kv_off < 0 for a layer that reads another layer's cache.
// qa: [tokens, heads, rank + rot]; this kernel fills the last rot columns of every head.
template <typename T>
__global__ void __launch_bounds__(128)
latent_prepare_kernel(const T* __restrict__ q, int ldq, const T* __restrict__ proj, int ld, int kv_off, T* __restrict__ qa,
                      const int32_t* __restrict__ positions, const int32_t* __restrict__ seq_of_token,
                      const int32_t* __restrict__ slot_mapping, const float* __restrict__ cos_table,
                      const float* __restrict__ sin_table, const float* __restrict__ latent_w, float eps,
                      T* __restrict__ latent_pages, T* __restrict__ krot_pages, int heads, int dim, int rot, int rot_dims, int rank) {
    pdl_trigger();
    pdl_wait();
    __shared__ float scratch[32];
    const int t = blockIdx.x;
    if (seq_of_token[t] < 0) return;
    const T* row = proj + static_cast<size_t>(t) * ld;
    const int half = rot_dims / 2;
    const float* cs = cos_table + static_cast<size_t>(positions[t]) * half;
    const float* sn = sin_table + static_cast<size_t>(positions[t]) * half;
    // rotated part of the queries
    T* qrow = qa + static_cast<size_t>(t) * heads * (rank + rot);
    for (int i = threadIdx.x; i < heads * rot; i += blockDim.x) {
        const int a = i / rot, j = i % rot;
        const T* src = q + static_cast<size_t>(t) * ldq + a * (dim + rot) + dim;
        float v = to_f32(src[j]);
        if (j < rot_dims) {
            const int pair = j >> 1;
            const float other = to_f32(src[j ^ 1]);
            v = (j & 1) ? fmaf(v, cs[pair], other * sn[pair]) : fmaf(v, cs[pair], -other * sn[pair]);
        }
        qrow[a * (rank + rot) + rank + j] = from_f32<T>(v);
    }
    if (kv_off < 0) return;
    const int slot = slot_mapping ? slot_mapping[t] : -1;
    const T* kv = row + kv_off;
    float sq = 0.f;
    for (int i = threadIdx.x; i < rank; i += blockDim.x) {
        const float x = to_f32(kv[i]);
        sq = fmaf(x, x, sq);
    }
    const float total = block_sum(sq, scratch);
    if (slot < 0) return;
    const float inv = rsqrtf(total / static_cast<float>(rank) + eps);
    T* lat = latent_pages + static_cast<size_t>(slot) * rank;
    for (int i = threadIdx.x; i < rank; i += blockDim.x) lat[i] = from_f32<T>(to_f32(kv[i]) * inv * latent_w[i]);
    T* kr = krot_pages + static_cast<size_t>(slot) * rot;
    for (int j = threadIdx.x; j < rot; j += blockDim.x) {
        float v = to_f32(kv[rank + j]);
        if (j < rot_dims) {
            const int pair = j >> 1;
            const float other = to_f32(kv[rank + (j ^ 1)]);
            v = (j & 1) ? fmaf(v, cs[pair], other * sn[pair]) : fmaf(v, cs[pair], -other * sn[pair]);
        }
        kr[j] = from_f32<T>(v);
    }
}

// ------------------------------------------------------------------------------------------------- gather
// The latents and rotated key parts of the first `num_seqs` requests, position 0 on, request after request, out of their pages into
// dense rows: what the product that expands keys and values reads. A warp a row, 16 bytes a lane. range (or null): 0 and the number of rows
// filled, which bound that product's work (a captured portion's `rows` are for the longest context that it may be replayed at).
__global__ void __launch_bounds__(256)
latent_gather_kernel(const uint4* __restrict__ latent_pages, const uint4* __restrict__ krot_pages, const int32_t* __restrict__ block_table,
                     int table_width, const int32_t* __restrict__ ctx_len, int num_seqs, int page_size, int rank16, int rot16, int rows,
                     uint4* __restrict__ latent, uint4* __restrict__ krot, int32_t* __restrict__ range) {
    pdl_trigger();
    pdl_wait();
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (range && blockIdx.x == 0 && threadIdx.x == 0) {
        int total = 0;
        for (int s = 0; s < num_seqs && total < rows; ++s) total += ctx_len[s];
        range[0] = 0;
        range[1] = min(total, rows);
    }
    if (row >= rows) return;
    int key = row, seq = 0;
    while (seq < num_seqs && key >= ctx_len[seq]) key -= ctx_len[seq++];
    if (seq == num_seqs || key / page_size >= table_width) return;      // past the last request's keys: nothing is read from there
    const int page = block_table[static_cast<size_t>(seq) * table_width + key / page_size];
    if (page < 0) return;
    const size_t slot = static_cast<size_t>(page) * page_size + key % page_size;
    for (int i = lane; i < rank16; i += 32) latent[static_cast<size_t>(row) * rank16 + i] = latent_pages[slot * rank16 + i];
    for (int i = lane; i < rot16; i += 32) krot[static_cast<size_t>(row) * rot16 + i] = krot_pages[slot * rot16 + i];
}

// ---------------------------------------------------------------------------------------------- head_gemm
// C[t, a, n] = (sum_k A[t * lda + a * a_hs + k] * B[a * b_hs + k * b_ks + n * b_ns]) * (gate ? sigmoid(gate[t * ldg + a * g_hs + n * g_ns]) : 1)
// (g_hs 1 and g_ns 0: one gate a head; g_hs N and g_ns 1: one gate an output)
constexpr int HM = 32, HN = 64, HK = 16;

template <typename T>
__global__ void __launch_bounds__(256)
head_gemm_kernel(const T* __restrict__ A, int lda, int a_hs, const T* __restrict__ B, long long b_hs, int b_ks, int b_ns,
                 T* __restrict__ C, int ldc, int c_hs, const T* __restrict__ gate, int ldg, int g_hs, int g_ns, int M, int N, int K) {
    pdl_trigger();
    pdl_wait();
    __shared__ float As[HK][HM + 1];
    __shared__ float Bs[HK][HN + 4];
    const int a = blockIdx.y;
    const int m0 = blockIdx.z * HM, n0 = blockIdx.x * HN;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;      // thread: rows ty*2..+1, columns tx*4..+3
    const T* Ah = A + static_cast<size_t>(a) * a_hs;
    const T* Bh = B + static_cast<size_t>(a) * b_hs;
    float acc[2][4] = {};
    for (int k0 = 0; k0 < K; k0 += HK) {
        for (int i = threadIdx.x; i < HM * HK; i += 256) {
            const int m = i / HK, k = i % HK;
            As[k][m] = (m0 + m < M && k0 + k < K) ? to_f32(Ah[static_cast<size_t>(m0 + m) * lda + k0 + k]) : 0.f;
        }
        for (int i = threadIdx.x; i < HN * HK; i += 256) {
            int n, k;
            if (b_ns == 1) { k = i / HN; n = i % HN; } else { n = i / HK; k = i % HK; }
            Bs[k][n] = (n0 + n < N && k0 + k < K)
                           ? to_f32(Bh[static_cast<size_t>(k0 + k) * b_ks + static_cast<size_t>(n0 + n) * b_ns]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < HK; ++k) {
            const float a0 = As[k][ty * 2], a1 = As[k][ty * 2 + 1];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float b = Bs[k][tx * 4 + j];
                acc[0][j] = fmaf(a0, b, acc[0][j]);
                acc[1][j] = fmaf(a1, b, acc[1][j]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int m = m0 + ty * 2 + i;
        if (m >= M) continue;
        float g = 1.f;
        if (gate && !g_ns) g = 1.f / (1.f + expf(-to_f32(gate[static_cast<size_t>(m) * ldg + static_cast<size_t>(a) * g_hs])));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            if (gate && g_ns) g = 1.f / (1.f + expf(-to_f32(gate[static_cast<size_t>(m) * ldg + static_cast<size_t>(a) * g_hs + static_cast<size_t>(n) * g_ns])));
            C[static_cast<size_t>(m) * ldc + static_cast<size_t>(a) * c_hs + n] = from_f32<T>(acc[i][j] * g);
        }
    }
}

// The same on the tensor cores for bfloat16 (mma_tile.cuh): 64 tokens x 64 columns of one head a CTA.
__global__ void __launch_bounds__(128)
head_gemm_tc_kernel(const __nv_bfloat16* __restrict__ A, int lda, int a_hs, const __nv_bfloat16* __restrict__ B, long long b_hs, int b_ks,
                    int b_ns, __nv_bfloat16* __restrict__ C, int ldc, int c_hs, const __nv_bfloat16* __restrict__ gate, int ldg, int g_hs,
                    int g_ns, int M, int N, int K) {
    pdl_trigger();
    if (blockIdx.z == 0) {      // the CTA's part of the weights, a row of 64 or of K numbers a thread
        const __nv_bfloat16* b = B + static_cast<size_t>(blockIdx.y) * b_hs + static_cast<size_t>(blockIdx.x) * TN * b_ns;
        const int cols = min(TN, N - static_cast<int>(blockIdx.x) * TN);
        if (b_ns == 1)
            for (int k = threadIdx.x; k < K; k += 128) prefetch_l2(b + static_cast<size_t>(k) * b_ks, cols * 2, 0, 1);
        else if (b_ks == 1)
            for (int n = threadIdx.x; n < cols; n += 128) prefetch_l2(b + static_cast<size_t>(n) * b_ns, static_cast<size_t>(K) * 2, 0, 1);
    }
    pdl_wait();
    __shared__ TileSmem sm;
    const int a = blockIdx.y;
    const int m0 = blockIdx.z * TM, n0 = blockIdx.x * TN;
    for (int r = threadIdx.x; r < TM; r += 128)
        sm.a_rows[r] = m0 + r < M ? A + static_cast<size_t>(m0 + r) * lda + static_cast<size_t>(a) * a_hs : nullptr;
    __syncthreads();
    float acc[2][4][4];
    mma_tile_64x64(sm, B + static_cast<size_t>(a) * b_hs, b_ns, b_ks, n0, N, K, acc);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int x = 0; x < 4; x += 2) {
            const int m = m0 + tile_row(i, x);
            if (m >= M) continue;
            float g = 1.f;
            if (gate && !g_ns) g = 1.f / (1.f + expf(-to_f32(gate[static_cast<size_t>(m) * ldg + static_cast<size_t>(a) * g_hs])));
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    const int n = n0 + tile_col(j, x + y);
                    if (n >= N) continue;
                    if (gate && g_ns) g = 1.f / (1.f + expf(-to_f32(gate[static_cast<size_t>(m) * ldg + static_cast<size_t>(a) * g_hs + static_cast<size_t>(n) * g_ns])));
                    C[static_cast<size_t>(m) * ldc + static_cast<size_t>(a) * c_hs + n] = __float2bfloat16_rn(acc[i][j][x + y] * g);
                }
        }
}

// The same for portions: 128 tokens x 128 columns a CTA, eight warps of 64 x 32, 64 columns of K at a time by cp.async, twice buffered;
// weights whose output index is the contiguous one stay as they lie and are read with transposing fragment loads (the kernel above takes them
// number by number). The terms come in the same order, so the bits are the same. 2,048 tokens of 16 heads, back to back: to 512
// columns from 128 24 us, 108 in tiles of 64 x 64; to 128 from 512 19 us and 48.
constexpr int WM = 128, WN = 128, WLD = TK + 8, WLDT = WN + 8;
constexpr int kWideStage = WM * WLD + (WN * WLD > TK * WLDT ? WN * WLD : TK * WLDT);       // elements
template <bool N_CONTIGUOUS>
__global__ void __launch_bounds__(256, 2)
head_gemm_wide_kernel(const __nv_bfloat16* __restrict__ A, int lda, int a_hs, const __nv_bfloat16* __restrict__ B, long long b_hs, int b_ld,
                      __nv_bfloat16* __restrict__ C, int ldc, int c_hs, const __nv_bfloat16* __restrict__ gate, int ldg, int g_hs, int g_ns, int M,
                      int N, int K) {
    extern __shared__ __align__(16) unsigned char wide_smem[];
    __nv_bfloat16* const sm = reinterpret_cast<__nv_bfloat16*>(wide_smem);
    pdl_trigger();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int a = blockIdx.y, m0 = blockIdx.z * WM, n0 = blockIdx.x * WN, wm = (warp >> 2) * 64, wn = (warp & 3) * 32;
    const __nv_bfloat16* const Ah = A + static_cast<size_t>(a) * a_hs;
    const __nv_bfloat16* const Bh = B + static_cast<size_t>(a) * b_hs;
    auto copy = [&](__nv_bfloat16* dst, const __nv_bfloat16* src, bool live) {      // 16 bytes, zeros past the end
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src), "r"(live ? 16 : 0)
                     : "memory");
    };
    auto load = [&](int k0, int buf) {
        __nv_bfloat16* const as = sm + buf * kWideStage;
        __nv_bfloat16* const bs = as + WM * WLD;
        for (int i = tid; i < WM * TCH; i += 256) {
            const int r = i / TCH, k = (i % TCH) * 8;
            const bool live = m0 + r < M && k0 + k < K;
            copy(as + r * WLD + k, live ? Ah + static_cast<size_t>(m0 + r) * lda + k0 + k : A, live);
        }
        if (N_CONTIGUOUS) {
            for (int i = tid; i < TK * (WN / 8); i += 256) {
                const int k = i / (WN / 8), n = (i % (WN / 8)) * 8;
                const bool live = n0 + n < N && k0 + k < K;
                copy(bs + k * WLDT + n, live ? Bh + static_cast<size_t>(k0 + k) * b_ld + n0 + n : B, live);
            }
        } else {
            for (int i = tid; i < WN * TCH; i += 256) {
                const int n = i / TCH, k = (i % TCH) * 8;
                const bool live = n0 + n < N && k0 + k < K;
                copy(bs + n * WLD + k, live ? Bh + static_cast<size_t>(n0 + n) * b_ld + k0 + k : B, live);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[4][4][4] = {};
    pdl_wait();
    load(0, 0);
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += TK, buf ^= 1) {
        if (k0 + TK < K) {
            load(k0 + TK, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const __nv_bfloat16* const as = sm + buf * kWideStage;
        const __nv_bfloat16* const bs = as + WM * WLD;
#pragma unroll
        for (int kk = 0; kk < TK; kk += 16) {
            uint32_t af[4][4], bf[4][2];
#pragma unroll
            for (int i = 0; i < 4; ++i) ldmatrix_x4(af[i], as + (wm + i * 16 + (lane & 15)) * WLD + kk + (lane >> 4) * 8);
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                uint32_t r[4];
                if (N_CONTIGUOUS) {
                    const uint32_t addr = static_cast<uint32_t>(__cvta_generic_to_shared(bs + (kk + (lane & 15)) * WLDT + wn + j * 8 + (lane >> 4) * 8));
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
                } else {
                    ldmatrix_x4(r, bs + (wn + j * 8 + (lane & 7) + ((lane >> 4) << 3)) * WLD + kk + ((lane >> 3) & 1) * 8);
                }
                bf[j][0] = r[0]; bf[j][1] = r[1]; bf[j + 1][0] = r[2]; bf[j + 1][1] = r[3];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) mma_bf16_16816(acc[i][j], af[i], bf[j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m = m0 + wm + i * 16 + g + 8 * h;
            if (m >= M) continue;
            float f = 1.f;
            if (gate && !g_ns) f = 1.f / (1.f + expf(-to_f32(gate[static_cast<size_t>(m) * ldg + static_cast<size_t>(a) * g_hs])));
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int n = n0 + wn + j * 8 + 2 * t;          // N is even: both columns or none
                if (n >= N) continue;
                float v[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (gate && g_ns) f = 1.f / (1.f + expf(-to_f32(gate[static_cast<size_t>(m) * ldg + static_cast<size_t>(a) * g_hs + static_cast<size_t>(n + e) * g_ns])));
                    v[e] = acc[i][j][2 * h + e] * f;
                }
                *reinterpret_cast<__nv_bfloat162*>(C + static_cast<size_t>(m) * ldc + static_cast<size_t>(a) * c_hs + n) = __floats2bfloat162_rn(v[0], v[1]);
            }
        }
}

// ------------------------------------------------------------------------------------------- exact attention
constexpr int kLatWarps = 4;
constexpr int kMaxRank = 512;          // latent width the exact kernel keeps in registers (rank / 32 per lane)

template <typename T>
__device__ __forceinline__ float dot_span(const float* __restrict__ q, const T* __restrict__ k, int n) {
    float acc = 0.f;
    int d = 0;
    if (sizeof(T) == 2) {
        if ((reinterpret_cast<uintptr_t>(k) & 15) == 0) {
            for (; d + 8 <= n; d += 8) {
                const uint4 raw = *reinterpret_cast<const uint4*>(k + d);
                const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 f = __bfloat1622float2(pairs[i]);
                    acc = fmaf(q[d + 2 * i], f.x, acc);
                    acc = fmaf(q[d + 2 * i + 1], f.y, acc);
                }
            }
        }
    } else {
        if ((reinterpret_cast<uintptr_t>(k) & 15) == 0) {
            for (; d + 4 <= n; d += 4) {
                const float4 kv = *reinterpret_cast<const float4*>(k + d);
                acc = fmaf(q[d], kv.x, acc);
                acc = fmaf(q[d + 1], kv.y, acc);
                acc = fmaf(q[d + 2], kv.z, acc);
                acc = fmaf(q[d + 3], kv.w, acc);
            }
        }
    }
    for (; d < n; ++d) acc = fmaf(q[d], to_f32(k[d]), acc);
    return acc;
}

// qa: [tokens, heads, rank + rot]; out: [tokens, heads, rank]; pages: latent [num_pages, page_size, rank], key part
// [num_pages, page_size, rot].
template <typename T>
__global__ void __launch_bounds__(kLatWarps * 32)
latent_attention_kernel(const T* __restrict__ qa, T* __restrict__ out, const T* __restrict__ latent_pages,
                        const T* __restrict__ krot_pages, const int32_t* __restrict__ block_table, int table_width,
                        const int32_t* __restrict__ seq_of_token, const int32_t* __restrict__ positions, int heads, int rank,
                        int rot, int page_size, float scale, const float* __restrict__ sinks) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) float q_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x;
    const int head = blockIdx.y * kLatWarps + warp;
    if (head >= heads) return;
    const int width = rank + rot;
    const int padded = (width + 3) & ~3;
    T* out_row = out + (static_cast<size_t>(t) * heads + head) * rank;
    const int seq = seq_of_token[t];
    if (seq < 0) {
        for (int d = lane; d < rank; d += 32) out_row[d] = from_f32<T>(0.f);
        return;
    }
    const int pos = positions[t];
    const int32_t* table = block_table + static_cast<size_t>(seq) * table_width;
    float* qs = q_smem + warp * padded;
    const T* q_row = qa + (static_cast<size_t>(t) * heads + head) * width;
    for (int d = lane; d < width; d += 32) qs[d] = to_f32(q_row[d]);
    __syncwarp();

    float m = -INFINITY, l = 0.f;
    float acc[kMaxRank / 32];
#pragma unroll
    for (int i = 0; i < kMaxRank / 32; ++i) acc[i] = 0.f;

    for (int base = 0; base <= pos; base += 32) {
        const int key = base + lane;
        const bool ok = key <= pos;
        float s = -INFINITY;
        if (ok) {
            const size_t slot = static_cast<size_t>(table[key / page_size]) * page_size + key % page_size;
            s = (dot_span<T>(qs, latent_pages + slot * rank, rank) + dot_span<T>(qs + rank, krot_pages + slot * rot, rot)) * scale;
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float p = ok ? expf(s - m_new) : 0.f;
        const float corr = expf(m - m_new);
        l = l * corr + warp_sum(p);
#pragma unroll
        for (int i = 0; i < kMaxRank / 32; ++i) acc[i] *= corr;
        const int count = min(32, pos - base + 1);
        for (int j = 0; j < count; ++j) {
            const float pj = __shfl_sync(0xffffffffu, p, j);
            const int kj = base + j;
            const T* v_row = latent_pages + (static_cast<size_t>(table[kj / page_size]) * page_size + kj % page_size) * rank;
#pragma unroll
            for (int i = 0; i < kMaxRank / 32; ++i) {
                const int d = lane + 32 * i;
                if (d < rank) acc[i] = fmaf(pj, to_f32(v_row[d]), acc[i]);
            }
        }
        m = m_new;
    }
    float inv = 1.f / l;
    if (sinks) {        // exp(sink_h) joins the denominator after the last key group: the order of the sums depends on the position only
        const float sink = sinks[head], top = fmaxf(m, sink);
        const float keep = expf(m - top);
        inv = keep / (l * keep + expf(sink - top));
    }
#pragma unroll
    for (int i = 0; i < kMaxRank / 32; ++i) {
        const int d = lane + 32 * i;
        if (d < rank) out_row[d] = from_f32<T>(acc[i] * inv);
    }
}

}  // namespace stride

using namespace stride;

extern "C" {

int stride_latent_prepare(const void* q, int ldq, const void* proj, int ld, int kv_off, void* qa, const int32_t* positions,
                          const int32_t* seq_of_token, const int32_t* slot_mapping, const float* cos_table, const float* sin_table,
                          const float* latent_w, float eps, void* latent_pages, void* krot_pages, int tokens, int heads, int dim,
                          int rot, int rot_dims, int rank, int dtype, cudaStream_t stream) {
    if (tokens < 0 || heads <= 0 || dim <= 0 || rot < 0 || rank <= 0 || rot_dims < 0 || rot_dims > rot || rot_dims % 2 || ld <= 0 || ldq <= 0 || !q)
        return STRIDE_BAD_ARGUMENT;
    if (kv_off >= 0 && (!latent_w || !latent_pages || (rot > 0 && !krot_pages))) return STRIDE_BAD_ARGUMENT;
    if (tokens == 0) return 0;
    if (dtype == STRIDE_DTYPE_F32)
        stride::launch(latent_prepare_kernel<float>, dim3(tokens), dim3(128), 0, stream, static_cast<const float*>(q), ldq,
                       static_cast<const float*>(proj), ld, kv_off,
                       static_cast<float*>(qa), positions, seq_of_token, slot_mapping, cos_table, sin_table, latent_w, eps,
                       static_cast<float*>(latent_pages), static_cast<float*>(krot_pages), heads, dim, rot, rot_dims, rank);
    else if (dtype == STRIDE_DTYPE_BF16)
        stride::launch(latent_prepare_kernel<__nv_bfloat16>, dim3(tokens), dim3(128), 0, stream, static_cast<const __nv_bfloat16*>(q), ldq,
                       static_cast<const __nv_bfloat16*>(proj), ld, kv_off, static_cast<__nv_bfloat16*>(qa), positions, seq_of_token, slot_mapping, cos_table, sin_table,
                       latent_w, eps, static_cast<__nv_bfloat16*>(latent_pages), static_cast<__nv_bfloat16*>(krot_pages), heads, dim,
                       rot, rot_dims, rank);
    else
        return STRIDE_BAD_ARGUMENT;
    return STRIDE_LAUNCH_STATUS();
}

int stride_head_gemm(const void* A, int lda, int a_hs, const void* B, long long b_hs, int b_ks, int b_ns, void* C, int ldc, int c_hs,
                     const void* gate, int ldg, int g_hs, int g_ns, int M, int heads, int N, int K, int dtype, cudaStream_t stream) {
    if (M < 0 || heads <= 0 || N <= 0 || K <= 0 || heads > 65535 || g_hs < 0 || g_ns < 0) return STRIDE_BAD_ARGUMENT;
    if (M == 0) return 0;
    const dim3 grid((N + HN - 1) / HN, heads, (M + HM - 1) / HM);
    if (grid.z > 65535) return STRIDE_UNSUPPORTED;
    if (dtype == STRIDE_DTYPE_F32)
        stride::launch(head_gemm_kernel<float>, grid, dim3(256), 0, stream, static_cast<const float*>(A), lda, a_hs,
                       static_cast<const float*>(B), b_hs, b_ks, b_ns, static_cast<float*>(C), ldc, c_hs, static_cast<const float*>(gate),
                       ldg, g_hs, g_ns, M, N, K);
    else if (dtype == STRIDE_DTYPE_BF16) {
        const long long b_ld = b_ns == 1 ? b_ks : b_ns;
        // A CTA of the wide kernel walks K alone: where K is long, lies contiguous (which the narrow kernel reads well too) and the tiles are
        // few, the narrow one's many CTAs win. 16 heads, to 128 columns from 512, wide / narrow: 128 tokens 12.5 / 9.8 us, 512 13.4 / 12.9,
        // 1,024 17.5 / 24.6; to 512 from 128, 128 tokens, 5.7 / 6.6.
        const long long wide_ctas = static_cast<long long>((N + WN - 1) / WN) * heads * ((M + WM - 1) / WM);
        const bool wide = M >= 128 && (b_ns == 1 || K <= 128 || wide_ctas >= 128) && (b_ns == 1 || b_ks == 1) && K % 8 == 0 && N % 8 == 0 && lda % 8 == 0 && a_hs % 8 == 0 && b_hs % 8 == 0 && b_ld % 8 == 0 &&
                          ldc % 2 == 0 && c_hs % 2 == 0 && (reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) % 16 == 0 &&
                          reinterpret_cast<uintptr_t>(C) % 4 == 0;
        if (wide) {
            constexpr int bytes = 2 * kWideStage * 2;
            const auto kernel = b_ks == 1 ? head_gemm_wide_kernel<false> : head_gemm_wide_kernel<true>;
            const cudaError_t e = b_ks == 1 ? allow_shared<head_gemm_wide_kernel<false>>(bytes) : allow_shared<head_gemm_wide_kernel<true>>(bytes);
            if (e != cudaSuccess) return static_cast<int>(e);
            stride::launch(kernel, dim3((N + WN - 1) / WN, heads, (M + WM - 1) / WM), dim3(256), bytes, stream, static_cast<const __nv_bfloat16*>(A), lda, a_hs,
                           static_cast<const __nv_bfloat16*>(B), b_hs, static_cast<int>(b_ld), static_cast<__nv_bfloat16*>(C), ldc, c_hs,
                           static_cast<const __nv_bfloat16*>(gate), ldg, g_hs, g_ns, M, N, K);
            return STRIDE_LAUNCH_STATUS();
        }
        const dim3 tc_grid((N + TN - 1) / TN, heads, (M + TM - 1) / TM);
        stride::launch(head_gemm_tc_kernel, tc_grid, dim3(128), 0, stream, static_cast<const __nv_bfloat16*>(A), lda, a_hs,
                       static_cast<const __nv_bfloat16*>(B), b_hs, b_ks, b_ns, static_cast<__nv_bfloat16*>(C), ldc, c_hs,
                       static_cast<const __nv_bfloat16*>(gate), ldg, g_hs, g_ns, M, N, K);
    }
    else
        return STRIDE_BAD_ARGUMENT;
    return STRIDE_LAUNCH_STATUS();
}

// Pages: latent [pages, page_size, rank], key part [pages, page_size, rot], bf16, rank and rot multiples of 8, 16-byte aligned.
int stride_latent_gather(const void* latent_pages, const void* krot_pages, const int32_t* block_table, int table_width, const int32_t* ctx_len,
                         int num_seqs, int page_size, int rank, int rot, int rows, void* latent, void* krot, int32_t* range,
                         cudaStream_t stream) {
    if (num_seqs < 0 || page_size <= 0 || table_width <= 0 || rank <= 0 || rot <= 0 || rows < 0) return STRIDE_BAD_ARGUMENT;
    if (rank % 8 || rot % 8 || (reinterpret_cast<uintptr_t>(latent_pages) | reinterpret_cast<uintptr_t>(krot_pages) | reinterpret_cast<uintptr_t>(latent) |
                                reinterpret_cast<uintptr_t>(krot)) % 16)
        return STRIDE_UNSUPPORTED;
    if (num_seqs == 0 || rows == 0) return 0;
    stride::launch(latent_gather_kernel, dim3((rows + 7) / 8), dim3(256), 0, stream, static_cast<const uint4*>(latent_pages),
                   static_cast<const uint4*>(krot_pages), block_table, table_width, ctx_len, num_seqs, page_size, rank / 8, rot / 8, rows,
                   static_cast<uint4*>(latent), static_cast<uint4*>(krot), range);
    return STRIDE_LAUNCH_STATUS();
}

int stride_latent_attention(const void* qa, void* out, const void* latent_pages, const void* krot_pages, const int32_t* block_table,
                            int table_width, const int32_t* seq_of_token, const int32_t* positions, int tokens, int heads, int rank,
                            int rot, int page_size, float scale, const float* sinks, int dtype, cudaStream_t stream) {
    if (tokens < 0 || heads <= 0 || rank <= 0 || rot < 0 || page_size <= 0 || table_width <= 0) return STRIDE_BAD_ARGUMENT;
    if (rank > kMaxRank) return STRIDE_UNSUPPORTED;
    if (tokens == 0) return 0;
    const size_t smem = static_cast<size_t>(kLatWarps) * ((rank + rot + 3) & ~3) * sizeof(float);
    if (smem > 48 * 1024) return STRIDE_UNSUPPORTED;
    const dim3 grid(tokens, (heads + kLatWarps - 1) / kLatWarps);
    if (dtype == STRIDE_DTYPE_F32)
        stride::launch(latent_attention_kernel<float>, grid, dim3(kLatWarps * 32), smem, stream, static_cast<const float*>(qa),
                       static_cast<float*>(out), static_cast<const float*>(latent_pages), static_cast<const float*>(krot_pages), block_table,
                       table_width, seq_of_token, positions, heads, rank, rot, page_size, scale, sinks);
    else if (dtype == STRIDE_DTYPE_BF16)
        stride::launch(latent_attention_kernel<__nv_bfloat16>, grid, dim3(kLatWarps * 32), smem, stream,
                       static_cast<const __nv_bfloat16*>(qa), static_cast<__nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(latent_pages),
                       static_cast<const __nv_bfloat16*>(krot_pages), block_table, table_width, seq_of_token, positions, heads, rank, rot,
                       page_size, scale, sinks);
    else
        return STRIDE_BAD_ARGUMENT;
    return STRIDE_LAUNCH_STATUS();
}

}  // extern "C"
