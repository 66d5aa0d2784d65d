// Latent attention of portions of prompts on the latents themselves, on the fifth-generation tensor cores (bfloat16 operands, float32
// accumulators): the folded form of latent_attention_tc.cu with its sums in the same order, tile by tile, 16 terms at a time, and so with the
// same bits, which a layer behind it that magnifies roundings (the matrix LSTM) would otherwise show.
//
// Every head of a token reads the same keys [latent | rotated part] and the same values (the latent), so the 128 rows of a tile are
// (token, head) pairs of one request. Their accumulator alone, rank 512 wide, would fill tensor memory; so a tile has two CTAs, each of
// which makes all scores and half of the output columns (1.5 times the products that are needed; half the rows a CTA would cost
// twice, because a tile of 64 rows takes the tensor cores as long as one of 128). Keys go by 64:
//
//   S = Q K^T      Q: the first 256 columns in tensor memory, the others in shared memory (all of Q there would leave room for one tile
//                  of keys only, and the reads of both operands from shared memory would bound the product)
//   softmax        a row a thread; P in bfloat16 over the place of its scores
//   O += P V       P from tensor memory; V is the latent part of the same tile of keys, read MN-major
//
//   warps 0-3   softmax, output;  4-11  copies of keys through the block table (16 bytes a thread, zeros past the last key), four warps a
//   stage of the ring of two;  12  tcgen05.mma and the tensor memory
//
// Tensor memory: O 0-255, two buffers of scores 256-383, Q 384-511. O is scaled down, after the products so far have ended, whenever a
// row's maximum grows: a row's largest probability is then 1 and not rounded (following the maximum only where it has grown by 2^8 is
// 5 % further from 64 bits). Tiles with the most keys are started first.
//
// 16 heads, rank 512, us (mma.sync there): 2,000 tokens 207 (717), 512 tokens 39 (94), 33 behind 2,000 109 (326), 2,048 behind 14,336 2,656
// (9,465), 64 requests of 8 20.5 (22.5), 16 tokens 18.5 (22.6). A tile of keys takes 2.3 us: its copy (72 KB, bound by the copying
// warps' instructions: with the addresses worked out piece by piece it took 7 us), scores, softmax and second product, two tiles in flight.
//
// Every wait on an mbarrier is bounded by a clock; a wait that runs out sets *status and the CTA winds down.
#include "tcgen05.cuh"

namespace stride {
namespace latent5 {

using namespace tc;

constexpr int kRows = 128, kKeys = 64, kThreads = 416;
constexpr int kChunkQ = kRows * 128, kChunkK = kKeys * 128;      // 64 columns of every row, 128-byte swizzle
constexpr int kTmemQ = 256;                                     // columns of Q in tensor memory, at most
constexpr uint32_t kTScores = 256, kTQ = 384;

__device__ __forceinline__ void copy16(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void warp_arrive(uint32_t bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}

// qa: [tokens, heads, rank + rot]; out: [tokens, heads, rank]. Grid: (2 * row tiles of the longest request, requests).
__global__ void __launch_bounds__(kThreads, 1)
latent_attention_tc5_kernel(const __nv_bfloat16* __restrict__ qa, __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ latent_pages,
                            const __nv_bfloat16* __restrict__ krot_pages, const int32_t* __restrict__ block_table, int table_width,
                            const int32_t* __restrict__ q_start, const int32_t* __restrict__ q_len, const int32_t* __restrict__ ctx_len,
                            int heads, int rank, int rot, int page_size, float scale, const float* __restrict__ sinks, int* __restrict__ status) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t k_full[2], k_empty[2], s_full[2], p_full[2], pv_done, q_full, ended;
    __shared__ uint32_t tmem_slot;
    pdl_trigger();
    pdl_wait();
    const int seq = blockIdx.y, n = q_len[seq], total_rows = n * heads;
    const int tile = static_cast<int>(gridDim.x / 2 - 1 - blockIdx.x / 2), r0 = tile * kRows, side = blockIdx.x & 1;
    if (n <= 0 || r0 >= total_rows) return;         // the whole CTA
    unsigned char* const smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int start = q_start[seq], pos0 = ctx_len[seq] - n, width = rank + rot;
    const int last_row = min(total_rows, r0 + kRows) - 1, keys = pos0 + last_row / heads + 1, tiles = (keys + kKeys - 1) / kKeys;
    const int q_cols = min(kTmemQ, rank), q_chunks = (rank - q_cols) / 64 + 1, k_chunks = rank / 64 + 1, half = rank / 2;
    unsigned char* const k_s = smem + q_chunks * kChunkQ;
    const int stage_bytes = k_chunks * kChunkK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(smem_u32(&k_full[s]), 4);
            mbar_init(smem_u32(&k_empty[s]), 1);
            mbar_init(smem_u32(&s_full[s]), 1);
            mbar_init(smem_u32(&p_full[s]), 4);
        }
        mbar_init(smem_u32(&pv_done), 1);
        mbar_init(smem_u32(&q_full), 4);
        mbar_init(smem_u32(&ended), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 12) tmem_alloc(smem_u32(&tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    if (warp < 4) {
        const int row = warp * 32 + lane, my_row = r0 + row;
        const uint32_t lanes = static_cast<uint32_t>(warp * 32) << 16;
        const bool live = my_row < total_rows;
        const size_t out_row = static_cast<size_t>(start) * heads + my_row;
        // ---- Q, this warp's 32 rows: what goes to tensor memory by way of the second stage of the ring, the other columns to their place
        const int pieces = width / 8, q_pieces = q_cols / 8;
        unsigned char* const staged = k_s + stage_bytes;
        const __nv_bfloat16* const q_first = qa + (static_cast<size_t>(start) * heads + r0 + warp * 32) * width;
        const int rows_here = min(32, total_rows - r0 - warp * 32);
#pragma unroll 4
        for (int r = 0; r < 32; ++r) {
            const int bytes = r < rows_here ? 16 : 0;               // past the last row: zeros
            const __nv_bfloat16* const from = r < rows_here ? q_first + static_cast<size_t>(r) * width : qa;
            const uint32_t line = (warp * 32 + r) * 128;
            for (int x = lane; x < pieces; x += 32) {
                const int y = x < q_pieces ? x : x - q_pieces;
                const uint32_t to = smem_u32(x < q_pieces ? staged : smem);
                copy16(to + (y >> 3) * kChunkQ + line + (((y & 7) ^ (r & 7)) * 16), from + x * 8, bytes);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        for (int c = 0; c < q_cols; c += 32) {
            float v[16];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int y = c / 8 + i;
                const float4 x = *reinterpret_cast<const float4*>(staged + (y >> 3) * kChunkQ + row * 128 + (((y & 7) ^ (row & 7)) * 16));
                v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
            }
            tmem_st16(tmem + lanes + kTQ + c / 2, v);
        }
        fence_proxy_async();
        tc_fence_before();
        warp_arrive(smem_u32(&q_full));

        const int pos = live ? pos0 + my_row / heads : -1;          // -1: no key is visible
        const int free_tiles = (pos0 + r0 / heads + 1) / kKeys;     // tiles that every row of the CTA sees whole
        float top = -INFINITY, sum = 0.f;
        bool ok = true;
        for (int j = 0; j < tiles; ++j) {
            const uint32_t t_s = tmem + lanes + kTScores + (j & 1) * kKeys;
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&s_full[j & 1]), (j >> 1) & 1, status, 73));
            if (!ok) break;
            tc_fence_after();
            float s[64];
            tmem_ld64(t_s, s);
            const int seen = pos - j * kKeys;                       // the last key of the tile that the row sees
            if (j < free_tiles) {
#pragma unroll
                for (int i = 0; i < 64; ++i) s[i] *= scale;
            } else {
#pragma unroll
                for (int i = 0; i < 64; ++i) s[i] = i <= seen ? s[i] * scale : -INFINITY;
            }
            float m0 = s[0], m1 = s[1];
#pragma unroll
            for (int i = 2; i < 62; i += 4) {
                m0 = max3(m0, s[i], s[i + 1]);
                m1 = max3(m1, s[i + 2], s[i + 3]);
            }
            const float now = fmaxf(max3(m0, s[62], s[63]), m1);
            const bool grown = top != -INFINITY && now > top;       // (without a key yet there is nothing to scale)
            if (top == -INFINITY) top = now;
            float f = 1.f;
            if (__any_sync(0xffffffffu, grown)) {
                if (grown) {
                    f = expf(top - now);
                    top = now;
                }
                // (This wait may skip phases, and one on phase j - 1 would pass while phase j - 2 is not over. It is: the scores of tile j, which
                // have been read above, were made from keys that came into the place of tile j - 2 only after its second product.)
                ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&pv_done), (j - 1) & 1, status, 73));
                if (!ok) break;
                tc_fence_after();
                for (int c = 0; c < half; c += 16) {
                    float v[16];
                    tmem_ld16(tmem + lanes + c, v);
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] *= f;
                    tmem_st16(tmem + lanes + c, v);
                }
            }
            const float base = top == -INFINITY ? 0.f : top;
            // the sum of what the second product uses, in the order of latent_attention_tc.cu: pairs, fours and eights of keys, then one after another
            float total = 0.f;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float p[16];
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    float pair[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float x = s[32 * h + 2 * (i + e)], y = s[32 * h + 2 * (i + e) + 1];
                        const __nv_bfloat162 b = __floats2bfloat162_rn(expf(x - base), expf(y - base));
                        pair[e] = __low2float(b) + __high2float(b);
                        p[i + e] = __uint_as_float(*reinterpret_cast<const uint32_t*>(&b));
                    }
                    total += (pair[0] + pair[1]) + (pair[2] + pair[3]);
                }
                tmem_st16(t_s + 16 * h, p);
            }
            sum = sum * f + total;
            tc_fence_before();
            warp_arrive(smem_u32(&p_full[j & 1]));
        }
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&pv_done), (tiles - 1) & 1, status, 73));
        tc_fence_after();
        if (ok) {
            float inv = 1.f / sum;
            if (sinks && live) {        // exp(sink) joins the sum; both terms relative to the larger of the maximum and the sink
                const float sink = sinks[my_row % heads], most = fmaxf(top, sink);
                const float keep = expf(top - most);
                inv = keep / (sum * keep + expf(sink - most));
            }
            __nv_bfloat16* const to = out + out_row * rank + side * half;
            for (int c = 0; c < half; c += 32) {
                float v[32];
                tmem_ld32(tmem + lanes + c, v);
                if (!live) continue;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const __nv_bfloat162 b = __floats2bfloat162_rn(v[8 * i + 2 * e] * inv, v[8 * i + 2 * e + 1] * inv);
                        w[e] = *reinterpret_cast<const uint32_t*>(&b);
                    }
                    *reinterpret_cast<uint4*>(to + c + 8 * i) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
        }
        tc_fence_before();
    } else if (warp < 12) {
        // four warps a stage, 16 keys each: a key a lane looks its place up, then the warp copies key after key
        const int s = (warp - 4) >> 2, first = ((warp - 4) & 3) * 16, rot_pieces = rot / 8;
        const int32_t* const table = block_table + static_cast<size_t>(seq) * table_width;
        const uint32_t stage = smem_u32(k_s + s * stage_bytes);
        // of a key's row a lane brings the pieces lane and lane + 32
        const bool near = lane * 8 < rank, far = lane * 8 + 256 < rank;
        const uint32_t chunk = (lane >> 3) * kChunkK;
        bool ok = s == 0 || mbar_wait(smem_u32(&q_full), 0, status, 71);         // the second stage held Q on its way
        for (int j = s; j < tiles; j += 2) {
            if (j >= 2) ok = ok && mbar_wait(smem_u32(&k_empty[s]), ((j >> 1) & 1) ^ 1, status, 71);
            if (!(ok = __all_sync(0xffffffffu, ok))) break;
            const int key0 = j * kKeys + first, read = min(key0 + (lane & 15), keys - 1);
            const unsigned slot = static_cast<unsigned>(table[read / page_size]) * page_size + read % page_size;
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const size_t at = __shfl_sync(0xffffffffu, slot, r);
                const int bytes = key0 + r < keys ? 16 : 0;         // past the last key: zeros
                const uint32_t to = stage + chunk + (first + r) * 128 + (((lane & 7) ^ (r & 7)) * 16);
                const __nv_bfloat16* const from = latent_pages + at * rank + lane * 8;
                if (near) copy16(to, from, bytes);
                if (far) copy16(to + 4 * kChunkK, from + 256, bytes);
            }
            for (int i = lane; i < 16 * rot_pieces; i += 32) {
                const int r = i / rot_pieces, x = i % rot_pieces;
                const size_t at = __shfl_sync(0xffffffffu, slot, r);
                copy16(stage + (k_chunks - 1) * kChunkK + (first + r) * 128 + ((x ^ (r & 7)) * 16), krot_pages + at * rot + x * 8,
                       key0 + r < keys ? 16 : 0);
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            fence_proxy_async();
            warp_arrive(smem_u32(&k_full[s]));
        }
    } else {
        const bool issuer = elect_one();
        const uint32_t idesc_s = instr_desc_bf16(kRows, kKeys, false), idesc_o = instr_desc_bf16(kRows, half, true);
        bool ok = mbar_wait(smem_u32(&q_full), 0, status, 72);
        auto scores = [&](int j) {
            ok = ok && mbar_wait(smem_u32(&k_full[j & 1]), (j >> 1) & 1, status, 72);
            if (!(ok = __all_sync(0xffffffffu, ok))) return;
            tc_fence_after();
            const uint32_t d = tmem + kTScores + (j & 1) * kKeys, k_addr = smem_u32(k_s + (j & 1) * stage_bytes), q_addr = smem_u32(smem);
            if (issuer) {
                for (int c = 0; c < q_cols / 64; ++c) {
                    const uint64_t b = smem_desc_sw128(k_addr + c * kChunkK);
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_bf16_tmem_a(d, tmem + kTQ + c * 32 + k * 8, b + 2 * k, idesc_s, c > 0 || k > 0 ? 1u : 0u);
                }
                for (int c = 0; c < q_chunks; ++c) {
                    const uint64_t a = smem_desc_sw128(q_addr + c * kChunkQ), b = smem_desc_sw128(k_addr + (q_cols / 64 + c) * kChunkK);
                    const int steps = c + 1 < q_chunks ? 4 : rot / 16;
                    for (int k = 0; k < steps; ++k) umma_bf16(d, a + 2 * k, b + 2 * k, idesc_s, 1u);
                }
                umma_commit(smem_u32(&s_full[j & 1]));
            }
            __syncwarp();
        };
        scores(0);
        for (int j = 0; j < tiles && ok; ++j) {
            if (j + 1 < tiles) scores(j + 1);           // the tensor cores work on these while P is made
            ok = ok && mbar_wait(smem_u32(&p_full[j & 1]), (j >> 1) & 1, status, 72);
            if (!(ok = __all_sync(0xffffffffu, ok))) break;
            tc_fence_after();
            const uint32_t v_addr = smem_u32(k_s + (j & 1) * stage_bytes + side * (half / 64) * kChunkK);
            if (issuer) {
#pragma unroll
                for (int k = 0; k < kKeys / 16; ++k)        // 16 keys: 16 rows of 128 bytes
                    umma_bf16_tmem_a(tmem, tmem + kTScores + (j & 1) * kKeys + k * 8, smem_desc(v_addr + k * 2048, kChunkK, 1024), idesc_o,
                                     j > 0 || k > 0 ? 1u : 0u);
                umma_commit(smem_u32(&k_empty[j & 1]));
                umma_commit(smem_u32(&pv_done));
            }
            __syncwarp();
        }
        // what was issued ends before the CTA does, also after a wait that ran out
        if (issuer) umma_commit(smem_u32(&ended));
        __syncwarp();
        mbar_wait(smem_u32(&ended), 0, status, 72);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 12) tmem_dealloc(tmem, 512);
}

inline int shared_bytes(int rank) {
    const int q_cols = rank < kTmemQ ? rank : kTmemQ, stage = (rank / 64 + 1) * kChunkK, staged = q_cols / 64 * kChunkQ;
    return ((rank - q_cols) / 64 + 1) * kChunkQ + stage + (stage > staged ? stage : staged) + 1024;
}

}  // namespace latent5
}  // namespace stride

using namespace stride;

// The step's first num_seqs requests, which bring up to max_q_len tokens each. Returns -2 for what it does not take.
extern "C" int stride_latent_attention_tc5(const void* qa, void* out, const void* latent_pages, const void* krot_pages, const int32_t* block_table,
                                           int table_width, const int32_t* q_start, const int32_t* q_len, const int32_t* ctx_len, int num_seqs,
                                           int max_q_len, int heads, int rank, int rot, int page_size, float scale, const float* sinks, int* status,
                                           cudaStream_t stream) {
    if (num_seqs < 0 || max_q_len <= 0 || page_size <= 0 || table_width <= 0 || heads <= 0 || status == nullptr) return STRIDE_BAD_ARGUMENT;
    if (rank <= 0 || rank % 128 || rank > 512 || rot <= 0 || rot % 16 || rot > 64 || num_seqs > 65535) return STRIDE_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(qa) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(latent_pages) | reinterpret_cast<uintptr_t>(krot_pages)) & 15)
        return STRIDE_UNSUPPORTED;
    if (num_seqs == 0) return 0;
    const cudaError_t e = allow_shared<latent5::latent_attention_tc5_kernel>(latent5::shared_bytes(512));
    if (e != cudaSuccess) return static_cast<int>(e);
    const long long row_tiles = (static_cast<long long>(max_q_len) * heads + latent5::kRows - 1) / latent5::kRows;
    const dim3 grid(static_cast<unsigned>(2 * row_tiles), num_seqs);
    stride::launch(latent5::latent_attention_tc5_kernel, grid, dim3(latent5::kThreads), latent5::shared_bytes(rank), stream,
                   static_cast<const __nv_bfloat16*>(qa), static_cast<__nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(latent_pages),
                   static_cast<const __nv_bfloat16*>(krot_pages), block_table, table_width, q_start, q_len, ctx_len, heads, rank, rot, page_size,
                   scale, sinks, status);
    return STRIDE_LAUNCH_STATUS();
}
