// Paged attention for any mix of prompt portions and decoded tokens, in float32
// or bfloat16 storage with float32 arithmetic, any head size up to 256. This is the exact, slower kernel:
// the whole 32-bit path runs on it, and the bfloat16 path falls back to it for
// head sizes or windows that the tensor-core kernels refuse.
//
// One warp owns one (token, query head). The token at absolute position p of its
// request reads the keys j <= p (and j > p - window when a window is set) through
// the request's block table: softmax(q k^T * scale) v with the causal rule of
// python/stride_worker/layers.py:109-149; query head h reads key head
// h / (nq / nkv). Keys are walked in groups of 32 aligned to absolute position 0,
// with an online softmax, so the order of every sum depends only on p: the result
// for a token is bitwise the same in a whole prompt, in a portion or as a single
// decoded token, whatever pages hold the keys.
//
// Two optional rules on top: a cap c on the scores, s <- c tanh(s / c) after the scale; and a sink per query head, a
// learned number whose exponential joins the softmax's denominator (it has no key and no value and is not scaled): it
// enters the running maximum and sum after the last group of keys, so the order of the sums stays a function of p.
// Values may be narrower or wider than keys (`vd` beside `hd`), and a head may take a penalty off a score in proportion
// to the key's distance: s <- s - slope_h (p - j), the slopes given per query head, or gain a learned number that depends on
// the distance: s <- s + rel[h, min(p - j, rel_len - 1)] (a table per query head whose last entry serves all farther keys).
#include "common.cuh"

namespace stride {

constexpr int kWarps = 4;
constexpr int kMaxHeadDim = 256;
constexpr int kMaxTileDim = 128;        // widths of keys and values of the kernel with the keys in shared memory

template <typename T>
__device__ __forceinline__ float dot_row(const float* __restrict__ q, const T* __restrict__ k, int hd);

template <>
__device__ __forceinline__ float dot_row<float>(const float* __restrict__ q, const float* __restrict__ k, int hd) {
    float acc = 0.f;
    if (hd & 3) {       // rows that do not start on 16-byte boundaries: one entry at a time
        for (int d = 0; d < hd; ++d) acc = fmaf(q[d], k[d], acc);
        return acc;
    }
    for (int d = 0; d < hd; d += 4) {
        const float4 kv = *reinterpret_cast<const float4*>(k + d);
        acc = fmaf(q[d], kv.x, acc);
        acc = fmaf(q[d + 1], kv.y, acc);
        acc = fmaf(q[d + 2], kv.z, acc);
        acc = fmaf(q[d + 3], kv.w, acc);
    }
    return acc;
}

template <>
__device__ __forceinline__ float dot_row<__nv_bfloat16>(const float* __restrict__ q, const __nv_bfloat16* __restrict__ k, int hd) {
    float acc = 0.f;
    if (hd & 7) {
        for (int d = 0; d < hd; ++d) acc = fmaf(q[d], __bfloat162float(k[d]), acc);
        return acc;
    }
    for (int d = 0; d < hd; d += 8) {
        const uint4 raw = *reinterpret_cast<const uint4*>(k + d);
        const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(pairs[i]);
            acc = fmaf(q[d + 2 * i], f.x, acc);
            acc = fmaf(q[d + 2 * i + 1], f.y, acc);
        }
    }
    return acc;
}

template <typename T>
__global__ void __launch_bounds__(kWarps * 32)
paged_attention_generic_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out, const T* __restrict__ k_pages,
                               const T* __restrict__ v_pages, const int32_t* __restrict__ block_table, int table_width,
                               const int32_t* __restrict__ seq_of_token, const int32_t* __restrict__ positions, int nq,
                               int nkv, int hd, int vd, int page_size, float scale, int window, float softcap,
                               const float* __restrict__ sinks, const float* __restrict__ slopes, const float* __restrict__ rel, int rel_len) {
    pdl_trigger();
    pdl_wait();
    __shared__ __align__(16) float q_smem[kWarps][kMaxHeadDim];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x;
    const int head = blockIdx.y * kWarps + warp;
    if (head >= nq) return;
    T* out_row = out + (static_cast<size_t>(t) * nq + head) * vd;
    const int seq = seq_of_token[t];
    if (seq < 0) {  // a padded token of a fixed-size batch
        for (int d = lane; d < vd; d += 32) out_row[d] = from_f32<T>(0.f);
        return;
    }
    const int pos = positions[t];
    const int kvh = head / (nq / nkv);
    const int first = window > 0 ? max(0, pos - window + 1) : 0;
    const int32_t* table = block_table + static_cast<size_t>(seq) * table_width;

    float* qs = q_smem[warp];
    const T* q_row = q + static_cast<size_t>(t) * q_stride + static_cast<size_t>(head) * hd;
    for (int d = lane; d < hd; d += 32) qs[d] = to_f32(q_row[d]);
    __syncwarp();

    const float slope = slopes ? slopes[head] : 0.f;
    float m = -INFINITY, l = 0.f;
    float acc[kMaxHeadDim / 32];
#pragma unroll
    for (int i = 0; i < kMaxHeadDim / 32; ++i) acc[i] = 0.f;

    for (int base = (first / 32) * 32; base <= pos; base += 32) {
        const int key = base + lane;
        const bool ok = key >= first && key <= pos;
        float s = -INFINITY;
        if (ok) {
            const int page = table[key / page_size];
            const T* k_row = k_pages + ((static_cast<size_t>(page) * nkv + kvh) * page_size + key % page_size) * hd;
            s = dot_row<T>(qs, k_row, hd) * scale;
            if (softcap > 0.f) s = softcap * tanhf(s / softcap);
            if (slopes) s = __fadd_rn(s, -__fmul_rn(slope, static_cast<float>(pos - key)));
            if (rel) s = __fadd_rn(s, rel[static_cast<size_t>(head) * rel_len + min(pos - key, rel_len - 1)]);
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float p = ok ? expf(s - m_new) : 0.f;
        const float corr = expf(m - m_new);
        l = l * corr + warp_sum(p);
#pragma unroll
        for (int i = 0; i < kMaxHeadDim / 32; ++i) acc[i] *= corr;
        unsigned valid = __ballot_sync(0xffffffffu, ok);
        while (valid) {
            const int j = __ffs(valid) - 1;
            valid &= valid - 1;
            const float pj = __shfl_sync(0xffffffffu, p, j);
            const int kj = base + j;
            const int page = table[kj / page_size];
            const T* v_row = v_pages + ((static_cast<size_t>(page) * nkv + kvh) * page_size + kj % page_size) * vd;
#pragma unroll
            for (int i = 0; i < kMaxHeadDim / 32; ++i) {
                const int d = lane + 32 * i;
                if (d < vd) acc[i] = fmaf(pj, to_f32(v_row[d]), acc[i]);
            }
        }
        m = m_new;
    }
    if (sinks) {
        const float sink = sinks[head];
        const float m_new = fmaxf(m, sink);
        const float corr = expf(m - m_new);
        l = l * corr + expf(sink - m_new);
#pragma unroll
        for (int i = 0; i < kMaxHeadDim / 32; ++i) acc[i] *= corr;
    }
    const float inv = 1.f / l;
#pragma unroll
    for (int i = 0; i < kMaxHeadDim / 32; ++i) {
        const int d = lane + 32 * i;
        if (d < vd) out_row[d] = from_f32<T>(acc[i] * inv);
    }
}

// The same in float32 with the keys in shared memory: a CTA owns TQ consecutive rows of the flat batch and up to GH query heads of one
// key head, a warp NR of those (token, head) rows; 32 keys and values at a time come in by cp.async, the next ones while these are
// worked through, and serve every row. A lane's chain over a key's numbers, the online softmax over a group of 32 keys and the order
// of the values are those of the kernel above, so every row has the same bits whichever ran it. Bound by the chains: head size 128
// costs 512 cycles a group, NR of them side by side. A prompt of 301 tokens, 24 heads on 8: 109 us (above: 342 us, where every (token, head)
// reads its keys itself, lane by lane, and waits for every page number), a single token behind 151: 33 us (84).
template <int TQ, int NW, int NR>
__global__ void __launch_bounds__(NW * 32)
paged_attention_tile_f32_kernel(const float* __restrict__ q, int q_stride, float* __restrict__ out, const float* __restrict__ k_pages,
                                const float* __restrict__ v_pages, const int32_t* __restrict__ block_table, int table_width,
                                const int32_t* __restrict__ seq_of_token, const int32_t* __restrict__ positions, int tokens, int nq, int nkv,
                                int hd, int vd, int page_size, float scale, int window, float softcap, const float* __restrict__ sinks,
                                const float* __restrict__ slopes, const float* __restrict__ rel, int rel_len, int GH) {
    constexpr int THREADS = NW * 32, MAXV = kMaxTileDim / 32;
    extern __shared__ __align__(16) float tile_smem[];
    const int kld = hd + 4;
    float* const ks = tile_smem;                        // [2][32][hd + 4]
    float* const vs = ks + 2 * 32 * kld;                // [2][32][vd]
    float* const qs = vs + 2 * 32 * vd;                 // [NW * NR][hd]
    pdl_trigger();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = nq / nkv, parts = (group + GH - 1) / GH;
    const int kvh = blockIdx.y / parts, head0 = kvh * group + (blockIdx.y % parts) * GH, heads = min(GH, (kvh + 1) * group - head0);
    const int t0 = blockIdx.x * TQ, t_end = min(tokens, t0 + TQ);
    auto row_token = [&](int row) { return t0 + row / GH; };
    auto row_head = [&](int row) { return head0 + row % GH; };
    auto row_used = [&](int row) { return row / GH < TQ && row_token(row) < t_end && row % GH < heads; };
    for (int i = threadIdx.x; i < NW * NR * hd; i += THREADS) {
        const int row = i / hd, d = i - row * hd;
        qs[i] = row_used(row) ? q[static_cast<size_t>(row_token(row)) * q_stride + static_cast<size_t>(row_head(row)) * hd + d] : 0.f;
    }
    for (int a = t0; a < t_end;) {                      // a run of rows of one request
        const int seq = seq_of_token[a];
        int b = a + 1, low = positions[a], high = low;
        while (b < t_end && seq_of_token[b] == seq) {
            low = min(low, positions[b]);
            high = max(high, positions[b]);
            ++b;
        }
        if (seq < 0) {                                  // padded tokens of a fixed-size batch
            for (int row = warp; row < TQ * GH; row += NW)
                if (row_used(row) && row_token(row) >= a && row_token(row) < b)
                    for (int d = lane; d < vd; d += 32) out[(static_cast<size_t>(row_token(row)) * nq + row_head(row)) * vd + d] = 0.f;
            a = b;
            continue;
        }
        const int32_t* table = block_table + static_cast<size_t>(seq) * table_width;
        const int lowest = window > 0 ? max(0, low - window + 1) : 0, begin = lowest / 32 * 32;       // pages before may have been given back
        int pos[NR];
        float m[NR], l[NR], acc[NR][MAXV];
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const int row = warp * NR + r;
            pos[r] = row_used(row) && row_token(row) >= a && row_token(row) < b ? positions[row_token(row)] : -1;       // -1: not of this run
            m[r] = -INFINITY;
            l[r] = 0.f;
#pragma unroll
            for (int i = 0; i < MAXV; ++i) acc[r][i] = 0.f;
        }
        auto load = [&](int base, int buf) {            // keys that no row of the run sees are left out: nobody looks at them
            const int kc = hd / 4, vc = vd / 4;
            for (int i = threadIdx.x; i < 32 * (kc + vc); i += THREADS) {
                const int j = i / (kc + vc), c = i - j * (kc + vc), key = base + j;
                if (key > high) break;
                if (key < lowest) continue;
                const size_t slot = (static_cast<size_t>(table[key / page_size]) * nkv + kvh) * page_size + key % page_size;
                float* dst = c < kc ? ks + (buf * 32 + j) * kld + 4 * c : vs + (buf * 32 + j) * vd + 4 * (c - kc);
                const float* src = c < kc ? k_pages + slot * hd + 4 * c : v_pages + slot * vd + 4 * (c - kc);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        load(begin, 0);
        int buf = 0;
        for (int base = begin; base <= high; base += 32, buf ^= 1) {
            if (base + 32 <= high) {
                load(base + 32, buf ^ 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
            const int key = base + lane;
            const float* k_row = ks + (buf * 32 + lane) * kld;
            float s[NR];
            unsigned valid[NR], any = 0;
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const int first = window > 0 ? max(0, pos[r] - window + 1) : 0;
                valid[r] = __ballot_sync(0xffffffffu, key >= first && key <= pos[r]);
                any |= valid[r];
                s[r] = 0.f;
            }
            if (any) {
                const float* q_row = qs + warp * NR * hd;
                for (int d = 0; d < hd; d += 4) {
                    const float4 kv = *reinterpret_cast<const float4*>(k_row + d);
#pragma unroll
                    for (int r = 0; r < NR; ++r) {
                        const float4 qv = *reinterpret_cast<const float4*>(q_row + r * hd + d);
                        s[r] = fmaf(qv.x, kv.x, s[r]);
                        s[r] = fmaf(qv.y, kv.y, s[r]);
                        s[r] = fmaf(qv.z, kv.z, s[r]);
                        s[r] = fmaf(qv.w, kv.w, s[r]);
                    }
                }
                float p[NR];
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    p[r] = 0.f;
                    if (!valid[r]) continue;
                    const bool ok = (valid[r] >> lane) & 1u;
                    const int head = row_head(warp * NR + r);
                    float z = s[r] * scale;
                    if (softcap > 0.f) z = softcap * tanhf(z / softcap);
                    if (slopes) z = __fadd_rn(z, -__fmul_rn(slopes[head], static_cast<float>(pos[r] - key)));
                    if (rel && ok) z = __fadd_rn(z, rel[static_cast<size_t>(head) * rel_len + min(pos[r] - key, rel_len - 1)]);
                    z = ok ? z : -INFINITY;
                    const float m_new = fmaxf(m[r], warp_max(z));
                    p[r] = ok ? expf(z - m_new) : 0.f;
                    const float corr = expf(m[r] - m_new);
                    l[r] = l[r] * corr + warp_sum(p[r]);
#pragma unroll
                    for (int i = 0; i < MAXV; ++i) acc[r][i] *= corr;
                    m[r] = m_new;
                }
                const float* v_tile = vs + buf * 32 * vd;
                for (unsigned left = any; left; left &= left - 1) {
                    const int j = __ffs(left) - 1;
                    float v[MAXV];
#pragma unroll
                    for (int i = 0; i < MAXV; ++i) v[i] = lane + 32 * i < vd ? v_tile[j * vd + lane + 32 * i] : 0.f;
#pragma unroll
                    for (int r = 0; r < NR; ++r) {
                        const float pj = __shfl_sync(0xffffffffu, p[r], j);
                        if ((valid[r] >> j) & 1u) {
#pragma unroll
                            for (int i = 0; i < MAXV; ++i) acc[r][i] = fmaf(pj, v[i], acc[r][i]);
                        }
                    }
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            if (pos[r] < 0) continue;
            const int row = warp * NR + r;
            if (sinks) {
                const float sink = sinks[row_head(row)];
                const float m_new = fmaxf(m[r], sink);
                const float corr = expf(m[r] - m_new);
                l[r] = l[r] * corr + expf(sink - m_new);
#pragma unroll
                for (int i = 0; i < MAXV; ++i) acc[r][i] *= corr;
            }
            const float inv = 1.f / l[r];
            float* out_row = out + (static_cast<size_t>(row_token(row)) * nq + row_head(row)) * vd;
#pragma unroll
            for (int i = 0; i < MAXV; ++i)
                if (lane + 32 * i < vd) out_row[lane + 32 * i] = acc[r][i] * inv;
        }
        a = b;
    }
}

template <int TQ, int NW, int NR>
int launch_tiles(const float* q, int q_stride, float* out, const float* k_pages, const float* v_pages, const int32_t* block_table, int table_width,
                 const int32_t* seq_of_token, const int32_t* positions, int tokens, int nq, int nkv, int hd, int vd, int page_size, float scale,
                 int window, float softcap, const float* sinks, const float* slopes, const float* rel, int rel_len, int gh, int ctas_y,
                 cudaStream_t stream) {
    const auto floats = [](int hd, int vd) { return 2 * 32 * (hd + 4) + 2 * 32 * vd + NW * NR * hd; };
    const cudaError_t e = allow_shared<paged_attention_tile_f32_kernel<TQ, NW, NR>>(floats(kMaxTileDim, kMaxTileDim) * 4);
    if (e != cudaSuccess) return static_cast<int>(e);
    stride::launch(paged_attention_tile_f32_kernel<TQ, NW, NR>, dim3((tokens + TQ - 1) / TQ, ctas_y), dim3(NW * 32), floats(hd, vd) * 4, stream, q,
                   q_stride, out, k_pages, v_pages, block_table, table_width, seq_of_token, positions, tokens, nq, nkv, hd, vd, page_size, scale,
                   window, softcap, sinks, slopes, rel, rel_len, gh);
    return STRIDE_LAUNCH_STATUS();
}

}  // namespace stride

using namespace stride;

// q: [tokens, q_stride] with head h at columns [h*hd, (h+1)*hd); out: [tokens, nq, vd];
// key pages: [num_pages, nkv, page_size, hd], value pages the same with vd; block_table: [seqs, table_width]. portions: which
// kernel a 32-bit step takes, 0 a row a CTA, 1 eight rows a CTA, 2 a (row, head) a warp; the results are the same.
extern "C" int stride_paged_attention_generic(const void* q, int q_stride, void* out, const void* k_pages, const void* v_pages,
                                              const int32_t* block_table, int table_width, const int32_t* seq_of_token,
                                              const int32_t* positions, int tokens, int nq, int nkv, int hd, int vd, int page_size,
                                              float scale, int window, float softcap, const float* sinks, const float* slopes,
                                              const float* rel, int rel_len, int portions, int dtype, cudaStream_t stream) {
    if (tokens < 0 || nq <= 0 || nkv <= 0 || hd <= 0 || vd <= 0 || page_size <= 0 || table_width <= 0 || window < 0 || softcap < 0.f ||
        (rel && rel_len <= 0)) return STRIDE_BAD_ARGUMENT;
    if (nq % nkv) return STRIDE_BAD_ARGUMENT;
    if (hd > kMaxHeadDim || vd > kMaxHeadDim) return STRIDE_UNSUPPORTED;
    if (tokens == 0) return 0;
    // a warp reads its keys in packs of 16 bytes where a row is whole packs
    if (hd % (dtype == STRIDE_DTYPE_F32 ? 4 : 8) == 0 && reinterpret_cast<uintptr_t>(k_pages) % 16) return STRIDE_UNSUPPORTED;
    const bool tile = portions != 2 && dtype == STRIDE_DTYPE_F32 && hd % 4 == 0 && vd % 4 == 0 && hd <= kMaxTileDim && vd <= kMaxTileDim &&
                      (reinterpret_cast<uintptr_t>(k_pages) | reinterpret_cast<uintptr_t>(v_pages)) % 16 == 0;
    if (tile) {
        const int gh = min(nq / nkv, 4), ctas_y = nkv * ((nq / nkv + gh - 1) / gh);
        if (ctas_y <= 65535) {
            return portions ? launch_tiles<8, 8, 4>(static_cast<const float*>(q), q_stride, static_cast<float*>(out), static_cast<const float*>(k_pages),
                                                    static_cast<const float*>(v_pages), block_table, table_width, seq_of_token, positions, tokens, nq,
                                                    nkv, hd, vd, page_size, scale, window, softcap, sinks, slopes, rel, rel_len, gh, ctas_y, stream)
                            : launch_tiles<1, 4, 1>(static_cast<const float*>(q), q_stride, static_cast<float*>(out), static_cast<const float*>(k_pages),
                                                    static_cast<const float*>(v_pages), block_table, table_width, seq_of_token, positions, tokens, nq,
                                                    nkv, hd, vd, page_size, scale, window, softcap, sinks, slopes, rel, rel_len, gh, ctas_y, stream);
        }
    }
    dim3 grid(tokens, (nq + kWarps - 1) / kWarps);
    if (dtype == STRIDE_DTYPE_F32)
        stride::launch(paged_attention_generic_kernel<float>, dim3(grid), dim3(kWarps * 32), 0, stream, 
            static_cast<const float*>(q), q_stride, static_cast<float*>(out), static_cast<const float*>(k_pages),
            static_cast<const float*>(v_pages), block_table, table_width, seq_of_token, positions, nq, nkv, hd, vd, page_size, scale, window, softcap, sinks, slopes, rel, rel_len);
    else if (dtype == STRIDE_DTYPE_BF16)
        stride::launch(paged_attention_generic_kernel<__nv_bfloat16>, dim3(grid), dim3(kWarps * 32), 0, stream, 
            static_cast<const __nv_bfloat16*>(q), q_stride, static_cast<__nv_bfloat16*>(out),
            static_cast<const __nv_bfloat16*>(k_pages), static_cast<const __nv_bfloat16*>(v_pages), block_table, table_width,
            seq_of_token, positions, nq, nkv, hd, vd, page_size, scale, window, softcap, sinks, slopes, rel, rel_len);
    else
        return STRIDE_BAD_ARGUMENT;
    return STRIDE_LAUNCH_STATUS();
}
