// Linear attention with a fading memory: per head a matrix S [D, DV] in float32 from zero and, per token,
//
//   channel decays     S <- diag(alpha_t) S + k v^T ;  o = S^T (q D^-1/2),  alpha_t = sigmoid(z_t + b)^(1 / tau) per key channel
//                      (Yang et al., "Gated Linear Attention Transformers with Hardware-Efficient Training")
//   constant decay     S <- decay_h S + silu(k) silu(v)^T ;  o = S^T silu(q)
//                      (Qin et al., "Lightning Attention-2: A Free Lunch for Handling Unlimited Sequence Lengths in Large
//                      Language Models")
//
// Three forms of the same recurrence:
//
//   decay_step    a single token of every request (decoding in bfloat16 models): one pass over S.
//   decay_scan    one token after the other (memory_scan.cuh): short portions, and the whole 32-bit path, where a token's
//                 output must not depend on how its prompt was cut.
//   decay_chunks  long portions, chunks of 64 tokens side by side. With g_t the running product of decays inside a chunk (from
//                 its first token on, so g <= 1), G the chunk's whole product and S_c the memory before the chunk:
//                     o_i = (q_i g_i)^T S_c + sum_{j <= i} ((q_i g_i) . (k_j / g_j)) v_j
//                     S_(c+1) = G S_c + sum_j (k_j G / g_j) v_j^T
//                 Four launches: the running logarithms of the decays (channel decays only), every chunk's own sum, the
//                 memories at the chunks' starts (memory_scan.cuh: pieces_combine), the outputs. All of it in float32 on the FMA
//                 pipe (the memory, the decays and what enters them are float32 by the designs' own rule, so the tensor cores,
//                 which would round the operands, are left out), as register-tiled products from shared memory.
//                 1 / g_j can overflow where a channel forgets nearly everything within a chunk: a CTA whose chunk has a
//                 channel with g below e^-60 forms its scores with exp(log g_i - log g_j) per channel instead, which only
//                 costs time. A constant decay never divides: decay^(i - j) is taken from a table of powers.
//
// The chunks also run the matrix LSTM of mlstm.cu (mlstm_chunks): its gates are one number a head and token, with a running
// maximum; n goes along as one more column. 2,000 tokens of 16 heads of 128 x 128: 131 us, 634 us token after token.
#include "memory_scan.cuh"

namespace stride {

constexpr int kChunk = 64;              // tokens a chunk
constexpr int kChunkCols = 128;         // columns of S a CTA works on
constexpr int kSumCols = 64;            // the same in the kernel of the chunks' own sums
constexpr int kChunkThreads = 256;
constexpr int kLd = kChunk + 4;         // row stride of the transposed tiles: 16-byte reads, stores without bank conflicts
constexpr float kSafeLog = -60.f;
// The matrix LSTM's sums over channels and over a chunk's tokens go in runs of this many terms, which are then added up: as one chain
// of 128 terms they were further from 64 bits than the token-by-token kernel, whose sums are spread over lanes (16 heads of 128 x 128,
// gates as a projection makes them: median error of a row 1.2 of that kernel's as one chain, 0.9 in runs; 2,000 tokens 122 us and
// 131 us).
constexpr int kRun = 16;

// The gates of a chunk's tokens of one head of the matrix LSTM (lstm_gates_kernel): with b the running sum of the forget gates'
// logarithms inside the chunk, li the input gates' logarithms, m the running maximum (m_0 at the chunk's start, m_e at its end), token
// j weighs exp(b_i - b_j + li_j - m_i) in token i's output, the memory at the start exp(b_i + m_0 - m_i).
struct LstmChunk {
    float b_hi[kChunk], b_lo[kChunk];   // b in two parts: a difference of two sums is as good as the sum of the logarithms between them
    float li[kChunk], m[kChunk];
    float carry[kChunk];                // exp(b_i + m_0 - m_i)
    float take[kChunk];                 // exp(b_e - b_j + li_j - m_e): token j's weight in the memory at the chunk's end
    float decay, pad[3];                // carry at the end
};

struct ChunkArgs {
    const void* q;          // [tokens, ld], head h at column h * D
    const void* k;
    const void* v;          // head h at column h * DV
    int ld, in_bf16;
    float* cum;             // channel decays: [tokens, H * D], the running logarithm of the decays inside the chunk
    const float* bias;      // channel decays: [H * D]
    const float* powers;    // constant decay: [H, kChunk + 1], decay^n
    // matrix LSTM: the chunks lie one request's behind the other's, records of them at most, so that a long portion beside many short
    // ones costs no room for chunks that are not there
    const LstmChunk* lstm;  // [records, H]
    float* piece_n;         // [records, H, D]
    const int2* where;      // [records]: a chunk's request and first token, -1 past the last chunk (null: of one request, in order)
    const int32_t* base;    // [seqs]: a request's first chunk (null: of one request)
    int records;
    float q_scale, inv_tau;
    float* o;               // [tokens, H * DV]
    float* piece_s;         // [seqs * max_pieces (matrix LSTM: records), H, D, DV]
    float* piece_p;         // [the same, H, D]
    const int32_t* q_start;
    const int32_t* q_len;
    int H, D, DV, max_pieces;
    int vec;                // bfloat16 rows that can be read in packs of 8
};

// z -> running sums of log(sigmoid(z + b)) / tau over the chunk's tokens, in place. One thread a (head, channel).
static __global__ void __launch_bounds__(128)
chunk_decay_kernel(const ChunkArgs p) {
    pdl_trigger();
    pdl_wait();
    const int z = blockIdx.y, seq = z / p.max_pieces, first = (z % p.max_pieces) * kChunk;
    const int nt = min(p.q_len[seq] - first, kChunk);
    const int c = blockIdx.x * blockDim.x + threadIdx.x, HD = p.H * p.D;
    if (nt <= 0 || c >= HD) return;
    float* at = p.cum + static_cast<size_t>(p.q_start[seq] + first) * HD + c;
    const float b = p.bias[c];
    float sum = 0.f, lost = 0.f;        // Kahan's sum: differences of these sums are the exponents of whole decays
    for (int t0 = 0; t0 < nt; t0 += 8) {
        float l[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) l[u] = t0 + u < nt ? at[static_cast<size_t>(t0 + u) * HD] : 0.f;
#pragma unroll
        for (int u = 0; u < 8; ++u) l[u] = log_sigmoid_f(l[u] + b) * p.inv_tau;
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (t0 + u < nt) {
                const float y = __fadd_rn(l[u], -lost), next = __fadd_rn(sum, y);
                lost = __fadd_rn(__fadd_rn(next, -sum), -y);
                sum = next;
                at[static_cast<size_t>(t0 + u) * HD] = sum;
            }
    }
}

struct LstmGates {
    const float* gates;     // [tokens, ld] float32: column h the input gate's projection, column H + h the forget gate's
    int ld;
    const float* bias_i;
    const float* bias_f;
    float cap;
    float* state;           // m of head h at m_off + h of a slot's row
    long long state_stride, m_off;
    const int32_t* state_slot;
    LstmChunk* chunks;
    int2* where;
    int32_t* base;
    int records;
};

// The gates' logarithms, their running sums in a chunk and the running maximum through a whole portion, m_t = max(lf_t + m_(t-1), li_t):
// with A the sum and B the largest contribution of a run of tokens, two runs make A = A1 + A2, B = max(B1 + A2, B2), and
// m = max(m_0 + A, B), so 256 tokens (four chunks) are one scan over a CTA. Sums and exponents in float64. Grid (heads, requests).
static __global__ void __launch_bounds__(256)
lstm_gates_kernel(const LstmGates p, const int32_t* __restrict__ q_start, const int32_t* __restrict__ q_len, int H) {
    __shared__ double w_sum[8], w_top[8], s_b[4], s_m[4];
    __shared__ int w_pieces[8];
    pdl_trigger();
    pdl_wait();
    const int h = blockIdx.x, seq = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int len = q_len[seq], start = q_start[seq], pieces = len > 0 ? (len + kChunk - 1) / kChunk : 0;
    int before_it = 0;                                  // chunks of the requests before this one
    for (int s = tid; s < seq; s += 256) before_it += max(0, q_len[s] + kChunk - 1) / kChunk;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before_it += __shfl_xor_sync(0xffffffffu, before_it, o);
    if (lane == 0) w_pieces[warp] = before_it;
    __syncthreads();
    int base = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) base += w_pieces[w];
    if (h == 0 && gridDim.y > 1) {
        if (tid == 0) p.base[seq] = base;
        for (int c = tid; c < pieces && base + c < p.records; c += 256) p.where[base + c] = make_int2(seq, c * kChunk);
        if (seq == static_cast<int>(gridDim.y) - 1)
            for (int c = base + pieces + tid; c < p.records; c += 256) p.where[c] = make_int2(-1, 0);
    }
    if (len <= 0) return;
    float* const m_g = p.state + static_cast<size_t>(p.state_slot[seq]) * p.state_stride + p.m_off + h;
    const float bi = p.bias_i[h], bf = p.bias_f[h];
    double m_in = *m_g;
    float zi = 0.f, zf = 0.f;
    auto fetch = [&](int t) {
        if (t >= len) return;
        const size_t row = static_cast<size_t>(start + t) * p.ld;
        zi = p.gates[row + h];
        zf = p.gates[row + H + h];
    };
    fetch(tid);
    for (int t0 = 0; t0 < len; t0 += 256) {
        const bool live = t0 + tid < len;
        const float li = live ? p.cap * tanhf((zi + bi) / p.cap) : -INFINITY;
        const float lf = live ? log_sigmoid_f(p.cap * tanhf((zf + bf) / p.cap)) : 0.f;      // a token past the end leaves m as it is
        fetch(t0 + 256 + tid);
        double sum = lf, top = li;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double s = __shfl_up_sync(0xffffffffu, sum, o), b = __shfl_up_sync(0xffffffffu, top, o);
            if (lane >= o) {
                top = fmax(b + sum, top);
                sum += s;
            }
        }
        if (lane == 31) { w_sum[warp] = sum; w_top[warp] = top; }
        __syncthreads();
        double b = sum;                                 // inside the chunk
        if (warp & 1) b += w_sum[warp - 1];
        double m_before = m_in, m_end = m_in;           // before this warp's tokens, behind the last of the 256
        for (int w = 0; w < 8; ++w) {
            m_end = fmax(m_end + w_sum[w], w_top[w]);
            if (w < warp) m_before = m_end;
        }
        const double m = fmax(m_before + sum, top);
        const int c = warp >> 1;                        // this thread's chunk of the four
        // the chunk's end is its last token, or the portion's; both hold b and m of it (tokens past the end add nothing)
        if ((warp & 1) && lane == 31) { s_b[c] = b; s_m[c] = m; }
        __syncthreads();
        const double m_start = c ? s_m[c - 1] : m_in, b_end = s_b[c], m_last = s_m[c];
        const int piece = t0 / kChunk + c;
        if (piece < pieces && base + piece < p.records) {
            LstmChunk& r = p.chunks[static_cast<size_t>(base + piece) * H + h];
            const int i = tid & (kChunk - 1);
            const float hi = static_cast<float>(b);
            r.b_hi[i] = hi;
            r.b_lo[i] = static_cast<float>(b - hi);
            r.li[i] = live ? li : 0.f;
            r.m[i] = static_cast<float>(m);
            r.carry[i] = live ? expf(static_cast<float>(b + m_start - m)) : 0.f;
            r.take[i] = live ? expf(static_cast<float>(b_end - b + li - m_last)) : 0.f;
            if (i == 0) r.decay = expf(static_cast<float>(b_end + m_start - m_last));
        }
        m_in = m_end;
        __syncthreads();
    }
    if (tid == 0) *m_g = static_cast<float>(m_in);
}

// Eight neighbouring values of a row of the projection.
__device__ __forceinline__ void unpack8(const uint4& r, float* v) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(h[i]);
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
}
__device__ __forceinline__ const uint4* row8(const void* base, size_t at) {
    return reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(base) + at);
}

// The values of a chunk [kChunk][COLS] from column col0 on into shared memory, zeros beyond the head; rows from nt on are left out.
template <int COLS, int RULE>
__device__ __forceinline__ void stage_values(const ChunkArgs& p, float* vs, size_t row0, int nt, int h, int col0) {
    if (p.vec) {
        constexpr int PACKS = kChunk * COLS / 8 / kChunkThreads;        // packs a thread
        uint4 raw[PACKS];
#pragma unroll
        for (int n = 0; n < PACKS; ++n) {
            const int idx = n * kChunkThreads + threadIdx.x, j = idx / (COLS / 8), c = (idx % (COLS / 8)) * 8;
            raw[n] = j < nt && col0 + c < p.DV ? *row8(p.v, (row0 + j) * p.ld + h * p.DV + col0 + c) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int n = 0; n < PACKS; ++n) {
            const int idx = n * kChunkThreads + threadIdx.x, j = idx / (COLS / 8), c = (idx % (COLS / 8)) * 8;
            float v[8];
            unpack8(raw[n], v);
            if (RULE == kConstantDecay) {
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = silu_quick(v[e]);
            }
            float4* dst = reinterpret_cast<float4*>(vs + j * COLS + c);
            dst[0] = make_float4(v[0], v[1], v[2], v[3]);
            dst[1] = make_float4(v[4], v[5], v[6], v[7]);
        }
        return;
    }
    for (int idx = threadIdx.x; idx < nt * COLS; idx += kChunkThreads) {
        const int j = idx / COLS, c = idx - j * COLS;
        float v = 0.f;
        if (col0 + c < p.DV) {
            v = load_any(p.v, (row0 + j) * p.ld + h * p.DV + col0 + c, p.in_bf16);
            if (RULE == kConstantDecay) v = silu_f(v);
        }
        vs[idx] = v;
    }
}

// Which request's chunk z is, and its first token there; false: none. (The matrix LSTM's table is written by the kernel before.)
template <int RULE>
__device__ __forceinline__ bool locate_chunk(const ChunkArgs& p, int z, int& seq, int& first) {
    if (RULE == kLstm && p.where) {
        pdl_wait();
        const int2 at = p.where[z];
        seq = at.x;
        first = at.y;
        return seq >= 0;
    }
    seq = z / p.max_pieces;
    first = (z % p.max_pieces) * kChunk;
    return true;
}

// piece_s[z, h] = sum_j (k_j G / g_j) v_j^T, piece_p[z, h] = G. DP: D padded. Grid (tiles of kSumCols columns, heads, chunks).
template <int DP, int RULE>
__global__ void __launch_bounds__(kChunkThreads)
chunk_sum_kernel(const ChunkArgs p) {
    constexpr int PASS_ROWS = DP < 128 ? DP : 128, R = PASS_ROWS / 16;      // rows of S a half warp holds at a time
    extern __shared__ __align__(16) float smem[];
    float* ks = smem;                       // [kChunk][DP]
    float* vs = smem + kChunk * DP;         // [kChunk][kSumCols]
    pdl_trigger();
    const int z = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * kSumCols;
    int seq, first;
    if (!locate_chunk<RULE>(p, z, seq, first)) return;
    const int nt = min(p.q_len[seq] - first, kChunk);
    if (nt <= 0) return;
    if (RULE != kLstm || !p.where) pdl_wait();
    const int D = p.D, DV = p.DV, HD = p.H * D;
    const size_t row0 = static_cast<size_t>(p.q_start[seq] + first);
    const float* powers = RULE == kConstantDecay ? p.powers + h * (kChunk + 1) : nullptr;
    const float* cum = RULE == kChannelDecay ? p.cum + row0 * HD + h * D : nullptr;
    const LstmChunk* lstm = RULE == kLstm ? p.lstm + static_cast<size_t>(z) * p.H + h : nullptr;
    if (p.vec) {
        constexpr int PACKS = kChunk * DP / 8 / kChunkThreads > 0 ? kChunk * DP / 8 / kChunkThreads : 1;
        uint4 raw[PACKS];
#pragma unroll
        for (int n = 0; n < PACKS; ++n) {
            const int idx = n * kChunkThreads + threadIdx.x, j = idx / (DP / 8), d = (idx % (DP / 8)) * 8;
            raw[n] = j < nt && d < D ? *row8(p.k, (row0 + j) * p.ld + h * D + d) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int n = 0; n < PACKS; ++n) {
            const int idx = n * kChunkThreads + threadIdx.x, j = idx / (DP / 8), d = (idx % (DP / 8)) * 8;
            float k[8];
            unpack8(raw[n], k);
            if (RULE == kConstantDecay) {
                const float f = j < nt ? powers[nt - 1 - j] : 0.f;
#pragma unroll
                for (int e = 0; e < 8; ++e) k[e] = silu_quick(k[e]) * f;
            } else if (RULE == kLstm) {
                const float f = j < kChunk ? lstm->take[j] : 0.f;
#pragma unroll
                for (int e = 0; e < 8; ++e) k[e] *= f;
            } else if (j < nt && d < D) {
                const float4* end = reinterpret_cast<const float4*>(cum + static_cast<size_t>(nt - 1) * HD + d);
                const float4* own = reinterpret_cast<const float4*>(cum + static_cast<size_t>(j) * HD + d);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float4 a = end[u], b = own[u];
                    k[4 * u] *= expf(a.x - b.x);
                    k[4 * u + 1] *= expf(a.y - b.y);
                    k[4 * u + 2] *= expf(a.z - b.z);
                    k[4 * u + 3] *= expf(a.w - b.w);
                }
            }
            if (j < kChunk) {
                float4* dst = reinterpret_cast<float4*>(ks + j * DP + d);
                dst[0] = make_float4(k[0], k[1], k[2], k[3]);
                dst[1] = make_float4(k[4], k[5], k[6], k[7]);
            }
        }
    } else {
        for (int idx = threadIdx.x; idx < nt * DP; idx += kChunkThreads) {
            const int j = idx / DP, d = idx - j * DP;
            float k = 0.f;
            if (d < D) {
                k = load_any(p.k, (row0 + j) * p.ld + h * D + d, p.in_bf16);
                k = RULE == kConstantDecay ? silu_f(k) * powers[nt - 1 - j]
                    : RULE == kLstm        ? k * lstm->take[j]
                                           : k * expf(cum[static_cast<size_t>(nt - 1) * HD + d] - cum[static_cast<size_t>(j) * HD + d]);
            }
            ks[idx] = k;
        }
    }
    stage_values<kSumCols, RULE>(p, vs, row0, nt, h, col0);
    if (blockIdx.x == 0)
        for (int d = threadIdx.x; d < D; d += kChunkThreads)
            p.piece_p[(static_cast<size_t>(z) * p.H + h) * D + d] =
                RULE == kConstantDecay ? powers[nt] : RULE == kLstm ? lstm->decay : expf(cum[static_cast<size_t>(nt - 1) * HD + d]);
    __syncthreads();
    if (RULE == kLstm && blockIdx.x == 0) {         // the chunk's own share of n: the weighted keys without values
        for (int d = threadIdx.x; d < D; d += kChunkThreads) {
            float n4[4] = {0.f, 0.f, 0.f, 0.f};
            int j = 0;
            for (; j + 4 <= nt; j += 4) {
#pragma unroll
                for (int e = 0; e < 4; ++e) n4[e] += ks[(j + e) * DP + d];
            }
            for (; j < nt; ++j) n4[0] += ks[j * DP + d];
            p.piece_n[(static_cast<size_t>(z) * p.H + h) * D + d] = (n4[0] + n4[1]) + (n4[2] + n4[3]);
        }
    }
    const int warp = threadIdx.x >> 5, cg = (threadIdx.x & 15) * 4, half = (threadIdx.x >> 4) & 1;
    float* out = p.piece_s + (static_cast<size_t>(z) * p.H + h) * D * DV;
    for (int pass = 0; pass < DP / PASS_ROWS; ++pass) {
        const int r0 = pass * PASS_ROWS + (2 * warp + half) * R;
        float acc[R][4];
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
#pragma unroll 4
        for (int j = 0; j < nt; ++j) {
            const float4 b = *reinterpret_cast<const float4*>(vs + j * kSumCols + cg);
            float a[R];
            if constexpr (R >= 4) {
#pragma unroll
                for (int r = 0; r < R; r += 4) {
                    const float4 a4 = *reinterpret_cast<const float4*>(ks + j * DP + r0 + r);
                    a[r] = a4.x; a[r + 1] = a4.y; a[r + 2] = a4.z; a[r + 3] = a4.w;
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) a[r] = ks[j * DP + r0 + r];
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                acc[r][0] = fmaf(a[r], b.x, acc[r][0]);
                acc[r][1] = fmaf(a[r], b.y, acc[r][1]);
                acc[r][2] = fmaf(a[r], b.z, acc[r][2]);
                acc[r][3] = fmaf(a[r], b.w, acc[r][3]);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (r0 + r >= D) continue;
            float* dst = out + static_cast<size_t>(r0 + r) * DV + col0 + cg;
            if (DV % 4 == 0) {
                if (col0 + cg < DV) *reinterpret_cast<float4*>(dst) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (col0 + cg + e < DV) dst[e] = acc[r][e];
            }
        }
    }
}

// Between the two: piece_s becomes the memory at every chunk's start, the state the memory after the last one. As
// pieces_combine_kernel, with four neighbouring columns a thread.
static __global__ void __launch_bounds__(256)
chunk_combine_kernel(float4* __restrict__ piece_s, const float* __restrict__ piece_p, float* __restrict__ state, long long state_stride,
                     const int32_t* __restrict__ q_len, const int32_t* __restrict__ state_slot, int H, int D, int DV, int max_pieces,
                     const int32_t* __restrict__ base) {
    pdl_trigger();
    const int seq = blockIdx.y;
    const int len = q_len[seq];
    const int entry = blockIdx.x * blockDim.x + threadIdx.x, entries = H * D * DV / 4;
    if (len <= 0 || entry >= entries) return;
    pdl_wait();
    const int row = entry * 4 / DV;                                      // h * D + i
    float4* S_g = reinterpret_cast<float4*>(state + static_cast<size_t>(state_slot[seq]) * state_stride) + entry;
    float4 S = *S_g;
    const int pieces = (len + kChunk - 1) / kChunk;
    const size_t z0 = base ? static_cast<size_t>(base[seq]) : static_cast<size_t>(seq) * max_pieces;
    constexpr int AHEAD = 8;        // chunks whose loads are in flight together
    for (int c0 = 0; c0 < pieces; c0 += AHEAD) {
        float4 own[AHEAD];
        float decay[AHEAD];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
            if (c0 + u < pieces) {
                const size_t z = z0 + c0 + u;
                own[u] = piece_s[z * entries + entry];
                decay[u] = piece_p[z * H * D + row];
            }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
            if (c0 + u < pieces) {
                piece_s[(z0 + c0 + u) * entries + entry] = S;
                S.x = fmaf(decay[u], S.x, own[u].x);
                S.y = fmaf(decay[u], S.y, own[u].y);
                S.z = fmaf(decay[u], S.z, own[u].z);
                S.w = fmaf(decay[u], S.w, own[u].w);
            }
    }
    *S_g = S;
}

// Outputs of a chunk from the memory at its start (piece_s by now). Grid (tiles of kChunkCols columns, heads, chunks).
template <int DP>
__host__ __device__ constexpr int chunk_second_floats() { return DP * kLd > kChunk * kChunkCols ? DP * kLd : kChunk * kChunkCols; }
template <int DP>
__host__ __device__ constexpr int chunk_out_floats() { return DP * kLd + chunk_second_floats<DP>() + kChunk * kLd; }

template <int DP, int RULE>
__global__ void __launch_bounds__(kChunkThreads, DP <= 128 ? 2 : 1)
chunk_out_kernel(const ChunkArgs p) {
    constexpr int SLAB = RULE == kLstm ? 32 : 64 < DP ? 64 : DP;        // rows of S staged at a time (the runs' sums take registers)
    constexpr int SLAB_PACKS = SLAB * kChunkCols / 4 / kChunkThreads;
    extern __shared__ __align__(16) float smem[];
    float* qT = smem;                               // [DP][kLd]: column i is token i's query (times g_i)
    float* kT = qT + DP * kLd;                      // [DP][kLd]; later slabs of S [SLAB][kChunkCols], then the values [kChunk][kChunkCols]
    float* aT = kT + chunk_second_floats<DP>();     // [kChunk j][kLd i]: scores
    pdl_trigger();
    const int z = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * kChunkCols;
    int seq, first;
    if (!locate_chunk<RULE>(p, z, seq, first)) return;
    const int nt = min(p.q_len[seq] - first, kChunk);
    if (nt <= 0) return;
    if (RULE != kLstm || !p.where) pdl_wait();
    const int D = p.D, DV = p.DV, HD = p.H * D;
    const size_t row0 = static_cast<size_t>(p.q_start[seq] + first);
    const float* powers = RULE == kConstantDecay ? p.powers + h * (kChunk + 1) : nullptr;
    const float* cum = RULE == kChannelDecay ? p.cum + row0 * HD + h * D : nullptr;
    const LstmChunk* lstm = RULE == kLstm ? p.lstm + static_cast<size_t>(z) * p.H + h : nullptr;
    __shared__ float den_s[RULE == kLstm ? 4 : 1][RULE == kLstm ? kChunk : 1];
    bool safe = true;
    if (RULE == kChannelDecay) {
        int low = 0;
        for (int d = threadIdx.x; d < D; d += kChunkThreads) low |= !(cum[static_cast<size_t>(nt - 1) * HD + d] >= kSafeLog);     // (no number: the tokens before it may lie low)
        safe = !__syncthreads_or(low);
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (p.vec) {
        // a warp takes packs of 8 channels, its lanes 32 neighbouring tokens: the transposed stores hit 32 banks
        constexpr int PACKS = DP / 8 * 2 / 8;       // (pack, half of the tokens) pairs a warp
        uint4 rq[PACKS], rk[PACKS];
#pragma unroll
        for (int n = 0; n < PACKS; ++n) {
            const int item = n * 8 + warp, d = (item >> 1) * 8, i = (item & 1) * 32 + lane;
            const bool ok = i < nt && d < D;
            const size_t at = (row0 + i) * p.ld + h * D + d;
            rq[n] = ok ? *row8(p.q, at) : make_uint4(0, 0, 0, 0);
            rk[n] = ok ? *row8(p.k, at) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int n = 0; n < PACKS; ++n) {
            const int item = n * 8 + warp, d = (item >> 1) * 8, i = (item & 1) * 32 + lane;
            float q[8], k[8];
            unpack8(rq[n], q);
            unpack8(rk[n], k);
            if (RULE == kConstantDecay) {
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    q[e] = silu_quick(q[e]);
                    k[e] = silu_quick(k[e]);
                }
            } else if (RULE == kLstm) {
#pragma unroll
                for (int e = 0; e < 8; ++e) q[e] *= p.q_scale;
            } else if (i < nt && d < D) {
                const float4* own = reinterpret_cast<const float4*>(cum + static_cast<size_t>(i) * HD + d);
                const float4 c0 = own[0], c1 = own[1];
                const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    q[e] *= safe ? p.q_scale * expf(c[e]) : p.q_scale;
                    if (safe) k[e] *= expf(-c[e]);
                }
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                qT[(d + e) * kLd + i] = q[e];
                kT[(d + e) * kLd + i] = k[e];
            }
        }
    } else {
        // lanes of a warp: 8 neighbouring channels of 4 neighbouring tokens
        for (int idx = threadIdx.x; idx < kChunk * DP; idx += kChunkThreads) {
            const int sub = idx & 31, blk = idx >> 5;
            const int d = (blk % (DP / 8)) * 8 + (sub & 7), i = (blk / (DP / 8)) * 4 + (sub >> 3);
            float q = 0.f, k = 0.f;
            if (d < D && i < nt) {
                const size_t at = (row0 + i) * p.ld + h * D + d;
                q = load_any(p.q, at, p.in_bf16);
                k = load_any(p.k, at, p.in_bf16);
                if (RULE == kConstantDecay) {
                    q = silu_f(q);
                    k = silu_f(k);
                } else {
                    q *= p.q_scale;
                    if (RULE == kChannelDecay && safe) {
                        const float c = cum[static_cast<size_t>(i) * HD + d];
                        q *= expf(c);
                        k *= expf(-c);
                    }
                }
            }
            qT[d * kLd + i] = q;
            kT[d * kLd + i] = k;
        }
    }
    // the first rows of S travel while the scores are worked out
    const float* S = p.piece_s + (static_cast<size_t>(z) * p.H + h) * D * DV;
    const bool s_vec = DV % 4 == 0;
    float4 ahead[SLAB_PACKS];
    auto fetch_slab = [&](int d0) {
#pragma unroll
        for (int n = 0; n < SLAB_PACKS; ++n) {
            const int idx = n * kChunkThreads + threadIdx.x, d = d0 + idx / (kChunkCols / 4), c = col0 + (idx % (kChunkCols / 4)) * 4;
            ahead[n] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (d < D && c < DV) {
                const float* at = S + static_cast<size_t>(d) * DV + c;
                if (s_vec) {
                    ahead[n] = *reinterpret_cast<const float4*>(at);
                } else {
                    ahead[n].x = at[0];
                    if (c + 1 < DV) ahead[n].y = at[1];
                    if (c + 2 < DV) ahead[n].z = at[2];
                    if (c + 3 < DV) ahead[n].w = at[3];
                }
            }
        }
    };
    fetch_slab(0);
    __syncthreads();
    {   // scores: thread (ty, tx) tokens i = 4 ty .. + 3 against j = 4 tx .. + 3
        const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
        float a[4][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) a[e][0] = a[e][1] = a[e][2] = a[e][3] = 0.f;
        if (RULE != kChannelDecay || safe) {
            if (tx <= ty) {
                float run[4][4] = {};
#pragma unroll 8
                for (int d = 0; d < DP; ++d) {
                    const float4 q4 = *reinterpret_cast<const float4*>(qT + d * kLd + 4 * ty);
                    const float4 k4 = *reinterpret_cast<const float4*>(kT + d * kLd + 4 * tx);
                    const float qv[4] = {q4.x, q4.y, q4.z, q4.w}, kv[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e)
#pragma unroll
                        for (int f = 0; f < 4; ++f) {
                            float& to = RULE == kLstm ? run[e][f] : a[e][f];
                            to = fmaf(qv[e], kv[f], to);
                        }
                    if (RULE == kLstm && d % kRun == kRun - 1) {
#pragma unroll
                        for (int e = 0; e < 4; ++e)
#pragma unroll
                            for (int f = 0; f < 4; ++f) {
                                a[e][f] += run[e][f];
                                run[e][f] = 0.f;
                            }
                    }
                }
            }
        } else if (tx <= ty) {
            for (int d = 0; d < D; ++d) {
                float ci[4], cj[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    ci[e] = 4 * ty + e < nt ? cum[static_cast<size_t>(4 * ty + e) * HD + d] : 0.f;
                    cj[e] = 4 * tx + e < nt ? cum[static_cast<size_t>(4 * tx + e) * HD + d] : 0.f;
                }
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int f = 0; f < 4; ++f)
                        if (4 * tx + f <= 4 * ty + e) a[e][f] = fmaf(qT[d * kLd + 4 * ty + e] * expf(ci[e] - cj[f]), kT[d * kLd + 4 * tx + f], a[e][f]);
            }
        }
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            float w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int n = 4 * ty + e - (4 * tx + f);
                if (RULE == kLstm) {
                    const int i = 4 * ty + e, j = 4 * tx + f;
                    w[e] = n < 0 || i >= nt ? 0.f : a[e][f] * expf((lstm->b_hi[i] - lstm->b_hi[j]) + (lstm->b_lo[i] - lstm->b_lo[j]) + (lstm->li[j] - lstm->m[i]));
                    continue;
                }
                w[e] = n < 0 ? 0.f : RULE == kConstantDecay ? a[e][f] * powers[n] : a[e][f];
            }
            *reinterpret_cast<float4*>(aT + (4 * tx + f) * kLd + 4 * ty) = make_float4(w[0], w[1], w[2], w[3]);
        }
    }
    __syncthreads();
    if (RULE == kChannelDecay && !safe) {
        for (int idx = threadIdx.x; idx < kChunk * DP; idx += kChunkThreads) {
            const int i = idx % kChunk, d = idx / kChunk;
            if (d < D && i < nt) qT[d * kLd + i] *= expf(cum[static_cast<size_t>(i) * HD + d]);
        }
    }
    if (RULE == kLstm) {            // n . q of every token, a quarter of its terms a thread
        const int i = threadIdx.x & (kChunk - 1), part = threadIdx.x / kChunk;
        const float* n = p.piece_n + (static_cast<size_t>(z) * p.H + h) * D;
        float own[2] = {0.f, 0.f}, past[2] = {0.f, 0.f};
        for (int j = part * (kChunk / 4); j < (part + 1) * (kChunk / 4); j += 2) {
            own[0] += aT[j * kLd + i];
            own[1] += aT[(j + 1) * kLd + i];
        }
        for (int d = part * (DP / 4); d < min(D, (part + 1) * (DP / 4)); d += 2) {
            past[0] = fmaf(qT[d * kLd + i], n[d], past[0]);
            if (d + 1 < D) past[1] = fmaf(qT[(d + 1) * kLd + i], n[d + 1], past[1]);
        }
        den_s[part][i] = (own[0] + own[1]) + lstm->carry[i] * (past[0] + past[1]);
    }
    // outputs: warp w tokens 8 w .. + 7, lane columns 4 lane .. + 3
    float acc[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
    auto step = [&](const float* a_row, const float* b_row, int from = 0) {     // the warp's tokens from ``from`` on
        const float4 lo = *reinterpret_cast<const float4*>(a_row), hi = *reinterpret_cast<const float4*>(a_row + 4);
        const float4 b = *reinterpret_cast<const float4*>(b_row);
        const float a[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            if (r < from) continue;
            acc[r][0] = fmaf(a[r], b.x, acc[r][0]);
            acc[r][1] = fmaf(a[r], b.y, acc[r][1]);
            acc[r][2] = fmaf(a[r], b.z, acc[r][2]);
            acc[r][3] = fmaf(a[r], b.w, acc[r][3]);
        }
    };
    float sum[8][4] = {};                           // matrix LSTM: the sums of the runs
    auto end_run = [&] {
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                sum[r][e] += acc[r][e];
                acc[r][e] = 0.f;
            }
    };
    for (int d0 = 0; d0 < DP && d0 < D; d0 += SLAB) {
#pragma unroll
        for (int n = 0; n < SLAB_PACKS; ++n) *reinterpret_cast<float4*>(kT + (n * kChunkThreads + threadIdx.x) * 4) = ahead[n];
        __syncthreads();
        if (d0 + SLAB < D) fetch_slab(d0 + SLAB);
        if constexpr (RULE == kLstm) {
            for (int d1 = 0; d1 < SLAB; d1 += kRun) {
#pragma unroll 4
                for (int d = d1; d < d1 + kRun; ++d) step(qT + (d0 + d) * kLd + 8 * warp, kT + d * kChunkCols + 4 * lane);
                end_run();
            }
        } else {
#pragma unroll 4
            for (int d = 0; d < SLAB; ++d) step(qT + (d0 + d) * kLd + 8 * warp, kT + d * kChunkCols + 4 * lane);
        }
        __syncthreads();
    }
    if (RULE == kConstantDecay) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float f = powers[8 * warp + r + 1];
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[r][e] *= f;
        }
    }
    if (RULE == kLstm) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float f = lstm->carry[8 * warp + r];
#pragma unroll
            for (int e = 0; e < 4; ++e) sum[r][e] *= f;
        }
    }
    stage_values<kChunkCols, RULE>(p, kT, row0, nt, h, col0);
    __syncthreads();
    // Tokens before this warp's eight, then the eight themselves: a later one of those has no weight in an earlier one's row and stays out of
    // it (0 times a value that is no number would be none).
    const int own = 8 * warp;
    if constexpr (RULE == kLstm) {
        for (int j0 = 0; j0 < own && j0 < nt; j0 += kRun) {
#pragma unroll 4
            for (int j = j0; j < min(min(nt, own), j0 + kRun); ++j) step(aT + j * kLd + own, kT + j * kChunkCols + 4 * lane);
            if (j0 + kRun <= own) end_run();        // (the run of 16 that the warp's own tokens begin in goes on below)
        }
    } else {
#pragma unroll 4
        for (int j = 0; j < min(nt, own); ++j) step(aT + j * kLd + own, kT + j * kChunkCols + 4 * lane);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
        if (own + u < nt) step(aT + (own + u) * kLd + own, kT + (own + u) * kChunkCols + 4 * lane, u);
    if constexpr (RULE == kLstm) end_run();
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int i = 8 * warp + r;
        if (i >= nt) break;
        if (RULE == kLstm) {
            const float dot = (den_s[0][i] + den_s[1][i]) + (den_s[2][i] + den_s[3][i]);
            const float f = 1.f / (fmaxf(fabsf(dot), expf(-lstm->m[i])) + 1e-6f);
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[r][e] = sum[r][e] * f;
        }
        float* dst = p.o + ((row0 + i) * p.H + h) * DV + col0 + 4 * lane;
        if (s_vec) {
            if (col0 + 4 * lane < DV) *reinterpret_cast<float4*>(dst) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (col0 + 4 * lane + e < DV) dst[e] = acc[r][e];
        }
    }
}

// A single token of every request: one pass over S, which is all there is to do. A warp reads whole rows of up to 128 columns, the
// eight warps of a CTA take every eighth row; their shares of S^T q meet in shared memory. Grid (tiles of 128 columns, heads, requests).
template <int RULE>
__global__ void __launch_bounds__(kChunkThreads)
decay_step_kernel(const ScanArgs p) {
    __shared__ float s_q[256], s_k[256], s_w[256];
    __shared__ __align__(16) float red[8][kChunkCols];
    pdl_trigger();
    const int seq = blockIdx.z, h = blockIdx.y, col = blockIdx.x * kChunkCols + 4 * (threadIdx.x & 31);
    if (p.q_len[seq] <= 0) return;
    pdl_wait();
    const int D = p.D, DV = p.DV, warp = threadIdx.x >> 5;
    const size_t row = static_cast<size_t>(p.q_start[seq]);
    float* S_g = p.state + static_cast<size_t>(p.state_slot[seq]) * p.state_stride + static_cast<size_t>(h) * D * DV + col;
    constexpr int AHEAD = 16;
    float4 S[AHEAD];
    const bool live = col < DV;
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
        if (live && warp + 8 * u < D) S[u] = *reinterpret_cast<const float4*>(S_g + static_cast<size_t>(warp + 8 * u) * DV);
    const int d = threadIdx.x;
    if (d < D) {
        const size_t at = row * p.lda + h * D + d;
        const float q = load_any(p.a, at, p.in_bf16), k = load_any(p.k, at, p.in_bf16);
        s_q[d] = RULE == kConstantDecay ? silu_f(q) : q * p.q_scale;
        s_k[d] = RULE == kConstantDecay ? silu_f(k) : k;
        s_w[d] = RULE == kConstantDecay ? p.fade[h] : expm1f(log_sigmoid_f(p.w[row * p.H * D + h * D + d] + p.w0[h * D + d]) * p.inv_tau);
    }
    float v[4] = {0.f, 0.f, 0.f, 0.f}, acc[4] = {0.f, 0.f, 0.f, 0.f};
    if (live) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            v[e] = load_any(p.v, row * p.ldv + h * DV + col + e, p.in_bf16);
            if (RULE == kConstantDecay) v[e] = silu_f(v[e]);
        }
    }
    __syncthreads();
    for (int d0 = 0; d0 < D; d0 += 8 * AHEAD) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const int i = d0 + warp + 8 * u;
            if (live && i < D) {
                const float w = s_w[i], k = s_k[i], q = s_q[i];
                float x[4] = {S[u].x, S[u].y, S[u].z, S[u].w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    x[e] = fmaf(k, v[e], fmaf(w, x[e], x[e]));
                    acc[e] = fmaf(q, x[e], acc[e]);
                }
                *reinterpret_cast<float4*>(S_g + static_cast<size_t>(i) * DV) = make_float4(x[0], x[1], x[2], x[3]);
            }
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const int i = d0 + 8 * AHEAD + warp + 8 * u;
            if (live && i < D) S[u] = *reinterpret_cast<const float4*>(S_g + static_cast<size_t>(i) * DV);
        }
    }
    *reinterpret_cast<float4*>(&red[warp][4 * (threadIdx.x & 31)]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    __syncthreads();
    if (threadIdx.x < kChunkCols && blockIdx.x * kChunkCols + threadIdx.x < DV) {
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) sum += red[w][threadIdx.x];
        p.o[(row * p.H + h) * DV + blockIdx.x * kChunkCols + threadIdx.x] = sum;
    }
}

template <typename... A>
cudaError_t more_shared_memory(void (*kernel)(A...), int bytes) {
    return bytes > 48 * 1024 ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) : cudaSuccess;
}

template <int DP, int RULE>
int launch_chunks(const ChunkArgs& p, float* state, long long state_stride, const int32_t* state_slot, int num_seqs, cudaStream_t stream) {
    const int zs = RULE == kLstm ? p.records : num_seqs * p.max_pieces;
    const dim3 grid((p.DV + kChunkCols - 1) / kChunkCols, p.H, zs), block(kChunkThreads);
    const dim3 sum_grid((p.DV + kSumCols - 1) / kSumCols, p.H, zs);
    constexpr int sum_bytes = (kChunk * DP + kChunk * kSumCols) * 4, out_bytes = chunk_out_floats<DP>() * 4;
    cudaError_t e = more_shared_memory(chunk_sum_kernel<DP, RULE>, sum_bytes);
    if (e == cudaSuccess) e = more_shared_memory(chunk_out_kernel<DP, RULE>, out_bytes);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (RULE == kChannelDecay) stride::launch(chunk_decay_kernel, dim3((p.H * p.D + 127) / 128, zs), dim3(128), 0, stream, p);
    stride::launch(chunk_sum_kernel<DP, RULE>, sum_grid, block, sum_bytes, stream, p);
    if (p.DV % 4 == 0 && state_stride % 4 == 0 && reinterpret_cast<uintptr_t>(state) % 16 == 0)
        stride::launch(chunk_combine_kernel, dim3((p.H * p.D * p.DV / 4 + 255) / 256, num_seqs), dim3(256), 0, stream,
                       reinterpret_cast<float4*>(p.piece_s), static_cast<const float*>(p.piece_p), state, state_stride, p.q_len, state_slot, p.H,
                       p.D, p.DV, p.max_pieces, p.base);
    else
        stride::launch(pieces_combine_kernel, dim3((p.H * p.D * p.DV + 255) / 256, num_seqs), dim3(256), 0, stream, p.piece_s,
                       static_cast<const float*>(p.piece_p), state, state_stride, p.q_len, state_slot, p.H, p.D, p.DV, kChunk, p.max_pieces, p.base);
    if (RULE == kLstm)      // n is one more column of the memory
        stride::launch(pieces_combine_kernel, dim3((p.H * p.D + 255) / 256, num_seqs), dim3(256), 0, stream, p.piece_n,
                       static_cast<const float*>(p.piece_p), state + static_cast<size_t>(p.H) * p.D * p.DV, state_stride, p.q_len, state_slot, p.H,
                       p.D, 1, kChunk, p.max_pieces, p.base);
    stride::launch(chunk_out_kernel<DP, RULE>, grid, block, out_bytes, stream, p);
    return STRIDE_LAUNCH_STATUS();
}

template <int RULE>
int dispatch_chunks(const ChunkArgs& p, float* state, long long state_stride, const int32_t* state_slot, int num_seqs, cudaStream_t stream) {
    if (p.D <= 32) return launch_chunks<32, RULE>(p, state, state_stride, state_slot, num_seqs, stream);
    if (p.D <= 64) return launch_chunks<64, RULE>(p, state, state_stride, state_slot, num_seqs, stream);
    if (p.D <= 128) return launch_chunks<128, RULE>(p, state, state_stride, state_slot, num_seqs, stream);
    if (p.D <= 256) return launch_chunks<256, RULE>(p, state, state_stride, state_slot, num_seqs, stream);
    return STRIDE_UNSUPPORTED;
}

inline ScanArgs decay_args(const void* q, const void* k, const void* v, int ld, const float* logit, const float* bias, const float* fade,
                           float q_scale, float inv_tau, float* o, float* state, long long state_stride, const int32_t* q_start,
                           const int32_t* q_len, const int32_t* state_slot, int H, int D, int DV, int dtype) {
    ScanArgs p = {};
    p.a = q;
    p.k = k;
    p.v = v;
    p.lda = p.ldv = ld;
    p.w = logit;
    p.w0 = bias;
    p.fade = fade;
    p.q_scale = q_scale;
    p.inv_tau = inv_tau;
    p.o = o;
    p.state = state;
    p.state_stride = state_stride;
    p.q_start = q_start;
    p.q_len = q_len;
    p.state_slot = state_slot;
    p.H = H;
    p.group = 1;
    p.D = D;
    p.DV = DV;
    p.in_bf16 = dtype == STRIDE_DTYPE_BF16 ? 1 : 0;
    return p;
}

}  // namespace stride

using namespace stride;

extern "C" {

// One token after the other. q, k [tokens, ld] with head h at column h * D, v with head h at column h * DV, all in the compute
// type. fade (constant decay): [H] float32, the decay minus one; null: channel decays from logit [tokens, H * D] and bias
// [H * D], float32. o [tokens, H * DV] float32; state: S of head h at h * D * DV floats into a slot's row.
int stride_decay_scan(const void* q, const void* k, const void* v, int ld, const float* logit, const float* bias, const float* fade,
                      float q_scale, float inv_tau, float* o, float* state, long long state_stride, const int32_t* q_start,
                      const int32_t* q_len, const int32_t* state_slot, int num_seqs, int H, int D, int DV, int dtype, cudaStream_t stream) {
    if (num_seqs < 0 || H <= 0 || D <= 0 || DV <= 0 || (!fade && (!logit || !bias))) return STRIDE_BAD_ARGUMENT;
    if (state_stride < static_cast<long long>(H) * D * DV) return STRIDE_BAD_ARGUMENT;
    if (dtype != STRIDE_DTYPE_F32 && dtype != STRIDE_DTYPE_BF16) return STRIDE_BAD_ARGUMENT;
    if (num_seqs > 65535 || H > 65535) return STRIDE_UNSUPPORTED;
    if (num_seqs == 0) return 0;
    const ScanArgs p = decay_args(q, k, v, ld, logit, bias, fade, q_scale, inv_tau, o, state, state_stride, q_start, q_len, state_slot, H, D, DV, dtype);
    return fade ? launch_scan<kConstantDecay>(p, num_seqs, stream) : launch_scan<kChannelDecay>(p, num_seqs, stream);
}

// The same for requests that bring exactly one token each (q_len 0: none); returns -2 for what it does not take (values in
// widths that are no multiple of 4, rows off 16-byte boundaries): decay_scan runs everything.
int stride_decay_step(const void* q, const void* k, const void* v, int ld, const float* logit, const float* bias, const float* fade,
                      float q_scale, float inv_tau, float* o, float* state, long long state_stride, const int32_t* q_start,
                      const int32_t* q_len, const int32_t* state_slot, int num_seqs, int H, int D, int DV, int dtype, cudaStream_t stream) {
    if (num_seqs < 0 || H <= 0 || D <= 0 || DV <= 0 || (!fade && (!logit || !bias))) return STRIDE_BAD_ARGUMENT;
    if (state_stride < static_cast<long long>(H) * D * DV) return STRIDE_BAD_ARGUMENT;
    if (dtype != STRIDE_DTYPE_F32 && dtype != STRIDE_DTYPE_BF16) return STRIDE_BAD_ARGUMENT;
    if (num_seqs > 65535 || H > 65535 || D > 256 || DV % 4 || state_stride % 4 || reinterpret_cast<uintptr_t>(state) % 16) return STRIDE_UNSUPPORTED;
    if (num_seqs == 0) return 0;
    ScanArgs p = decay_args(q, k, v, ld, logit, bias, fade, q_scale, inv_tau, o, state, state_stride, q_start, q_len, state_slot, H, D, DV, dtype);
    const dim3 grid((DV + kChunkCols - 1) / kChunkCols, H, num_seqs);
    stride::launch(fade ? decay_step_kernel<kConstantDecay> : decay_step_kernel<kChannelDecay>, grid, dim3(kChunkThreads), 0, stream, p);
    return STRIDE_LAUNCH_STATUS();
}

// Chunk by chunk. powers (constant decay): [H, 65] float32, decay^0 .. decay^64; null: channel decays, whose logits are
// overwritten. scratch: float32, num_seqs * max_pieces * H * D * (DV + 1), max_pieces = ceil(longest portion / 64).
int stride_decay_chunks(const void* q, const void* k, const void* v, int ld, float* logit, const float* bias, const float* powers,
                        float q_scale, float inv_tau, float* o, float* state, long long state_stride, const int32_t* q_start,
                        const int32_t* q_len, const int32_t* state_slot, int num_seqs, int H, int D, int DV, int dtype, int max_pieces,
                        float* scratch, cudaStream_t stream) {
    if (num_seqs < 0 || H <= 0 || D <= 0 || DV <= 0 || max_pieces <= 0 || !scratch || (!powers && (!logit || !bias))) return STRIDE_BAD_ARGUMENT;
    if (state_stride < static_cast<long long>(H) * D * DV) return STRIDE_BAD_ARGUMENT;
    if (dtype != STRIDE_DTYPE_F32 && dtype != STRIDE_DTYPE_BF16) return STRIDE_BAD_ARGUMENT;
    if (static_cast<long long>(num_seqs) * max_pieces > 65535 || H > 65535 || reinterpret_cast<uintptr_t>(scratch) % 16) return STRIDE_UNSUPPORTED;
    if (num_seqs == 0) return 0;
    ChunkArgs p = {};
    p.q = q;
    p.k = k;
    p.v = v;
    p.ld = ld;
    p.in_bf16 = dtype == STRIDE_DTYPE_BF16 ? 1 : 0;
    p.cum = logit;
    p.bias = bias;
    p.powers = powers;
    p.q_scale = q_scale;
    p.inv_tau = inv_tau;
    p.o = o;
    p.piece_s = scratch;
    p.piece_p = scratch + static_cast<size_t>(num_seqs) * max_pieces * H * D * DV;
    p.q_start = q_start;
    p.q_len = q_len;
    p.H = H;
    p.D = D;
    p.DV = DV;
    p.max_pieces = max_pieces;
    auto aligned = [](const void* x) { return reinterpret_cast<uintptr_t>(x) % 16 == 0; };
    p.vec = p.in_bf16 && D % 8 == 0 && DV % 8 == 0 && ld % 8 == 0 && aligned(q) && aligned(k) && aligned(v) && (powers || aligned(logit));
    return powers ? dispatch_chunks<kConstantDecay>(p, state, state_stride, state_slot, num_seqs, stream)
                  : dispatch_chunks<kChannelDecay>(p, state, state_stride, state_slot, num_seqs, stream);
}

// Scratch of stride_mlstm_chunks in floats for `records` chunks in all.
static long long lstm_table_floats(int num_seqs, int records) { return (2LL * records + 3) / 4 * 4 + (num_seqs + 3LL) / 4 * 4; }
long long stride_mlstm_chunks_scratch(int num_seqs, int records, int H, int D, int DV) {
    return static_cast<long long>(records) * H * (static_cast<long long>(D) * (DV + 2) + static_cast<long long>(sizeof(LstmChunk) / 4)) +
           lstm_table_floats(num_seqs, records);
}

// The matrix LSTM (mlstm.cu has the recurrence and the layout of the state) over long portions, chunk by chunk. Arguments as
// stride_mlstm_scan; records: the sum of the requests' chunks (of 64 tokens, the last one broken) at least; scratch: 16-byte aligned. Returns -2 for more than 256 rows a head or too many chunks.
int stride_mlstm_chunks(const void* proj, int ld, int q_off, int k_off, int v_off, const float* gates, int ld_gates, const float* bias_i,
                        const float* bias_f, float cap, float q_scale, float* o, float* state, long long state_stride, const int32_t* q_start,
                        const int32_t* q_len, const int32_t* state_slot, int num_seqs, int H, int D, int DV, int dtype, int records, float* scratch,
                        cudaStream_t stream) {
    if (num_seqs < 0 || H <= 0 || D <= 0 || DV <= 0 || ld <= 0 || ld_gates < 2 * H || !(cap > 0.f) || q_off < 0 || k_off < 0 || v_off < 0 ||
        records <= 0 || !scratch)
        return STRIDE_BAD_ARGUMENT;
    if (dtype != STRIDE_DTYPE_F32 && dtype != STRIDE_DTYPE_BF16) return STRIDE_BAD_ARGUMENT;
    if (state_stride < static_cast<long long>(H) * D * DV + static_cast<long long>(H) * D + H) return STRIDE_BAD_ARGUMENT;
    if (D > 256 || records > 65535 || num_seqs > 65535 || H > 65535 || reinterpret_cast<uintptr_t>(scratch) % 16) return STRIDE_UNSUPPORTED;
    if (num_seqs == 0) return 0;
    const int item = dtype == STRIDE_DTYPE_BF16 ? 2 : 4;
    const size_t rows = static_cast<size_t>(records) * H;
    auto at = [&](int off) { return static_cast<const unsigned char*>(proj) + static_cast<size_t>(off) * item; };
    ChunkArgs p = {};
    p.q = at(q_off);
    p.k = at(k_off);
    p.v = at(v_off);
    p.ld = ld;
    p.in_bf16 = dtype == STRIDE_DTYPE_BF16 ? 1 : 0;
    p.q_scale = q_scale;
    p.o = o;
    LstmChunk* chunks = reinterpret_cast<LstmChunk*>(scratch);
    p.lstm = chunks;
    int2* where = reinterpret_cast<int2*>(scratch + rows * (sizeof(LstmChunk) / 4));
    int32_t* base = reinterpret_cast<int32_t*>(where) + (2LL * records + 3) / 4 * 4;
    p.where = num_seqs > 1 ? where : nullptr;
    p.base = num_seqs > 1 ? base : nullptr;
    p.records = records;
    p.piece_s = scratch + rows * (sizeof(LstmChunk) / 4) + lstm_table_floats(num_seqs, records);
    p.piece_p = p.piece_s + rows * D * DV;
    p.piece_n = p.piece_p + rows * D;
    p.q_start = q_start;
    p.q_len = q_len;
    p.H = H;
    p.D = D;
    p.DV = DV;
    p.max_pieces = records;
    auto aligned = [](const void* x) { return reinterpret_cast<uintptr_t>(x) % 16 == 0; };
    p.vec = p.in_bf16 && D % 8 == 0 && DV % 8 == 0 && ld % 8 == 0 && aligned(p.q) && aligned(p.k) && aligned(p.v);
    const LstmGates g{gates, ld_gates, bias_i, bias_f, cap, state, state_stride, static_cast<long long>(H) * D * DV + static_cast<long long>(H) * D, state_slot, chunks, where, base, records};
    stride::launch(lstm_gates_kernel, dim3(H, num_seqs), dim3(256), 0, stream, g, q_start, q_len, H);
    return dispatch_chunks<kLstm>(p, state, state_stride, state_slot, num_seqs, stream);
}

}  // extern "C"
