// Recurrent block with a real-gated linear recurrent unit (the recurrent layer of Griffin: De et al., "Griffin:
// Mixing Gated Linear Recurrences with Local Attention for Efficient Language Models").
//
// Per token, from the two projections of the layer's input (y~ and x~, both [width], in one matrix `xy`):
//   x  = x~ + bias_x ;  u = conv_b + sum_j conv[c, j] * x(t - (taps - 1) + j)         causal, per channel
//   r  = sigmoid(Wa[b] u_b + ba) ; i = sigmoid(Wi[b] u_b + bi)                        per block b of width / blocks channels
//   a  = exp(-decay * r * softplus(lam)) ;  S_t = a S_(t-1) + sqrt(1 - a^2) * i * u   S in float32, zero at the start
//   out = S_t * gelu_tanh(y~ + bias_y)
// Everything after the projections is float32. Per request the state slot holds taps rows of [width] float32: rows
// 0 .. taps-2 are the last taps-1 inputs x (oldest first; zero before the sequence starts, which is what a fresh slot
// holds), row taps-1 is S. Three kernels, run in this order on any mix of portions and single tokens:
//   rglru_conv    u for every token (reads the tail of the state, writes nothing to it)
//   rglru_gates   the block-diagonal products, with a - 1 and the gated input in the epilogue. a - 1 = expm1(log a) is
//                 what is handed on: for a channel that forgets slowly a is 1 - 1e-4 or closer, where float32 has
//                 steps of 6e-8, and the error of a rounded (and, with a biased exponential, shifted) a grows with
//                 every token of a long sequence
//   rglru_scan    the recurrence over each request's tokens, the output, and the new state (S and the tail)
#include <type_traits>

#include "common.cuh"
#include "mma.cuh"

namespace stride {

constexpr int kMaxTaps = 16;

__device__ __forceinline__ float gelu_tanh_f(float z) {
    // z / 2 (1 + tanh y) = z sigmoid(2 y): an exponential and a quotient, and no 1 + tanh that nearly vanishes where y is far below zero
    return z / (1.f + expf(-1.5957691216057308f * (z + 0.044715f * z * z * z)));
}
__device__ __forceinline__ float sigmoid_f(float z) { return 1.f / (1.f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// A long step with four taps: a thread owns four channels of eight consecutive tokens and keeps the last three rows in registers,
// so that a row is read once and not four times. 2,048 tokens x 2,560 channels: 12 us, 41 us with a thread a number.
constexpr int CT = 8;
__global__ void __launch_bounds__(128)
rglru_conv_rows_kernel(const __nv_bfloat16* __restrict__ xy, int ld, int x_off, const float* __restrict__ bias_x, const __nv_bfloat16* __restrict__ conv_w,
                       const float* __restrict__ conv_b, const float* __restrict__ state, const int32_t* __restrict__ seq_of_token,
                       const int32_t* __restrict__ q_start, const int32_t* __restrict__ state_slot, float* __restrict__ u, int tokens, int width) {
    constexpr int TAPS = 4;
    pdl_trigger();
    const int c = (blockIdx.x * 128 + threadIdx.x) * 4, t0 = blockIdx.y * CT;
    if (c >= width) return;
    float w[4][TAPS], bias[4], first[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
#pragma unroll
        for (int j = 0; j < TAPS; ++j) w[e][j] = to_f32(conv_w[static_cast<size_t>(c + e) * TAPS + j]);
        bias[e] = bias_x[c + e];
        first[e] = conv_b[c + e];
    }
    pdl_wait();
    uint2 raw[CT + TAPS - 1];
#pragma unroll
    for (int i = 0; i < CT + TAPS - 1; ++i) {
        const int t = t0 + i - (TAPS - 1);
        raw[i] = t >= 0 && t < tokens ? *reinterpret_cast<const uint2*>(xy + static_cast<size_t>(t) * ld + x_off + c) : make_uint2(0, 0);
    }
#pragma unroll
    for (int i = 0; i < CT; ++i) {
        const int t = t0 + i;
        if (t >= tokens) break;
        const int seq = seq_of_token[t];
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        if (seq >= 0) {
            const int local = t - q_start[seq];
            const float* tail = state + static_cast<size_t>(state_slot[seq]) * TAPS * width;
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[e] = first[e];
#pragma unroll
            for (int j = 0; j < TAPS; ++j) {
                const int src = local - (TAPS - 1) + j;
                float v[4];
                if (src >= 0) {
                    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[i + j].x));
                    const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[i + j].y));
                    v[0] = lo.x + bias[0]; v[1] = lo.y + bias[1]; v[2] = hi.x + bias[2]; v[3] = hi.y + bias[3];
                } else {
                    const float4 q = *reinterpret_cast<const float4*>(tail + static_cast<size_t>(TAPS - 1 + src) * width + c);
                    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[e] = fmaf(w[e][j], v[e], acc[e]);
            }
        }
        *reinterpret_cast<float4*>(u + static_cast<size_t>(t) * width + c) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    }
}

template <typename T>
__global__ void __launch_bounds__(256)
rglru_conv_kernel(const T* __restrict__ xy, int ld, int x_off, const float* __restrict__ bias_x, const T* __restrict__ conv_w,
                  const float* __restrict__ conv_b, const float* __restrict__ state, const int32_t* __restrict__ seq_of_token,
                  const int32_t* __restrict__ q_start, const int32_t* __restrict__ state_slot, float* __restrict__ u, int width,
                  int taps) {
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x;
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    if (c >= width) return;
    const int seq = seq_of_token[t];
    if (seq < 0) {
        u[static_cast<size_t>(t) * width + c] = 0.f;
        return;
    }
    const int start = q_start[seq];
    const int local = t - start;
    const float* tail = state + static_cast<size_t>(state_slot[seq]) * taps * width;
    float acc = conv_b[c];
    for (int j = 0; j < taps; ++j) {
        const int src = local - (taps - 1) + j;
        const float v = src >= 0 ? to_f32(xy[static_cast<size_t>(start + src) * ld + x_off + c]) + bias_x[c]
                                 : tail[static_cast<size_t>(taps - 1 + src) * width + c];
        acc = fmaf(to_f32(conv_w[static_cast<size_t>(c) * taps + j]), v, acc);
    }
    u[static_cast<size_t>(t) * width + c] = acc;
}

// wa_t / wi_t: the gate matrices transposed per block, [blocks, in, out], so that threads of neighbouring output
// channels read neighbouring addresses. One CTA: GT tokens x 32 output channels of one block, the sum over the block's
// inputs cut into four slices (one a warp) that are added in the order of the slices: many small CTAs, so that a step of
// a few tokens still spreads the weights' read over the device.
constexpr int GT = 8, GC = 32, GS = 4;

template <typename T>
__global__ void __launch_bounds__(GC * GS)
rglru_gates_kernel(const float* __restrict__ u, const T* __restrict__ wa_t, const T* __restrict__ wi_t, const float* __restrict__ ba,
                   const float* __restrict__ bi, const float* __restrict__ lam, float decay, float* __restrict__ a_out,
                   float* __restrict__ gx_out, int tokens, int width, int bw) {
    pdl_trigger();
    if (blockIdx.z == 0) {      // the CTA's columns of both matrices, a row a thread
        const size_t at = static_cast<size_t>(blockIdx.y) * bw * bw + blockIdx.x * GC;
        const int cols = min(GC, bw - static_cast<int>(blockIdx.x) * GC);
        for (int k = threadIdx.x; k < bw; k += GC * GS) {
            prefetch_l2(wa_t + at + static_cast<size_t>(k) * bw, cols * sizeof(T), 0, 1);
            prefetch_l2(wi_t + at + static_cast<size_t>(k) * bw, cols * sizeof(T), 0, 1);
        }
    }
    pdl_wait();
    extern __shared__ float us[];                   // [GT][bw], then the slices' sums [GS][2][GT][GC]
    float* part = us + GT * bw;
    const int b = blockIdx.y;
    const int t0 = blockIdx.z * GT;
    const int lane = threadIdx.x & (GC - 1), slice = threadIdx.x / GC;
    const int oc = blockIdx.x * GC + lane;          // output channel inside the block
    for (int i = threadIdx.x; i < GT * bw; i += GC * GS) {
        const int tt = i / bw, k = i % bw;
        us[i] = t0 + tt < tokens ? u[static_cast<size_t>(t0 + tt) * width + b * bw + k] : 0.f;
    }
    __syncthreads();
    float accr[GT], acci[GT];
#pragma unroll
    for (int tt = 0; tt < GT; ++tt) accr[tt] = acci[tt] = 0.f;
    const int per = (bw + GS - 1) / GS;
    const int k_lo = slice * per, k_hi = min(bw, k_lo + per);
    if (oc < bw) {
        const T* wa = wa_t + static_cast<size_t>(b) * bw * bw + oc;
        const T* wi = wi_t + static_cast<size_t>(b) * bw * bw + oc;
#pragma unroll 16       // 32 loads in flight: 3 tokens of 10 blocks of 256 in 11.7 us, 19.6 with 8
        for (int k = k_lo; k < k_hi; ++k) {
            const float wr = to_f32(wa[static_cast<size_t>(k) * bw]), wg = to_f32(wi[static_cast<size_t>(k) * bw]);
#pragma unroll
            for (int tt = 0; tt < GT; ++tt) {
                const float x = us[tt * bw + k];
                accr[tt] = fmaf(wr, x, accr[tt]);
                acci[tt] = fmaf(wg, x, acci[tt]);
            }
        }
    }
#pragma unroll
    for (int tt = 0; tt < GT; ++tt) {
        part[((slice * 2 + 0) * GT + tt) * GC + lane] = accr[tt];
        part[((slice * 2 + 1) * GT + tt) * GC + lane] = acci[tt];
    }
    __syncthreads();
    if (oc >= bw) return;
    const int c = b * bw + oc;
    const float rate = decay * softplus_f(lam[c]);
    const float br = ba[c], bg = bi[c];
    // warp `slice` finishes the tokens slice, slice + GS, ...
    for (int tt = slice; tt < GT; tt += GS) {
        if (t0 + tt >= tokens) break;
        float sr = 0.f, sg = 0.f;
#pragma unroll
        for (int s2 = 0; s2 < GS; ++s2) {
            sr += part[((s2 * 2 + 0) * GT + tt) * GC + lane];
            sg += part[((s2 * 2 + 1) * GT + tt) * GC + lane];
        }
        const float r = sigmoid_f(sr + br), g = sigmoid_f(sg + bg);
        const float log_a = -rate * r;
        const size_t at = static_cast<size_t>(t0 + tt) * width + c;
        a_out[at] = expm1f(log_a);      // a - 1: a itself, rounded to float32, would lose the rate of a slowly decaying channel
        gx_out[at] = sqrtf(-expm1f(2.f * log_a)) * g * us[tt * bw + oc];
    }
}

// The same products for a long step in bfloat16 mode, on the tensor cores. The inputs are float32: each is cut into three bfloat16
// numbers that add up to it (24 bits), the weights are bfloat16 as stored. The tensor cores cut off what falls below their
// accumulator's last place, always towards zero, which over a long sum is twice the error of rounded multiply-adds (2.4e-7 against
// 1.2e-7 at 72 inputs): so the first parts' products of 16 inputs start from zero and are added up with rounded additions, and only
// those of the second and third parts, 2^-8 and less of them, stay in an accumulator. A CTA: 64 tokens x 64 output channels
// of one block, both gates; eight warps, 32 tokens x 16 channels each; 64 inputs at a time through shared memory. Bound by
// the exponentials of its epilogue (22 us) and the products; 2,048 tokens x 10 blocks of 256: 102 us with the next 64 inputs on their way
// during the products, 117 without, 243 us with multiply-adds (8 tokens x 128 channels a CTA).
template <bool VEC>
__global__ void __launch_bounds__(256, 2)
rglru_gates_mma_kernel(const float* __restrict__ u, const __nv_bfloat16* __restrict__ wa_t, const __nv_bfloat16* __restrict__ wi_t,
                       const float* __restrict__ ba, const float* __restrict__ bi, const float* __restrict__ lam, float decay,
                       float* __restrict__ a_out, float* __restrict__ gx_out, int tokens, int width, int bw) {
    constexpr int LD = 72;                              // 64 numbers and 16 bytes: rows of a fragment meet no bank twice
    __shared__ __align__(16) __nv_bfloat16 us[3][64][LD];      // [part][token][input]
    __shared__ __align__(16) __nv_bfloat16 ws[2][64][LD];      // [gate][input][channel]
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int b = blockIdx.y, t0 = blockIdx.z * 64, c0 = blockIdx.x * 64;
    const int wm = (warp >> 2) * 32, wn = (warp & 3) * 16;
    const __nv_bfloat16* const wg[2] = {wa_t + static_cast<size_t>(b) * bw * bw, wi_t + static_cast<size_t>(b) * bw * bw};
    const float* const ub = u + static_cast<size_t>(b) * bw;
    float acc[2][4][4] = {}, low[2][4][4] = {};         // [16 tokens][gate, 8 channels][fragment]
    pdl_wait();
    float4 next_u[4];           // pieces of 4 inputs of a token
    uint4 next_w[4];            // pieces of 8 channels of an input
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int p = tid + i * 256, r = p >> 4, k = k0 + (p & 15) * 4;
            float x[4] = {0.f, 0.f, 0.f, 0.f};
            if (t0 + r < tokens) {
                const float* src = ub + static_cast<size_t>(t0 + r) * width + k;
                if (VEC) {
                    if (k < bw) {
                        const float4 v = *reinterpret_cast<const float4*>(src);
                        x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (k + e < bw) x[e] = src[e];
                }
            }
            next_u[i] = make_float4(x[0], x[1], x[2], x[3]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int p = tid + i * 256, gate = p >> 9, k = k0 + ((p >> 3) & 63), c = (p & 7) * 8;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (k < bw) {
                const __nv_bfloat16* src = wg[gate] + static_cast<size_t>(k) * bw + c0 + c;
                if (VEC) {
                    if (c0 + c < bw) v = *reinterpret_cast<const uint4*>(src);
                } else {
                    __nv_bfloat16* e = reinterpret_cast<__nv_bfloat16*>(&v);
#pragma unroll
                    for (int n = 0; n < 8; ++n)
                        if (c0 + c + n < bw) e[n] = src[n];
                }
            }
            next_w[i] = v;
        }
    };
    fetch(0);
    for (int k0 = 0; k0 < bw; k0 += 64) {
        if (k0) __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int p = tid + i * 256, r = p >> 4, k = (p & 15) * 4;
            float x[4] = {next_u[i].x, next_u[i].y, next_u[i].z, next_u[i].w};
#pragma unroll
            for (int part = 0; part < 3; ++part) {
                __nv_bfloat162 h[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    h[e] = __floats2bfloat162_rn(x[2 * e], x[2 * e + 1]);
                    const float lo = __bfloat162float(h[e].x), hi = __bfloat162float(h[e].y);
                    x[2 * e] = isinf(lo) ? 0.f : x[2 * e] - lo;             // an infinity is whole in its first part
                    x[2 * e + 1] = isinf(hi) ? 0.f : x[2 * e + 1] - hi;
                }
                *reinterpret_cast<uint2*>(&us[part][r][k]) = make_uint2(*reinterpret_cast<uint32_t*>(&h[0]), *reinterpret_cast<uint32_t*>(&h[1]));
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int p = tid + i * 256, gate = p >> 9, k = (p >> 3) & 63, c = (p & 7) * 8;
            *reinterpret_cast<uint4*>(&ws[gate][k][c]) = next_w[i];
        }
        if (k0 + 64 < bw) fetch(k0 + 64);           // on their way while the products run
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 64; k += 16) {
            uint32_t bf[2][4];                          // per gate: (channels 0-7: inputs 0-7, 8-15), (channels 8-15: the same)
#pragma unroll
            for (int gate = 0; gate < 2; ++gate) ldmatrix_x4_trans(bf[gate], smem_addr(&ws[gate][k + (lane & 15)][wn + (lane >> 4) * 8]));
#pragma unroll
            for (int part = 2; part >= 0; --part)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    uint32_t af[4];
                    ldmatrix_x4(af, smem_addr(&us[part][wm + i * 16 + (lane & 15)][k + (lane >> 4) * 8]));
#pragma unroll
                    for (int n = 0; n < 4; ++n) {
                        if (part) {
                            mma_bf16_16816(low[i][n], af, bf[n >> 1][(n & 1) * 2], bf[n >> 1][(n & 1) * 2 + 1]);
                        } else {
                            float d[4] = {0.f, 0.f, 0.f, 0.f};
                            mma_bf16_16816(d, af, bf[n >> 1][(n & 1) * 2], bf[n >> 1][(n & 1) * 2 + 1]);
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[i][n][e] += d[e];
                        }
                    }
                }
        }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int oc = c0 + wn + n * 8 + 2 * t + e;
            if (oc >= bw) continue;
            const int c = b * bw + oc;
            const float rate = decay * softplus_f(lam[c]), br = ba[c], bg = bi[c];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int row = t0 + wm + i * 16 + g + 8 * h;
                    if (row >= tokens) continue;
                    const float r = sigmoid_f(acc[i][n][2 * h + e] + low[i][n][2 * h + e] + br);
                    const float q = sigmoid_f(acc[i][2 + n][2 * h + e] + low[i][2 + n][2 * h + e] + bg);
                    const float log_a = -rate * r;
                    const size_t at = static_cast<size_t>(row) * width + c;
                    a_out[at] = expm1f(log_a);
                    gx_out[at] = sqrtf(-expm1f(2.f * log_a)) * q * u[at];
                }
        }
}

template <typename T>
__global__ void __launch_bounds__(64)
rglru_scan_kernel(const float* __restrict__ a /* a - 1 */, const float* __restrict__ gx, const T* __restrict__ xy, int ld, int x_off, int y_off,
                  const float* __restrict__ bias_x, const float* __restrict__ bias_y, float* __restrict__ state,
                  const int32_t* __restrict__ q_start, const int32_t* __restrict__ q_len, const int32_t* __restrict__ state_slot,
                  T* __restrict__ out, int width, int taps) {
    pdl_trigger();
    pdl_wait();
    const int seq = blockIdx.y;
    const int n = q_len[seq];
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (n <= 0 || c >= width) return;
    const int start = q_start[seq];
    float* rows = state + static_cast<size_t>(state_slot[seq]) * taps * width;
    float s = rows[static_cast<size_t>(taps - 1) * width + c];
    const float by = bias_y[c];
    // Nothing the loop loads depends on s: eight tokens' values are fetched into registers before the chain of s runs
    // over them, so their latencies overlap. The order of the arithmetic is the token order either way.
    constexpr int AHEAD = 8;
    int i = 0;
    for (; i + AHEAD <= n; i += AHEAD) {
        float am1[AHEAD], g[AHEAD], yp[AHEAD];
#pragma unroll
        for (int j = 0; j < AHEAD; ++j) {
            const size_t at = static_cast<size_t>(start + i + j) * width + c;
            am1[j] = a[at];
            g[j] = gx[at];
            yp[j] = to_f32(xy[static_cast<size_t>(start + i + j) * ld + y_off + c]);
        }
#pragma unroll
        for (int j = 0; j < AHEAD; ++j) {
            s = fmaf(am1[j], s, s) + g[j];      // a S + gx with a - 1 stored
            out[static_cast<size_t>(start + i + j) * width + c] = from_f32<T>(s * gelu_tanh_f(yp[j] + by));
        }
    }
    for (; i < n; ++i) {
        const size_t at = static_cast<size_t>(start + i) * width + c;
        s = fmaf(a[at], s, s) + gx[at];
        const float y = gelu_tanh_f(to_f32(xy[static_cast<size_t>(start + i) * ld + y_off + c]) + by);
        out[at] = from_f32<T>(s * y);
    }
    rows[static_cast<size_t>(taps - 1) * width + c] = s;
    // the last taps-1 inputs, oldest first: from this step's tokens where it has them, else from the old tail
    float tail[kMaxTaps];
    const float bx = bias_x[c];
    for (int r = 0; r < taps - 1; ++r) {
        const int src = n - (taps - 1) + r;
        tail[r] = src >= 0 ? to_f32(xy[static_cast<size_t>(start + src) * ld + x_off + c]) + bx
                           : rows[static_cast<size_t>(taps - 1 + src) * width + c];
    }
    for (int r = 0; r < taps - 1; ++r) rows[static_cast<size_t>(r) * width + c] = tail[r];
}

// ---- the recurrence of a long portion in three passes, parallel over pieces of SEG tokens (bfloat16 mode; the 32-bit
// path keeps the one chain in token order above). With S_t = a_t S_(t-1) + g_t a piece maps the state at its start to
// the state at its end as S -> P S + B, P the product of its a and B its own scan from zero:
//   rglru_piece_kernel   P and B of every piece                      (parallel over pieces and channels)
//   rglru_carry_kernel   the state at the start of every piece        (per request and channel, one step a piece),
//                        the request's new state and convolution tail
//   rglru_apply_kernel   the scan of every piece from its start state, times the gelu branch
// 2,048 tokens of 2,560 channels, among the kernels of a step: 30, 27 and 44 us; 33, 34 and 68 with eight tokens, one piece and eight tokens asked
// for at a time and tanhf in the gelu branch, whose instructions bound the last (tanhf as an exponential and a quotient: 44 of 67).
constexpr int SEG = 64;
constexpr int SEG_AHEAD = 16;       // tokens (pieces) whose inputs a thread has asked for before it works on the first of them

__global__ void __launch_bounds__(64)
rglru_piece_kernel(const float* __restrict__ a, const float* __restrict__ gx, const int32_t* __restrict__ q_start,
                   const int32_t* __restrict__ q_len, float* __restrict__ piece /* [tokens / SEG + seqs][2][width] by first row */,
                   int width) {
    pdl_trigger();
    pdl_wait();
    const int seq = blockIdx.y, j = blockIdx.z;
    const int n = q_len[seq];
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (j * SEG >= n || c >= width) return;
    const int first = q_start[seq] + j * SEG, count = min(SEG, n - j * SEG);
    float p = 1.f, b = 0.f;
    for (int i0 = 0; i0 < count; i0 += SEG_AHEAD) {
        float am1[SEG_AHEAD], g[SEG_AHEAD];
#pragma unroll
        for (int i = 0; i < SEG_AHEAD; ++i)
            if (i0 + i < count) {
                const size_t at = static_cast<size_t>(first + i0 + i) * width + c;
                am1[i] = a[at];
                g[i] = gx[at];
            }
#pragma unroll
        for (int i = 0; i < SEG_AHEAD; ++i)
            if (i0 + i < count) {
                b = fmaf(am1[i], b, b) + g[i];
                p = fmaf(am1[i], p, p);
            }
    }
    // a piece is named by the row of its first token: pieces of different requests never share one
    float* dst = piece + static_cast<size_t>(first / SEG + seq) * 2 * width;
    dst[c] = p;
    dst[width + c] = b;
}

template <typename T>
__global__ void __launch_bounds__(64)
rglru_carry_kernel(float* __restrict__ piece, const T* __restrict__ xy, int ld, int x_off, const float* __restrict__ bias_x,
                   float* __restrict__ state, const int32_t* __restrict__ q_start, const int32_t* __restrict__ q_len,
                   const int32_t* __restrict__ state_slot, int width, int taps) {
    pdl_trigger();
    pdl_wait();
    const int seq = blockIdx.y;
    const int n = q_len[seq];
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (n <= 0 || c >= width) return;
    const int start = q_start[seq];
    float* rows = state + static_cast<size_t>(state_slot[seq]) * taps * width;
    float s = rows[static_cast<size_t>(taps - 1) * width + c];
    auto at = [&](int j) { return piece + static_cast<size_t>((start + j * SEG) / SEG + seq) * 2 * width + c; };
    for (int j0 = 0; j0 * SEG < n; j0 += SEG_AHEAD) {
        float p[SEG_AHEAD], b[SEG_AHEAD];
#pragma unroll
        for (int j = 0; j < SEG_AHEAD; ++j)
            if ((j0 + j) * SEG < n) {
                p[j] = at(j0 + j)[0];
                b[j] = at(j0 + j)[width];
            }
#pragma unroll
        for (int j = 0; j < SEG_AHEAD; ++j)
            if ((j0 + j) * SEG < n) {
                at(j0 + j)[0] = s;          // the piece's start state takes the place of its P
                s = fmaf(p[j], s, b[j]);
            }
    }
    rows[static_cast<size_t>(taps - 1) * width + c] = s;
    float tail[kMaxTaps];
    const float bx = bias_x[c];
    for (int r = 0; r < taps - 1; ++r) {
        const int src = n - (taps - 1) + r;
        tail[r] = src >= 0 ? to_f32(xy[static_cast<size_t>(start + src) * ld + x_off + c]) + bx
                           : rows[static_cast<size_t>(taps - 1 + src) * width + c];
    }
    for (int r = 0; r < taps - 1; ++r) rows[static_cast<size_t>(r) * width + c] = tail[r];
}

template <typename T>
__global__ void __launch_bounds__(64, 9)
rglru_apply_kernel(const float* __restrict__ a, const float* __restrict__ gx, const float* __restrict__ piece, const T* __restrict__ xy,
                   int ld, int y_off, const float* __restrict__ bias_y, const int32_t* __restrict__ q_start,
                   const int32_t* __restrict__ q_len, T* __restrict__ out, int width) {
    pdl_trigger();
    pdl_wait();
    const int seq = blockIdx.y, j = blockIdx.z;
    const int n = q_len[seq];
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (j * SEG >= n || c >= width) return;
    const int first = q_start[seq] + j * SEG, count = min(SEG, n - j * SEG);
    float s = piece[static_cast<size_t>(first / SEG + seq) * 2 * width + c];
    const float by = bias_y[c];
    constexpr int AHEAD = 8;
    auto batch = [&](int i0, auto whole) {
        float am1[AHEAD], g[AHEAD], yp[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (decltype(whole)::value || i0 + i < count) {
                const size_t at = static_cast<size_t>(first + i0 + i) * width + c;
                am1[i] = a[at];
                g[i] = gx[at];
                yp[i] = to_f32(xy[static_cast<size_t>(first + i0 + i) * ld + y_off + c]);
            }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (decltype(whole)::value || i0 + i < count) {
                s = fmaf(am1[i], s, s) + g[i];
                out[static_cast<size_t>(first + i0 + i) * width + c] = from_f32<T>(s * gelu_tanh_f(yp[i] + by));
            }
    };
    for (int i0 = 0; i0 < count; i0 += AHEAD) {
        if (i0 + AHEAD <= count) batch(i0, std::true_type{});
        else batch(i0, std::false_type{});
    }
}

}  // namespace stride

using namespace stride;

extern "C" {

int stride_rglru_conv(const void* xy, int ld, int x_off, const float* bias_x, const void* conv_w, const float* conv_b, const float* state,
                      const int32_t* seq_of_token, const int32_t* q_start, const int32_t* state_slot, float* u, int tokens, int width,
                      int taps, int dtype, cudaStream_t stream) {
    if (tokens < 0 || width <= 0 || taps <= 0 || ld <= 0 || x_off < 0) return STRIDE_BAD_ARGUMENT;
    if (taps > kMaxTaps) return STRIDE_UNSUPPORTED;
    if (tokens == 0) return 0;
    // Short steps and narrow layers spread better with a thread a number. Rows in registers / a thread a number, 216
    // channels: 512 tokens 3.7 / 2.8 us, 2,048 4.1 / 5.1; 2,560 channels: 128 tokens 3.9 / 4.1, 200 4.1 / 5.4.
    if (dtype == STRIDE_DTYPE_BF16 && taps == 4 && static_cast<long long>(tokens) * width >= 1 << 18 && (tokens + CT - 1) / CT <= 65535 && width % 4 == 0 && ld % 4 == 0 && x_off % 4 == 0 &&
        (reinterpret_cast<uintptr_t>(xy) | reinterpret_cast<uintptr_t>(u) | reinterpret_cast<uintptr_t>(state)) % 16 == 0) {
        stride::launch(rglru_conv_rows_kernel, dim3((width / 4 + 127) / 128, (tokens + CT - 1) / CT), dim3(128), 0, stream,
                       static_cast<const __nv_bfloat16*>(xy), ld, x_off, bias_x, static_cast<const __nv_bfloat16*>(conv_w), conv_b, state, seq_of_token,
                       q_start, state_slot, u, tokens, width);
        return STRIDE_LAUNCH_STATUS();
    }
    const dim3 grid(tokens, (width + 255) / 256);
    if (dtype == STRIDE_DTYPE_F32)
        stride::launch(rglru_conv_kernel<float>, grid, dim3(256), 0, stream, static_cast<const float*>(xy), ld, x_off, bias_x,
                       static_cast<const float*>(conv_w), conv_b, state, seq_of_token, q_start, state_slot, u, width, taps);
    else if (dtype == STRIDE_DTYPE_BF16)
        stride::launch(rglru_conv_kernel<__nv_bfloat16>, grid, dim3(256), 0, stream, static_cast<const __nv_bfloat16*>(xy), ld, x_off,
                       bias_x, static_cast<const __nv_bfloat16*>(conv_w), conv_b, state, seq_of_token, q_start, state_slot, u, width, taps);
    else
        return STRIDE_BAD_ARGUMENT;
    return STRIDE_LAUNCH_STATUS();
}

int stride_rglru_gates(const float* u, const void* wa_t, const void* wi_t, const float* ba, const float* bi, const float* lam, float decay,
                       float* a_out, float* gx_out, int tokens, int width, int blocks, int dtype, cudaStream_t stream) {
    if (tokens < 0 || width <= 0 || blocks <= 0 || width % blocks) return STRIDE_BAD_ARGUMENT;
    if (tokens == 0) return 0;
    const int bw = width / blocks;
    const size_t smem = (static_cast<size_t>(GT) * bw + GS * 2 * GT * GC) * sizeof(float);
    if (smem > 200 * 1024) return STRIDE_UNSUPPORTED;
    if (smem > 48 * 1024) {     // blocks of more than 1,280 channels: ask for the shared memory beyond the default limit
        const int want = static_cast<int>(smem);
        if (cudaFuncSetAttribute(rglru_gates_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, want) != cudaSuccess ||
            cudaFuncSetAttribute(rglru_gates_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, want) != cudaSuccess)
            return STRIDE_UNSUPPORTED;
    }
    const dim3 grid((bw + GC - 1) / GC, blocks, (tokens + GT - 1) / GT);
    if (grid.z > 65535 || grid.y > 65535) return STRIDE_UNSUPPORTED;
    // Blocks narrower than a tile leave most of it empty: they stay with the multiply-adds until the work counts. Tensor cores /
    // multiply-adds, 3 blocks of 72: 512 tokens 12.8 / 7.2 us, 2,048 17.7 / 20.1; a block of 8: 2,048 7.1 / 3.3; 10 blocks of 256: 128 22 / 28.
    if (dtype == STRIDE_DTYPE_BF16 && tokens > 64 && (bw >= 128 || static_cast<long long>(tokens) * width * bw >= 1 << 24)) {
        // Long steps in bfloat16 mode. (The 32-bit path keeps one form for every step, so that a token's sums have the same order
        // however the step was cut.)
        const dim3 tiles((bw + 63) / 64, blocks, (tokens + 63) / 64);
        const bool vec = bw % 8 == 0 && (reinterpret_cast<uintptr_t>(u) | reinterpret_cast<uintptr_t>(wa_t) | reinterpret_cast<uintptr_t>(wi_t)) % 16 == 0;
        const auto kernel = vec ? rglru_gates_mma_kernel<true> : rglru_gates_mma_kernel<false>;
        stride::launch(kernel, tiles, dim3(256), 0, stream, u, static_cast<const __nv_bfloat16*>(wa_t), static_cast<const __nv_bfloat16*>(wi_t), ba, bi,
                       lam, decay, a_out, gx_out, tokens, width, bw);
        return STRIDE_LAUNCH_STATUS();
    }
    if (dtype == STRIDE_DTYPE_F32)
        stride::launch(rglru_gates_kernel<float>, grid, dim3(GC * GS), smem, stream, u, static_cast<const float*>(wa_t),
                       static_cast<const float*>(wi_t), ba, bi, lam, decay, a_out, gx_out, tokens, width, bw);
    else if (dtype == STRIDE_DTYPE_BF16)
        stride::launch(rglru_gates_kernel<__nv_bfloat16>, grid, dim3(GC * GS), smem, stream, u, static_cast<const __nv_bfloat16*>(wa_t),
                       static_cast<const __nv_bfloat16*>(wi_t), ba, bi, lam, decay, a_out, gx_out, tokens, width, bw);
    else
        return STRIDE_BAD_ARGUMENT;
    return STRIDE_LAUNCH_STATUS();
}

int stride_rglru_scan(const float* a, const float* gx, const void* xy, int ld, int x_off, int y_off, const float* bias_x,
                      const float* bias_y, float* state, const int32_t* q_start, const int32_t* q_len, const int32_t* state_slot, void* out,
                      int num_seqs, int width, int taps, int dtype, cudaStream_t stream) {
    if (num_seqs < 0 || width <= 0 || taps <= 0 || num_seqs > 65535) return STRIDE_BAD_ARGUMENT;
    if (taps > kMaxTaps) return STRIDE_UNSUPPORTED;
    if (num_seqs == 0) return 0;
    const dim3 grid((width + 63) / 64, num_seqs);
    if (dtype == STRIDE_DTYPE_F32)
        stride::launch(rglru_scan_kernel<float>, grid, dim3(64), 0, stream, a, gx, static_cast<const float*>(xy), ld, x_off, y_off, bias_x,
                       bias_y, state, q_start, q_len, state_slot, static_cast<float*>(out), width, taps);
    else if (dtype == STRIDE_DTYPE_BF16)
        stride::launch(rglru_scan_kernel<__nv_bfloat16>, grid, dim3(64), 0, stream, a, gx, static_cast<const __nv_bfloat16*>(xy), ld, x_off,
                       y_off, bias_x, bias_y, state, q_start, q_len, state_slot, static_cast<__nv_bfloat16*>(out), width, taps);
    else
        return STRIDE_BAD_ARGUMENT;
    return STRIDE_LAUNCH_STATUS();
}

// The same as stride_rglru_scan in three passes over pieces of 64 tokens (bfloat16 activations). `piece`: float32 scratch of
// (tokens / 64 + num_seqs + 1) * 2 * width. max_q_len: the most tokens a request brings (sizes the grid).
int stride_rglru_scan_pieces(const float* a, const float* gx, const void* xy, int ld, int x_off, int y_off, const float* bias_x,
                             const float* bias_y, float* state, const int32_t* q_start, const int32_t* q_len, const int32_t* state_slot,
                             void* out, float* piece, int num_seqs, int max_q_len, int width, int taps, int dtype, cudaStream_t stream) {
    if (num_seqs < 0 || width <= 0 || taps <= 0 || num_seqs > 65535 || max_q_len <= 0 || !piece) return STRIDE_BAD_ARGUMENT;
    if (taps > kMaxTaps || dtype != STRIDE_DTYPE_BF16) return STRIDE_UNSUPPORTED;
    if (num_seqs == 0) return 0;
    const int pieces = (max_q_len + SEG - 1) / SEG;
    if (pieces > 65535) return STRIDE_UNSUPPORTED;
    const dim3 wide((width + 63) / 64, num_seqs, pieces), narrow((width + 63) / 64, num_seqs);
    const __nv_bfloat16* x = static_cast<const __nv_bfloat16*>(xy);
    stride::launch(rglru_piece_kernel, wide, dim3(64), 0, stream, a, gx, q_start, q_len, piece, width);
    stride::launch(rglru_carry_kernel<__nv_bfloat16>, narrow, dim3(64), 0, stream, piece, x, ld, x_off, bias_x, state, q_start, q_len,
                   state_slot, width, taps);
    stride::launch(rglru_apply_kernel<__nv_bfloat16>, wide, dim3(64), 0, stream, a, gx, static_cast<const float*>(piece), x, ld, y_off,
                   bias_y, q_start, q_len, static_cast<__nv_bfloat16*>(out), width);
    return STRIDE_LAUNCH_STATUS();
}

}  // extern "C"
