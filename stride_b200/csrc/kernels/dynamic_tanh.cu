// Dynamic Tanh norm fused with the residual sum, and the scaled residual sum on its own.
//
// The norm computes no statistic: y = tanh(alpha * x) * w + b per element, with a scalar alpha. For row r
// (source row s = rows ? rows[r] : r):
//   x = residual[s] + scale * delta[s]     (float32; delta may be absent)
//   residual[s] = x                        (only when rows == nullptr)
//   out[r] = tanh(alpha * x) * w + b       (float32, one rounding at the end)
// `scale` is the multiplier an architecture puts on every sum into its stream (1 where it has none).
#include "common.cuh"

namespace stride {

template <typename T>
__global__ void add_dyt_kernel(float* __restrict__ residual, const T* __restrict__ delta, float scale,
                               const float* __restrict__ weight, const float* __restrict__ bias, float alpha,
                               T* __restrict__ out, const int32_t* __restrict__ rows, int hidden) {
    pdl_trigger();
    pdl_wait();
    const int r = blockIdx.x;
    const size_t s = rows ? static_cast<size_t>(rows[r]) : static_cast<size_t>(r);
    float* res = residual + s * hidden;
    const T* del = delta ? delta + s * hidden : nullptr;
    T* dst = out + static_cast<size_t>(r) * hidden;
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < hidden; i += gridDim.y * blockDim.x) {
        float x = res[i];
        if (del) {
            x = __fmaf_rn(scale, to_f32(del[i]), x);
            if (!rows) res[i] = x;
        }
        dst[i] = from_f32<T>(__fmaf_rn(tanhf(alpha * x), weight[i], bias[i]));
    }
}

// Four neighbouring elements of type T.
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, const float4& v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
__device__ __forceinline__ float4 add_scaled4(float scale, const float4& d, const float4& x) {
    return make_float4(__fmaf_rn(scale, d.x, x.x), __fmaf_rn(scale, d.y, x.y), __fmaf_rn(scale, d.z, x.z), __fmaf_rn(scale, d.w, x.w));
}

// Both with a pack of four elements a thread, where rows are whole packs on their boundaries: the same numbers; an element a thread was bound by
// its instructions and by 2- and 4-byte accesses. 2,048 tokens of 2,048, among the kernels of a step: sum and norm 7.6 us (12.6), sum 9.0 (15.0).
template <typename T>
__global__ void __launch_bounds__(256)
add_dyt_vec_kernel(float* __restrict__ residual, const T* __restrict__ delta, float scale, const float* __restrict__ weight,
                   const float* __restrict__ bias, float alpha, T* __restrict__ out, const int32_t* __restrict__ rows, int hidden) {
    pdl_trigger();
    const int r = blockIdx.x, i = (blockIdx.y * 256 + threadIdx.x) * 4;
    if (i >= hidden) return;
    const float4 w = load4(weight + i), b = load4(bias + i);
    pdl_wait();
    const size_t s = (rows ? static_cast<size_t>(rows[r]) : static_cast<size_t>(r)) * hidden + i;
    float4 x = load4(residual + s);
    if (delta) {
        x = add_scaled4(scale, load4(delta + s), x);
        if (!rows) store4(residual + s, x);
    }
    store4(out + static_cast<size_t>(r) * hidden + i,
           make_float4(__fmaf_rn(tanhf(alpha * x.x), w.x, b.x), __fmaf_rn(tanhf(alpha * x.y), w.y, b.y), __fmaf_rn(tanhf(alpha * x.z), w.z, b.z),
                       __fmaf_rn(tanhf(alpha * x.w), w.w, b.w)));
}

template <typename T>
__global__ void __launch_bounds__(256)
add_scaled_vec_kernel(float* __restrict__ residual, const T* __restrict__ delta, float scale, size_t n) {
    pdl_trigger();
    pdl_wait();
    const size_t i = (blockIdx.x * static_cast<size_t>(256) + threadIdx.x) * 4;
    if (i < n) store4(residual + i, add_scaled4(scale, load4(delta + i), load4(residual + i)));
}

template <typename T>
__global__ void add_scaled_kernel(float* __restrict__ residual, const T* __restrict__ delta, float scale, size_t n) {
    pdl_trigger();
    pdl_wait();
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += static_cast<size_t>(gridDim.x) * blockDim.x)
        residual[i] = __fmaf_rn(scale, to_f32(delta[i]), residual[i]);
}

}  // namespace stride

using namespace stride;

extern "C" {

int stride_add_dyt(float* residual, const void* delta, float scale, const float* weight, const float* bias, float alpha,
                   void* out, const int32_t* rows, int num_rows, int hidden, int dtype, cudaStream_t stream) {
    if (num_rows < 0 || hidden <= 0) return STRIDE_BAD_ARGUMENT;
    if (num_rows == 0) return 0;
    const int pack = dtype == STRIDE_DTYPE_F32 ? 16 : 8;        // bytes of four elements
    if (hidden % 4 == 0 && hidden / 4 <= 65535 * 256 && (dtype == STRIDE_DTYPE_F32 || dtype == STRIDE_DTYPE_BF16) &&
        (reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(weight) | reinterpret_cast<uintptr_t>(bias)) % 16 == 0 &&
        (reinterpret_cast<uintptr_t>(delta) | reinterpret_cast<uintptr_t>(out)) % pack == 0) {
        const dim3 vec(num_rows, (hidden / 4 + 255) / 256);
        if (dtype == STRIDE_DTYPE_F32)
            stride::launch(add_dyt_vec_kernel<float>, vec, dim3(256), 0, stream, residual, static_cast<const float*>(delta), scale, weight, bias, alpha,
                           static_cast<float*>(out), rows, hidden);
        else
            stride::launch(add_dyt_vec_kernel<__nv_bfloat16>, vec, dim3(256), 0, stream, residual, static_cast<const __nv_bfloat16*>(delta), scale,
                           weight, bias, alpha, static_cast<__nv_bfloat16*>(out), rows, hidden);
        return STRIDE_LAUNCH_STATUS();
    }
    const int threads = 256;
    const int per_row = hidden >= 4096 ? 4 : (hidden >= 1024 ? 2 : 1);
    const dim3 grid(num_rows, per_row);
    if (dtype == STRIDE_DTYPE_F32)
        stride::launch(add_dyt_kernel<float>, grid, dim3(threads), 0, stream, residual, static_cast<const float*>(delta), scale, weight,
                       bias, alpha, static_cast<float*>(out), rows, hidden);
    else if (dtype == STRIDE_DTYPE_BF16)
        stride::launch(add_dyt_kernel<__nv_bfloat16>, grid, dim3(threads), 0, stream, residual,
                       static_cast<const __nv_bfloat16*>(delta), scale, weight, bias, alpha, static_cast<__nv_bfloat16*>(out), rows, hidden);
    else
        return STRIDE_BAD_ARGUMENT;
    return STRIDE_LAUNCH_STATUS();
}

int stride_add_scaled(float* residual, const void* delta, float scale, long long n, int dtype, cudaStream_t stream) {
    if (n < 0) return STRIDE_BAD_ARGUMENT;
    if (n == 0) return 0;
    const int pack = dtype == STRIDE_DTYPE_F32 ? 16 : 8;
    if (n % 4 == 0 && n / 1024 < 0x7fffffff && (dtype == STRIDE_DTYPE_F32 || dtype == STRIDE_DTYPE_BF16) && reinterpret_cast<uintptr_t>(residual) % 16 == 0 &&
        reinterpret_cast<uintptr_t>(delta) % pack == 0) {
        const dim3 vec(static_cast<unsigned>((n / 4 + 255) / 256));
        if (dtype == STRIDE_DTYPE_F32)
            stride::launch(add_scaled_vec_kernel<float>, vec, dim3(256), 0, stream, residual, static_cast<const float*>(delta), scale, static_cast<size_t>(n));
        else
            stride::launch(add_scaled_vec_kernel<__nv_bfloat16>, vec, dim3(256), 0, stream, residual, static_cast<const __nv_bfloat16*>(delta), scale,
                           static_cast<size_t>(n));
        return STRIDE_LAUNCH_STATUS();
    }
    const unsigned blocks = static_cast<unsigned>(n / 256 >= 4096 ? 4096 : (n + 255) / 256);
    if (dtype == STRIDE_DTYPE_F32)
        stride::launch(add_scaled_kernel<float>, dim3(blocks), dim3(256), 0, stream, residual, static_cast<const float*>(delta), scale,
                       static_cast<size_t>(n));
    else if (dtype == STRIDE_DTYPE_BF16)
        stride::launch(add_scaled_kernel<__nv_bfloat16>, dim3(blocks), dim3(256), 0, stream, residual,
                       static_cast<const __nv_bfloat16*>(delta), scale, static_cast<size_t>(n));
    else
        return STRIDE_BAD_ARGUMENT;
    return STRIDE_LAUNCH_STATUS();
}

}  // extern "C"
