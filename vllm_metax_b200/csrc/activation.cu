// Gated and plain activations, optionally fused with fp8 quantisation.
//   act_and_mul:  out[t, :d] = act(x[t, :d]) * x[t, d:]      (silu, gelu, gelu_tanh, fatrelu, relu2)
//   mul_and_silu, swigluoai (interleaved gate/up with clamp), swiglustep (clamped)
//   plain: gelu_new / gelu_fast / gelu_quick / silu / relu2
//   fused: act_and_mul + static fp8, act_and_mul + per-128 block fp8 (optionally ue8m0 scales)
// Parity: csrc/activation_kernels.cu:102-561, quantization/activation_kernels.cu:43,
// quantization/fused_kernels/fused_silu_mul_block_quant.cu:15 of the reference.
#include "common.cuh"
#include "pdl.cuh"

namespace b200 {

enum Act : int {
  kSilu = 0, kGelu = 1, kGeluTanh = 2, kFatRelu = 3, kRelu2 = 4, kMulSilu = 5, kSwigluOai = 6, kSwigluStep = 7,
  kGeluNew = 8, kGeluFast = 9, kGeluQuick = 10
};

__device__ __forceinline__ float silu_f(float x) { return x / (1.f + __expf(-x)); }
__device__ __forceinline__ float gelu_f(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_tanh_f(float x) {
  return 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
}

__device__ __forceinline__ float unary_act(int act, float x, float p0) {
  switch (act) {
    case kSilu: return silu_f(x);
    case kGelu: return gelu_f(x);
    case kGeluTanh: return gelu_tanh_f(x);
    case kFatRelu: return x > p0 ? x : 0.f;
    case kRelu2: { float r = fmaxf(x, 0.f); return r * r; }
    case kGeluNew: return gelu_tanh_f(x);
    case kGeluFast: return 0.5f * x * (1.f + tanhf(x * 0.7978845608f * (1.f + 0.044715f * x * x)));
    case kGeluQuick: return x / (1.f + __expf(-1.702f * x));
    default: return x;
  }
}

// gate/up combination for one element pair
__device__ __forceinline__ float gated(int act, float g, float u, float p0, float p1) {
  switch (act) {
    case kMulSilu: return g * silu_f(u);
    case kSwigluOai: {  // p0 = alpha, p1 = limit
      g = fminf(g, p1);
      u = fminf(fmaxf(u, -p1), p1);
      return (u + 1.f) * g / (1.f + __expf(-p0 * g));
    }
    case kSwigluStep: {  // p1 = limit
      float s = fminf(silu_f(g), p1);
      u = fminf(fmaxf(u, -p1), p1);
      return s * u;
    }
    default: return unary_act(act, g, p0) * u;
  }
}

// y[t, :] *= sigmoid(x[t, :] . w): the gate of a shared expert.  A CTA per token; its part of y is on its way while the product is
// summed (fp32).  As a library product of one column and five elementwise passes it took 16 us for 64 x 2048 and
// 57 us for 3949 rows; 2.3 and 15 us here, bound by its launch and by the rows' bytes.
template <typename T>
__global__ void __launch_bounds__(256)
sigmoid_dot_scale_kernel(T* out, const T* x, const T* w, const T* y, int K, int N, int64_t x_stride, int64_t y_stride) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[32];
  const int64_t t = blockIdx.x;
  const uint4 *xr = reinterpret_cast<const uint4*>(x + t * x_stride), *yr = reinterpret_cast<const uint4*>(y + t * y_stride);
  uint4 mine = make_uint4(0u, 0u, 0u, 0u);
  if ((int)threadIdx.x < N / 8) mine = yr[threadIdx.x];
  float dot = 0.f;
  for (int i = threadIdx.x; i < K / 8; i += blockDim.x) {
    float a[8], b[8];
    unpack8<T>(xr[i], a);
    unpack8<T>(reinterpret_cast<const uint4*>(w)[i], b);
#pragma unroll
    for (int e = 0; e < 8; ++e) dot = fmaf(a[e], b[e], dot);
  }
  dot = block_sum(dot, red);
  const float s = 1.f / (1.f + __expf(-dot));
  for (int i = threadIdx.x; i < N / 8; i += blockDim.x) {
    float f[8];
    unpack8<T>(i == (int)threadIdx.x ? mine : yr[i], f);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] *= s;
    reinterpret_cast<uint4*>(out + t * N)[i] = pack8<T>(f);
  }
}

template <typename T>
__global__ void act_and_mul_kernel(T* __restrict__ out, const T* __restrict__ x, int d, int64_t x_stride,
                                   int64_t out_stride, int act, float p0, float p1) {
  const int64_t t = blockIdx.x;
  const T* row = x + t * x_stride;
  T* o = out + t * out_stride;
  if (act == kSwigluOai) {  // interleaved: gate = x[2i], up = x[2i+1]
    for (int i = threadIdx.x; i < d; i += blockDim.x)
      o[i] = from_f<T>(gated(act, to_f(row[2 * i]), to_f(row[2 * i + 1]), p0, p1));
    return;
  }
  const int nvec = ((d & 7) == 0 && (x_stride & 7) == 0 && (out_stride & 7) == 0) ? d >> 3 : 0;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    float g[8], u[8];
    unpack8<T>(reinterpret_cast<const uint4*>(row)[v], g);
    unpack8<T>(reinterpret_cast<const uint4*>(row + d)[v], u);
#pragma unroll
    for (int i = 0; i < 8; ++i) g[i] = gated(act, g[i], u[i], p0, p1);
    reinterpret_cast<uint4*>(o)[v] = pack8<T>(g);
  }
  for (int i = (nvec << 3) + threadIdx.x; i < d; i += blockDim.x)
    o[i] = from_f<T>(gated(act, to_f(row[i]), to_f(row[d + i]), p0, p1));
}

template <typename T>
__global__ void activation_kernel(T* __restrict__ out, const T* __restrict__ x, int64_t n, int act, float p0) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = from_f<T>(unary_act(act, to_f(x[i]), p0));
}

// act_and_mul followed by fp8 quantisation.  group == 0: static scale (scale_in[0]);
// group > 0: one dynamic scale per `group` outputs, written to scale_out[t, d/group].
// The activation output is rounded to T before quantisation, as the unfused pipeline would.
// With sorted_ids, rows of padding (ids from numel on) are left out.  Groups of 128 go 8 entries a lane, 16 lanes a group: bound
// by the rows' bytes (22912 rows of 2 x 2048, a third of them padding: 121 us entry by entry with all rows, 47 us so).
template <typename T>
__global__ void __launch_bounds__(256)
act_and_mul_quant128_kernel(uint8_t* __restrict__ out_q, float* __restrict__ scale_out, const T* __restrict__ x, int d, int act,
                            float p0, float p1, int ue8m0, const int* __restrict__ sorted_ids, int numel) {
  const int64_t t = blockIdx.x;
  if (sorted_ids != nullptr && sorted_ids[t] >= numel) return;
  const T* row = x + t * (int64_t)(2 * d);
  for (int c0 = 0; c0 < d; c0 += 256 * 8) {
    const int c = c0 + threadIdx.x * 8;
    const bool live = c < d;                         // (d is a multiple of 128: whole groups of lanes)
    float a[8] = {}, b[8] = {}, m = 0.f;
    if (live) {
      unpack8<T>(*reinterpret_cast<const uint4*>(row + c), a);
      unpack8<T>(*reinterpret_cast<const uint4*>(row + d + c), b);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      a[i] = to_f(from_f<T>(gated(act, a[i], b[i], p0, p1)));
      if (live) m = fmaxf(m, fabsf(a[i]));
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    m = fmaxf(m, 1e-10f);
    float s = m / 448.f;
    if (ue8m0) s = ue8m0_ceil(s);
    if (!live) continue;
    if ((threadIdx.x & 15) == 0) scale_out[t * (d / 128) + c / 128] = s;
    uint8_t q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = float_to_fp8_e4m3(a[i] / s);
    *reinterpret_cast<uint2*>(out_q + t * (int64_t)d + c) =
        make_uint2(q[0] | q[1] << 8 | q[2] << 16 | (uint32_t)q[3] << 24, q[4] | q[5] << 8 | q[6] << 16 | (uint32_t)q[7] << 24);
  }
}

template <typename T>
__global__ void act_and_mul_quant_kernel(uint8_t* __restrict__ out_q, float* __restrict__ scale_out,
                                         const float* __restrict__ scale_in, const T* __restrict__ x, int d, int act,
                                         float p0, float p1, int group, int ue8m0, const int* __restrict__ sorted_ids,
                                         int numel) {
  const int64_t t = blockIdx.x;
  if (sorted_ids != nullptr && sorted_ids[t] >= numel) return;
  const T* row = x + t * (int64_t)(2 * d);
  uint8_t* o = out_q + t * (int64_t)d;
  if (group == 0) {
    const float inv = 1.f / scale_in[0];
    for (int i = threadIdx.x; i < d; i += blockDim.x) {
      const float y = to_f(from_f<T>(gated(act, to_f(row[i]), to_f(row[d + i]), p0, p1)));
      o[i] = float_to_fp8_e4m3(y * inv);
    }
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int ngroups = d / group;
  for (int g = warp; g < ngroups; g += nw) {
    float y[8];  // group <= 256
    float m = 0.f;
    const int per = group / 32;
    for (int j = 0; j < per; ++j) {
      const int i = g * group + lane + 32 * j;
      y[j] = to_f(from_f<T>(gated(act, to_f(row[i]), to_f(row[d + i]), p0, p1)));
      m = fmaxf(m, fabsf(y[j]));
    }
    m = fmaxf(warp_max(m), 1e-10f);
    float s = m / 448.f;
    if (ue8m0) s = ue8m0_ceil(s);
    if (lane == 0) scale_out[t * ngroups + g] = s;
    for (int j = 0; j < per; ++j) o[g * group + lane + 32 * j] = float_to_fp8_e4m3(y[j] / s);
  }
}

void act_and_mul(void* out, const void* x, int tokens, int d, int64_t x_stride, int64_t out_stride, int act, float p0,
                 float p1, int dtype, cudaStream_t stream) {
  if (tokens <= 0) return;
  int th = d / 8;
  th = th < 64 ? 64 : (th > 1024 ? 1024 : (th + 31) / 32 * 32);
  if (dtype == 0)
    act_and_mul_kernel<__nv_bfloat16><<<tokens, th, 0, stream>>>((__nv_bfloat16*)out, (const __nv_bfloat16*)x, d,
                                                                 x_stride, out_stride, act, p0, p1);
  else
    act_and_mul_kernel<__half><<<tokens, th, 0, stream>>>((__half*)out, (const __half*)x, d, x_stride, out_stride, act,
                                                          p0, p1);
}

void activation(void* out, const void* x, int64_t n, int act, float p0, int dtype, cudaStream_t stream) {
  if (n <= 0) return;
  const int th = 256;
  int64_t blocks = (n + th - 1) / th;
  if (blocks > 148 * 16) blocks = 148 * 16;
  if (dtype == 0)
    activation_kernel<__nv_bfloat16><<<(int)blocks, th, 0, stream>>>((__nv_bfloat16*)out, (const __nv_bfloat16*)x, n, act, p0);
  else
    activation_kernel<__half><<<(int)blocks, th, 0, stream>>>((__half*)out, (const __half*)x, n, act, p0);
}

void act_and_mul_quant(void* out_q, float* scale_out, const float* scale_in, const void* x, int tokens, int d, int act,
                       float p0, float p1, int group, int ue8m0, const int* sorted_ids, int numel, int dtype,
                       cudaStream_t stream) {
  if (tokens <= 0) return;
  const int th = 256;
  if (group == 128 && d % 128 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(out_q) & 7) == 0) {
    if (dtype == 0)
      act_and_mul_quant128_kernel<__nv_bfloat16><<<tokens, th, 0, stream>>>((uint8_t*)out_q, scale_out, (const __nv_bfloat16*)x, d,
                                                                            act, p0, p1, ue8m0, sorted_ids, numel);
    else
      act_and_mul_quant128_kernel<__half><<<tokens, th, 0, stream>>>((uint8_t*)out_q, scale_out, (const __half*)x, d, act, p0, p1,
                                                                     ue8m0, sorted_ids, numel);
    return;
  }
  if (dtype == 0)
    act_and_mul_quant_kernel<__nv_bfloat16><<<tokens, th, 0, stream>>>((uint8_t*)out_q, scale_out, scale_in,
                                                                       (const __nv_bfloat16*)x, d, act, p0, p1, group, ue8m0, sorted_ids, numel);
  else
    act_and_mul_quant_kernel<__half><<<tokens, th, 0, stream>>>((uint8_t*)out_q, scale_out, scale_in, (const __half*)x,
                                                                d, act, p0, p1, group, ue8m0, sorted_ids, numel);
}

// Rows of 16-byte pieces; out is packed.  Returns 0, or 1 for other alignments.
int sigmoid_dot_scale(void* out, const void* x, const void* w, const void* y, int64_t rows, int K, int N, int64_t x_stride,
                      int64_t y_stride, int dtype, cudaStream_t stream) {
  auto wide = [](const void* at) { return (reinterpret_cast<uintptr_t>(at) & 15) == 0; };
  if (K % 8 || N % 8 || x_stride % 8 || y_stride % 8 || !wide(out) || !wide(x) || !wide(w) || !wide(y)) return 1;
  if (rows <= 0) return 0;
#define SDS(T) pdl_run(sigmoid_dot_scale_kernel<T>, (unsigned)rows, 256, 0, stream, (T*)out, (const T*)x, (const T*)w, (const T*)y, K, N, \
                       x_stride, y_stride)
  if (dtype == 0) SDS(__nv_bfloat16); else SDS(__half);
#undef SDS
  return 0;
}

}  // namespace b200
