// Scales from data: the per-tensor scale of a matrix about to be packed, and the calibration helper.
//
// Calibration helper: the largest post-activation magnitude of a first-projection result.
//
// The hidden-activation scale of a layer is amax(act(fc1 output)) / 2688.  The fc1 result of the
// calibration batch is kept as BF16 (rows x N, gate/up interleaved for the gated activations);
// this kernel applies the activation in FP32 with exact exp / tanh and reduces |value| to one
// float, so the host needs neither FP32 copies of the matrix nor a synchronisation.
#include "common.cuh"

namespace lm {
namespace {

constexpr int kThreads = 256;

struct AmaxParams {
  const __nv_bfloat16* preact;
  int64_t elements;  // rows * n
  int activation;
  float clamp_limit;
  float sigmoid_alpha;
  float up_bias;
  float* out;  // non-negative floats order like their bit patterns: atomicMax on the bits
};

__device__ __forceinline__ float post_activation(float g, float u, const AmaxParams& p) {
  if (p.activation == LM_ACT_RELU2) {
    const float x = fmaxf(g, 0.0f);
    return x * x;
  }
  if (p.clamp_limit > 0.0f) {
    g = fminf(g, p.clamp_limit);
    u = fmaxf(fminf(u, p.clamp_limit), -p.clamp_limit);
  }
  switch (p.activation) {
    case LM_ACT_SWIGLU:
    case LM_ACT_SWIGLU_OAI:
      return g * (1.0f / (1.0f + expf(-p.sigmoid_alpha * g))) * (u + p.up_bias);
    case LM_ACT_GEGLU: {
      const float inner = 0.7978845608028654f * (g + 0.044715f * g * g * g);
      return 0.5f * g * (1.0f + tanhf(inner)) * u;
    }
    default:  // reglu
      return fmaxf(g, 0.0f) * u;
  }
}

__global__ void __launch_bounds__(kThreads) activation_amax_kernel(AmaxParams p) {
  // eight BF16 values (four gate/up pairs, or eight unary inputs) per thread and step
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kThreads * 8;
  float best = 0.0f;
  for (int64_t i = (static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x) * 8; i < p.elements; i += stride) {
    const uint4 raw = __ldg(reinterpret_cast<const uint4*>(p.preact + i));
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float lo = __uint_as_float(w[j] << 16), hi = __uint_as_float(w[j] & 0xFFFF0000u);
      if (p.activation == LM_ACT_RELU2) {
        best = fmaxf(best, fmaxf(post_activation(lo, 0.0f, p), post_activation(hi, 0.0f, p)));
      } else {
        best = fmaxf(best, fabsf(post_activation(lo, hi, p)));
      }
    }
  }
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) best = fmaxf(best, __shfl_xor_sync(0xFFFFFFFFu, best, d));
  __shared__ float s_best[kThreads / 32];
  if ((threadIdx.x & 31) == 0) s_best[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < kThreads / 32; ++i) best = fmaxf(best, s_best[i]);
    atomicMax(reinterpret_cast<unsigned int*>(p.out), __float_as_uint(best));
  }
}

// ------------------------------------------------ scale of a matrix: amax / 2688
// Bound by reading the matrix once: four 16-byte loads a thread in flight, five blocks an SM at a time for
// BF16 (42 registers) and four for FP32 (50), one atomic a block.  The grid is eight blocks an SM, so
// the last three or four of each run in a second, emptier round; that is left as it is.
// 128 x 1024 x 2048 BF16 weights: 88 us (6.1 TB/s) where the torch chain took 330 us, because it
// wrote the magnitudes to memory and read them back before it reduced them.
struct TensorScaleParams {
  const uint4* x;
  int64_t vecs;  // 16-byte vectors
  uint32_t* pair;  // [amax bits, finished blocks] on the way, [scale, 1 / scale] at the end
};

// Running maximum of the magnitudes in one 32-bit word of the input: of both BF16 halves, or of
// the FP32 value.  NaN wins, as in torch.amax.
template <bool kBf16>
__device__ __forceinline__ uint32_t max_magnitude(uint32_t m, uint32_t w) {
  if (kBf16) {
    asm("max.NaN.bf16x2 %0, %0, %1;" : "+r"(m) : "r"(w & 0x7FFF7FFFu));
  } else {
    asm("{\n\t.reg .f32 a, b;\n\tmov.b32 a, %0;\n\tmov.b32 b, %1;\n\tmax.NaN.f32 a, a, b;\n\tmov.b32 %0, a;\n\t}"
        : "+r"(m)
        : "r"(w & 0x7FFFFFFFu));
  }
  return m;
}

template <bool kBf16>
__global__ void __launch_bounds__(kThreads) tensor_scale_kernel(TensorScaleParams p) {
  constexpr int kLoads = 4;
  uint32_t m[4] = {0, 0, 0, 0};
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kThreads * kLoads;
  for (int64_t base = static_cast<int64_t>(blockIdx.x) * kThreads * kLoads + threadIdx.x; base < p.vecs;
       base += stride) {
    uint4 v[kLoads];
#pragma unroll
    for (int j = 0; j < kLoads; ++j) {
      const int64_t i = base + j * kThreads;
      v[j] = i < p.vecs ? __ldg(p.x + i) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int j = 0; j < kLoads; ++j) {
      m[0] = max_magnitude<kBf16>(m[0], v[j].x);
      m[1] = max_magnitude<kBf16>(m[1], v[j].y);
      m[2] = max_magnitude<kBf16>(m[2], v[j].z);
      m[3] = max_magnitude<kBf16>(m[3], v[j].w);
    }
  }
  m[0] = max_magnitude<kBf16>(max_magnitude<kBf16>(m[0], m[1]), max_magnitude<kBf16>(m[2], m[3]));
  // as FP32 bits: non-negative floats order like their bits, and a NaN lies above infinity
  uint32_t best = kBf16 ? max(m[0] << 16, m[0] & 0xFFFF0000u) : m[0];
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) best = max(best, __shfl_xor_sync(0xFFFFFFFFu, best, d));
  __shared__ uint32_t s_best[kThreads / 32];
  if ((threadIdx.x & 31) == 0) s_best[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int i = 1; i < kThreads / 32; ++i) best = max(best, s_best[i]);
  atomicMax(p.pair, best);
  __threadfence();
  if (atomicAdd(p.pair + 1, 1u) != gridDim.x - 1) return;
  // the last block: every other block's maximum is in
  __threadfence();
  const float amax = __uint_as_float(atomicMax(p.pair, 0u));
  // torch divides by a constant as a product with its reciprocal; the floor lets a NaN through
  float scale = __fmul_rn(amax, 1.0f / 2688.0f);
  if (scale < 1e-30f) scale = 1e-30f;
  p.pair[0] = __float_as_uint(scale);
  p.pair[1] = __float_as_uint(__fdiv_rn(1.0f, scale));
}

}  // namespace
}  // namespace lm

extern "C" int lm_tensor_scale(const void* x, int x_dtype, int64_t count, float* scale_pair, lm_stream_t stream) {
  using namespace lm;
  LM_REQUIRE(x && scale_pair, "tensor_scale: null pointer");
  LM_REQUIRE(x_dtype == LM_DTYPE_BF16 || x_dtype == LM_DTYPE_F32, "tensor_scale: x must be BF16 or FP32");
  LM_REQUIRE(count > 0 && count % 8 == 0, "tensor_scale: the element count must be a positive multiple of 8");
  LM_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0, "tensor_scale: the matrix must be 16-byte aligned");
  TensorScaleParams p{static_cast<const uint4*>(x), count / (x_dtype == LM_DTYPE_BF16 ? 8 : 4),
                      reinterpret_cast<uint32_t*>(scale_pair)};
  LM_CUDA(cudaMemsetAsync(scale_pair, 0, 2 * sizeof(float), as_stream(stream)));
  constexpr int kPerBlock = kThreads * 4;  // vectors of one step
  const int64_t blocks = (p.vecs + kPerBlock - 1) / kPerBlock;
  const int64_t most = 8ll * sm_count();
  const int grid = static_cast<int>(blocks < most || most <= 0 ? (blocks < 65535 ? blocks : 65535) : most);
  if (x_dtype == LM_DTYPE_BF16) {
    tensor_scale_kernel<true><<<grid, kThreads, 0, as_stream(stream)>>>(p);
  } else {
    tensor_scale_kernel<false><<<grid, kThreads, 0, as_stream(stream)>>>(p);
  }
  note_launch();
  LM_CUDA(cudaGetLastError());
  return LM_OK;
}

extern "C" int lm_activation_amax(const void* preact, int64_t rows, int n, int activation, float clamp_limit,
                                  float sigmoid_alpha, float up_bias, float* out, lm_stream_t stream) {
  using namespace lm;
  LM_REQUIRE(preact && out, "activation_amax: null pointer");
  LM_REQUIRE(activation >= LM_ACT_SWIGLU && activation <= LM_ACT_RELU2, "activation_amax: unknown activation");
  LM_REQUIRE(rows >= 0 && n > 0 && n % 8 == 0, "activation_amax: N must be a multiple of 8");
  LM_REQUIRE((reinterpret_cast<uintptr_t>(preact) & 15) == 0, "activation_amax: the matrix must be 16-byte aligned");
  LM_CUDA(cudaMemsetAsync(out, 0, sizeof(float), as_stream(stream)));
  if (rows == 0) return LM_OK;
  AmaxParams p{static_cast<const __nv_bfloat16*>(preact), rows * n, activation, clamp_limit, sigmoid_alpha,
               up_bias, out};
  const int64_t steps = (p.elements / 8 + kThreads - 1) / kThreads;
  const int sms = sm_count();
  const int grid = static_cast<int>(steps < 8ll * sms ? (steps > 0 ? steps : 1) : 8ll * sms);
  activation_amax_kernel<<<grid, kThreads, 0, as_stream(stream)>>>(p);
  note_launch();
  LM_CUDA(cudaGetLastError());
  return LM_OK;
}
