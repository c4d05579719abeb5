// Deterministic top-k combine (HBM-bound gather-reduce).
//
// One thread owns eight BF16 columns (16 bytes) of one token: it loads the
// token's rows a batch of routes at a time, adds them in route order to an FP32 sum in
// registers and stores the BF16 result once.  The product with the routing weight is rounded before the
// add (mul.rn then add.rn, never fused), so the result is independent of the
// launch shape and bit-identical from run to run.
//
// What bounds it: reading the routed rows once.  Compiled for the exact route count (no predicates
// or idle registers for routes that do not exist), with two FP32 sums an instruction and every
// thread of a block on a vector, it takes (B200, device time, against a block of eight-route
// batches per token and 2048 columns): 32768 tokens x 6 routes x 4096 350 -> 285 us (6.6 TB/s, a
// plain copy's rate), 16384 x 4 x 6144 226 -> 168 us, 8192 x 10 x 4096 143 -> 116 us, 1777 x 6 x
// 2688 14.4 -> 9.9 us.  The launch bounds matter: without them the compiler aims at full
// occupancy in 32 registers and takes the loads of a batch one after another.
#include "common.cuh"

namespace lm {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxTopK = 32;

struct CombineParams {
  const __nv_bfloat16* rows;
  const int32_t* slots;
  const float* weights;
  __nv_bfloat16* out;
  uint32_t vecs;  // tokens * vec_per_row
  int top_k;
  int64_t row_stride;
  int64_t out_stride;
  uint32_t vec_per_row;
  const int32_t* valid;  // optional: 0 = the rows were not computed this step, write zeros
};

// Two FP32 sums in one instruction, each rounded on its own.  (The products stay scalar: a packed
// product whose result goes into a packed sum came out fused, rounded once instead of twice.)
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t pair2(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}

// kRoutes = the routes of one batch; kExact: top_k == kRoutes, one batch and no remainder.
template <bool kWeighted, int kRoutes, bool kExact>
__global__ void __launch_bounds__(kThreads, 4) combine_kernel(CombineParams p) {
  // As a programmatic dependent the kernel may start while its predecessor drains.  The routed
  // rows are that kernel's output and are read after the wait below; slots and weights are older
  // (the dispatch wrote them before the GEMMs began) and are read while it still runs.
  const uint32_t id = blockIdx.x * kThreads + threadIdx.x;
  if (id >= p.vecs) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    return;
  }
  // vectors are numbered through all tokens, so every thread of a block has one whatever the
  // row length (a block per token and 256 vectors left a quarter of the threads of a 2688-wide
  // row idle)
  const uint32_t token = id / p.vec_per_row;
  const uint32_t col = (id - token * p.vec_per_row) * 8;
  const bool live = p.valid == nullptr || __ldg(p.valid) != 0;
  uint64_t acc[4] = {0, 0, 0, 0};

  const int top_k = kExact ? kRoutes : p.top_k;
  const int32_t* slot_ptr = p.slots + static_cast<int64_t>(token) * top_k;
  const __nv_bfloat16* rows = p.rows + col;
  // A batch's slots, then its rows and weights, are loaded together and summed in route order
  // afterwards: two memory round trips per batch instead of two per route (a decode step is a
  // handful of tokens: nothing else hides them).
  for (int j0 = 0; j0 < top_k; j0 += kRoutes) {
    int slot[kRoutes];
    uint4 row[kRoutes];
    float w[kRoutes];
#pragma unroll
    for (int j = 0; j < kRoutes; ++j)
      slot[j] = (live && (kExact || j0 + j < top_k)) ? __ldg(slot_ptr + j0 + j) : -1;
#pragma unroll
    for (int j = 0; j < kRoutes; ++j) {
      w[j] = 0.0f;
      if (kWeighted && slot[j] >= 0) w[j] = __ldg(p.weights + slot[j]);
    }
    if (j0 == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
    // Plain loads in volatile asm, not __ldg: a load the compiler knows as invariant may be
    // hoisted above the wait now that its address (the slot) is known before it, and would
    // then read rows the previous kernel has not written yet.
#pragma unroll
    for (int j = 0; j < kRoutes; ++j)
      asm volatile(
          "{\n\t.reg .pred live;\n\tsetp.ge.s32 live, %5, 0;\n\t"
          "mov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
          "@live ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
          : "=&r"(row[j].x), "=&r"(row[j].y), "=&r"(row[j].z), "=&r"(row[j].w)
          : "l"(rows + slot[j] * p.row_stride), "r"(slot[j])
          : "memory");
    // A dropped route is a row of zeros with weight zero: adding +0 changes no sum, because a
    // sum that starts at +0 and rounds to nearest is never -0.
#pragma unroll
    for (int j = 0; j < kRoutes; ++j) {
      const uint32_t words[4] = {row[j].x, row[j].y, row[j].z, row[j].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float lo = __uint_as_float(words[i] << 16);
        float hi = __uint_as_float(words[i] & 0xFFFF0000u);
        if (kWeighted) {
          lo = __fmul_rn(lo, w[j]);
          hi = __fmul_rn(hi, w[j]);
        }
        acc[i] = add2(acc[i], pair2(lo, hi));
      }
    }
    if (kExact) break;
  }
  uint4 packed;
  uint32_t* pw = reinterpret_cast<uint32_t*>(&packed);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc[i]));
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    pw[i] = *reinterpret_cast<uint32_t*>(&v);
  }
  *reinterpret_cast<uint4*>(p.out + token * p.out_stride + col) = packed;
}

template <bool kWeighted>
cudaError_t launch_combine(const cudaLaunchConfig_t& config, const CombineParams& p) {
  // The route counts of real routers are compiled in: no predicates and no idle registers for
  // routes that do not exist.  Others go through batches of eight.
  switch (p.top_k) {
    case 1: return cudaLaunchKernelEx(&config, combine_kernel<kWeighted, 1, true>, p);
    case 2: return cudaLaunchKernelEx(&config, combine_kernel<kWeighted, 2, true>, p);
    case 3: return cudaLaunchKernelEx(&config, combine_kernel<kWeighted, 3, true>, p);
    case 4: return cudaLaunchKernelEx(&config, combine_kernel<kWeighted, 4, true>, p);
    case 5: return cudaLaunchKernelEx(&config, combine_kernel<kWeighted, 5, true>, p);
    case 6: return cudaLaunchKernelEx(&config, combine_kernel<kWeighted, 6, true>, p);
    case 7: return cudaLaunchKernelEx(&config, combine_kernel<kWeighted, 7, true>, p);
    case 8: return cudaLaunchKernelEx(&config, combine_kernel<kWeighted, 8, true>, p);
    case 9: return cudaLaunchKernelEx(&config, combine_kernel<kWeighted, 9, true>, p);
    case 10: return cudaLaunchKernelEx(&config, combine_kernel<kWeighted, 10, true>, p);
    default: return cudaLaunchKernelEx(&config, combine_kernel<kWeighted, 8, false>, p);
  }
}

}  // namespace
}  // namespace lm

extern "C" int lm_finalize(const void* routed_out, const int32_t* slots, const float* weights,
                           void* out, int64_t tokens, int top_k, int hidden,
                           int64_t routed_row_stride, int64_t out_row_stride, const int32_t* valid,
                           int use_pdl, lm_stream_t stream) {
  using namespace lm;
  LM_REQUIRE(routed_out && slots && out, "finalize: null pointer");
  LM_REQUIRE(hidden > 0 && hidden % 8 == 0, "finalize: hidden must be a multiple of 8");
  LM_REQUIRE(routed_row_stride % 8 == 0 && out_row_stride % 8 == 0,
             "finalize: row strides must keep 16-byte alignment");
  LM_REQUIRE(top_k > 0 && top_k <= kMaxTopK, "finalize: top_k must be in 1..32");
  LM_REQUIRE(tokens >= 0 && tokens < (1ll << 31), "finalize: bad token count");
  if (tokens == 0) return LM_OK;
  const uint32_t vec_per_row = static_cast<uint32_t>(hidden / 8);
  // vectors are counted in 32 bits: batches beyond that go in slices of whole tokens
  const int64_t slice = 0xFFFF0000ll / vec_per_row;
  for (int64_t t0 = 0; t0 < tokens; t0 += slice) {
    const int64_t count = tokens - t0 < slice ? tokens - t0 : slice;
    CombineParams p{static_cast<const __nv_bfloat16*>(routed_out),
                    slots + t0 * top_k,
                    weights,
                    static_cast<__nv_bfloat16*>(out) + t0 * out_row_stride,
                    static_cast<uint32_t>(count * vec_per_row),
                    top_k,
                    routed_row_stride,
                    out_row_stride,
                    vec_per_row,
                    valid};
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((p.vecs + kThreads - 1) / kThreads);
    config.blockDim = dim3(kThreads);
    config.stream = as_stream(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attr;
    config.numAttrs = use_pdl ? 1 : 0;
    LM_CUDA(weights != nullptr ? launch_combine<true>(config, p) : launch_combine<false>(config, p));
    note_launch();
    LM_CUDA(cudaGetLastError());
  }
  return LM_OK;
}
