// Row-wise BF16/FP32 -> NVFP4 quantization (HBM-bound).
//
// One CTA covers one 128-row scale-factor atom row and 512 features.  A warp
// streams row slices of 512 features: each lane owns one 16-element group (32 B of
// BF16), so a warp reads 1 KB contiguous and writes 256 B of packed codes.
// Scale factors are staged in shared memory in atom order and leave the CTA as
// 16-byte stores, so every 512-byte atom is written whole.
#include "common.cuh"
#include "quantize_math.cuh"

namespace lm {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kTileRows = 128;
constexpr int kTileCols = 512;  // 32 lanes x 16 elements

struct QuantParams {
  const void* x;
  int64_t rows;
  int features;
  const int32_t* m_indptr;
  int experts;
  int64_t rows_per_group;
  int tiles_per_group;
  const float* scale_pair;
  int scale_alone;  // scale_pair holds the scale only: its reciprocal is taken here
  const int32_t* gather;
  uint8_t* q;
  uint8_t* sf;
  int sf_mode;
  int te_math;
  uint32_t col_chunks;  // 512-feature chunks of a row
  int wide_loads;       // x is 32-byte aligned
};

// What bounds it: one read of the input, one write of the codes.  Each warp keeps a ring of row
// slices whose loads are in flight while it converts the oldest one, and the first loads leave
// before anything else is looked up; consecutive CTAs take the column chunks of the same rows.
// Instructions come close behind: the two divisions of a group's scale factor and the one behind it
// were a third of them, so the byte is decided by a product wherever that is certain
// (`divided_scale_factor`) and the codes' factor, one of 126 values, is read from a table.
// 128 x 1024 x 2048 BF16 weights with their 8192 x 2048 activations 154 -> 129 us (5.7 TB/s), 8192
// x 4096 24.5 -> 21.4 us, 4730 x 4288 with 6 x 640 x 4288 36.5 -> 24.7 us.
template <typename In, bool kGather, bool kTe>
__global__ void __launch_bounds__(kThreads, 4) quantize_rowwise_kernel(QuantParams p) {
  // an atom every 528 bytes: the eight atoms a warp writes one byte quad to lie in eight banks
  constexpr int kAtomPitch = 512 + 16;
  __shared__ __align__(16) uint8_t s_sf[(kTileCols / 64) * kAtomPitch];
  __shared__ int s_group[2];  // varlen: first row, valid rows
  __shared__ float s_factor[128];  // the codes' factor for every scale-factor byte

  const int tid = threadIdx.x;
  const uint32_t chunk = blockIdx.x % p.col_chunks;
  const int64_t atom_row = blockIdx.x / p.col_chunks;
  const int col0 = static_cast<int>(chunk) * kTileCols;

  // ---- which rows does this atom row hold?
  int64_t row0;
  int valid;
  if (p.sf_mode == LM_SF_VARLEN) {
    if (tid == 0) s_group[1] = 0;
    __syncthreads();
    for (int e = tid; e < p.experts; e += kThreads) {
      int lo = __ldg(p.m_indptr + e);
      int hi = __ldg(p.m_indptr + e + 1);
      int64_t first = lo / kTileRows + e;
      int64_t next = hi / kTileRows + e + 1;
      if (atom_row >= first && atom_row < next) {
        int lt = static_cast<int>(atom_row - first);
        int remaining = (hi - lo) - lt * kTileRows;
        if (remaining > 0) {
          s_group[0] = lo + lt * kTileRows;
          s_group[1] = remaining < kTileRows ? remaining : kTileRows;
        }
      }
    }
    __syncthreads();
    row0 = s_group[0];
    valid = s_group[1];
    if (valid == 0) return;
  } else {
    const int64_t group = p.sf_mode == LM_SF_BATCHED ? atom_row / p.tiles_per_group : 0;
    const int64_t lt = atom_row - group * p.tiles_per_group;
    const int64_t group_rows = p.sf_mode == LM_SF_BATCHED ? p.rows_per_group : p.rows;
    const int64_t remaining = group_rows - lt * kTileRows;
    row0 = group * p.rows_per_group + lt * kTileRows;
    valid = remaining < kTileRows ? static_cast<int>(remaining) : kTileRows;
  }

  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int col = col0 + lane * 16;
  const bool col_ok = col < p.features;
  const In* x = static_cast<const In*>(p.x) + col;

  // The warp owns rows warp, warp + 8, ...; with a gather lane i fetches the source row of the
  // i-th of them up front, so no row load waits on an index load.
  constexpr int kRowsPerWarp = kTileRows / kWarps;
  int64_t my_src = 0;
  if (kGather) {
    const int r = warp + lane * kWarps;
    if (lane < kRowsPerWarp && r < valid) my_src = __ldg(p.gather + row0 + r);
  }
  constexpr int kRing = Slice<In>::kRing;
  Slice<In> v[kRing];
  auto fetch = [&](Slice<In>& s, int i) {
    const int r = warp + i * kWarps;
    const int64_t src = kGather ? __shfl_sync(0xFFFFFFFFu, my_src, i) : row0 + r;
    if (col_ok && r < valid) s.load(x + src * p.features, p.wide_loads);
  };
#pragma unroll
  for (int i = 0; i < kRing; ++i) fetch(v[i], i);

  const float pts = __ldg(p.scale_pair);
  const float inv_pts = p.scale_alone ? __fdiv_rn(1.0f, pts) : __ldg(p.scale_pair + 1);
  const bool blocked = p.sf_mode != LM_SF_LINEAR;
  const int groups_per_row = p.features >> 4;
  if (blocked && valid < kTileRows) {
    uint4* z = reinterpret_cast<uint4*>(s_sf);
    for (int i = tid; i < static_cast<int>(sizeof(s_sf) / 16); i += kThreads) z[i] = make_uint4(0, 0, 0, 0);
  }
  if (tid < 128) s_factor[tid] = group_factor(e4m3_to_f32(tid), pts, inv_pts, kTe);
  const float approx = kTe ? __fmul_rn(inv_pts, inv6()) : __fdiv_rn(1.0f, __fmul_rn(kF4Max, pts));
  const bool fast = pts >= 1e-30f && pts <= 1e30f;
  __syncthreads();

  uint8_t* const sf_lane = s_sf + (lane >> 2) * kAtomPitch + (lane & 3);
  uint8_t* q_row = p.q + (row0 + warp) * (p.features >> 1) + (col >> 1);
#pragma unroll
  for (int i = 0; i < kRowsPerWarp; ++i) {
    const int r = warp + i * kWarps;
    if (col_ok && r < valid) {
      const float amax = v[i % kRing].amax();
      const uint32_t sf_byte = kTe ? f32_to_e4m3(fmaxf(fminf(__fmul_rn(amax, approx), kE4M3Max), kE4M3MinSf))
                                   : divided_scale_factor(amax, pts, approx, fast);
      *reinterpret_cast<uint2*>(q_row) = group_codes(v[i % kRing], s_factor[sf_byte]);
      if (blocked) {
        sf_lane[(r & 31) * 16 + (r >> 5) * 4] = static_cast<uint8_t>(sf_byte);
      } else {
        p.sf[(row0 + r) * groups_per_row + (col >> 4)] = static_cast<uint8_t>(sf_byte);
      }
    }
    q_row += static_cast<int64_t>(kWarps) * (p.features >> 1);
    if (i + kRing < kRowsPerWarp) fetch(v[i % kRing], i + kRing);
  }
  if (!blocked) return;
  __syncthreads();

  // ---- atoms leave as 16-byte stores: thread i -> atom i / 32, piece i % 32
  const int atom_cols = p.features >> 6;
  const int atom = tid >> 5;
  const int atom_col = (col0 >> 6) + atom;
  if (atom_col < atom_cols) {
    const uint4 piece = *reinterpret_cast<const uint4*>(s_sf + atom * kAtomPitch + lane * 16);
    uint8_t* dst = p.sf + (atom_row * atom_cols + atom_col) * 512 + lane * 16;
    *reinterpret_cast<uint4*>(dst) = piece;
  }
}

template <typename In>
void launch_rowwise(unsigned grid, cudaStream_t stream, const QuantParams& p) {
  if (p.gather != nullptr) {
    if (p.te_math) {
      quantize_rowwise_kernel<In, true, true><<<grid, kThreads, 0, stream>>>(p);
    } else {
      quantize_rowwise_kernel<In, true, false><<<grid, kThreads, 0, stream>>>(p);
    }
  } else if (p.te_math) {
    quantize_rowwise_kernel<In, false, true><<<grid, kThreads, 0, stream>>>(p);
  } else {
    quantize_rowwise_kernel<In, false, false><<<grid, kThreads, 0, stream>>>(p);
  }
}

// ------------------------------------------------- quantize once, scatter to slots
// A warp owns 1024 features of one token: it works out the token's destinations (one row per
// route), quantizes its features once -- 32 neighbouring ones a lane -- and writes the packed
// codes (512 B, one store of 16 B a lane) and the scale factors (sixteen 4-byte words, one per
// 64-feature atom) to every expert-major row the token was routed to.
// What bounds it: the instructions around the stores (shuffles that hand the destinations round,
// and the load/store unit's work on the scattered scale-factor words), then the writes.  So a warp
// takes as many features per destination as its lanes can store in one instruction each, and the
// slices of a token are dealt to different warps, which also fills the chip for short batches.
// Against a warp a token in 512-feature slices: 320 tokens x 4 routes x 6144 10.9 -> 4.7 us, 270 x 6 x
// 3840 8.3 -> 3.6 us, 16384 x 4 x 6144 88 -> 83 us, 32768 x 6 x 4096 183 -> 173 us (4.2 TB/s).
struct ScatterQuantParams {
  const __nv_bfloat16* x;
  int64_t tokens;
  int features;
  int top_k;
  const int32_t* slots;
  const int32_t* topk_ids;
  const int32_t* m_indptr;
  const float* scale_pair;
  uint8_t* q;
  uint8_t* sf;
  uint32_t slices;  // 1024-feature slices of a row
  int wide_loads;   // x is 32-byte aligned
  int wide_stores;  // q is 16-byte aligned (8 is all that callers promise)
  uint8_t* sf_tokens;  // token-major scale factors, (tokens, features / 16)
};

constexpr int64_t kTokenSfWords = 7 << 16;  // 4-byte words to save before scale factors go by way of the tokens
constexpr int kScatterCols = 1024;  // features of a warp: 32 lanes x two groups of 16

// kTokenSf: the scale factors are written once a token, token-major; `sf_gather_kernel` takes them to
// the atoms of its rows.
// kChained: a programmatic dependent of the dispatch.  The token is read and quantized beside it;
// slots and bounds, which it writes, are read after the wait.  (Otherwise they are read first: their
// round trips hide behind the token's.)
template <bool kTokenSf, bool kChained>
__global__ void __launch_bounds__(kThreads) quantize_scatter_kernel(ScatterQuantParams p) {
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // consecutive blocks take the slices of the same eight tokens
  const uint32_t token_block = blockIdx.x / p.slices;
  const int64_t token = static_cast<int64_t>(token_block) * kWarps + warp;
  if (token >= p.tokens) return;
  const int col = static_cast<int>(blockIdx.x - token_block * p.slices) * kScatterCols + lane * 32;
  const bool col_ok = col < p.features;
  Slice<__nv_bfloat16> v[2];
  if (col_ok) {
    const __nv_bfloat16* src = p.x + token * p.features + col;
    v[0].load(src, p.wide_loads);
    v[1].load(src + 16, p.wide_loads);
  }
  // Destination of route `lane` (lanes beyond top_k idle): its row, and the atom row and the
  // 4-byte word inside each 512-byte atom that hold the row's scale factors.
  const int atom_cols = p.features >> 6;
  int my_slot = -1;
  uint32_t my_sf = 0;
  auto find_rows = [&]() {
    if (lane >= p.top_k) return;
    // (chained: volatile loads, one that the compiler knows as invariant could move above the wait)
    auto load = [](const int32_t* at) {
      return kChained ? *reinterpret_cast<const volatile int32_t*>(at) : __ldg(at);
    };
    my_slot = load(p.slots + token * p.top_k + lane);
    const int e = __ldg(p.topk_ids + token * p.top_k + lane);
    if (my_slot >= 0) {
      const int lo = load(p.m_indptr + e);
      const int local = my_slot - lo;
      const uint32_t atom_row = lo / kTileRows + e + local / kTileRows;
      const int r = local % kTileRows;
      my_sf = atom_row * 128 + (r & 31) * 4 + (r >> 5);
    }
  };
  if (!kChained) find_rows();
  const float pts = __ldg(p.scale_pair);
  const float inv_pts = __ldg(p.scale_pair + 1);
  uint2 packed[2] = {make_uint2(0, 0), make_uint2(0, 0)};
  uint32_t word = 0;
  if (col_ok) {
    word = quantize_group(v[0], pts, inv_pts, true, &packed[0]);
    word |= quantize_group(v[1], pts, inv_pts, true, &packed[1]) << 8;
  }
  // two neighbouring lanes hold the four factors of one atom word
  word |= __shfl_down_sync(0xFFFFFFFFu, word, 1) << 16;
  if (kChained) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    find_rows();
  }
  uint8_t* const q = p.q + (col >> 1);
  uint8_t* const sf = p.sf + static_cast<int64_t>(col >> 6) * 512;
  const int64_t q_pitch = p.features >> 1;
  const int64_t sf_pitch = static_cast<int64_t>(atom_cols) * 512;
  const bool sf_lane = col_ok && (lane & 1) == 0;
  if (kTokenSf && sf_lane)
    *reinterpret_cast<uint32_t*>(p.sf_tokens + token * (p.features >> 4) + (col >> 4)) = word;
#pragma unroll 2
  for (int j = 0; j < p.top_k; ++j) {
    const int slot = __shfl_sync(0xFFFFFFFFu, my_slot, j);
    const uint32_t at = kTokenSf ? 0 : __shfl_sync(0xFFFFFFFFu, my_sf, j);
    if (slot < 0) continue;
    if (col_ok) {
      uint8_t* const dst = q + slot * q_pitch;
      if (p.wide_stores) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(packed[0].x, packed[0].y, packed[1].x, packed[1].y);
      } else {
        reinterpret_cast<uint2*>(dst)[0] = packed[0];
        reinterpret_cast<uint2*>(dst)[1] = packed[1];
      }
    }
    if (!kTokenSf && sf_lane) *reinterpret_cast<uint32_t*>(sf + (at >> 7) * sf_pitch + (at & 127) * 4) = word;
  }
}

// ------------------------------------------------- scale factors of tokens to the atoms of their rows
// A block makes 32 atoms (2048 features) of one 128-row atom row: a warp reads the factors of rows
// r, r + 32, r + 64 and r + 96 (128 bytes a row, 4 bytes a lane = one atom's word), which are the 16
// bytes of unit r of every atom, and the atoms leave whole.  The scattered 4-byte words that
// this stands in for cost as much as all other bytes of the quantizer: sixteen partial sectors a
// route and slice.  Both launches together against the scattered words: 32768 tokens x 6 x 4096 171 ->
// 120 us, 16384 x 4 x 6144 83 -> 70 us, 8192 x 10 x 4096 57 -> 44 us, 8192 x 8 x 2048 24 -> 20 us.
struct SfGatherParams {
  const uint8_t* sf_tokens;
  const int32_t* gather;
  const int32_t* m_indptr;
  int experts;
  int atom_cols;
  uint32_t chunks;  // 32-atom chunks of an atom row
  uint8_t* sf;
};

__global__ void __launch_bounds__(kThreads) sf_gather_kernel(SfGatherParams p) {
  constexpr int kAtoms = 32;
  constexpr int kPitch = 512 + 16;  // sixteen-byte units of neighbouring atoms in neighbouring bank groups
  __shared__ __align__(16) uint8_t s_sf[kAtoms * kPitch];
  __shared__ int s_token[kTileRows];
  __shared__ int s_group[2];  // first row, valid rows
  const int tid = threadIdx.x;
  const int64_t atom_row = blockIdx.x / p.chunks;
  const int atom0 = static_cast<int>(blockIdx.x % p.chunks) * kAtoms;
  if (tid == 0) s_group[1] = 0;
  __syncthreads();
  for (int e = tid; e < p.experts; e += kThreads) {
    const int lo = __ldg(p.m_indptr + e), hi = __ldg(p.m_indptr + e + 1);
    const int64_t first = lo / kTileRows + e;
    if (atom_row >= first && atom_row < hi / kTileRows + e + 1) {
      const int lt = static_cast<int>(atom_row - first);
      const int remaining = (hi - lo) - lt * kTileRows;
      if (remaining > 0) {
        s_group[0] = lo + lt * kTileRows;
        s_group[1] = min(remaining, kTileRows);
      }
    }
  }
  __syncthreads();
  const int row0 = s_group[0], valid = s_group[1];
  if (valid == 0) return;
  if (tid < kTileRows) s_token[tid] = tid < valid ? __ldg(p.gather + row0 + tid) : -1;
  __syncthreads();

  const int warp = tid >> 5, lane = tid & 31;
  const int atom = atom0 + lane;
  const int64_t pitch = static_cast<int64_t>(p.atom_cols) * 4;
  const uint8_t* src = p.sf_tokens + static_cast<int64_t>(atom) * 4;
  uint32_t w[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int token = s_token[warp + i * kWarps + j * 32];
      w[i][j] = token >= 0 && atom < p.atom_cols ? __ldg(reinterpret_cast<const uint32_t*>(src + token * pitch)) : 0;
    }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<uint4*>(s_sf + lane * kPitch + (warp + i * kWarps) * 16) =
        make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kAtoms / kWarps; ++i) {
    const int a = warp + i * kWarps;
    if (atom0 + a < p.atom_cols)
      *reinterpret_cast<uint4*>(p.sf + (atom_row * p.atom_cols + atom0 + a) * 512 + lane * 16) =
          *reinterpret_cast<const uint4*>(s_sf + a * kPitch + lane * 16);
  }
}

}  // namespace
}  // namespace lm

namespace lm {
namespace {

int quantize_rows(const void* x, int x_dtype, int64_t rows, int features, const int32_t* m_indptr, int experts,
                  int64_t rows_per_group, const float* scale_pair, int scale_alone, const int32_t* gather_idx,
                  uint8_t* q, uint8_t* sf, int sf_mode, int te_math, lm_stream_t stream) {
  LM_REQUIRE(x && scale_pair && q && sf, "quantize: null pointer");
  LM_REQUIRE(x_dtype == LM_DTYPE_BF16 || x_dtype == LM_DTYPE_F32, "quantize: x must be BF16 or FP32");
  LM_REQUIRE(features > 0 && features % 64 == 0, "quantize: features must be a multiple of 64");
  LM_REQUIRE(rows >= 0, "quantize: negative row count");
  LM_REQUIRE(sf_mode >= LM_SF_VARLEN && sf_mode <= LM_SF_LINEAR, "quantize: unknown sf_mode");
  if (rows == 0) return LM_OK;
  QuantParams p{};
  p.x = x;
  p.rows = rows;
  p.features = features;
  p.m_indptr = m_indptr;
  p.experts = experts;
  p.rows_per_group = rows_per_group;
  p.scale_pair = scale_pair;
  p.scale_alone = scale_alone;
  p.gather = gather_idx;
  p.q = q;
  p.sf = sf;
  p.sf_mode = sf_mode;
  p.te_math = te_math;
  int64_t atom_rows;
  if (sf_mode == LM_SF_VARLEN) {
    LM_REQUIRE(m_indptr != nullptr && experts > 0, "quantize: varlen layout needs m_indptr");
    atom_rows = (rows + 127) / 128 + experts;
  } else if (sf_mode == LM_SF_BATCHED) {
    LM_REQUIRE(rows_per_group > 0 && rows % rows_per_group == 0,
               "quantize: rows must be a multiple of rows_per_group");
    p.tiles_per_group = static_cast<int>((rows_per_group + 127) / 128);
    atom_rows = (rows / rows_per_group) * p.tiles_per_group;
  } else {
    atom_rows = (rows + 127) / 128;
  }
  p.col_chunks = static_cast<uint32_t>((features + kTileCols - 1) / kTileCols);
  LM_REQUIRE(atom_rows * p.col_chunks < (1ll << 31), "quantize: too many rows");
  p.wide_loads = (reinterpret_cast<uintptr_t>(x) & 31) == 0;
  const unsigned grid = static_cast<unsigned>(atom_rows * p.col_chunks);
  if (x_dtype == LM_DTYPE_BF16) {
    launch_rowwise<__nv_bfloat16>(grid, as_stream(stream), p);
  } else {
    launch_rowwise<float>(grid, as_stream(stream), p);
  }
  note_launch();
  LM_CUDA(cudaGetLastError());
  return LM_OK;
}

}  // namespace
}  // namespace lm

extern "C" int lm_quantize_rowwise(const void* x, int x_dtype, int64_t rows, int features,
                                   const int32_t* m_indptr, int experts, int64_t rows_per_group,
                                   const float* scale_pair, const int32_t* gather_idx, uint8_t* q,
                                   uint8_t* sf, int sf_mode, int te_math, lm_stream_t stream) {
  return lm::quantize_rows(x, x_dtype, rows, features, m_indptr, experts, rows_per_group, scale_pair, 0, gather_idx,
                           q, sf, sf_mode, te_math, stream);
}

extern "C" int lm_quantize_rowwise_scale(const void* x, int x_dtype, int64_t rows, int features,
                                         const int32_t* m_indptr, int experts, int64_t rows_per_group,
                                         const float* scale, const int32_t* gather_idx, uint8_t* q,
                                         uint8_t* sf, int sf_mode, int te_math, lm_stream_t stream) {
  return lm::quantize_rows(x, x_dtype, rows, features, m_indptr, experts, rows_per_group, scale, 1, gather_idx, q,
                           sf, sf_mode, te_math, stream);
}

extern "C" int lm_quantize_decode(const void* x, int64_t tokens, int features, int top_k,
                                  const int32_t* slots, const int32_t* topk_ids,
                                  const int32_t* m_indptr, int experts, const float* scale_pair,
                                  uint8_t* q, uint8_t* sf, lm_stream_t stream) {
  return lm::quantize_scatter(x, tokens, features, top_k, slots, topk_ids, m_indptr, experts, scale_pair, q, sf,
                              nullptr, nullptr, stream);
}

int lm::quantize_scatter(const void* x, int64_t tokens, int features, int top_k, const int32_t* slots,
                         const int32_t* topk_ids, const int32_t* m_indptr, int experts, const float* scale_pair,
                         uint8_t* q, uint8_t* sf, const int32_t* gather, uint8_t* sf_tokens, lm_stream_t stream) {
  LM_REQUIRE(x && slots && topk_ids && m_indptr && scale_pair && q && sf, "quantize_decode: null pointer");
  LM_REQUIRE(features > 0 && features % 64 == 0, "quantize_decode: features must be a multiple of 64");
  LM_REQUIRE(top_k > 0 && tokens >= 0, "quantize_decode: bad sizes");
  if (tokens == 0) return LM_OK;
  LM_REQUIRE(top_k <= 32, "quantize_decode: top_k must be at most 32");
  const int64_t slices = (features + kScatterCols - 1) / kScatterCols;
  const int64_t blocks = (tokens + kWarps - 1) / kWarps * slices;
  LM_REQUIRE(blocks < (1ll << 31), "quantize_decode: too many tokens");
  ScatterQuantParams p{static_cast<const __nv_bfloat16*>(x), tokens, features, top_k, slots,
                       topk_ids, m_indptr, scale_pair, q, sf, static_cast<uint32_t>(slices),
                       (reinterpret_cast<uintptr_t>(x) & 31) == 0, (reinterpret_cast<uintptr_t>(q) & 15) == 0,
                       sf_tokens};
  // Scale factors by way of the tokens take a second launch, about 2 us of a step beside the chained
  // form below.  What they save grows with the 4-byte words a step would scatter, a share of
  // 1 - 2 / top_k of them: each token's own words are written and read back instead.  Whole steps, hidden
  // 1024 to 6144, scattered against by way of the tokens: two routes never gain (1 us lost at 2 M
  // words); three break even at 1.1 M words and gain 1 to 3 us at 1.5 M; four break even at 0.75 M
  // (16384 rows x 1024, 0.25 M: 45.1 / 47.2 us; 65536 x 2048, 2 M: 180.2 / 176.6 us); eight and ten at about
  // 0.5 M (16384 x 2048, 0.5 M: 63.4 / 65.0 us; 8192 x 6144, 0.75 M: 96.4 / 92.3 us).
  const int64_t rows = tokens * top_k;
  const bool by_token = sf_tokens != nullptr && gather != nullptr &&
                        rows * (features / 64) * (top_k - 2) >= kTokenSfWords * top_k;
  if (by_token) {
    quantize_scatter_kernel<true, false><<<static_cast<unsigned>(blocks), kThreads, 0, as_stream(stream)>>>(p);
    note_launch();
    LM_CUDA(cudaGetLastError());
    SfGatherParams g{sf_tokens, gather, m_indptr, experts, features / 64,
                     static_cast<uint32_t>((features / 64 + 31) / 32), sf};
    const int64_t atom_rows = (rows + kTileRows - 1) / kTileRows + experts;
    LM_REQUIRE(atom_rows * g.chunks < (1ll << 31), "quantize_decode: too many tokens");
    sf_gather_kernel<<<static_cast<unsigned>(atom_rows * g.chunks), kThreads, 0, as_stream(stream)>>>(g);
  } else if (gather != nullptr && blocks <= 6ll * sm_count()) {
    // Inside a layer step (`gather`: the dispatch that fills the slots has just been launched, and x is
    // older), chained to the dispatch while all blocks are resident at once: they then wait with
    // their codes ready.  In a larger grid the waiting blocks take issue slots from the dispatch and
    // hide nothing of the rest (8192 tokens x 8 on 256 experts: a step 2 % slower).  1777 tokens x 6 on 8
    // experts: a step 103.5 -> 101.8 us.
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(static_cast<unsigned>(blocks));
    config.blockDim = dim3(kThreads);
    config.stream = as_stream(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attr;
    config.numAttrs = 1;
    LM_CUDA(cudaLaunchKernelEx(&config, quantize_scatter_kernel<false, true>, p));
  } else {
    quantize_scatter_kernel<false, false><<<static_cast<unsigned>(blocks), kThreads, 0, as_stream(stream)>>>(p);
  }
  note_launch();
  LM_CUDA(cudaGetLastError());
  return LM_OK;
}
