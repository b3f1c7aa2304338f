// Fused RMSNorm / residual-add RMSNorm + NVFP4 quantisation for sm_100a.
//
// Replaces the flashinfer CuTe-DSL operators the reference runs verbatim
// (call sites tests/python/test_flashinfer_norm_verbatim.py:134,155-164); the
// arithmetic contract is the reference's torch golden (same file, lines 58-99).
//
// One pass over HBM: a row is read once (x, and residual for the add variant), kept in registers across the row
// reduction, and written once (residual, e2m1 codes, e4m3 scale factors).  Each thread owns kVec adjacent 16-element
// scale blocks (one 256-bit load per block and tensor), so a block's amax, scale factor and code bytes never leave the
// thread; neighbouring lanes merge their scale bytes into one 32-bit store, which is contiguous both in the row-major
// and in the 128x4 tiled scale-factor layout.
//
// One block per row, in hardware order: several blocks share an SM, so one row's loads overlap another's reduction and
// quantisation, and the last rows spread over all SMs.  (A persistent grid that looped over rows with the weights parked
// in shared memory as f32 was 10 % slower on the largest shapes and 40 % on middle ones: a last wave that was nearly
// empty, and a launch that had to load the weights first.)  What bounds it: DRAM for the add variant -- [8192, 7168]
// bf16, 385 MB: 61 us = 6.3 TB/s as a burst (66 before), 66 in a long loop (72).  The plain one ([4096, 5120] fp16: 22.6 -> 13.7
// us; [8192, 7168] bf16: 45 -> 34 us) fills neither DRAM (3.9 TB/s, 61 % of a copy) nor the issue slots (64 % busy).
#include "common.cuh"

namespace b200fp4 {
namespace {

constexpr int kMaxUnitsPerThread = 2;    // strided units per thread per row
constexpr int kMaxThreads = 512;

struct NormParams {
  const void* x;
  void* residual;           // in/out, null for plain rmsnorm
  const void* weight;
  uint8_t* y;               // [rows, hidden/2]
  uint8_t* sf_swizzled;     // 128x4 tiled, or null
  uint8_t* sf_rowmajor;     // [rows, hidden/16], or null
  const float* global_scale;
  float eps;
  int64_t rows;
  int hidden;
  int64_t x_row_stride;     // elements
  int64_t res_row_stride;   // elements
  bool y_vec16;             // rows of y are 16-byte aligned
  bool sf_rows_vec4;        // rows of sf_rowmajor are 4-byte aligned
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Rows that only pad the last 128-row tile of tiled scale factors: their bytes read as zero.  Blocks past the last row
// of data write them, so that a call is one launch (a separate memset cost a decode-sized call a third of its time).
__device__ __forceinline__ void zero_padding_row(const NormParams& p, int64_t row, int rk, int tid, int team) {
  for (int i = tid; i < rk; i += team)
    *reinterpret_cast<uint32_t*>(p.sf_swizzled + sf_swizzled_offset(row, 4 * i, rk)) = 0u;
}

// The sum over all 32 slots of red[] in the order of a butterfly over 32 lanes (distance 16, 8, 4, 2, 1), of which only
// the first kN can be non-zero; every thread adds for itself from broadcast reads, without shuffles.
template <int kN>
__device__ __forceinline__ float butterfly_sum(const float* red) {
  float v[kN];
#pragma unroll
  for (int i = 0; i < kN; i += 4) {
    const float4 q = *reinterpret_cast<const float4*>(red + i);
    v[i] = q.x, v[i + 1] = q.y, v[i + 2] = q.z, v[i + 3] = q.w;
  }
#pragma unroll
  for (int o = kN / 2; o > 0; o >>= 1) {
#pragma unroll
    for (int i = 0; i < o; ++i) v[i] = __fadd_rn(v[i], v[i + o]);
  }
  return v[0];
}

// A "unit" is kVec adjacent 16-element chunks; thread t of a row's team handles units
// t, t+team, ... (kUnits of them).  kWarpRow: the team is one warp and a block
// works on one row per warp (hidden <= 1024); otherwise the team is the block.
template <typename T, bool kAdd, int kVec, int kUnits, bool kWarpRow, int kCap, int kMinCtas>
__global__ void __launch_bounds__(kCap, kMinCtas) norm_quant_kernel(const NormParams p) {
  constexpr int kSlots = kCap <= 256 ? 8 : 16;             // warps of a team
  __shared__ __align__(16) float red[kSlots];

  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nchunks = p.hidden >> 4;
  const int team = kWarpRow ? 32 : blockDim.x;
  const int tid = kWarpRow ? lane : threadIdx.x;
  const int rk = (nchunks + 3) >> 2;
  const int64_t row = kWarpRow ? static_cast<int64_t>(blockIdx.x) * (kCap / 32) + warp : blockIdx.x;
  if constexpr (!kWarpRow) {
    if (tid < kSlots && tid >= (team >> 5)) red[tid] = 0.0f;       // slots without a warp
  }
  // (the other way round the blocks of several calls to come line up and hold the slots: add, [128, 16384] bf16, one call after
  // the other in a graph, 6.2 us instead of 4.8)
  grid_dependency_wait();
  let_dependents_launch();
  if (row >= p.rows) {                       // only tiled outputs have blocks past the data
    if (p.sf_swizzled != nullptr && row < ((p.rows + 127) & ~int64_t{127})) zero_padding_row(p, row, rk, tid, team);
    return;
  }
  const T* xrow = static_cast<const T*>(p.x) + row * p.x_row_stride;
  T* rrow = static_cast<T*>(p.residual) + (kAdd ? row * p.res_row_stride : 0);
  const T* wg = static_cast<const T*>(p.weight);

  // ---- phase 1: load, (add, round, write residual), sum of squares; all f32 math on register pairs.  Everything the
  // thread reads from DRAM is requested before anything is used.
  U32x8 xin[kUnits * kVec], rin[kAdd ? kUnits * kVec : 1], win[kUnits * kVec];
#pragma unroll
  for (int u = 0; u < kUnits; ++u) {
#pragma unroll
    for (int v = 0; v < kVec; ++v) {
      const int c = u * kVec + v, chunk = (tid + u * team) * kVec + v;
      if (chunk < nchunks) {
        xin[c] = ld_stream_32B(xrow + chunk * 16);
        if constexpr (kAdd) rin[c] = ld_stream_32B(rrow + chunk * 16);
        else win[c] = ld_cached_32B(wg + chunk * 16);
      }
    }
  }
  const float gs = ld_word(p.global_scale);
  // what phase 2 normalises, kept as packed 16-bit pairs so that few registers live across the row reduction
  uint32_t h[kUnits * kVec][8];
  uint64_t ssq2 = 0;                         // {0.0f, 0.0f}
#pragma unroll
  for (int u = 0; u < kUnits; ++u) {
#pragma unroll
    for (int v = 0; v < kVec; ++v) {
      const int c = u * kVec + v, chunk = (tid + u * team) * kVec + v;
      if (chunk < nchunks) {
        if constexpr (kAdd) {
          U32x8 outv;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint64_t s2 = f32x2_add(pair16_to_f32x2<T>(xin[c].v[i]), pair16_to_f32x2<T>(rin[c].v[i]));
            ssq2 = f32x2_fma(s2, s2, ssq2);
            outv.v[i] = f32x2_to_pair16<T>(s2);
            h[c][i] = outv.v[i];             // the normalised value is built from the ROUNDED residual
          }
          st_32B(rrow + chunk * 16, outv);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint64_t x2 = pair16_to_f32x2<T>(xin[c].v[i]);
            ssq2 = f32x2_fma(x2, x2, ssq2);
            h[c][i] = Pack16<T>::mul(xin[c].v[i], win[c].v[i]);   // x*w is rounded to the input type before the scaling
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) h[c][i] = 0;
      }
    }
  }
  if constexpr (kAdd) {
#pragma unroll
    for (int u = 0; u < kUnits; ++u) {
#pragma unroll
      for (int v = 0; v < kVec; ++v) {
        const int c = u * kVec + v, chunk = (tid + u * team) * kVec + v;
        if (chunk < nchunks) {
          win[c] = ld_cached_32B(wg + chunk * 16);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) win[c].v[i] = 0;
        }
      }
    }
  }

  // ---- row reduction: lanes, then (CTA teams) warps through shared memory
  float ssq = warp_sum(__fadd_rn(f32x2_lo(ssq2), f32x2_hi(ssq2)));
  if constexpr (!kWarpRow) {
    if (lane == 0) red[warp] = ssq;
    __syncthreads();
    ssq = butterfly_sum<kSlots>(red);
  }
  // 1/sqrt(mean + eps) with IEEE division and square root
  const float rstd = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ssq, static_cast<float>(p.hidden)), p.eps)));
  const uint64_t rstd2 = f32x2_pack(rstd, rstd);

  // ---- phase 2: scale, quantise, store
#pragma unroll
  for (int u = 0; u < kUnits; ++u) {
    uint32_t codes[kVec][2];
    uint32_t sfb[kVec];
    const int chunk0 = (tid + u * team) * kVec;
#pragma unroll
    for (int v = 0; v < kVec; ++v) {
      const int c = u * kVec + v;
      if constexpr (kAdd) {
        uint64_t val[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
          val[i] = f32x2_mul(f32x2_mul(pair16_to_f32x2<T>(h[c][i]), rstd2), pair16_to_f32x2<T>(win[c].v[i]));
        quantize_block16<false, true>(val, gs, codes[v][0], codes[v][1], sfb[v]);
      } else {
        // h * rstd rounds monotonically in |h|, so the block's largest value comes from its largest |h|, which packed
        // 16-bit maxima find; the common factor rstd goes into the quantiser's scale.  A row with a NaN or an infinity has an
        // rstd of NaN or 0, a row of zeros with eps = 0 one of infinity: their values are NaN or zero, and a NaN is no
        // largest value (fmaxf drops it) as it is none in the other variant
        uint32_t m = Pack16<T>::max_abs(h[c][0], h[c][1]);
#pragma unroll
        for (int i = 2; i < 8; ++i) m = Pack16<T>::max_abs(m, h[c][i]);
        const float amax = fmaxf(__fmul_rn(fmaxf(Pair16<T>::lo(m), Pair16<T>::hi(m)), rstd), 0.0f);
        quantize_block16<false, true>([&](int i) { return pair16_to_f32x2<T>(h[c][i]); },
                                [&](int i) { return f32x2_mul(pair16_to_f32x2<T>(h[c][i]), rstd2); }, amax, rstd * gs, 0.0f * rstd,
                                gs, codes[v][0], codes[v][1], sfb[v]);
      }
      if (chunk0 + v >= nchunks) sfb[v] = 0;
    }
    // codes: kVec * 8 contiguous bytes per thread
    uint8_t* yrow = p.y + row * (p.hidden >> 1);
    if constexpr (kVec == 2) {
      if (chunk0 + 1 < nchunks) {
        if (p.y_vec16) {
          *reinterpret_cast<uint4*>(yrow + chunk0 * 8) = make_uint4(codes[0][0], codes[0][1], codes[1][0], codes[1][1]);
        } else {
          *reinterpret_cast<uint2*>(yrow + chunk0 * 8) = make_uint2(codes[0][0], codes[0][1]);
          *reinterpret_cast<uint2*>(yrow + chunk0 * 8 + 8) = make_uint2(codes[1][0], codes[1][1]);
        }
      } else if (chunk0 < nchunks) {
        *reinterpret_cast<uint2*>(yrow + chunk0 * 8) = make_uint2(codes[0][0], codes[0][1]);
      }
    } else {
      if (chunk0 < nchunks) *reinterpret_cast<uint2*>(yrow + chunk0 * 8) = make_uint2(codes[0][0], codes[0][1]);
    }
    // scale bytes: the lane whose first chunk is a multiple of 4 collects four K-blocks
    uint32_t quad;
    bool leader;
    if constexpr (kVec == 2) {
      const uint32_t pair = sfb[0] | (sfb[1] << 8);
      quad = pair | (__shfl_down_sync(0xffffffffu, pair, 1) << 16);
      leader = (lane & 1) == 0;
    } else {
      quad = sfb[0];
      quad |= __shfl_down_sync(0xffffffffu, sfb[0], 1) << 8;
      quad |= __shfl_down_sync(0xffffffffu, sfb[0], 2) << 16;
      quad |= __shfl_down_sync(0xffffffffu, sfb[0], 3) << 24;
      leader = (lane & 3) == 0;
    }
    if (leader && chunk0 < nchunks) {
      if (p.sf_swizzled != nullptr) *reinterpret_cast<uint32_t*>(p.sf_swizzled + sf_swizzled_offset(row, chunk0, rk)) = quad;
      if (p.sf_rowmajor != nullptr) {
        uint8_t* dst = p.sf_rowmajor + row * nchunks + chunk0;
        if (p.sf_rows_vec4) {
          *reinterpret_cast<uint32_t*>(dst) = quad;
        } else {
          for (int j = 0; j < 4 && chunk0 + j < nchunks; ++j) dst[j] = static_cast<uint8_t>(quad >> (8 * j));
        }
      }
    }
  }
}

template <typename T, bool kAdd, int kVec, int kUnits, bool kWarpRow, int kCap, int kMinCtas>
int launch_one(const NormParams& p, int threads, cudaStream_t stream) {
  const int64_t per_cta = kWarpRow ? kCap / 32 : 1;
  if (p.rows > (0x7fffffffLL - 128) * per_cta) return fail(kUnsupported, "too many rows");      // blocks of a grid
  const int64_t rows = p.sf_swizzled != nullptr ? (p.rows + 127) / 128 * 128 : p.rows;
  return check_cuda(launch_dependent(norm_quant_kernel<T, kAdd, kVec, kUnits, kWarpRow, kCap, kMinCtas>,
                                     dim3(static_cast<unsigned>((rows + per_cta - 1) / per_cta)),
                                     dim3(kWarpRow ? kCap : threads), 0, stream, p),
                    "norm_quant_kernel launch");
}

template <typename T, bool kAdd>
int dispatch(const NormParams& p, cudaStream_t stream) {
  const int nchunks = p.hidden / 16;
  // up to 1024 columns a warp holds a row (one chunk per lane, or two) and a block of four warps four rows: blocks of a
  // single warp would leave half of an SM's warp slots empty ([16384, 1024]: 18.3 -> 11.1 us plain, 21.8 -> 20.3 add)
  if (nchunks <= 32) return launch_one<T, kAdd, 1, 1, true, 128, 1>(p, 32, stream);
  const int nunits = (nchunks + 1) / 2;                       // two adjacent chunks per unit
  const int units = (nunits + kMaxThreads - 1) / kMaxThreads;
  const int threads = (((nunits + units - 1) / units) + 31) / 32 * 32;
  switch (units) {
    case 1:
      if (threads == 32) return launch_one<T, kAdd, 2, 1, true, 128, 8>(p, threads, stream);
      // resident blocks: 64 registers for the add variant (five blocks of 48 are no faster, six spill), 48 for the plain
      // one, which has half the loads ([8192, 7168]: 34 us against 38 with 64 registers)
      return threads <= 256 ? launch_one<T, kAdd, 2, 1, false, 256, kAdd ? 4 : 5>(p, threads, stream)
                            : launch_one<T, kAdd, 2, 1, false, kMaxThreads, 2>(p, threads, stream);
    case 2: return launch_one<T, kAdd, 2, 2, false, kMaxThreads, 1>(p, threads, stream);
    default: return fail(kUnsupported, "hidden=%d exceeds the supported maximum of %d", p.hidden,
                         32 * kMaxThreads * kMaxUnitsPerThread);
  }
}

}  // namespace

// sf_layout: 0 = row-major [rows, hidden/16], 1 = 128x4 tiled, 2 = both
// (tiled into block_scale, row-major into block_scale_unswizzled)
int norm_fp4quant_launch(const void* x, void* residual, const void* weight, void* y_fp4, void* block_scale,
                         void* block_scale_unswizzled, const float* global_scale, float eps, int64_t rows,
                         int hidden, int64_t x_row_stride, int64_t res_row_stride, int dtype, int sf_layout,
                         cudaStream_t stream) {
  if (x == nullptr || weight == nullptr || y_fp4 == nullptr || block_scale == nullptr || global_scale == nullptr)
    return fail(kInvalidArgument, "null pointer argument");
  if (rows < 0) return fail(kInvalidArgument, "rows=%lld is negative", static_cast<long long>(rows));
  if (hidden < 64 || hidden % 16 != 0)
    return fail(kInvalidArgument, "hidden=%d must be a multiple of 16 and at least 64", hidden);
  if (x_row_stride % 16 != 0 || (residual != nullptr && res_row_stride % 16 != 0))
    return fail(kInvalidArgument, "row strides must be multiples of 16 elements (32-byte rows)");
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(weight)) & 31)
    return fail(kInvalidArgument, "input, residual and weight must be 32-byte aligned");
  if ((reinterpret_cast<uintptr_t>(y_fp4) & 7) || (reinterpret_cast<uintptr_t>(block_scale) & 3))
    return fail(kInvalidArgument, "y_fp4 must be 8-byte and block_scale 4-byte aligned");
  if (dtype != 0 && dtype != 1) return fail(kUnsupported, "dtype code %d (0 = fp16, 1 = bf16)", dtype);
  if (sf_layout < 0 || sf_layout > 2) return fail(kInvalidArgument, "sf_layout=%d", sf_layout);
  if (sf_layout == 2 && block_scale_unswizzled == nullptr)
    return fail(kInvalidArgument, "sf_layout=2 needs block_scale_unswizzled");
  if (rows == 0) return kOk;

  NormParams p{};
  p.x = x;
  p.residual = residual;
  p.weight = weight;
  p.y = static_cast<uint8_t*>(y_fp4);
  p.sf_swizzled = sf_layout >= 1 ? static_cast<uint8_t*>(block_scale) : nullptr;
  p.sf_rowmajor = sf_layout == 0 ? static_cast<uint8_t*>(block_scale)
                                 : (sf_layout == 2 ? static_cast<uint8_t*>(block_scale_unswizzled) : nullptr);
  p.global_scale = global_scale;
  p.eps = eps;
  p.rows = rows;
  p.hidden = hidden;
  p.x_row_stride = x_row_stride;
  p.res_row_stride = res_row_stride;

  p.y_vec16 = hidden % 32 == 0 && (reinterpret_cast<uintptr_t>(y_fp4) & 15) == 0;
  p.sf_rows_vec4 = hidden % 64 == 0 && (reinterpret_cast<uintptr_t>(p.sf_rowmajor) & 3) == 0;
  const bool add = residual != nullptr;
  if (dtype == 1) return add ? dispatch<__nv_bfloat16, true>(p, stream) : dispatch<__nv_bfloat16, false>(p, stream);
  return add ? dispatch<__half, true>(p, stream) : dispatch<__half, false>(p, stream);
}

}  // namespace b200fp4
