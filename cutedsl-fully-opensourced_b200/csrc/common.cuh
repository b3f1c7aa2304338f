// Shared device helpers for the sm_100a NVFP4 kernels: error plumbing, wide
// global-memory accesses, scalar-format conversions and the 16-element NVFP4
// block quantiser whose rounding rules follow the reference's torch golden
// (tests/python/test_flashinfer_norm_verbatim.py:47-68 and, for the MoE
// activation packer, tests/python/test_flashinfer_b12x_verbatim.py:28-65).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp4.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200fp4 {

// ---------------------------------------------------------------------------
// host-side error reporting (defined in capi.cu)
// ---------------------------------------------------------------------------
enum Status : int {
  kOk = 0,
  kInvalidArgument = 1,
  kUnsupported = 2,
  kCudaError = 3,
  kDeviceTimeout = 4,
  kNotInitialised = 5,
};

int fail(int code, const char* fmt, ...);
int check_cuda(cudaError_t e, const char* what);

#define B200_CUDA(call)                                         \
  do {                                                          \
    int _rc = ::b200fp4::check_cuda((call), #call);             \
    if (_rc) return _rc;                                        \
  } while (0)

// ---------------------------------------------------------------------------
// 32-byte global accesses (one instruction per 16 half-precision elements)
// ---------------------------------------------------------------------------
struct alignas(32) U32x8 {
  uint32_t v[8];
};

// No load here is .nc (nor __ldg, nor through a const __restrict__ parameter of a kernel that is launched as a dependent):
// such a kernel is already running while its predecessor still writes, and a load that is promised read-only data may be
// moved above the wait for that predecessor.
// streamed once: bypass L1 allocation
__device__ __forceinline__ U32x8 ld_stream_32B(const void* p) {
  U32x8 r;
  asm volatile("ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
                 "=r"(r.v[6]), "=r"(r.v[7])
               : "l"(p)
               : "memory");
  return r;
}

// one word of a table or a scale
template <typename T>
__device__ __forceinline__ T ld_word(const T* p) {
  static_assert(sizeof(T) == 4, "words");
  uint32_t v;
  asm volatile("ld.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  T r;
  memcpy(&r, &v, 4);
  return r;
}

// What a kernel reads BEFORE its own grid_dependency_wait() (see there): from L2, whatever a line of an earlier launch in
// this SM's L1 may hold.
template <typename T>
__device__ __forceinline__ T ld_early_word(const T* p) {
  static_assert(sizeof(T) == 4, "words");
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  T r;
  memcpy(&r, &v, 4);
  return r;
}
__device__ __forceinline__ U32x8 ld_early_32B(const void* p) {
  U32x8 r;
  asm volatile("ld.relaxed.gpu.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
                 "=r"(r.v[6]), "=r"(r.v[7])
               : "l"(p)
               : "memory");
  return r;
}

// read again by other blocks of the SM: through L1
__device__ __forceinline__ U32x8 ld_cached_32B(const void* p) {
  U32x8 r;
  asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
                 "=r"(r.v[6]), "=r"(r.v[7])
               : "l"(p)
               : "memory");
  return r;
}

// 16 bytes that nobody reads again: they leave L2 first (the per-slot rows of a prefill step are larger than L2, and what
// of them is still there need not push out the next step's data: 0.6 % of the step)
__device__ __forceinline__ uint4 ld_once_16B(const void* p) {
  uint4 r;
  uint64_t policy;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v4.b32 {%0, %1, %2, %3}, [%4], %5;"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "l"(p), "l"(policy)
               : "memory");
  return r;
}

// the 128-byte line at p (aligned) holds nothing that anybody will read: if it is dirty in L2 it need not go to DRAM
__device__ __forceinline__ void discard_l2_line(const void* p) {
  asm volatile("discard.global.L2 [%0], 128;" ::"l"(p) : "memory");
}

__device__ __forceinline__ void st_32B(void* p, const U32x8& r) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r.v[0]), "r"(r.v[1]),
               "r"(r.v[2]), "r"(r.v[3]), "r"(r.v[4]), "r"(r.v[5]), "r"(r.v[6]), "r"(r.v[7])
               : "memory");
}

// ---------------------------------------------------------------------------
// 16-bit float pairs <-> f32
// ---------------------------------------------------------------------------
template <typename T>
struct Pair16;

template <>
struct Pair16<__nv_bfloat16> {
  static __device__ __forceinline__ float lo(uint32_t u) { return __uint_as_float(u << 16); }
  static __device__ __forceinline__ float hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }
  // two f32 -> packed pair, round-to-nearest-even each
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
  }
};

template <>
struct Pair16<__half> {
  static __device__ __forceinline__ float lo(uint32_t u) {
    return __half2float(__ushort_as_half(static_cast<unsigned short>(u & 0xffffu)));
  }
  static __device__ __forceinline__ float hi(uint32_t u) {
    return __half2float(__ushort_as_half(static_cast<unsigned short>(u >> 16)));
  }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
  }
};

// both halves of a packed 16-bit pair as one f32x2 register pair (defined after f32x2_pack)
template <typename T>
__device__ __forceinline__ uint64_t pair16_to_f32x2(uint32_t u);

template <typename T>
__device__ __forceinline__ T to_out(float v);
template <>
__device__ __forceinline__ __nv_bfloat16 to_out<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ __half to_out<__half>(float v) { return __float2half_rn(v); }

// ---------------------------------------------------------------------------
// packed f32x2 arithmetic (sm_100): two IEEE round-to-nearest f32 operations per instruction,
// operands are register pairs viewed as one 64-bit value {lo, hi}
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t f32x2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float f32x2_lo(uint64_t v) { return __uint_as_float(static_cast<uint32_t>(v)); }
__device__ __forceinline__ float f32x2_hi(uint64_t v) { return __uint_as_float(static_cast<uint32_t>(v >> 32)); }
__device__ __forceinline__ uint64_t f32x2_mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f32x2_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f32x2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

template <typename T>
__device__ __forceinline__ uint64_t pair16_to_f32x2(uint32_t u) {
  return f32x2_pack(Pair16<T>::lo(u), Pair16<T>::hi(u));
}
// f32x2 -> packed 16-bit pair, round-to-nearest-even each
template <typename T>
__device__ __forceinline__ uint32_t f32x2_to_pair16(uint64_t v) {
  return Pair16<T>::pack(f32x2_lo(v), f32x2_hi(v));
}

// ---------------------------------------------------------------------------
// packed 16-bit arithmetic: a product of two 16-bit floats rounded once to the type (the same bits as the f32 product,
// which is exact, rounded to the type), and the largest magnitudes of two pairs
// ---------------------------------------------------------------------------
template <typename T>
struct Pack16;
template <>
struct Pack16<__nv_bfloat16> {
  static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
  }
  static __device__ __forceinline__ uint32_t max_abs(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("{\n.reg .b32 x, y;\nabs.bf16x2 x, %1;\nabs.bf16x2 y, %2;\nmax.bf16x2 %0, x, y;\n}" : "=r"(r) : "r"(a), "r"(b));
    return r;
  }
};
template <>
struct Pack16<__half> {
  static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
  }
  static __device__ __forceinline__ uint32_t max_abs(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("{\n.reg .b32 x, y;\nabs.f16x2 x, %1;\nabs.f16x2 y, %2;\nmax.f16x2 %0, x, y;\n}" : "=r"(r) : "r"(a), "r"(b));
    return r;
  }
};

// ---------------------------------------------------------------------------
// programmatic dependent launch: a kernel launched with the attribute may start while the kernel before it in the
// stream drains.  grid_dependency_wait() returns when that kernel is complete and its writes are visible: nothing that
// an earlier kernel may write or read is touched before it.  let_dependents_launch() lets the next kernel's blocks be
// scheduled as soon as every block of this one has called it (or has exited).
// A few reads come before a kernel's own wait: block tables, weights and tokens, all written before its predecessor
// started.  They rely on every kernel here calling grid_dependency_wait() before let_dependents_launch(): when a dependent
// may start, the kernels before its predecessor are complete and their writes in L2.  The wait makes those writes visible
// to the kernel that executes it, not to its dependents, so such words are read past L1 (ld_early_*; TMA reads L2 anyway).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_dependents_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// launch with that attribute
template <typename... Params, typename... Args>
cudaError_t launch_dependent(void (*kern)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                             Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);
}

// ---------------------------------------------------------------------------
// e4m3 scale factors
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t e4m3_encode_rn(float x) {   // 0 <= x <= 448
  return static_cast<uint32_t>(__nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3));
}

__device__ __forceinline__ float e4m3_decode(uint32_t bits) {
  __half_raw h = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(bits & 0xffu), __NV_E4M3);
  return __half2float(__half(h));
}

// every non-zero code read as 2^(e-7) * (1 + m/8), exponent-0 codes included
__device__ __forceinline__ float e4m3_decode_implicit_one(uint32_t bits) {
  bits &= 0x7fu;
  return bits == 0 ? 0.0f : __uint_as_float((((bits >> 3) + 120u) << 23) | ((bits & 7u) << 20));
}

// ---------------------------------------------------------------------------
// e2m1 codes
// ---------------------------------------------------------------------------
// Exact code of q = t / s (s > 0): nearest grid value; a value half way
// between two grid points takes the smaller magnitude; a result of zero is +0.
// t > c*s  <=>  fl(t/s) > c  for every midpoint c, because c*s is exact in f32.
__device__ __forceinline__ uint32_t e2m1_code_exact(float t, float s) {
  const float mag = fabsf(t);
  uint32_t idx = (mag > 0.25f * s) + (mag > 0.75f * s) + (mag > 1.25f * s) + (mag > 1.75f * s) +
                 (mag > 2.5f * s) + (mag > 3.5f * s) + (mag > 5.0f * s);
  return (t < 0.0f && idx != 0) ? (idx | 8u) : idx;
}

// hardware round-to-nearest-even conversion of eight values; element i lands
// in nibble i (cvt's first source operand goes to the high nibble)
__device__ __forceinline__ uint32_t e2m1x8_hw(const float* u) {
  uint32_t r;
  asm("{\n"
      ".reg .b8 b0, b1, b2, b3;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n"
      "mov.b32 %0, {b0, b1, b2, b3};\n"
      "}"
      : "=r"(r)
      : "f"(u[0]), "f"(u[1]), "f"(u[2]), "f"(u[3]), "f"(u[4]), "f"(u[5]), "f"(u[6]), "f"(u[7]));
  return r;
}

// -0 (code 8) -> +0 (code 0) in all eight nibbles
__device__ __forceinline__ uint32_t e2m1x8_drop_negative_zero(uint32_t x) {
  const uint32_t nonzero = ((x & 0x77777777u) + 0x77777777u) & 0x88888888u;
  return x & (0x77777777u | nonzero);
}

// a / 6 rounded to nearest, without the division routine: q = a*c, one exact
// residual and one correction with c = RN(1/6) (division by a constant known in
// advance: Brisebarre, Muller, Raina, IEEE Trans. Computers 53(8), 2004).  Checked against a/6.0f for
// every positive float whose quotient is a normal number; for denormal
// quotients (far below the smallest scale factor) it may be one ulp off,
// which the e4m3 rounding to zero hides.
__device__ __forceinline__ float div_by_6(float a) {
  const float c = 0.16666667163372039794921875f;
  const float q = __fmul_rn(a, c);
  return __fmaf_rn(__fmaf_rn(-6.0f, q, a), c, q);
}

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// ---------------------------------------------------------------------------
// NVFP4 quantisation of one 16-element block held in registers
//   sf   = min((amax*gs)/6, 448) -> e4m3 (RN-even)
//   code = nearest_e2m1((v*gs) / sf_q), ties to the smaller magnitude
// The codes come from the hardware converter applied to two brackets of the
// quotient, v*k*(1+2^-19) and v*k*(1-2^-19) with k ~ gs/sf_q.  The exact
// quotient lies strictly between them, so when both brackets convert to the
// same eight codes that is the exact answer; the rare group where they differ
// (a value within 2^-18 of a midpoint, exact ties included) is redone with the
// division-free exact comparison above.
// kImplicitOne selects the MoE activation packer, which divides by the
// implicit-one reading of the scale byte instead of its true value.
// ---------------------------------------------------------------------------
// The arithmetic runs on the packed f32x2 instructions of sm_100 (two IEEE round-to-nearest f32
// operations per instruction): a block is eight register pairs.
//
// pair(i): elements 2i and 2i + 1 of the block as an f32x2, in a form that `scale` turns into the values times gs up to
// a few ulp; exact(i): the same two values exactly as the golden computes them (only evaluated when a bracket is
// open: one warp in a hundred; a loop over the open values instead of sixteen copies of the exact rounding made the norm
// kernel 20 to 40 % slower, it keeps the compiler from interleaving a thread's blocks); amax: the exact largest
// magnitude, NaN ignored; nothing: what `scale` becomes where the scale factor is zero (0, or NaN where it stands for
// values that are NaN all by themselves, so that their codes are a NaN's).  kOneBranch: one branch for the block instead
// of one per eight values (2 to 3 % faster in the norm kernel, 1 % slower in the epilogue of the MoE's first GEMM).
template <bool kImplicitOne, bool kOneBranch, typename Pair, typename Exact>
__device__ __forceinline__ void quantize_block16(Pair&& pair, Exact&& exact, float amax, float scale, float nothing,
                                                 float gs, uint32_t& codes_lo, uint32_t& codes_hi, uint32_t& sf_bits) {
  const float sf = fminf(div_by_6(__fmul_rn(amax, gs)), 448.0f);
  sf_bits = e4m3_encode_rn(sf);
  const float div = kImplicitOne ? e4m3_decode_implicit_one(sf_bits) : e4m3_decode(sf_bits);
  // k only has to be within a few ulp of scale / div: the brackets are 2^-19 wide
  const float k = div > 0.0f ? scale * rcp_approx(div) : nothing;
  const float k_hi = k * 1.0000019073486328125f;   // 1 + 2^-19
  const float k_lo = k * 0.9999980926513671875f;   // 1 - 2^-19
  const uint64_t k_hi2 = f32x2_pack(k_hi, k_hi);
  const uint64_t k_lo2 = f32x2_pack(k_lo, k_lo);
  uint32_t ch[2], cl[2];
  auto redo = [&](int g) {
    ch[g] = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint64_t v = exact(4 * g + i);
      ch[g] |= e2m1_code_exact(__fmul_rn(f32x2_lo(v), gs), div) << (8 * i);
      ch[g] |= e2m1_code_exact(__fmul_rn(f32x2_hi(v), gs), div) << (8 * i + 4);
    }
  };
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    float uh[8], ul[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint64_t v = pair(4 * g + i);
      const uint64_t h = f32x2_mul(v, k_hi2);
      const uint64_t l = f32x2_mul(v, k_lo2);
      uh[2 * i] = f32x2_lo(h);
      uh[2 * i + 1] = f32x2_hi(h);
      ul[2 * i] = f32x2_lo(l);
      ul[2 * i + 1] = f32x2_hi(l);
    }
    ch[g] = e2m1x8_hw(uh);
    cl[g] = e2m1x8_hw(ul);
    if constexpr (!kOneBranch) {
      if (ch[g] != cl[g]) redo(g);
    }
  }
  if constexpr (kOneBranch) {
    if (((ch[0] ^ cl[0]) | (ch[1] ^ cl[1])) != 0) {
      redo(0);
      redo(1);
    }
  }
  codes_lo = e2m1x8_drop_negative_zero(ch[0]);
  codes_hi = e2m1x8_drop_negative_zero(ch[1]);
}

// the values themselves in registers
template <bool kImplicitOne, bool kOneBranch = false>
__device__ __forceinline__ void quantize_block16(const uint64_t (&v2)[8], float gs, uint32_t& codes_lo,
                                                 uint32_t& codes_hi, uint32_t& sf_bits) {
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) amax = fmaxf(fmaxf(amax, fabsf(f32x2_lo(v2[i]))), fabsf(f32x2_hi(v2[i])));
  auto value = [&](int i) { return v2[i]; };
  quantize_block16<kImplicitOne, kOneBranch>(value, value, amax, gs, 0.0f, gs, codes_lo, codes_hi, sf_bits);
}

// ---------------------------------------------------------------------------
// The MoE activation packer (implicit-one reading of the scale byte) on sixteen bf16 values, eight packed pairs.
//
// When gs is a power of two -- 1 for the tokens, and for activations unless the caller calibrated a scale -- one
// conversion is exact.  v * gs is then a bf16 number, 8 significant bits, and a midpoint c (2 or 3 bits) times the divisor
// s (4 bits) is one too: two of them that differ, differ by more than 2^-8 of either.  So with u = v * gs / s * (1 - 2^-12),
// the factor approximated to a few ulp, v * gs > c * s puts u above c, v * gs < c * s below it, and a tie, which the golden
// gives to the smaller magnitude, also below: u is never half way between two codes and the hardware's nearest one is the
// golden's.  Half of the general routine's multiplications and conversions, and no second path.
// ---------------------------------------------------------------------------
struct Block16Codes {
  uint32_t lo, hi, sf;
};
static __device__ __noinline__ Block16Codes quantize_bf16x16_any_scale(uint4 a, uint4 b, float gs) {
  const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  uint64_t v2[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v2[i] = pair16_to_f32x2<__nv_bfloat16>(w[i]);
  Block16Codes r;
  quantize_block16<true>(v2, gs, r.lo, r.hi, r.sf);
  return r;
}
__device__ __forceinline__ bool is_power_of_two(float v) {        // positive and normal
  const uint32_t u = __float_as_uint(v);
  return (u & 0x807fffffu) == 0u && u != 0u && u != 0x7f800000u;
}
__device__ __forceinline__ Block16Codes quantize_bf16x16_pow2(const uint32_t (&w)[8], float gs) {
  uint32_t m = Pack16<__nv_bfloat16>::max_abs(w[0], w[1]);
#pragma unroll
  for (int i = 2; i < 8; ++i) m = Pack16<__nv_bfloat16>::max_abs(m, w[i]);
  // (not below zero: the largest of sixteen NaN is a NaN, which is no largest value, here as in the general routine)
  const float amax = fmaxf(fmaxf(Pair16<__nv_bfloat16>::lo(m), Pair16<__nv_bfloat16>::hi(m)), 0.0f);
  Block16Codes r;
  r.sf = e4m3_encode_rn(fminf(div_by_6(__fmul_rn(amax, gs)), 448.0f));
  const float div = e4m3_decode_implicit_one(r.sf);
  const float k = div > 0.0f ? gs * rcp_approx(div) * 0.999755859375f : 0.0f;      // 1 - 2^-12
  const uint64_t k2 = f32x2_pack(k, k);
  uint32_t out[2];
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    float u[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint64_t v = f32x2_mul(pair16_to_f32x2<__nv_bfloat16>(w[4 * g + i]), k2);
      u[2 * i] = f32x2_lo(v);
      u[2 * i + 1] = f32x2_hi(v);
    }
    out[g] = e2m1x8_drop_negative_zero(e2m1x8_hw(u));
  }
  r.lo = out[0];
  r.hi = out[1];
  return r;
}
// pow2: is_power_of_two(gs)
__device__ __forceinline__ Block16Codes quantize_bf16x16(const uint32_t (&w)[8], float gs, bool pow2) {
  if (pow2) return quantize_bf16x16_pow2(w, gs);
  return quantize_bf16x16_any_scale(make_uint4(w[0], w[1], w[2], w[3]), make_uint4(w[4], w[5], w[6], w[7]), gs);
}

// exchange buffers of the ranks of an expert-parallel group, as mapped into this process
constexpr int kMaxPeers = 16;
struct PeerPtrs {
  uint8_t* p[kMaxPeers];
};

// ---------------------------------------------------------------------------
// cross-rank signalling of the expert-parallel kernels
// ---------------------------------------------------------------------------
enum CtrlWord : int {
  kCtrlEpoch = 0,            // completed steps; every kernel of a step signals / waits for epoch + 1
  kCtrlTicketCount = 1,      // CTAs of the count kernel that have finished
  kCtrlTicketPlace = 2,
  kCtrlTicketCombine = 3,
  kCtrlAbort = 4,            // a cross-rank wait expired
  kCtrlTicketGemm = 5,       // CTAs of the row-pushing FC2 that have finished
  kCtrlWords = 16,
};
constexpr int kStatusPeerWaitExpired = 16;
constexpr int kSignalPhases = 3;       // 0: counts published, 1: rows placed, 2: output rows delivered

__device__ __forceinline__ int ld_acquire_sys(const int* p) {
  int v;
  asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_sys(int* p, int v) {
  asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// wait until *flag has reached `epoch`; gives up after limit_ns
__device__ __forceinline__ bool wait_flag(const int* flag, int epoch, unsigned long long limit_ns) {
  if (ld_acquire_sys(flag) - epoch >= 0) return true;
  const unsigned long long t0 = globaltimer_ns();
  for (;;) {
    if (ld_acquire_sys(flag) - epoch >= 0) return true;
    if (globaltimer_ns() - t0 > limit_ns) return false;
    __nanosleep(64);
  }
}
// offset of scale factor (row m, K-block kb) in the 128x4 tiled layout with rk
// K-tiles per row tile (python/cutlass_compat/cutlass/utils/blockscaled_layout.py:37-42)
__device__ __host__ __forceinline__ int64_t sf_swizzled_offset(int64_t m, int kb, int rk) {
  return (m & 31) * 16 + ((m >> 5) & 3) * 4 + (kb & 3) + static_cast<int64_t>(kb >> 2) * 512 +
         (m >> 7) * static_cast<int64_t>(rk) * 512;
}

}  // namespace b200fp4
