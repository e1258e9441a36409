// Stand-alone group quantiser / dequantiser, master-weight split and maxabs.
//
// These run at checkpoint save/load, fp32 export/import and when a state is set from a
// full-precision tensor, never inside a training step, and reproduce the PyTorch formulation in
// ops/oracle.py bit for bit.  The quantiser takes an approximate reciprocal where its error cannot
// change the code and the formula's IEEE operations elsewhere; the dequantiser's quotients are
// corrected by their exact remainders; the master-weight kernels use round-to-nearest intrinsics,
// which the compiler never contracts into FMAs.  What they compute matches
// flashoptim/optimizers.py:2610-2676 (quantise), :2541-2607 (dequantise),
// :2726-2776 (error-correction encode / decode).
#include <type_traits>

#include "fo_api.h"
#include "fo_common.cuh"

namespace fo {

constexpr int kQThreads = 256;
// Register budgets (launch bounds) that measured best at 2^28 elements: 40 registers (6 CTAs per SM)
// for the quantiser (bf16, companded: 151 us; 158 with 48, 172 with 64), 32 (8 CTAs) for the
// dequantiser (to bf16: 172 us; 193 with 40, 205 with 48), 40 for the master-weight kernels.
constexpr int kQuantMinBlocks = 6;
constexpr int kDequantMinBlocks = 8;
constexpr int kEccMinBlocks = 6;

// ---------------------------------------------------------------- memory access
// Read-once data through the non-coherent path with default caching: measured 2-3 % faster in
// these kernels than L1::no_allocate loads.
__device__ __forceinline__ uint4 ldg16(const void* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }
__device__ __forceinline__ uint2 ldg8(const void* p) { return __ldg(reinterpret_cast<const uint2*>(p)); }
__device__ __forceinline__ uint32_t ldg4(const void* p) { return __ldg(reinterpret_cast<const uint32_t*>(p)); }

// 256-bit accesses (sm_100 and later): a unit of eight fp32 values is one request.
struct Words8 {
  uint32_t w[8];
};
__device__ __forceinline__ bool aligned32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31) == 0; }
__device__ __forceinline__ Words8 ldg32(const void* p) {
  Words8 v;
  asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]), "=r"(v.w[6]),
                 "=r"(v.w[7])
               : "l"(p));
  return v;
}
__device__ __forceinline__ void st32(void* p, const Words8& v) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v.w[0]), "r"(v.w[1]), "r"(v.w[2]),
               "r"(v.w[3]), "r"(v.w[4]), "r"(v.w[5]), "r"(v.w[6]), "r"(v.w[7])
               : "memory");
}

template <typename T>
__device__ __forceinline__ float load_as_float(const T* p, int64_t i) {
  if constexpr (sizeof(T) == 4) return p[i];
  else if constexpr (std::is_same<T, __half>::value) return __half2float(p[i]);
  else return __bfloat162float(p[i]);
}

template <typename T>
__device__ __forceinline__ bool aligned_for_units(const T* p) {
  constexpr uintptr_t need = sizeof(T) * kUnit >= 16 ? 16 : sizeof(T) * kUnit;
  return (reinterpret_cast<uintptr_t>(p) & (need - 1)) == 0;
}

// 8 elements of any supported float type -> fp32 (exact widening); zero beyond n.
template <typename T>
__device__ __forceinline__ void load8f(const T* p, int64_t base, int64_t n, bool vec, float (&v)[kUnit]) {
  if (vec && base + kUnit <= n) {
    if constexpr (sizeof(T) == 4) {
      if (aligned32(p + base)) {
        const Words8 a = ldg32(p + base);
#pragma unroll
        for (int i = 0; i < kUnit; ++i) v[i] = __uint_as_float(a.w[i]);
      } else {
        const uint4 a = ldg16(p + base), b = ldg16(p + base + 4);
        v[0] = __uint_as_float(a.x); v[1] = __uint_as_float(a.y); v[2] = __uint_as_float(a.z); v[3] = __uint_as_float(a.w);
        v[4] = __uint_as_float(b.x); v[5] = __uint_as_float(b.y); v[6] = __uint_as_float(b.z); v[7] = __uint_as_float(b.w);
      }
    } else {
      const uint4 a = ldg16(p + base);
      const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if constexpr (std::is_same<T, __half>::value) {
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
          v[2 * i] = f.x;
          v[2 * i + 1] = f.y;
        } else {
          v[2 * i] = __uint_as_float(w[i] << 16);
          v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < kUnit; ++i) v[i] = base + i < n ? load_as_float(p, base + i) : 0.0f;
  }
}
// ---------------------------------------------------------------- lists of tensors
//
// A call covers a list of tensors (the states of a whole checkpoint): their addresses travel in
// the kernel parameters, kMaxRows to a launch, and CTAs take chunks of kConvChunk elements off the
// concatenated list.  A CTA's chunk numbers only grow, so it steps through the rows.
constexpr int kSpan = 16;  // elements per thread and chunk
constexpr int kConvChunk = kQThreads * kSpan;
constexpr int kMaxRows = 12;  // 0.6 KB of parameters; the 2.8 KB of 64 rows made a small launch 1 us longer
struct ConvBatch {
  FoConvRow rows[kMaxRows];
  int32_t begin[kMaxRows + 1];  // first chunk of each row
  int total;
};
__device__ __forceinline__ void seek_row(const ConvBatch& B, int c, int& r) {
  while (c >= B.begin[r + 1]) ++r;
}
__device__ __forceinline__ bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// 16 elements of any supported float type -> fp32 (exact widening); zero beyond n.
template <typename T>
__device__ __forceinline__ void load_span(const T* p, int64_t base, int64_t n, float2 (&v)[8]) {
  constexpr int kWords = sizeof(T) * 4;
  if (aligned16(p) && base + kSpan <= n) {
    uint32_t w[kWords];
    if (aligned32(p + base)) {
#pragma unroll
      for (int k = 0; k < kWords / 8; ++k) {
        const Words8 a = ldg32(reinterpret_cast<const uint32_t*>(p + base) + 8 * k);
#pragma unroll
        for (int i = 0; i < 8; ++i) w[8 * k + i] = a.w[i];
      }
    } else {
#pragma unroll
      for (int k = 0; k < kWords / 4; ++k) {
        const uint4 a = ldg16(reinterpret_cast<const uint32_t*>(p + base) + 4 * k);
        w[4 * k] = a.x; w[4 * k + 1] = a.y; w[4 * k + 2] = a.z; w[4 * k + 3] = a.w;
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if constexpr (sizeof(T) == 4)
        v[i] = make_float2(__uint_as_float(w[2 * i]), __uint_as_float(w[2 * i + 1]));
      else if constexpr (std::is_same<T, __half>::value)
        v[i] = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      else
        v[i] = make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[i].x = base + 2 * i < n ? load_as_float(p, base + 2 * i) : 0.0f;
      v[i].y = base + 2 * i + 1 < n ? load_as_float(p, base + 2 * i + 1) : 0.0f;
    }
  }
}

// ---------------------------------------------------------------- quantiser

// One code as the written-down formula has it: correctly rounded square root and divisions.
template <bool kSigned, bool kSqrt, bool kSoftsign>
__device__ __forceinline__ uint32_t exact_code(float x, float a) {
  if (kSqrt) x = __fsqrt_rn(x);
  float t = __fdiv_rn(x, a);
  if (kSoftsign) t = __fdiv_rn(__fmul_rn(t, 2.0f), __fadd_rn(fabsf(t), 1.0f));
  return (uint32_t)(int)floorf(__fadd_rn(__fmul_rn(t, kSigned ? 127.0f : 255.0f), 0.5f));
}

// A thread takes half a group: one shuffle per group maximum, 16-byte code vectors.
//
// The formula's two correctly rounded divisions (and square root) per element made the kernel
// issue bound at a third of the memory bandwidth (2^28 elements, bf16: companded 357 us, sqrt domain
// 314; now 152 and 183, 5.4 and 4.5 TB/s).  Here a code is first computed with one
// approximate reciprocal (or square root) per element; its distance to the nearest rounding
// boundary then says whether the formula's own rounding errors could have led to the neighbouring
// code, and only then (about one element in 4000) the formula is evaluated.
//   Bound, in units of 2^-24 relative to the scaled value s: approximation <= 6 with the compander
//   (constant, its product, FMA, reciprocal 2, product) or 6 without (square root 2, reciprocal 2,
//   two products), formula <= 4 with it or 3 without, plus half an ulp of s + 0.5.  With |s| <= 127
//   that is at most 8e-5, with |s| <= 255 at most 1.6e-4 or 1.45e-4; kNear lies above each.  NaN fails the comparison, so
//   that everything that is not finite takes the formula too; an infinite group maximum gives
//   zero on both ways.
// The square root is monotonic: the root of the group maximum is the maximum of the roots.
template <typename T, bool kSigned, bool kSqrt, bool kSoftsign>
__global__ void __launch_bounds__(kQThreads, kQuantMinBlocks)
    quantize_kernel(const __grid_constant__ ConvBatch B) {
  constexpr float kMax = kSigned ? 127.0f : 255.0f;
  constexpr float kNear = kSigned ? 0x1p-13f : kSoftsign ? 0x1p-12f : 0x1.4p-13f;
  int r = 0;
  for (int c = blockIdx.x; c < B.total; c += gridDim.x) {
    seek_row(B, c, r);
    const int64_t n = B.rows[r].n;
    const int64_t base = (int64_t)(c - B.begin[r]) * kConvChunk + threadIdx.x * kSpan;
    float2 x[8];
    load_span(static_cast<const T*>(B.rows[r].src), base, n, x);  // zero beyond the tensor: padding cannot raise the absmax
    float a = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      a = kSqrt ? fmaxf(a, fmaxf(x[i].x, x[i].y)) : fmaxf(a, fmaxf(fabsf(x[i].x), fabsf(x[i].y)));
    a = fmaxf(a, __shfl_xor_sync(kFullMask, a, 1));
    if (kSqrt) a = __fsqrt_rn(a);
    a = fmaxf(a, 1e-12f);

    constexpr float kInv = 1.0f / (2.0f * kMax);
    // scaled by 2^-32 so that the reciprocal of the largest maxima does not underflow
    const float k = kSoftsign ? __fmul_rn(a, kInv) : __fmul_rn(fast_rcp(a * 0x1p-32f), kMax * 0x1p-32f);
    const float2 magic = splat2(kRoundMagic), neg1 = splat2(-1.0f);
    uint32_t w[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float2 s[4];
      uint32_t z[8];
      bool sure = true;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float2 v = x[4 * h + i];
        if (kSqrt) v = make_float2(fast_sqrt(v.x), fast_sqrt(v.y));
        // with the compander, MAX * 2n / (1 + |n|) for n = v / a is v / ((a + |v|) / (2 MAX))
        const float2 f = kSoftsign ? make_float2(fast_rcp(fmaf(fabsf(v.x), kInv, k)), fast_rcp(fmaf(fabsf(v.y), kInv, k)))
                                   : splat2(k);
        s[i] = mul2(v, f);
        const float2 q = add2(s[i], magic);
        const float2 off = add2(s[i], fma2(q, neg1, magic));  // from the nearest integer
        sure = sure && fabsf(off.x) < 0.5f - kNear && fabsf(off.y) < 0.5f - kNear;
        z[2 * i] = __float_as_uint(q.x);
        z[2 * i + 1] = __float_as_uint(q.y);
      }
      if (!sure) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float si = (i & 1) ? s[i >> 1].y : s[i >> 1].x;
          const float xi = (i & 1) ? x[4 * h + (i >> 1)].y : x[4 * h + (i >> 1)].x;
          const float off = __fsub_rn(si, __fsub_rn(__uint_as_float(z[i]), kRoundMagic));
          if (!(fabsf(off) < 0.5f - kNear)) z[i] = exact_code<kSigned, kSqrt, kSoftsign>(xi, a);
        }
      }
      w[2 * h] = __byte_perm(__byte_perm(z[0], z[1], 0x0040), __byte_perm(z[2], z[3], 0x0040), 0x5410);
      w[2 * h + 1] = __byte_perm(__byte_perm(z[4], z[5], 0x0040), __byte_perm(z[6], z[7], 0x0040), 0x5410);
    }
    uint8_t* q = static_cast<uint8_t*>(B.rows[r].dst);
    if (base + kSpan <= n && aligned16(q)) {
      st16(q + base, make_uint4(w[0], w[1], w[2], w[3]));
    } else {
#pragma unroll
      for (int i = 0; i < kSpan; ++i)
        if (base + i < n) q[base + i] = (uint8_t)(w[i >> 2] >> (8 * (i & 3)));
    }
    if ((threadIdx.x & 1) == 0 && base < n) static_cast<__half*>(B.rows[r].dst2)[base >> 5] = __float2half_rn(a);
  }
}

// ---------------------------------------------------------------- dequantiser

// a / b from an approximate reciprocal of b, the product and one correction by its exact remainder
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990).
__device__ __forceinline__ float2 corrected_quotient2(float2 a, float2 neg_b, float2 rcp_b) {
  const float2 q = mul2(a, rcp_b);
  return fma2(fma2(q, neg_b, a), rcp_b, q);
}
// What the formula divides depends on the code alone, so that 256 codes are all there is to check:
// equal to IEEE division for each of them (tests/test_quantizer_boundaries_gpu.py).  With IEEE
// divisions 2^28 elements took 326-367 us (companded, to fp32), with these 213 (6.3 TB/s), with a
// table of the values in shared memory, one copy per bank, 277.
template <bool kSigned, bool kSoftsign>
__device__ __forceinline__ float2 code_value2(float2 c) {
  constexpr float kMax = kSigned ? 127.0f : 255.0f;
  const float2 t = corrected_quotient2(c, splat2(-kMax), splat2(1.0f / kMax));
  if (!kSoftsign) return t;
  const float2 neg_d = make_float2(__fsub_rn(fabsf(t.x), 2.0f), __fsub_rn(fabsf(t.y), 2.0f));
  return corrected_quotient2(t, neg_d, make_float2(fast_rcp(-neg_d.x), fast_rcp(-neg_d.y)));
}

// An access takes the codes of 8 elements per lane, contiguous over the warp.
template <typename T, bool kSigned, bool kSqrt, bool kSoftsign>
__global__ void __launch_bounds__(kQThreads, kDequantMinBlocks)
    dequantize_kernel(const __grid_constant__ ConvBatch B) {
  constexpr int kAccesses = kSpan / kUnit;
  int r = 0;
  for (int c = blockIdx.x; c < B.total; c += gridDim.x) {
    seek_row(B, c, r);
    const int64_t n = B.rows[r].n;
    const uint8_t* q = static_cast<const uint8_t*>(B.rows[r].src);
    const __half* scales = static_cast<const __half*>(B.rows[r].aux);
    T* out = static_cast<T*>(B.rows[r].dst);
    const int64_t first = (int64_t)(c - B.begin[r]) * kConvChunk + threadIdx.x * kUnit;
    const bool vec = (reinterpret_cast<uintptr_t>(q) & 7) == 0;
    uint32_t w[kAccesses][2];
    float sc[kAccesses];
#pragma unroll
    for (int k = 0; k < kAccesses; ++k) {
      const int64_t base = first + k * (kQThreads * kUnit);
      sc[k] = base < n ? __half2float(scales[base >> 5]) : 0.0f;
      if (base + kUnit <= n && vec) {
        const uint2 a = ldg8(q + base);
        w[k][0] = a.x;
        w[k][1] = a.y;
      } else {
        ld_partial<1, 2>(q + base, (int)min(n - base, (int64_t)kUnit), w[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < kAccesses; ++k) {
      const int64_t base = first + k * (kQThreads * kUnit);
      float2 x[4];
      if (kSigned) s8_to_float(make_uint2(w[k][0], w[k][1]), x);
      else u8_to_float(make_uint2(w[k][0], w[k][1]), x);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[i] = mul2(code_value2<kSigned, kSoftsign>(x[i]), splat2(sc[k]));
        if (kSqrt) x[i] = mul2(x[i], x[i]);
      }
      const int left = (int)min(n - base, (int64_t)kUnit);
      if constexpr (sizeof(T) == 4) {
        Words8 o;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          o.w[2 * i] = __float_as_uint(x[i].x);
          o.w[2 * i + 1] = __float_as_uint(x[i].y);
        }
        if (left == kUnit && aligned32(out)) {
          st32(out + base, o);
        } else if (left == kUnit && aligned16(out)) {
          st16(out + base, make_uint4(o.w[0], o.w[1], o.w[2], o.w[3]));
          st16(out + base + 4, make_uint4(o.w[4], o.w[5], o.w[6], o.w[7]));
        } else {
          st_partial<4, 8>(out + base, left, o.w);
        }
      } else {
        uint32_t o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const __nv_bfloat162 b = __floats2bfloat162_rn(x[i].x, x[i].y);
          o[i] = *reinterpret_cast<const uint32_t*>(&b);
        }
        if (left == kUnit && aligned16(out)) st16(out + base, make_uint4(o[0], o[1], o[2], o[3]));
        else st_partial<2, 4>(out + base, left, o);
      }
    }
  }
}

// ---------------------------------------------------------------- master-weight split / merge

// Exact 2^e for e in [-126, 127].
__device__ __forceinline__ float pow2i(int e) { return __int_as_float((e + 127) << 23); }

// c / smax, correctly rounded, for an integer code |c| <= smax in {127, 32767}: the rounded
// reciprocal, one product and one FMA-corrected refinement.  Equal to IEEE division for every
// code (checked exhaustively against fp32 division; tests/test_kernels_gpu.py compares the
// kernel with the PyTorch formulation over all codes) at a third of its instructions.
__device__ __forceinline__ float div_by_code_range(float c, float smax) {
  const float r = smax == 127.0f ? (1.0f / 127.0f) : (1.0f / 32767.0f);
  const float q0 = __fmul_rn(c, r);
  const float rem = __fmaf_rn(-q0, smax, c);
  return __fmaf_rn(rem, r, q0);
}

template <typename T>
__device__ __forceinline__ int ecc_log_scale_bits(uint16_t bits) {
  constexpr int M = Elem<T>::kMant;
  constexpr int bias = std::is_same<T, __half>::value ? 15 : 127;
  const int field = (bits & 0x7FFF) >> M;
  const int e = field == 0 ? 1 - bias : field - bias;
  return e - M - 1;
}
template <typename T>
__device__ __forceinline__ float narrow_bits_to_float(uint16_t bits) {
  if constexpr (std::is_same<T, __half>::value) return __half2float(__ushort_as_half(bits));
  else return __uint_as_float((uint32_t)bits << 16);
}

// 2^ls and 2^-ls (ls = E(w) - M - 1) as single floats, straight from the exponent field of the
// narrow value.  The PyTorch formulation scales by two powers of two so that nothing under- or
// overflows on the way; one factor gives the same bits whenever it is itself a normal number and
// the scaled correction is (an exact scaling then, and `code * 2^ls + w` rounds once either
// way).  fp16: always (E >= -14; subnormals and zero share the smallest normal's exponent, the
// clamp).  bf16: for |w| >= 2^-94; smaller values, zero included, take the two-factor form.
template <typename T>
__device__ __forceinline__ bool single_scale_ok(float w) {
  if constexpr (std::is_same<T, __half>::value) return true;
  else return fabsf(w) >= 5.048709793414476e-29f;  // 2^-94; false for NaN
}
template <typename T>
__device__ __forceinline__ float ecc_scale(uint16_t bits) {
  if constexpr (std::is_same<T, __half>::value)
    return __uint_as_float((max((uint32_t)bits & 0x7C00u, 0x0400u) << 13) + ((127u - 15u - 11u) << 23));
  else
    return __uint_as_float((((uint32_t)bits << 16) & 0x7F800000u) - (8u << 23));
}
template <typename T>
__device__ __forceinline__ float ecc_inv_scale(uint16_t bits) {
  if constexpr (std::is_same<T, __half>::value)
    return __uint_as_float(((127u + 15u + 11u) << 23) - (max((uint32_t)bits & 0x7C00u, 0x0400u) << 13));
  else
    return __uint_as_float(((254u + 8u) << 23) - (((uint32_t)bits << 16) & 0x7F800000u));
}

// The split / merge kernels use an interleaved layout: a warp owns a tile of 256 consecutive
// elements and a lane moves elements [4 * lane, 4 * lane + 4) of each half, so that every
// warp-wide access covers one contiguous span (512 / 256 / 128 bytes for 4- / 2- / 1-byte
// elements).  Measured against 8 consecutive elements per lane (32-byte fp32 accesses at a
// 32-byte stride): 4-15 % faster.
template <typename T>
__device__ __forceinline__ bool aligned_for_quads(const T* p) {
  return (reinterpret_cast<uintptr_t>(p) & (sizeof(T) * 4 - 1)) == 0;
}
// Four elements as sizeof(T) packed words; zero beyond n.
template <typename T>
__device__ __forceinline__ void load4raw(const T* p, int64_t base, int64_t n, bool vec, uint32_t (&w)[sizeof(T)]) {
  if (vec && base + 4 <= n) {
    if constexpr (sizeof(T) == 4) {
      const uint4 a = ldg16(p + base);
      w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
    } else if constexpr (sizeof(T) == 2) {
      const uint2 a = ldg8(p + base);
      w[0] = a.x; w[1] = a.y;
    } else {
      w[0] = ldg4(p + base);
    }
  } else {
#pragma unroll
    for (int k = 0; k < (int)sizeof(T); ++k) w[k] = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (base + i < n) {
        if constexpr (sizeof(T) == 4) w[i] = reinterpret_cast<const uint32_t*>(p)[base + i];
        else if constexpr (sizeof(T) == 2)
          w[i >> 1] |= (uint32_t) reinterpret_cast<const uint16_t*>(p)[base + i] << (16 * (i & 1));
        else w[0] |= (uint32_t) reinterpret_cast<const uint8_t*>(p)[base + i] << (8 * i);
      }
    }
  }
}
template <typename T>
__device__ __forceinline__ void store4raw(T* p, int64_t base, int64_t n, bool vec, const uint32_t (&w)[sizeof(T)]) {
  if (vec && base + 4 <= n) {
    if constexpr (sizeof(T) == 4) st16(p + base, make_uint4(w[0], w[1], w[2], w[3]));
    else if constexpr (sizeof(T) == 2) st8(p + base, make_uint2(w[0], w[1]));
    else *reinterpret_cast<uint32_t*>(p + base) = w[0];
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (base + i < n) {
        if constexpr (sizeof(T) == 4) reinterpret_cast<uint32_t*>(p)[base + i] = w[i];
        else if constexpr (sizeof(T) == 2)
          reinterpret_cast<uint16_t*>(p)[base + i] = (uint16_t)(w[i >> 1] >> (16 * (i & 1)));
        else reinterpret_cast<uint8_t*>(p)[base + i] = (uint8_t)(w[0] >> (8 * i));
      }
    }
  }
}
// Element i of a packed quad of signed codes as an exact float.  The caller has flipped the sign
// bit of every code in the packed word (code + 128, or + 32768, as an unsigned field); one byte
// permute drops that field into the mantissa of 2^23 and subtracting 2^23 + the offset leaves
// the code: no integer-to-float conversion and no sign extension per element.
template <typename E>
__device__ __forceinline__ float quad_code_f(const uint32_t (&w)[sizeof(E)], int i) {
  if constexpr (sizeof(E) == 1)
    return __fsub_rn(__uint_as_float(__byte_perm(w[0], 0x4B000000u, 0x7440u | i)), 8388736.0f);
  else
    return __fsub_rn(__uint_as_float(__byte_perm(w[i >> 1], 0x4B000000u, (i & 1) ? 0x7432u : 0x7410u)), 8421376.0f);
}

// The tiles of a warp: a CTA takes chunks off the list, warp w of it the tiles w, w + 8, ... of each.
struct TileWalk {
  int chunk = blockIdx.x, tile = -1;
  int64_t base = 0;  // first element of this lane's first quad
  __device__ __forceinline__ bool next(const ConvBatch& B, int& row) {
    if (++tile == kConvChunk / (kQThreads * 8)) {
      tile = 0;
      chunk += gridDim.x;
    }
    if (chunk >= B.total) return false;
    if (tile == 0) seek_row(B, chunk, row);
    base = (int64_t)(chunk - B.begin[row]) * kConvChunk + tile * (kQThreads * 8) + (threadIdx.x >> 5) * 256 +
           (threadIdx.x & 31) * 4;
    return true;
  }
};

template <typename T, typename E>
__global__ void __launch_bounds__(kQThreads, kEccMinBlocks)
    ecc_decode_kernel(const __grid_constant__ ConvBatch B) {
  const float smax = sizeof(E) == 1 ? 127.0f : 32767.0f;
  const uint32_t flip = sizeof(E) == 1 ? 0x80808080u : 0x80008000u;
  int row = 0;
  for (TileWalk t; t.next(B, row);) {
    const T* w = static_cast<const T*>(B.rows[row].src);
    const E* ecc = static_cast<const E*>(B.rows[row].aux);
    float* out = static_cast<float*>(B.rows[row].dst);
    const int64_t n = B.rows[row].n;
    const bool vec = aligned_for_quads(w) && aligned_for_quads(ecc) && aligned_for_quads(out);
    const int64_t b[2] = {t.base, t.base + 128};
    uint32_t wn[2][2], wc[2][sizeof(E)];
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      load4raw(w, b[hf], n, vec, wn[hf]);
      load4raw(ecc, b[hf], n, vec, wc[hf]);
    }
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
      for (int k = 0; k < (int)sizeof(E); ++k) wc[hf][k] ^= flip;
      uint32_t r[4];
      uint16_t hb[4];
      float wf[4];
      bool single = true;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        hb[i] = (uint16_t)(wn[hf][i >> 1] >> (16 * (i & 1)));
        wf[i] = narrow_bits_to_float<T>(hb[i]);
        single = single && single_scale_ok<T>(wf[i]);
      }
      if (single) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float corr = div_by_code_range(quad_code_f<E>(wc[hf], i), smax);
          r[i] = __float_as_uint(__fmaf_rn(corr, ecc_scale<T>(hb[i]), wf[i]));
        }
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int ls = ecc_log_scale_bits<T>(hb[i]);
          const int hh = ls >> 1;  // floor(ls / 2)
          const float corr = div_by_code_range(quad_code_f<E>(wc[hf], i), smax);
          const float e = __fmul_rn(__fmul_rn(corr, pow2i(hh)), pow2i(ls - hh));
          r[i] = __float_as_uint(__fadd_rn(wf[i], e));
        }
      }
      store4raw(out, b[hf], n, vec, r);
    }
  }
}

// Rounds two fp32 values to the narrow type, packed.
template <typename T>
__device__ __forceinline__ uint32_t narrow_pair(float lo, float hi) {
  if constexpr (std::is_same<T, __half>::value) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  } else {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
}

// Correction codes of fp32 values against their narrow roundings, which are read (kSplit false:
// aux holds them, dst takes the codes) or made here (kSplit true: dst takes them, dst2 the codes).
// Importing fp32 weights as a rounding, its copy into the parameter and the encoding, three
// kernels, moved 17 bytes per element where this moves 7.
template <typename T, typename E, bool kSplit>
__global__ void __launch_bounds__(kQThreads, kEccMinBlocks)
    ecc_encode_kernel(const __grid_constant__ ConvBatch B) {
  const float smax = sizeof(E) == 1 ? 127.0f : 32767.0f;
  int row = 0;
  for (TileWalk t; t.next(B, row);) {
    const float* x = static_cast<const float*>(B.rows[row].src);
    const T* w = static_cast<const T*>(kSplit ? B.rows[row].dst : B.rows[row].aux);
    E* ecc = static_cast<E*>(kSplit ? B.rows[row].dst2 : B.rows[row].dst);
    const int64_t n = B.rows[row].n;
    const bool vec = aligned_for_quads(x) && aligned_for_quads(w) && aligned_for_quads(ecc);
    const int64_t b[2] = {t.base, t.base + 128};
    uint32_t wn[2][2], wx[2][4];
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      load4raw(x, b[hf], n, vec, wx[hf]);
      if constexpr (!kSplit) load4raw(w, b[hf], n, vec, wn[hf]);
    }
    if constexpr (kSplit) {
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        wn[hf][0] = narrow_pair<T>(__uint_as_float(wx[hf][0]), __uint_as_float(wx[hf][1]));
        wn[hf][1] = narrow_pair<T>(__uint_as_float(wx[hf][2]), __uint_as_float(wx[hf][3]));
        store4raw(const_cast<T*>(w), b[hf], n, vec, wn[hf]);
      }
    }
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      uint32_t o[sizeof(E)];
#pragma unroll
      for (int k = 0; k < (int)sizeof(E); ++k) o[k] = 0;
      uint16_t hb[4];
      float wf[4];
      bool single = true;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        hb[i] = (uint16_t)(wn[hf][i >> 1] >> (16 * (i & 1)));
        wf[i] = narrow_bits_to_float<T>(hb[i]);
        single = single && single_scale_ok<T>(wf[i]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float e = __fsub_rn(__uint_as_float(wx[hf][i]), wf[i]);
        float en;
        if (single) {
          en = __fmul_rn(e, ecc_inv_scale<T>(hb[i]));
        } else {
          const int neg = -ecc_log_scale_bits<T>(hb[i]);
          const int hh = neg >> 1;
          en = __fmul_rn(__fmul_rn(e, pow2i(hh)), pow2i(neg - hh));
        }
        en = fminf(fmaxf(en, -1.0f), 1.0f);  // a NaN difference becomes -1
        const float s = __fmul_rn(en, smax);
        // copysign(floor(|s| + 0.5), s) without a float-to-int conversion: for 0 <= t < 2^23,
        // t + 2^23 rounded down leaves floor(t) in the mantissa
        const float t = __fadd_rn(fabsf(s), 0.5f);
        const int mag = __float_as_int(__fadd_rd(t, 8388608.0f)) & 0x7FFFFF;
        const int c = s < 0.0f ? -mag : mag;
        if constexpr (sizeof(E) == 1) o[0] |= (uint32_t)(c & 0xff) << (8 * i);
        else o[i >> 1] |= (uint32_t)(c & 0xffff) << (16 * (i & 1));
      }
      store4raw(ecc, b[hf], n, vec, o);
    }
  }
}

// ---------------------------------------------------------------- one-byte codes in the parameter's dtype
//
// Checkpoints carry the one-byte corrections as values of the parameter's dtype.  3 bytes per
// element, bound by memory; torch's own conversions between int8 and the 16-bit floats reach
// 1.1 TB/s (585 and 574 us for 218 M elements).
__device__ __forceinline__ uint32_t signed_bytes(float lo, float hi) {
  return (uint32_t)(uint8_t) static_cast<int8_t>(lo) | (uint32_t)(uint8_t) static_cast<int8_t>(hi) << 8;
}
template <typename T, bool kToNarrow>
__global__ void __launch_bounds__(kQThreads) code_cast_kernel(const __grid_constant__ ConvBatch B) {
  constexpr int kAccesses = kSpan / kUnit;
  int r = 0;
  for (int c = blockIdx.x; c < B.total; c += gridDim.x) {
    seek_row(B, c, r);
    const int64_t n = B.rows[r].n;
    const void* src = B.rows[r].src;
    void* dst = B.rows[r].dst;
    const int8_t* q = static_cast<const int8_t*>(kToNarrow ? src : dst);
    const T* v = static_cast<const T*>(kToNarrow ? dst : src);
    const bool vec = (reinterpret_cast<uintptr_t>(q) & 7) == 0 && aligned16(v);
    const int64_t first = (int64_t)(c - B.begin[r]) * kConvChunk + threadIdx.x * kUnit;
    uint32_t in[kAccesses][kToNarrow ? 2 : 4];
#pragma unroll
    for (int k = 0; k < kAccesses; ++k) {
      const int64_t base = first + k * (kQThreads * kUnit);
      const int left = (int)min(n - base, (int64_t)kUnit);
      if constexpr (kToNarrow) {
        if (left == kUnit && vec) {
          const uint2 a = ldg8(q + base);
          in[k][0] = a.x; in[k][1] = a.y;
        } else {
          ld_partial<1, 2>(q + base, left, in[k]);
        }
      } else {
        if (left == kUnit && vec) {
          const uint4 a = ldg16(v + base);
          in[k][0] = a.x; in[k][1] = a.y; in[k][2] = a.z; in[k][3] = a.w;
        } else {
          ld_partial<2, 4>(v + base, left, in[k]);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kAccesses; ++k) {
      const int64_t base = first + k * (kQThreads * kUnit);
      const int left = (int)min(n - base, (int64_t)kUnit);
      if constexpr (kToNarrow) {
        float2 f[4];
        s8_to_float(make_uint2(in[k][0], in[k][1]), f);
        uint32_t o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = narrow_pair<T>(f[i].x, f[i].y);
        T* out = static_cast<T*>(dst) + base;
        if (left == kUnit && vec) st16(out, make_uint4(o[0], o[1], o[2], o[3]));
        else st_partial<2, 4>(out, left, o);
      } else {
        uint32_t o[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t a = in[k][2 * j], b = in[k][2 * j + 1];
          o[j] = signed_bytes(narrow_bits_to_float<T>((uint16_t)a), narrow_bits_to_float<T>((uint16_t)(a >> 16))) |
                 signed_bytes(narrow_bits_to_float<T>((uint16_t)b), narrow_bits_to_float<T>((uint16_t)(b >> 16))) << 16;
        }
        int8_t* out = static_cast<int8_t*>(dst) + base;
        if (left == kUnit && vec) st8(out, make_uint2(o[0], o[1]));
        else st_partial<1, 2>(out, left, o);
      }
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kQThreads) maxabs_kernel(const T* __restrict__ x, int64_t n, float* out) {
  float a = 0.0f;
  const int64_t n_units = (n + kUnit - 1) / kUnit;
  const bool vec = aligned_for_units(x);
  for (int64_t unit = (int64_t)blockIdx.x * kQThreads + threadIdx.x; unit < n_units;
       unit += (int64_t)gridDim.x * kQThreads) {
    float v[kUnit];
    load8f(x, unit * kUnit, n, vec, v);
#pragma unroll
    for (int i = 0; i < kUnit; ++i) a = fmaxf(a, fabsf(v[i]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a = fmaxf(a, __shfl_xor_sync(kFullMask, a, o));
  // non-negative floats order like their bit patterns; NaN inputs are dropped by fmaxf
  if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<unsigned int*>(out), __float_as_uint(a));
}

// Grids: a loop over chunks by at most 64 CTAs per SM (the SM count is read once per device), never
// more than the work.  Several times the resident CTAs, because the SMs do not all run at the same
// pace and equal fixed shares wait for the slowest (quantiser at 2^28 elements: 168 us with 16 CTAs
// per SM, 158 with 64, 166 with 256).  maxabs, whose units are half as large, takes twice as many;
// -DFO_QUANT_BLOCKS_PER_SM=k changes that for tuning builds.
constexpr int kListCtasPerSm = 64;
#ifndef FO_QUANT_BLOCKS_PER_SM
#define FO_QUANT_BLOCKS_PER_SM 128
#endif
static int sm_count() {
  static int sms[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 148;
  if (sms[dev] == 0) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
    sms[dev] = v;
  }
  return sms[dev];
}
static int blocks_for(int64_t units) {
  int64_t b = (units + kQThreads - 1) / kQThreads;
  const int64_t cap = (int64_t)sm_count() * FO_QUANT_BLOCKS_PER_SM;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}
template <auto kKernel, typename... Args>
static void launch_strided(int64_t units, cudaStream_t st, Args... args) {
  kKernel<<<blocks_for(units), kQThreads, 0, st>>>(args...);
}

// Cuts a list of tensors into launches of at most kMaxRows rows.
template <typename Launch>
static int for_batches(const FoConvRow* rows, int n_rows, Launch launch) {
  for (int i = 0; i < n_rows;) {
    ConvBatch B;
    int k = 0;
    int64_t total = 0;
    for (; i < n_rows && k < kMaxRows; ++i) {
      if (rows[i].n <= 0) continue;
      const int64_t more = (rows[i].n + kConvChunk - 1) / kConvChunk;
      if (total + more > INT32_MAX / 2) {
        if (k == 0) return (int)cudaErrorInvalidValue;
        break;
      }
      B.rows[k] = rows[i];
      B.begin[k++] = (int32_t)total;
      total += more;
    }
    if (k == 0) break;
    for (int j = k; j <= kMaxRows; ++j) B.begin[j] = (int32_t)total;
    B.total = (int)total;
    const int cap = sm_count() * kListCtasPerSm;
    launch(B, B.total < cap ? B.total : cap);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}
template <auto kKernel>
static int launch_rows(const FoConvRow* rows, int n_rows, cudaStream_t st) {
  return for_batches(rows, n_rows, [&](const ConvBatch& B, int grid) { kKernel<<<grid, kQThreads, 0, st>>>(B); });
}

// Calls f with the three recipe flags as template arguments.
template <typename F>
static int with_recipe(int is_signed, int do_sqrt, int softsign, F f) {
  using Y = std::true_type;
  using N = std::false_type;
  if (is_signed) {
    if (do_sqrt) return softsign ? f(Y(), Y(), Y()) : f(Y(), Y(), N());
    return softsign ? f(Y(), N(), Y()) : f(Y(), N(), N());
  }
  if (do_sqrt) return softsign ? f(N(), Y(), Y()) : f(N(), Y(), N());
  return softsign ? f(N(), N(), Y()) : f(N(), N(), N());
}
template <typename T>
static int quantize_rows(const FoConvRow* rows, int n_rows, int is_signed, int do_sqrt, int softsign, cudaStream_t st) {
  return with_recipe(is_signed, do_sqrt, softsign, [&](auto a, auto b, auto c) {
    return launch_rows<quantize_kernel<T, decltype(a)::value, decltype(b)::value, decltype(c)::value>>(rows, n_rows, st);
  });
}
template <typename T>
static int dequantize_rows(const FoConvRow* rows, int n_rows, int is_signed, int do_sqrt, int softsign, cudaStream_t st) {
  return with_recipe(is_signed, do_sqrt, softsign, [&](auto a, auto b, auto c) {
    return launch_rows<dequantize_kernel<T, decltype(a)::value, decltype(b)::value, decltype(c)::value>>(rows, n_rows, st);
  });
}

template <typename T, bool kSplit>
static int encode_rows(const FoConvRow* rows, int n_rows, int err_bytes, cudaStream_t st) {
  if (err_bytes == 1) return launch_rows<ecc_encode_kernel<T, int8_t, kSplit>>(rows, n_rows, st);
  if (err_bytes == 2) return launch_rows<ecc_encode_kernel<T, int16_t, kSplit>>(rows, n_rows, st);
  return (int)cudaErrorInvalidValue;
}
template <bool kSplit>
static int encode_rows_of(const FoConvRow* rows, int n_rows, int dtype, int err_bytes, cudaStream_t st) {
  if (dtype == FO_BF16) return encode_rows<__nv_bfloat16, kSplit>(rows, n_rows, err_bytes, st);
  if (dtype == FO_FP16) return encode_rows<__half, kSplit>(rows, n_rows, err_bytes, st);
  return (int)cudaErrorInvalidValue;
}
template <typename T>
static int decode_rows(const FoConvRow* rows, int n_rows, int err_bytes, cudaStream_t st) {
  if (err_bytes == 1) return launch_rows<ecc_decode_kernel<T, int8_t>>(rows, n_rows, st);
  if (err_bytes == 2) return launch_rows<ecc_decode_kernel<T, int16_t>>(rows, n_rows, st);
  return (int)cudaErrorInvalidValue;
}
template <typename T>
static void launch_maxabs(const void* x, int64_t n, float* out, cudaStream_t st) {
  launch_strided<maxabs_kernel<T>>((n + kUnit - 1) / kUnit, st, (const T*)x, n, out);
}

}  // namespace fo

extern "C" int fo_quantize_many(const FoConvRow* rows, int n_rows, int dtype, int is_signed, int do_sqrt, int softsign,
                                void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case FO_BF16: return fo::quantize_rows<__nv_bfloat16>(rows, n_rows, is_signed, do_sqrt, softsign, st);
    case FO_FP16: return fo::quantize_rows<__half>(rows, n_rows, is_signed, do_sqrt, softsign, st);
    case FO_FP32: return fo::quantize_rows<float>(rows, n_rows, is_signed, do_sqrt, softsign, st);
  }
  return (int)cudaErrorInvalidValue;
}

extern "C" int fo_dequantize_many(const FoConvRow* rows, int n_rows, int out_dtype, int is_signed, int do_sqrt,
                                  int softsign, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (out_dtype) {
    case FO_FP32: return fo::dequantize_rows<float>(rows, n_rows, is_signed, do_sqrt, softsign, st);
    case FO_BF16: return fo::dequantize_rows<__nv_bfloat16>(rows, n_rows, is_signed, do_sqrt, softsign, st);
  }
  return (int)cudaErrorInvalidValue;
}

extern "C" int fo_quantize(const void* x, int dtype, void* q, void* scales, int64_t n, int is_signed,
                           int do_sqrt, int softsign, void* stream) {
  if (n <= 0) return 0;
  const FoConvRow row = {x, nullptr, q, scales, n};
  return fo_quantize_many(&row, 1, dtype, is_signed, do_sqrt, softsign, stream);
}

extern "C" int fo_dequantize(const void* q, const void* scales, float* out, int64_t n, int is_signed,
                             int do_sqrt, int softsign, void* stream) {
  if (n <= 0) return 0;
  const FoConvRow row = {q, scales, out, nullptr, n};
  return fo_dequantize_many(&row, 1, FO_FP32, is_signed, do_sqrt, softsign, stream);
}

extern "C" int fo_ecc_decode_many(const FoConvRow* rows, int n_rows, int dtype, int err_bytes, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == FO_BF16) return fo::decode_rows<__nv_bfloat16>(rows, n_rows, err_bytes, st);
  if (dtype == FO_FP16) return fo::decode_rows<__half>(rows, n_rows, err_bytes, st);
  return (int)cudaErrorInvalidValue;
}
extern "C" int fo_ecc_split_many(const FoConvRow* rows, int n_rows, int dtype, int err_bytes, void* stream) {
  return fo::encode_rows_of<true>(rows, n_rows, dtype, err_bytes, static_cast<cudaStream_t>(stream));
}
extern "C" int fo_codes_to_narrow_many(const FoConvRow* rows, int n_rows, int dtype, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == FO_BF16) return fo::launch_rows<fo::code_cast_kernel<__nv_bfloat16, true>>(rows, n_rows, st);
  if (dtype == FO_FP16) return fo::launch_rows<fo::code_cast_kernel<__half, true>>(rows, n_rows, st);
  return (int)cudaErrorInvalidValue;
}
extern "C" int fo_narrow_to_codes_many(const FoConvRow* rows, int n_rows, int dtype, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == FO_BF16) return fo::launch_rows<fo::code_cast_kernel<__nv_bfloat16, false>>(rows, n_rows, st);
  if (dtype == FO_FP16) return fo::launch_rows<fo::code_cast_kernel<__half, false>>(rows, n_rows, st);
  return (int)cudaErrorInvalidValue;
}

extern "C" int fo_ecc_decode(const void* narrow, int dtype, const void* ecc, int err_bytes, float* out,
                             int64_t n, void* stream) {
  if (n <= 0) return 0;
  const FoConvRow row = {narrow, ecc, out, nullptr, n};
  return fo_ecc_decode_many(&row, 1, dtype, err_bytes, stream);
}

extern "C" int fo_ecc_encode(const float* x, const void* narrow, int dtype, void* ecc, int err_bytes,
                             int64_t n, void* stream) {
  if (n <= 0) return 0;
  const FoConvRow row = {x, narrow, ecc, nullptr, n};
  return fo::encode_rows_of<false>(&row, 1, dtype, err_bytes, static_cast<cudaStream_t>(stream));
}

extern "C" int fo_maxabs(const void* x, int dtype, int64_t n, float* out, void* stream) {
  if (n <= 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case FO_BF16: fo::launch_maxabs<__nv_bfloat16>(x, n, out, st); break;
    case FO_FP16: fo::launch_maxabs<__half>(x, n, out, st); break;
    case FO_FP32: fo::launch_maxabs<float>(x, n, out, st); break;
    default: return (int)cudaErrorInvalidValue;
  }
  return (int)cudaGetLastError();
}
