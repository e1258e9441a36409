// Bulk-copy staged variants of the fused steps (8-bit states).
// Same arithmetic as the reference's step kernels (flashoptim/optimizers.py:1587-1719,
// :2256-2443); the data path below has no counterpart there.
//
// The register-path kernels hold at most 32 warps x 56 B of loads in flight per
// SM and sit at about one eligible warp per scheduler.  Here a producer warp
// streams whole chunks (parameter, gradient, correction codes, state codes and
// their scales: 14-21 KB) into a ring of shared-memory stages with
// cp.async.bulk (the TMA unit's untiled copy; no multicast, no tensor map),
// completion is tracked by one mbarrier per stage, and four consumer warps read
// 16 elements per thread from shared memory, release the stage and run the same
// update as the register path.  Up to kStages - 1 chunks per CTA are in
// flight regardless of what the consumers are doing.
//
// A chunk that is not a full 2048-element block (a tail), or whose parameter or
// states do not start on 16 bytes, skips the copy engine: the producer completes
// the stage's phase with a plain arrive and the consumers load it directly.  The
// gradient may start anywhere (chunk_is_staged).
//
// Every mbarrier wait is bounded (wall clock); a wait that runs out records a
// code in StepParams.status (when given), and the waiting warp leaves its loop.
#include "fo_stage.cuh"
#include "fo_step_table.cuh"

namespace fo {

// A consumer thread owns kSpan = 16 consecutive elements of a chunk, half a quantisation group:
// the group's absmax takes one shuffle, codes move as 16-byte vectors, and what a thread spends per
// chunk outside the arithmetic (barrier, addresses, constants, scales) is shared by 16 elements.
// These kernels are bound by instruction issue (43 per AdamW element, 67 % of the issue slots) and,
// through it, by the power cap: 1.53-1.56 of 1.965 GHz at 998 W over 150 steps of 8.03 B elements.
constexpr int kSpan = 16;
constexpr int kStagedChunk = kChunk;  // elements; the chunk prefix is shared with the register path
constexpr int kConsumerThreads = kStagedChunk / kSpan;
constexpr int kConsumerWarps = kConsumerThreads / 32;
constexpr int kStagedThreads = kConsumerThreads + 32;

// Ring depth and CTAs per SM.  -DFO_STAGES / -DFO_STAGED_CTAS_PER_SM override both for tuning builds
// (-DFO_STAGES_FP32 / -DFO_STAGED_CTAS_PER_SM_FP32 for fp32 parameters, whose stages are larger).
// AdamW, fp32, 124 M elements in 148 tensors: register path 377 us, 3 stages on 3 CTAs 377, 4 on 2
// 366, 2 on 4 322 (6.3 TB/s): the consumers need the warps more than the copies need the depth.
#ifndef FO_STAGES
#define FO_STAGES 3
#endif
#ifndef FO_STAGED_CTAS_PER_SM
#define FO_STAGED_CTAS_PER_SM 4
#endif
#ifndef FO_STAGES_FP32
#define FO_STAGES_FP32 2
#endif
#ifndef FO_STAGED_CTAS_PER_SM_FP32
#define FO_STAGED_CTAS_PER_SM_FP32 4
#endif
template <typename T>
struct StageConfig {
  static constexpr int kStages = sizeof(T) == 4 ? FO_STAGES_FP32 : FO_STAGES;
  static constexpr int kCtasPerSm = sizeof(T) == 4 ? FO_STAGED_CTAS_PER_SM_FP32 : FO_STAGED_CTAS_PER_SM;
};

template <typename T, int kErr, int kStates>
struct StageLayout {
  static constexpr int kP = 0;
  static constexpr int kEcc = kP + kStagedChunk * (int)sizeof(T);
  static constexpr int kQ0 = kEcc + kStagedChunk * kErr;
  static constexpr int kQ1 = kQ0 + kStagedChunk;
  static constexpr int kS0 = kQ0 + kStagedChunk * kStates;
  static constexpr int kS1 = kS0 + (kStagedChunk / kGroup) * 2;
  // gradient last: 16 bytes more when it does not start on a 16-byte boundary
  static constexpr int kG = kS0 + kStates * (kStagedChunk / kGroup) * 2;
  static constexpr int kBytes = kG + kStagedChunk * (int)sizeof(T);
  static constexpr int kStride = (kBytes + 16 + 127) / 128 * 128;
};

// A chunk goes through the copy engine when it is a full block of a segment whose
// streams (including the scale vectors) are 16-byte aligned.  The gradient may start anywhere:
// the copy then begins at the 16-byte boundary below it and ends at the one above its last byte
// (both inside the 16-byte blocks that the gradient itself touches), and the consumers shift.
// Element-wise global loads instead cost three times the whole update (0.79 against 0.26 ms for
// 108 M fp16 elements).
__device__ __forceinline__ bool chunk_is_staged(const ChunkWalker& w, int c) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(w.S.s0s) | reinterpret_cast<uintptr_t>(w.S.s1s);
  const int64_t base = (int64_t)(c - w.seg_begin) * kStagedChunk;
  return w.vec && (a & 15) == 0 && base + kStagedChunk <= w.S.n;
}

// 32 bytes: one 256-bit store where the address allows.
__device__ __forceinline__ void st32(void* p, const uint4& lo, const uint4& hi) {
  if ((reinterpret_cast<uintptr_t>(p) & 31) == 0) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(lo.x), "r"(lo.y), "r"(lo.z),
                 "r"(lo.w), "r"(hi.x), "r"(hi.y), "r"(hi.z), "r"(hi.w)
                 : "memory");
  } else {
    st16(p, lo);
    st16(static_cast<char*>(p) + 16, hi);
  }
}

// kVecs 16-byte vectors that start kWord words and `bits` (0 or 16) bits into one more of them.
template <int kWord, int kVecs>
__device__ __forceinline__ void shift_words(const uint32_t (&w)[4 * kVecs + 4], int bits, uint4 (&out)[kVecs]) {
  uint32_t o[4 * kVecs];
#pragma unroll
  for (int i = 0; i < 4 * kVecs; ++i) o[i] = __funnelshift_r(w[i + kWord], w[i + kWord + 1], bits);
#pragma unroll
  for (int i = 0; i < kVecs; ++i) out[i] = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
}
// A span of a gradient whose first element lies `skew` bytes (2 ... 14) behind `src`.
template <int kVecs>
__device__ __forceinline__ void load_skewed(const unsigned char* src, int skew, uint4 (&out)[kVecs]) {
  uint32_t w[4 * kVecs + 4];
#pragma unroll
  for (int i = 0; i < kVecs + 1; ++i) {
    const uint4 x = *reinterpret_cast<const uint4*>(src + i * 16);
    w[4 * i] = x.x, w[4 * i + 1] = x.y, w[4 * i + 2] = x.z, w[4 * i + 3] = x.w;
  }
  const int bits = (skew & 3) * 8;
  switch (skew >> 2) {
    case 0: shift_words<0>(w, bits, out); break;
    case 1: shift_words<1>(w, bits, out); break;
    case 2: shift_words<2>(w, bits, out); break;
    default: shift_words<3>(w, bits, out); break;
  }
}

// Half h of a span.
template <typename T, int kVecs>
__device__ __forceinline__ Raw8<T> raw8_of(const uint4 (&span)[kVecs], int h) {
  Raw8<T> r;
  r.v = span[h * kVecs / 2];
  if constexpr (sizeof(T) == 4) r.w = span[h * kVecs / 2 + 1];
  return r;
}

// One span out of shared memory, updated and stored.
template <typename T, int kErr, int kStates, typename Hyper, typename Update>
__device__ __forceinline__ void staged_span(const FoSeg& S, int64_t chunk_base, const unsigned char* st,
                                            uint64_t* empty_bar, const Hyper& H, Update update) {
  using L = StageLayout<T, kErr, kStates>;
  constexpr int kSpanBytes = kSpan * sizeof(T), kVecs = kSpanBytes / 16;
  const int t = threadIdx.x;
  uint4 rp[kVecs], rg[kVecs], ecc[2], q[2];
  float sc[2];
  const int skew = (int)(reinterpret_cast<uintptr_t>(S.g) & 15);
#pragma unroll
  for (int i = 0; i < kVecs; ++i) rp[i] = *reinterpret_cast<const uint4*>(st + L::kP + t * kSpanBytes + i * 16);
  if (skew == 0) {
#pragma unroll
    for (int i = 0; i < kVecs; ++i) rg[i] = *reinterpret_cast<const uint4*>(st + L::kG + t * kSpanBytes + i * 16);
  } else {
    load_skewed(st + L::kG + t * kSpanBytes, skew, rg);
  }
  if constexpr (kErr == 1) {
    const uint4 e = *reinterpret_cast<const uint4*>(st + L::kEcc + t * 16);
    ecc[0] = make_uint4(e.x, e.y, 0, 0);
    ecc[1] = make_uint4(e.z, e.w, 0, 0);
  } else if constexpr (kErr == 2) {
#pragma unroll
    for (int h = 0; h < 2; ++h) ecc[h] = *reinterpret_cast<const uint4*>(st + L::kEcc + t * 32 + h * 16);
  }
#pragma unroll
  for (int k = 0; k < kStates; ++k) {
    q[k] = *reinterpret_cast<const uint4*>(st + (k == 0 ? L::kQ0 : L::kQ1) + t * 16);
    sc[k] = __half2float(*reinterpret_cast<const __half*>(st + (k == 0 ? L::kS0 : L::kS1) + (t >> 1) * 2));
  }
  __syncwarp();
  if ((t & 31) == 0) mbar_arrive(empty_bar);  // this warp holds its spans in registers now

  float2 m[2][4], v[2][4];
  Raw8<T> pn[2];
  uint4 en[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float2 p[4], g[4], back[4], res[4];
    unpack8<T>(raw8_of<T>(rp, h), p);
    unpack8<T>(raw8_of<T>(rg, h), g);
    if constexpr (kErr != 0) {
      float2 c[4];
      ecc_codes_scaled<T, kErr>(ecc[h], c);
      ecc_apply8<T>(p, c);
    }
    dequant_softsign8(h == 0 ? make_uint2(q[0].x, q[0].y) : make_uint2(q[0].z, q[0].w), sc[0], m[h]);
    if constexpr (kStates == 2)
      dequant_sqrt8(h == 0 ? make_uint2(q[1].x, q[1].y) : make_uint2(q[1].z, q[1].w), sc[1], v[h]);
    update(p, g, m[h], v[h], H);
    pack8<T>(p, pn[h], back);
    if constexpr (kErr == 1) {
      ecc_residual8<T, 1>(p, back, res);
      const uint2 c = round_to_bytes(res);
      if (h == 0) en[0].x = c.x, en[0].y = c.y;
      else en[0].z = c.x, en[0].w = c.y;
    } else if constexpr (kErr == 2) {
      ecc_residual8<T, 2>(p, back, res);
      en[h] = round_to_shorts(res);
    }
  }
  const int64_t base = chunk_base + t * kSpan;
  char* out = static_cast<char*>(S.p) + base * (int)sizeof(T);
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int h = 0; h < 2; ++h) st32(out + h * 32, pn[h].v, pn[h].w);
  } else {
    st32(out, pn[0].v, pn[1].v);
  }
  if constexpr (kErr == 1) st16(static_cast<char*>(S.ecc) + base, en[0]);
  else if constexpr (kErr == 2) st32(static_cast<char*>(S.ecc) + base * 2, en[0], en[1]);
  uint4 codes;
  const float a0 = quant_softsign16(m, codes);
  st16(static_cast<char*>(S.s0) + base, codes);
  if ((t & 1) == 0) static_cast<__half*>(S.s0s)[base >> 5] = __float2half_rn(a0);
  if constexpr (kStates == 2) {
    const float a1 = quant_sqrt16_pre(v, codes);
    st16(static_cast<char*>(S.s1) + base, codes);
    if ((t & 1) == 0) static_cast<__half*>(S.s1s)[base >> 5] = __float2half_rn(a1);
  }
}

template <typename T, int kErr, int kStates, typename Hyper, typename Update>
__device__ __forceinline__ void staged_body(const StepParams& P, const Hyper& H, Update update) {
  using L = StageLayout<T, kErr, kStates>;
  using Regs = UnitRegs<T, kErr, kStates, true>;
  constexpr int kStages = StageConfig<T>::kStages;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t full[kStages], empty[kStages];

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kConsumerWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  grid_begin();
  ChunkWalker w(P);  // its barrier also publishes the mbarriers

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int s = 0;           // ring position and the parity of its current round
  uint32_t parity = 0;
  if (warp == kConsumerWarps) {
    // ---------------------------------------------------------------- producer
    if (lane != 0) return;  // a whole warp walking along costs 2 % of the time under the power cap
    int round = 0;
    for (int c = blockIdx.x; c < w.total; c += gridDim.x) {
      if (round > 0 && !mbar_wait(&empty[s], parity ^ 1)) {
        report_timeout(P.status, 0);
        // the consumers of stage s never came; the other stages' copies must have landed before
        // this CTA may end
        for (int k = 0; k < kStages; ++k)
          if (k != s) mbar_wait(&full[k], k < s ? parity : parity ^ 1);
        return;
      }
      w.seek(c);
      if (!chunk_is_staged(w, c)) {
        mbar_arrive(&full[s]);
      } else {
        const int64_t base = (int64_t)(c - w.seg_begin) * kStagedChunk;
        unsigned char* st = smem + s * L::kStride;
        const char* g = static_cast<const char*>(w.S.g) + base * (int)sizeof(T);
        const uint32_t skew = (uint32_t)(reinterpret_cast<uintptr_t>(g) & 15), more = skew ? 16 : 0;
        constexpr uint32_t kValueBytes = kStagedChunk * sizeof(T);
        constexpr uint32_t kScaleBytes = (kStagedChunk / kGroup) * 2;
        mbar_arrive_expect_tx(&full[s], L::kBytes + more);
        bulk_load(st + L::kP, static_cast<const char*>(w.S.p) + base * (int)sizeof(T), kValueBytes, &full[s]);
        bulk_load(st + L::kG, g - skew, kValueBytes + more, &full[s]);
        if constexpr (kErr > 0)
          bulk_load(st + L::kEcc, static_cast<const char*>(w.S.ecc) + base * kErr, kStagedChunk * kErr, &full[s]);
        bulk_load(st + L::kQ0, static_cast<const char*>(w.S.s0) + base, kStagedChunk, &full[s]);
        bulk_load(st + L::kS0, static_cast<const char*>(w.S.s0s) + (base >> 5) * 2, kScaleBytes, &full[s]);
        if constexpr (kStates == 2) {
          bulk_load(st + L::kQ1, static_cast<const char*>(w.S.s1) + base, kStagedChunk, &full[s]);
          bulk_load(st + L::kS1, static_cast<const char*>(w.S.s1s) + (base >> 5) * 2, kScaleBytes, &full[s]);
        }
      }
      if (++s == kStages) s = 0, parity ^= 1, round = 1;
    }
    return;
  }

  // ------------------------------------------------------------------ consumers
  for (int c = blockIdx.x; c < w.total; c += gridDim.x) {
    w.seek(c);
    const int64_t chunk_base = (int64_t)(c - w.seg_begin) * kStagedChunk;
    // one verdict per warp: at the deadline lanes may disagree, and the group shuffles need all
    // 32 lanes
    if (!__all_sync(kFullMask, mbar_wait(&full[s], parity))) {
      if (lane == 0) report_timeout(P.status, 1);
      return;
    }
    if (chunk_is_staged(w, c)) {
      staged_span<T, kErr, kStates>(w.S, chunk_base, smem + s * L::kStride, &empty[s], H, update);
    } else {
      if (lane == 0) mbar_arrive(&empty[s]);  // nothing was staged
#pragma unroll 1
      for (int u = 0; u < kSpan / kUnit; ++u) {
        const int64_t base = chunk_base + (int64_t)(u * kConsumerThreads + threadIdx.x) * kUnit;
        Regs r;
        load_unit_state(r, w.S, base, w.vec);
        load_unit_grad(r, w.S, base, w.vec_grad);
        float2 p[4], g[4], m[4], v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) m[i] = v[i] = make_float2(0.f, 0.f);
        unpack8<T>(r.g, g);
        widen_unit(r, p, m, v);
        update(p, g, m, v, H);
        store_unit(r, w.S, base, w.vec, p, m, v);
      }
    }
    if (++s == kStages) s = 0, parity ^= 1;
  }
}

struct AdamUpdate {
  __device__ __forceinline__ void operator()(float2 (&p)[4], const float2 (&g)[4], float2 (&m)[4], float2 (&v)[4],
                                             const FoAdamHyper& H) const {
    adam_update8<true>(p, g, m, v, H);
  }
};
struct MomentumUpdate {
  __device__ __forceinline__ void operator()(float2 (&p)[4], const float2 (&g)[4], float2 (&m)[4], float2 (&v)[4],
                                             const FoMomentumHyper& H) const {
    momentum_update8(p, g, m, H, true);
  }
};

template <typename T, int kErr>
__global__ void __launch_bounds__(kStagedThreads, StageConfig<T>::kCtasPerSm)
    adam_staged_kernel(const __grid_constant__ StepParams P, const __grid_constant__ FoAdamHyper H) {
  staged_body<T, kErr, 2>(P, H, AdamUpdate());
}
template <typename T, int kErr>
__global__ void __launch_bounds__(kStagedThreads, StageConfig<T>::kCtasPerSm)
    momentum_staged_kernel(const __grid_constant__ StepParams P, const __grid_constant__ FoMomentumHyper H) {
  staged_body<T, kErr, 1>(P, H, MomentumUpdate());
}

// Grid = resident CTAs x up to this factor: the hardware hands out the later CTAs as earlier
// ones finish, which evens out SMs that run at different paces (equal fixed shares wait for
// the slowest).  On the 291-tensor Llama-3-8B list, sustained under the power cap: AdamW-24
// 2.30 -> 2.24 ms per 1 B parameters, AdamW-32 2.54 -> 2.40, Lion-24 1.83 -> 1.78 for a factor of
// 6-12; 32 loses part of it again.  A CTA keeps at least kMinChunksPerCta chunks so that its
// ring fills: launches below about 60 M elements keep one round.
#ifndef FO_STAGED_ROUNDS
#define FO_STAGED_ROUNDS 8
#endif
static int g_staged_rounds = FO_STAGED_ROUNDS;
constexpr int kMinChunksPerCta = 16;

template <typename T, int kErr, int kStates, typename Kernel, typename Hyper>
static int launch_staged(Kernel kernel, const StepParams& P, const Hyper& H, int sm_count, cudaStream_t st) {
  constexpr int smem_bytes = StageConfig<T>::kStages * StageLayout<T, kErr, kStates>::kStride;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
  if (e != cudaSuccess) return (int)e;
  const int64_t resident = (int64_t)sm_count * StageConfig<T>::kCtasPerSm;
  int64_t rounds = P.total_chunks / (resident * kMinChunksPerCta);
  if (rounds > g_staged_rounds) rounds = g_staged_rounds;
  if (rounds < 1) rounds = 1;
  int64_t grid = resident * rounds;
  if (P.total_chunks < grid) grid = P.total_chunks;
  return launch_overlapped(kernel, (int)grid, kStagedThreads, smem_bytes, st, P, H);
}

template <typename T>
static int staged_adam_t(const StepParams& P, const FoAdamHyper& H, int err, int sms, cudaStream_t st) {
  switch (err) {
    case 0: return launch_staged<T, 0, 2>(adam_staged_kernel<T, 0>, P, H, sms, st);
    case 1: return launch_staged<T, 1, 2>(adam_staged_kernel<T, 1>, P, H, sms, st);
    case 2: return launch_staged<T, 2, 2>(adam_staged_kernel<T, 2>, P, H, sms, st);
  }
  return -1;
}
template <typename T>
static int staged_momentum_t(const StepParams& P, const FoMomentumHyper& H, int err, int sms, cudaStream_t st) {
  switch (err) {
    case 0: return launch_staged<T, 0, 1>(momentum_staged_kernel<T, 0>, P, H, sms, st);
    case 1: return launch_staged<T, 1, 1>(momentum_staged_kernel<T, 1>, P, H, sms, st);
    case 2: return launch_staged<T, 2, 1>(momentum_staged_kernel<T, 2>, P, H, sms, st);
  }
  return -1;
}

int staged_adam_launch(const StepParams& P, const FoAdamHyper& H, int dtype, int err_bytes, int quantized,
                       int sm_count, cudaStream_t st) {
  if (!quantized) return -1;
  if (dtype == FO_BF16) return staged_adam_t<__nv_bfloat16>(P, H, err_bytes, sm_count, st);
  if (dtype == FO_FP16) return staged_adam_t<__half>(P, H, err_bytes, sm_count, st);
  if (dtype == FO_FP32 && err_bytes == 0) return launch_staged<float, 0, 2>(adam_staged_kernel<float, 0>, P, H, sm_count, st);
  return -1;
}

int staged_momentum_launch(const StepParams& P, const FoMomentumHyper& H, int dtype, int err_bytes,
                           int state_mode, int sm_count, cudaStream_t st) {
  if (state_mode != FO_STATE_Q8) return -1;
  if (dtype == FO_BF16) return staged_momentum_t<__nv_bfloat16>(P, H, err_bytes, sm_count, st);
  if (dtype == FO_FP16) return staged_momentum_t<__half>(P, H, err_bytes, sm_count, st);
  if (dtype == FO_FP32 && err_bytes == 0) return launch_staged<float, 0, 1>(momentum_staged_kernel<float, 0>, P, H, sm_count, st);
  return -1;
}

}  // namespace fo

extern "C" void fo_set_staged_rounds(int rounds) { fo::g_staged_rounds = rounds < 1 ? 1 : (rounds > 1024 ? 1024 : rounds); }
extern "C" int fo_get_staged_rounds(void) { return fo::g_staged_rounds; }

