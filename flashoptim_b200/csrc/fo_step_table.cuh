// Launch configuration, segment table and chunk walker shared by the step kernels.
//
// No counterpart in the reference, which launches one Triton kernel per parameter tensor
// (flashoptim/optimizers.py:1535-1583, :2203-2252; grid from _make_grid, :2984-2996): here one
// launch walks a table of all tensors of a step.
#pragma once

#include "fo_step_core.cuh"

namespace fo {

#ifndef FO_UNROLL
#define FO_UNROLL 1
#endif
#ifndef FO_CTAS_PER_SM
#define FO_CTAS_PER_SM 4
#endif
#ifndef FO_THREADS
#define FO_THREADS 256
#endif
constexpr int kThreads = FO_THREADS;
constexpr int kUnroll = FO_UNROLL;  // units per thread per chunk; all loads of a chunk are issued before any math
constexpr int kChunk = kThreads * kUnit * kUnroll;
constexpr int kCtasPerSm = FO_CTAS_PER_SM;

// Step kernels are launched with programmatic stream serialisation: a grid may become resident
// while the one before it drains.  It touches no memory before grid_begin() returns, which is when
// everything before it on the stream has completed; grid_begin() also lets the next such grid
// become resident as this one's CTAs retire.  Nine launches of gradient release 260 -> 245 us, two
// launches over ResNet-18 29.3 -> 25.8, four small tensors 6.6 -> 6.0; single large launches unchanged.
__device__ __forceinline__ void grid_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
}
template <typename... Params, typename... Args>
static int launch_overlapped(void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t st,
                             const Args&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  if (e != cudaSuccess) cudaGetLastError();  // reported here, not by somebody's next check
  return (int)e;
}

struct InlineTable {
  FoSeg segs[FO_MAX_INLINE_SEGS];
  int32_t chunk_begin[FO_MAX_INLINE_SEGS + 1];
};

struct StepParams {
  const FoSeg* segs;           // device table (null when inline)
  const int32_t* chunk_begin;  // device table (null when inline)
  int n_seg;
  int total_chunks;
  unsigned int* status;  // optional pair of words where a kernel records a wait that ran out
  InlineTable inl;
};

// Records a wait that ran out in word `who` (0: producer, 1: consumer).  Plain stores: the words
// usually live in host memory, where read-modify-write operations of a GPU are not atomic.
__device__ __forceinline__ void report_timeout(unsigned int* status, int who) {
  if (!status) return;
  reinterpret_cast<volatile unsigned int*>(status)[who] = 1u << who;
  __threadfence_system();
}

// Walks the chunk list of one CTA: chunk c belongs to the segment s with
// chunk_begin[s] <= c < chunk_begin[s + 1]; a CTA visits chunks in increasing
// order, so the segment index only ever moves forward.
//
// A CTA's first look-up is a search by one of its warps: each round narrows the segments 32-fold,
// two rounds for a thousand.  Stepping through the table from segment 0 instead is a chain of
// dependent loads that every CTA pays: with 200 tensors of 1024 elements it took 13.2 us of which
// 3 us are the update.  The result goes through shared memory so that the compiler sees a value
// that is the same for all lanes and keeps segment and addresses out of the vector registers
// (taken from the ballot directly, a large launch was 4 % slower: these kernels are power bound).
// Later look-ups step, usually to the same or the next segment (a binary search there had the same
// effect on the registers, and cost as much).
struct ChunkWalker {
  const FoSeg* segs;
  const int32_t* cb;
  int total;
  int n_seg, seg, seg_begin, seg_end;
  FoSeg S;
  bool vec, vec_grad;

  // The whole CTA constructs its walker together (one barrier).
  __device__ __forceinline__ ChunkWalker(const StepParams& P)
      : segs(P.segs ? P.segs : P.inl.segs), cb(P.chunk_begin ? P.chunk_begin : P.inl.chunk_begin),
        total(P.total_chunks), n_seg(P.n_seg) {
    __shared__ int first;
    if (threadIdx.x < 32) {
      const int lane = threadIdx.x, c = blockIdx.x;
      int lo = 0, hi = n_seg;  // the segment of chunk c is in [lo, hi)
      while (hi - lo > 1) {
        const int stride = (hi - lo + 31) >> 5;
        const int last = lo + (lane + 1) * stride - 1;  // last segment of this lane's share
        const unsigned past = __ballot_sync(kFullMask, last >= hi - 1 || cb[last + 1] > c);
        lo += (__ffs(past) - 1) * stride;
        hi = min(lo + stride, hi);
      }
      if (lane == 0) first = lo;
    }
    __syncthreads();
    seg = first;
    enter();
  }
  __device__ __forceinline__ void enter() {
    S = segs[seg];
    seg_begin = cb[seg];
    seg_end = cb[seg + 1];
    vec = seg_state_vector_safe(S);
    vec_grad = seg_grad_vector_safe(S);
  }
  __device__ __forceinline__ void seek(int c) {
    if (c < seg_end) return;
    do { ++seg; } while (c >= cb[seg + 1]);
    enter();
  }
  __device__ __forceinline__ int64_t unit_base(int c, int u) const {
    return (int64_t)(c - seg_begin) * kChunk + (int64_t)(u * kThreads + threadIdx.x) * kUnit;
  }
};


// Bulk-copy staged variants (fo_step_staged.cu).  Return -1 when the combination is not
// served by a staged kernel (the caller then uses the register-path kernel).
int staged_adam_launch(const StepParams& P, const FoAdamHyper& H, int dtype, int err_bytes, int quantized,
                       int sm_count, cudaStream_t st);
int staged_momentum_launch(const StepParams& P, const FoMomentumHyper& H, int dtype, int err_bytes,
                           int state_mode, int sm_count, cudaStream_t st);

}  // namespace fo
