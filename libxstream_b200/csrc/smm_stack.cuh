/*
 * Device building blocks shared by the stack-kernel translation units: programmatic dependent launch,
 * the FP64 tensor instruction, warp tiles of C and their write-back, the description of one stack
 * (StackTask) and the L2 prefetch of its operands.
 */
#pragma once

#include "internal.h"
#include "tc_ptx.cuh"
#include <cuda_runtime.h>
#include <stdint.h>

namespace xs_stack {

/* Programmatic dependent launch: a kernel launched with pdl_launch may be scheduled while the
   kernel before it in the stream is still running (once that kernel's CTAs have all passed
   pdl_trigger or exited); it must call pdl_wait before it reads anything its predecessor writes.
   Both are no-ops for a kernel launched the ordinary way. */
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" :::); }

template <typename... KArgs, typename... Args>
cudaError_t pdl_launch(void (*kernel)(KArgs...), int grid, int block, size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

/* Release/acquire fence at GPU scope: orders this thread's piece stores before its (relaxed) arrival
   increment, and a CTA's reads of the other CTAs' pieces after the increment that found them all
   published. Lighter than the sequentially consistent __threadfence(). */
__device__ __forceinline__ void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

/* Bring a block of `count` contiguous doubles into L2 (one prefetch per 128-byte line, by 32 lanes). */
__device__ __forceinline__ void prefetch_block_l2(const double* p, int count, int lane) {
  for (int x = 16 * lane; x < count + 15; x += 16 * 32) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p + (x < count ? x : count - 1)));
  }
}

__device__ __forceinline__ void dmma_m8n8k4(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

/* Per-lane geometry of a warp sub-tile (8*MT x 8*NT of C): which fragment rows/columns it loads. */
template <int MT, int NT>
struct Tile {
  bool rok[MT], cok[NT];
  int r0, c0;
  __device__ __forceinline__ void init(int sub, int nsub_n, int m, int n, int g) {
    const int sm = sub / nsub_n, sn = sub - sm * nsub_n;
    r0 = sm * 8 * MT;
    c0 = sn * 8 * NT;
#pragma unroll
    for (int i = 0; i < MT; ++i) rok[i] = r0 + 8 * i + g < m;
#pragma unroll
    for (int j = 0; j < NT; ++j) cok[j] = c0 + 8 * j + g < n;
  }
};

/* Write-back of a finished C sub-tile: each element has exactly one writer (red.global.add.f64). */
template <int MT, int NT>
__device__ __forceinline__ void commit_tile(double* __restrict__ C, size_t coff, const double (&acc)[MT][NT][2], int m,
  int n, int g, int t, const Tile<MT, NT>& tl, double alpha) {
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    const int r = tl.r0 + 8 * i + g;
    if (r < m) {
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int cc = tl.c0 + 8 * j + 2 * t;
        if (cc < n) atomicAdd(C + coff + (size_t)cc * m + r, alpha * acc[i][j][0]);
        if (cc + 1 < n) atomicAdd(C + coff + (size_t)(cc + 1) * m + r, alpha * acc[i][j][1]);
      }
    }
  }
}

/* What the stack kernel needs to know about one stack: one task for a single call, one per stack
   for a batch. keys/vals are the stack's grouped entries, pieces its CTA-level piece slots. */
struct StackTask {
  const double* a;
  const double* b;
  double* c;
  const unsigned* keys;
  const unsigned long long* vals;
  double* pieces;
  int S, m, n, k;
  int L, nchunks, ngroups, nsub_n, nsub;
  int item_begin; /* first work item of this stack (batch) */
  int cls;        /* tile class (MT - 1) * 4 + (NT - 1) (batch) */
  int sid;        /* stack index within the call: tag of its segment-list entries */
  int kind;       /* unified batch kernel: 0 = register kernel of tile class cls, else 1 + staged shape index */
  double alpha;   /* C += alpha * A * B (1 for the LIBSMM ABI) */
  int* arrive;    /* per (CTA group, sub-tile) arrival counters of CTA-crossing segments, zero at launch:
                     the stack kernel combines them itself; nullptr: they go to the combine kernel */
  const int* raw; /* the caller's parameter stack (input of the grouping), for the L2 prefetch */
  int rstride;    /* ints per parameter record (3 or 6) */
  int rbase;      /* a-offset position within a record (b follows) */
  int rshift;     /* added to a record's offsets to make them 0-based (-1: 1-based, 0: 0-based) */
  int npf;        /* records whose A and B blocks are prefetched into L2 (0: none) */
  int Ls[3];      /* entries per chunk in the CTA groups [0, slotn), [slotn, 2 slotn), [2 slotn, ...) */
  int slotn;      /* CTA groups per length class (the SM count when the lengths differ) */
};

/* Bulk prefetch into L2 of the A and B blocks of the first tk.npf parameter records, dealt round-robin
   over the CTAs (record i to CTA i mod grid), so that every SM's copy unit issues a share. It reads only the caller's inputs (the raw stack and the pools), so a stack kernel
   runs it before pdl_wait, while the grouping that precedes it in the stream still runs and the
   pools would otherwise be fetched only at the first copy. A block's window is widened to 16-byte
   boundaries (the bulk-copy granule); a widened window never leaves the block's page. */
__device__ __forceinline__ void prefetch_block(const double* p, uint32_t bytes) {
  const uint64_t s = (uint64_t)p, s0 = s & ~15ull, s1 = (s + bytes + 15ull) & ~15ull;
  xs_tc::bulk_prefetch_l2((const void*)s0, (uint32_t)(s1 - s0));
}
__device__ __forceinline__ void prefetch_operands(const StackTask& tk) {
  if (0 >= tk.npf) return;
  const uint32_t abytes = (uint32_t)(tk.m * tk.k * sizeof(double)), bbytes = (uint32_t)(tk.k * tk.n * sizeof(double));
  const int nthreads = (int)(gridDim.x * blockDim.x);
  for (int i = (int)(blockIdx.x + gridDim.x * threadIdx.x); i < tk.npf; i += nthreads) {
    const int* const e = tk.raw + (size_t)tk.rstride * i + tk.rbase;
    prefetch_block(tk.a + (e[0] + tk.rshift), abytes);
    prefetch_block(tk.b + (e[1] + tk.rshift), bbytes);
  }
}

}  // namespace xs_stack
