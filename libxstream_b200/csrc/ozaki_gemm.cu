/*
 * Ozaki scheme-1 FP64 GEMM on the int8 tensor cores (tcgen05 with tensor-memory accumulators).
 *
 * C = alpha * op(A) * op(B) + beta * C, FP64, column-major (BLAS conventions). Each row of op(A)
 * and each column of op(B) is scaled by its largest power of two (the biased exponent of its
 * largest entry) and split into `nslices` signed 7-bit digits of the aligned 53-bit significand,
 * as the reference does (samples/ozaki/kernels/ozaki_common.cl:789-834 digit rule,
 * samples/ozaki/kernels/ozaki1_int8.cl:428-589 preprocessing): digit s holds bits
 * [46-7s, 52-7s] of the aligned significand; the eighth digit (bits [0,3]) is stored multiplied by
 * 8, so that every digit s carries weight 2^(46-7s) and a slice pair (sa, sb) weighs
 * 2^(92-7(sa+sb)). All pairs with sa + sb <= cutoff are multiplied on the tensor cores (int8 x int8
 * -> exact int32 sums); pairs of one anti-diagonal d = sa + sb share one tensor-memory
 * accumulator (their scales are equal), so one FP64 recombination per diagonal suffices:
 *   C(i,j) += alpha * 2^(ea_i + eb_j - 2058 - 7d) * D_d(i,j)        (ozaki1_int8.cl:740-790).
 * Exactness of the int32 sums: |digit| <= 127 and a diagonal holds at most 8 pairs, so a K range
 * of at most 16384 keeps |D_d| < 8 * 16384 * 127^2 < 2^31; longer K runs in chunks of 16384.
 *
 * Device layout: digit panels, the order in which the GEMM reads them. Rows of op(A) in blocks of 128
 * and columns of op(B) in blocks of 64 (one block of 8 or 16 rows' granularity when there are fewer), k in blocks of 32:
 * panel (row block, k block) holds all slices one after the other, each as core matrices of 8 rows x 16 bytes (row
 * group g at 256 g, k half h at 128 h, row r % 8 at 16 (r % 8)); K zero padded; exponents ea[M], eb[N] (int32).
 *
 * GEMM kernel: persistent, one CTA per SM, 10 warps, tiles of 128 x 64 of C with ALL anti-diagonals (up to
 * eight at a time: 8 x 64 = 512 tensor-memory columns) accumulated at once. A stage takes the A and the B panels of
 * as many k blocks as fit 36 KB, one at least, with one bulk copy each; as the B slices lie one after the other, one
 * tcgen05.mma (M = 128, N = 64 w, K = 32) of A slice sa against the w slices from sb on adds the pairs (sa, sb + i) to
 * diagonals sa + sb + i. So every digit is read once per tile instead of once per pair, and C once:
 * 42 KB per 28 pairs of a 32-wide k block at 7 slices, 47 bytes per cycle and SM (128 x 256 tiles, one pair at a
 * time, took 96, more than the L2 delivers, and added every diagonal into C or tensor memory). Warp 0
 * copies, warp 1 issues the MMAs, warps 2-9 (two per tensor-memory lane quarter) combine the diagonals of a
 * finished tile in FP64, smallest weight first, and write C. The MMAs of a tile wait for the epilogue of
 * the one before (tensor memory is full): about 3 % at K = 4096. More than eight diagonals (no trim) run as
 * several launches that add into C.
 * Measured on B200 (whole calls, pairs up to the diagonal, 4096^3; slice-pair tiles -> this): 7 slices 2319 -> 1563 us, 88
 * TFLOP/s FP64-equivalent, tensor pipe 63 % busy; 4 slices 1034 -> 923, 3 slices 743 -> 674 (with stages of one k block and
 * MMAs put together by the issuing thread from packed fields 1611, 980, 879: that thread bounds forms of few slices).
 * Every mbarrier wait is bounded: a stalled pipeline ends the kernel with an error status (per-call
 * abort word and the library's device error word) instead of a hang.
 */
#include "internal.h"
#include "tc_ptx.cuh"
#include "ozaki_digits.cuh"
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

extern "C" unsigned* xs_device_error_ptr(void);

namespace {
using namespace xs_tc;
using namespace xs_oz;

constexpr int kBM = 128, kBN = 64, kBK = 32;
constexpr int kMaxSlices = 8;
constexpr int kMaxDiag = 512 / kBN;       /* diagonals in tensor memory at a time */
constexpr int kMaxStages = 9;
constexpr int kStageBytes = 36 * 1024;    /* k blocks share a stage as long as it does not pass this size */
constexpr int kRegOps = 4;
constexpr int kMaxOps = 3 * kMaxSlices;   /* MMAs per k block */
constexpr int kKChunkBlocks = 16384 / kBK; /* k blocks per launch: keeps every diagonal's int32 sum exact */
constexpr int kEpiWarps = 8;
constexpr int kGemmThreads = 64 + 32 * kEpiWarps;
constexpr int kGroupM = 8; /* row panels per rasterization group */
constexpr unsigned kErrOzakiTimeout = 4u; /* device error word bit: an Ozaki pipeline wait timed out */

/* ------------------------------------------------------------------------------ slicing */

/* Row maxima of the biased exponent, rows contiguous in memory: element (r, k) at x[r + k*ld].
   Grid (ceil(R/256), k-chunks), eight loads in flight per thread; partial maxima meet in emax[] (zeroed by
   the caller) by atomicMax. */
__global__ void xs_oz_rowexp_rc(const double* __restrict__ x, long long ld, int R, int K, int kchunk, int* __restrict__ emax) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= R) return;
  const int k0 = blockIdx.y * kchunk, k1 = min(K, k0 + kchunk);
  int e = 0;
  for (int k = k0; k < k1; k += 8) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = (k + u < k1) ? x[r + (long long)(k + u) * ld] : 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) e = max(e, biased_exp(v[u]));
  }
  if (0 != e) atomicMax(emax + r, e);
}

/* Row maxima with k contiguous: element (r, k) at x[k + r*ld]; one warp per row. */
__global__ void xs_oz_rowexp_kc(const double* __restrict__ x, long long ld, int R, int K, int* __restrict__ emax) {
  const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= R) return;
  const double* const row = x + (long long)r * ld;
  int e = 0;
  for (int k = lane; k < K; k += 32) e = max(e, biased_exp(row[k]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
  if (0 == lane) emax[r] = e;
}

/* Digits of 16 consecutive k of one row into the slices of its panel (16 bytes of a core matrix each),
   `slice` bytes apart. */
__device__ __forceinline__ void slice16(const double (&v)[16], int erow, int ns, signed char* __restrict__ d, int slice) {
  unsigned long long al[16];
  unsigned sg[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    int be;
    unsigned long long mt;
    ieee_split(v[j], sg[j], be, mt);
    const int sh = erow - be;
    al[j] = (0 != mt && sh <= 52) ? (mt >> sh) : 0ull;
  }
  for (int s = 0; s < ns; ++s) {
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t x = 0;
#pragma unroll
      for (int b = 0; b < 4; ++b) x |= ((uint32_t)(slice_digit(al[q * 4 + b], sg[q * 4 + b], s) & 0xFF)) << (8 * b);
      w[q] = x;
    }
    *reinterpret_cast<uint4*>(d + s * slice) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

/* Bytes from the start of the digit panels to row r, k group kg (of 16) of slice 0; rb rows per block. */
__device__ __forceinline__ long long panel_offset(int r, int kg, int Kp, int ns, int rb) {
  const int blk = r / rb, rr = r - blk * rb;
  return ((long long)blk * (Kp / kBK) + (kg >> 1)) * ns * (rb * kBK) + (rr >> 3) * 256 + (kg & 1) * 128 + (rr & 7) * 16;
}

/* Slicing with k contiguous (element (r, k) at x[k + r*ld]): one thread per (row, 16 k), eight rows of one
   k group side by side, so that they write whole core matrices. */
__global__ void xs_oz_slice_kc(const double* __restrict__ x, long long ld, int R, int K, int Kp, const int* __restrict__ emax,
  int ns, int rb, signed char* __restrict__ d) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int ng = Kp / 16, r = (int)(t / (8 * ng)) * 8 + (int)(t & 7), kg = (int)((t >> 3) % ng), k0 = kg * 16;
  if (r >= R) return;
  const double* const row = x + (long long)r * ld;
  double v[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = (k0 + j < K) ? row[k0 + j] : 0.0;
  slice16(v, emax[r], ns, d + panel_offset(r, kg, Kp, ns, rb), rb * kBK);
}

/* Slicing with rows contiguous (element (r, k) at x[r + k*ld]): threads of a block run over rows
   (coalesced reads, whole core matrices written), blockIdx.y over groups of 16 k. */
__global__ void xs_oz_slice_rc(const double* __restrict__ x, long long ld, int R, int K, int Kp, const int* __restrict__ emax,
  int ns, int rb, signed char* __restrict__ d) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= R) return;
  const int k0 = blockIdx.y * 16;
  double v[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = (k0 + j < K) ? x[r + (long long)(k0 + j) * ld] : 0.0;
  slice16(v, emax[r], ns, d + panel_offset(r, blockIdx.y, Kp, ns, rb), rb * kBK);
}

/* C = beta * C (K == 0 or alpha == 0). */
__global__ void xs_oz_scale_c(double* __restrict__ c, long long ldc, int M, int N, double beta) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)M * N) return;
  const int j = (int)(t / M), i = (int)(t - (long long)j * M);
  double* const p = c + i + (long long)j * ldc;
  *p = (0.0 == beta) ? 0.0 : beta * *p;
}

/* ------------------------------------------------------------------------------ GEMM */

/* One MMA of a k block: an A slice against adjacent B slices, into the columns of the first pair's diagonal. As the
   issuing thread needs it, so that an MMA costs it one 16-byte read and a few additions. */
struct alignas(16) OzOp {
  uint32_t a, b;  /* offset of the A slice, of the first B slice in the k block, / 16 */
  uint32_t d;     /* tensor-memory column; bit 31: add to the columns, else write them */
  uint32_t idesc; /* instruction descriptor */
};

struct OzGemmArgs {
  int M, N, kb0, kb1, KB; /* k blocks [kb0, kb1) of KB */
  int ns, nstages;
  int rows, cols;         /* of a digit panel of A, of B */
  int kps;                /* k blocks per stage */
  int ndiag, eshift;      /* diagonals of the launch, -2058 - 7 d of the first */
  int first;              /* 1: this launch applies beta to C, later ones add to it */
  double alpha, beta;
  const unsigned char* dA;
  const unsigned char* dB;
  const int* ea;
  const int* eb;
  double* C;
  long long ldc;
  unsigned* abort; /* per-call abort word (zeroed by the host before the first launch) */
  unsigned* dev_err;
  long long wait_limit; /* bound of every pipeline wait, clock cycles */
  int nops[2];          /* MMAs of the first k block, of the others */
  OzOp op[2][kMaxOps];
};

/* Shared memory: 128 bytes of alignment slack, the ring, its barriers, the tensor-memory address; and what the MMAs, which
   take 128 rows, read past the last slice of a panel with fewer (for rows of C that there are not). */
size_t oz_gemm_smem(const OzGemmArgs& g) {
  return 128 + (size_t)g.nstages * g.kps * g.ns * (g.rows + g.cols) * kBK + (kBM - g.rows) * kBK + (2 * kMaxStages + 2) * sizeof(uint64_t) + 16;
}

/* Tile t: groups of kGroupM row panels sweep the column panels together, so that the CTAs running at one
   time share their panels in L2. */
__device__ __forceinline__ void oz_tile(int t, int ntm, int ntn, int& bm, int& bn) {
  const int per_group = kGroupM * ntn, g = t / per_group, first = g * kGroupM;
  const int gsize = min(kGroupM, ntm - first), r = t - g * per_group;
  bm = first + r % gsize;
  bn = r / gsize;
}

template <bool FEW>
__global__ void __launch_bounds__(kGemmThreads, 1) xs_ozaki_gemm_kernel(const __grid_constant__ OzGemmArgs args) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* const smem = (unsigned char*)(((uintptr_t)smem_raw + 127) & ~(uintptr_t)127);
  const int ns = args.ns, nst = args.nstages, kps = args.kps;
  const uint32_t abytes = (uint32_t)(ns * args.rows * kBK), bbytes = (uint32_t)(ns * args.cols * kBK); /* of a k block */
  const uint32_t stage_bytes = (uint32_t)kps * (abytes + bbytes), stage_b = (uint32_t)kps * abytes;
  uint64_t* const bars = (uint64_t*)(smem + (size_t)nst * stage_bytes);
  uint64_t* const full = bars;
  uint64_t* const empty = bars + kMaxStages;
  uint64_t* const accf = bars + 2 * kMaxStages;
  uint64_t* const acce = accf + 1;
  uint32_t* const tmem_slot = (uint32_t*)(acce + 1);
  unsigned* const abort = args.abort;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ntm = (args.M + kBM - 1) / kBM, ntn = (args.N + kBN - 1) / kBN, ntiles = ntm * ntn;
  if (0 == threadIdx.x) {
    for (int i = 0; i < nst; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(accf, 1);
    mbar_init(acce, 32 * kEpiWarps);
    fence_barrier_init();
  }
  if (1 == warp) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (0 == warp) { /* producer */
    if (0 == lane) {
      int stage = 0;
      uint32_t ph = 0u;
      bool ok = true;
      for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
        int bm, bn;
        oz_tile(t, ntm, ntn, bm, bn);
        const unsigned char* const pa = args.dA + (size_t)bm * args.KB * abytes;
        const unsigned char* const pb = args.dB + (size_t)bn * args.KB * bbytes;
        for (int kb = args.kb0; kb < args.kb1; kb += kps) {
          const uint32_t nkb = (uint32_t)min(kps, args.kb1 - kb);
          if (!(ok = mbar_wait(&empty[stage], ph ^ 1u, abort, 1u, args.wait_limit))) break;
          unsigned char* const st = smem + (size_t)stage * stage_bytes;
          mbar_arrive_expect_tx(&full[stage], nkb * (abytes + bbytes));
          bulk_load(st, pa + (size_t)kb * abytes, nkb * abytes, &full[stage]);
          bulk_load(st + stage_b, pb + (size_t)kb * bbytes, nkb * bbytes, &full[stage]);
          if (++stage == nst) {
            stage = 0;
            ph ^= 1u;
          }
        }
      }
    }
  }
  else if (1 == warp) { /* MMA issuer */
    if (0 == lane) {
      int stage = 0;
      uint32_t ph = 0u, use = 0u;
      bool ok = true;
      OzOp few[kRegOps]; /* the MMAs of a k block, when they are that few, stay in registers */
#pragma unroll
      for (int i = 0; i < kRegOps; ++i) few[i] = args.op[1][i];
      const int nfew = args.nops[1];
      for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, ++use) {
        if (!(ok = mbar_wait(acce, (use & 1u) ^ 1u, abort, 2u, args.wait_limit))) break;
        tc_fence_after();
        for (int kb = args.kb0; kb < args.kb1; kb += kps) {
          const int nkb = min(kps, args.kb1 - kb);
          if (!(ok = mbar_wait(&full[stage], ph, abort, 2u, args.wait_limit))) break;
          tc_fence_after();
          const uint32_t s0 = smem_u32(smem + (size_t)stage * stage_bytes);
          uint64_t da = desc_k_noswz(s0, 128, 256), db = desc_k_noswz(s0 + stage_b, 128, 256);
          for (int j = 0; j < nkb; ++j, da += abytes >> 4, db += bbytes >> 4) {
            if (FEW && kb + j != args.kb0) {
#pragma unroll
              for (int i = 0; i < kRegOps; ++i) {
                if (i < nfew) mma_i8(tmem + (few[i].d & 0x7FFFFFFFu), da + few[i].a, db + few[i].b, few[i].idesc, 1u);
              }
              continue;
            }
            const int which = (kb + j == args.kb0) ? 0 : 1, n = args.nops[which];
            const OzOp* const op = args.op[which];
#pragma unroll 2
            for (int i = 0; i < n; ++i) {
              const OzOp o = op[i];
              mma_i8(tmem + (o.d & 0x7FFFFFFFu), da + o.a, db + o.b, o.idesc, o.d >> 31);
            }
          }
          mma_commit(&empty[stage]);
          if (++stage == nst) {
            stage = 0;
            ph ^= 1u;
          }
        }
        if (ok) mma_commit(accf);
      }
    }
  }
  else { /* epilogue: tensor-memory lane quarter warp % 4, column half (warp - 2) / 4; thread = one row, 32 columns */
    const int q = warp & 3, cb = ((warp - 2) >> 2) * 32;
    const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)cb;
    uint32_t use = 0u;
    const double w_last = __longlong_as_double((long long)(1023 - 7 * (args.ndiag - 1)) << 52);
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++use) {
      int bm, bn;
      oz_tile(t, ntm, ntn, bm, bn);
      const int row = bm * kBM + q * 32 + lane, n0 = bn * kBN + cb;
      const bool rok = row < args.M;
      const int er = (rok ? args.ea[row] : 0) + args.eshift, ec = (n0 + lane < args.N) ? args.eb[n0 + lane] : 0;
      if (!mbar_wait(accf, use & 1u, abort, 8u, args.wait_limit)) break;
      tc_fence_after();
      double sum[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) sum[j] = 0.0;
      double w = w_last;
      uint32_t at = tbase + (uint32_t)(args.ndiag * args.cols);
      for (int d = args.ndiag - 1; d >= 0; --d, w *= 128.0) {
        uint32_t v[32];
        at -= (uint32_t)args.cols;
        tmem_ld32(at, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) { /* exact int32 -> double: 2^52 + 2^31 + v, minus the offset */
          const double dv = __hiloint2double(0x43300000, (int)(v[j] ^ 0x80000000u)) - 4503601774854144.0;
          sum[j] = fma(dv, w, sum[j]);
        }
      }
      tc_fence_before();
      mbar_arrive(acce); /* the accumulators are read: the next tile's MMAs may start */
      double* const crow = args.C + row + (long long)n0 * args.ldc;
      const bool read_c = (0 == args.first) || 0.0 != args.beta;
      const double beta = (0 != args.first) ? args.beta : 1.0;
#pragma unroll
      for (int j0 = 0; j0 < 32; j0 += 8) {
        double old[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          old[j] = (rok && read_c && n0 + j0 + j < args.N) ? crow[(long long)(j0 + j) * args.ldc] : 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int E = er + __shfl_sync(0xffffffffu, ec, j0 + j);
          const double x = sum[j0 + j];
          const double sc = (E >= -1022 && E <= 1023) ? x * __longlong_as_double((long long)(E + 1023) << 52) : ldexp(x, E);
          if (rok && n0 + j0 + j < args.N) crow[(long long)(j0 + j) * args.ldc] = fma(args.alpha, sc, read_c ? beta * old[j] : 0.0);
        }
      }
    }
  }
  if (0 != *(volatile unsigned*)abort) { /* let copies and MMAs still in flight land before TMEM goes */
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (1 == warp) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  if (0 == threadIdx.x && 0 != *(volatile unsigned*)abort) atomicOr(args.dev_err, kErrOzakiTimeout);
}

/* ------------------------------------------------------------------------------ host */

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

/* Exponents and digit panels of op(X) viewed as R rows of K entries, rb rows per block: element (r, k)
   at x[r + k*ld] when rows_contiguous, else at x[k + r*ld]. */
int slice_operand(const double* x, long long ld, bool rows_contiguous, int R, int K, int Kp, int ns, int rb, int* emax,
  signed char* panels, cudaStream_t s) {
  if (rows_contiguous) {
    /* k ranges short enough that small operands fill the device too */
    const int nrb = (R + 255) / 256, want = 4 * xs_sm_count() / nrb + 1, kchunk = max(16, min(256, (K + want - 1) / want));
    xs_oz_rowexp_rc<<<dim3(nrb, (K + kchunk - 1) / kchunk), 256, 0, s>>>(x, ld, R, K, kchunk, emax);
    xs_oz_slice_rc<<<dim3((R + 127) / 128, Kp / 16), 128, 0, s>>>(x, ld, R, K, Kp, emax, ns, rb, panels);
  }
  else {
    xs_oz_rowexp_kc<<<(R + 7) / 8, 256, 0, s>>>(x, ld, R, K, emax);
    const long long n = (long long)((R + 7) / 8 * 8) * (Kp / 16);
    xs_oz_slice_kc<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(x, ld, R, K, Kp, emax, ns, rb, panels);
  }
  return (int)cudaGetLastError();
}

/* The MMAs of a k block for the diagonals [d0, d0 + nd): per A slice its run of B slices, in pieces of at
   most 256 columns of nearly equal width. first: a diagonal's first MMA writes its columns
   (a piece never mixes written and added columns). */
int make_ops(int ns, int rows, int cols, int d0, int nd, bool first, OzOp* op) {
  const int wmax = 256 / cols; /* slices per MMA */
  int n = 0, fresh = d0; /* diagonals from here on have not been written */
  for (int sa = 0; sa < ns; ++sa) {
    const int lo = max(0, d0 - sa), hi = min(ns - 1, d0 + nd - 1 - sa); /* B slices */
    for (int b = lo; b <= hi;) {
      const bool acc = !first || sa + b < fresh;
      int e = hi; /* last slice of the run with the same accumulate flag */
      if (first && acc && sa + e >= fresh) e = fresh - 1 - sa;
      const int len = e - b + 1, parts = (len + wmax - 1) / wmax, w = (len + parts - 1) / parts;
      op[n].a = (uint32_t)(sa * rows * kBK) >> 4;
      op[n].b = (uint32_t)(b * cols * kBK) >> 4;
      op[n].d = (uint32_t)((sa + b - d0) * cols) | (acc ? 1u << 31 : 0u);
      op[n].idesc = idesc_i8(kBM, w * cols);
      ++n;
      b += w;
    }
    if (lo <= hi) fresh = max(fresh, sa + hi + 1);
  }
  return n;
}

/* Rows of a panel of A and columns of one of B: fewer than a tile's when there are no more (a panel's rows are
   read and kept for every k, which for a product of a few rows and a long k would be most of the call). */
int panel_rows(int M) { return M < kBM ? (M + 7) / 8 * 8 : kBM; }
int panel_cols(int N) { return N < kBN ? (N + 15) / 16 * 16 : kBN; }

}  // namespace

extern "C" {

size_t xs_ozaki_gemm_scratch_bytes(int M, int N, int K, int nslices) {
  const size_t Kp = align_up((size_t)(K > 0 ? K : 1), kBK);
  return align_up((size_t)nslices * align_up(M, panel_rows(M)) * Kp, 1024) +
         align_up((size_t)nslices * align_up(N, panel_cols(N)) * Kp, 1024) + align_up(sizeof(int) * M, 256) + align_up(sizeof(int) * N, 256) + 256;
}

int xs_ozaki_gemm(char transa, char transb, int M, int N, int K, double alpha, const double* a, int lda, const double* b,
  int ldb, double beta, double* c, int ldc, int nslices, int cutoff, void* scratch, size_t scratch_bytes, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const bool ta = ('T' == transa || 't' == transa || 'C' == transa || 'c' == transa);
  const bool tb = ('T' == transb || 't' == transb || 'C' == transb || 'c' == transb);
  if (M < 0 || N < 0 || K < 0 || nslices < 1 || nslices > kMaxSlices || ldc < (M > 1 ? M : 1)) return (int)cudaErrorInvalidValue;
  if (0 == M || 0 == N) return 0;
  if (0 == K || 0.0 == alpha) {
    if (1.0 == beta) return 0;
    const long long n = (long long)M * N;
    xs_oz_scale_c<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(c, ldc, M, N, beta);
    return (int)cudaGetLastError();
  }
  if (lda < (ta ? K : M) || ldb < (tb ? N : K)) return (int)cudaErrorInvalidValue;
  if (nullptr == scratch || scratch_bytes < xs_ozaki_gemm_scratch_bytes(M, N, K, nslices)) return (int)cudaErrorInvalidValue;
  const int maxcut = 2 * (nslices - 1);
  if (cutoff < 0 || cutoff > maxcut) cutoff = maxcut;
  const int Kp = (int)align_up((size_t)K, kBK), rows = panel_rows(M), cols = panel_cols(N);
  char* p = (char*)scratch;
  signed char* const dA = (signed char*)p;
  p += align_up((size_t)nslices * align_up(M, rows) * Kp, 1024);
  signed char* const dB = (signed char*)p;
  p += align_up((size_t)nslices * align_up(N, cols) * Kp, 1024);
  int* const ea = (int*)p;
  p += align_up(sizeof(int) * M, 256);
  int* const eb = (int*)p;
  p += align_up(sizeof(int) * N, 256);
  unsigned* const abort = (unsigned*)p;
  int r = (int)cudaMemsetAsync(ea, 0, (size_t)(p - (char*)ea) + 256, s);
  if (0 != r) return r;
  /* rows of op(A): A(i, k) at a[i + k*lda] ('N') or a[k + i*lda] ('T'); columns of op(B): B(k, j)
     at b[k + j*ldb] ('N', k contiguous) or b[j + k*ldb] ('T') */
  void* prof = xs_profile_begin(stream);
  if (0 != (r = slice_operand(a, lda, !ta, M, K, Kp, nslices, rows, ea, dA, s))) return r;
  if (0 != (r = slice_operand(b, ldb, tb, N, K, Kp, nslices, cols, eb, dB, s))) return r;
  xs_profile_end(prof, "ozaki_slice", 0.0, 8.0 * ((double)M * K + (double)K * N), stream);
  OzGemmArgs args;
  memset(&args, 0, sizeof(args));
  args.M = M;
  args.N = N;
  args.alpha = alpha;
  args.beta = beta;
  args.ea = ea;
  args.eb = eb;
  args.C = c;
  args.ldc = ldc;
  args.abort = abort;
  args.dev_err = xs_device_error_ptr();
  args.wait_limit = xs_wait_limit();
  if (nullptr == args.dev_err) return (int)cudaErrorInvalidValue;
  args.dA = (const unsigned char*)dA;
  args.dB = (const unsigned char*)dB;
  args.ns = nslices;
  args.KB = Kp / kBK;
  args.rows = rows;
  args.cols = cols;
  args.kps = max(1, kStageBytes / (nslices * (rows + cols) * kBK));
  args.nstages = kMaxStages;
  while (oz_gemm_smem(args) > 227 * 1024) --args.nstages;
  /* at least 120 KB, so that an SM takes one CTA: it owns all tensor-memory columns */
  const size_t smem = max((size_t)120 * 1024, oz_gemm_smem(args));
  const int ntiles = ((N + kBN - 1) / kBN) * ((M + kBM - 1) / kBM);
  for (int kb0 = 0; kb0 < args.KB; kb0 += kKChunkBlocks) {
    args.kb0 = kb0;
    args.kb1 = (kb0 + kKChunkBlocks < args.KB) ? kb0 + kKChunkBlocks : args.KB;
    for (int d0 = 0; d0 <= cutoff; d0 += kMaxDiag) {
      args.ndiag = min(kMaxDiag, cutoff + 1 - d0);
      args.eshift = -2058 - 7 * d0;
      args.first = (0 == kb0 && 0 == d0) ? 1 : 0;
      args.nops[0] = make_ops(nslices, rows, cols, d0, args.ndiag, true, args.op[0]);
      args.nops[1] = make_ops(nslices, rows, cols, d0, args.ndiag, false, args.op[1]);
      prof = xs_profile_begin(stream);
      const auto kernel = (kRegOps >= args.nops[1]) ? &xs_ozaki_gemm_kernel<true> : &xs_ozaki_gemm_kernel<false>;
      if (0 != (r = xs_func_smem((const void*)kernel, smem))) return r;
      kernel<<<min(ntiles, xs_sm_count()), kGemmThreads, smem, s>>>(args);
      if (0 != (r = (int)cudaGetLastError())) return r;
      const double kc = (double)(args.kb1 - args.kb0) * kBK;
      xs_profile_end(prof, "ozaki_gemm", 2.0 * M * N * (kc < K ? kc : K), 0.0, stream);
    }
  }
  return 0;
}

}  // extern "C"
