/*
 * The tile stack kernel: the FP64 stack multiply of any block shape, with the A and B block of each
 * stack entry staged once in shared memory for a team of warps that hold one C block between them.
 *
 * What bounds the path: the FP64 tensor pipe (a DMMA m8n8k4 occupies a scheduler for 16 cycles) as long
 * as fragments arrive in time. The register kernel (smm_kernels.cu) loads every fragment from L2, once
 * per warp tile that needs it: an A block of 64 x 64 is read twice, and each k panel waits for L2. Here
 *   - a team of T = 1..10 warps, one per warp tile of the block, shares a ring of two stages in shared
 *     memory. A stage holds a panel of k indices (all of them where they fit) of one entry's A and B:
 *     a panel is contiguous in memory (A is column-major, B row-major), so one thread brings each operand
 *     with one bulk copy (cp.async.bulk, counted in bytes on the stage's mbarrier);
 *   - the four k indices of a DMMA step lie Q apart (1, 2 or 4, the same for A and B): the columns that a
 *     warp reads at once then start on different banks although they are not padded. Columns of a
 *     multiple of 16 doubles start on one bank whatever Q is; those operands are copied by the team with
 *     16-byte cp.async into padded columns (one bulk copy per column was measured much slower:
 *     64^3 8.1 ms against 4.0);
 *   - a chunk of the grouped stack belongs to one team; pieces of the segments that cross its ends go to
 *     scratch, and the last team to arrive sums them in chunk order (at most kFan pieces at a time, in two
 *     levels), so results are bitwise reproducible.
 * Longer panels won over deeper rings (45^3: 265 us with two stages of whole entries, 290 with three of 32
 * indices), and 8 to 12 warps per SM with long panels over 16 with short ones (280 us).
 * Measured on B200 (whole calls, S entries, c Zipf(1.1)), register kernel -> this one: 45^3, 30000: 459 ->
 * 259 us (DMMA pipe 75 % busy); 64^3, 200000 (operands from HBM): 6.25 -> 4.37 ms; 17x29x11, 20000: 64.5 ->
 * 54.5 us; 45x26x22, 42000: 245 -> 159 us; 66^3, 50000: 3.9 -> 1.6 ms.
 */
#include "smm_stack.cuh"
#include "smm_tile.h"

namespace {
using namespace xs_stack;

constexpr int kMaxThreads = 320; /* 10 warps: a team of up to 10 warp tiles */
constexpr int kStages = 2;
constexpr int kMaxTeams = 8;
constexpr int kSmemMax = 227 * 1024; /* shared memory of an SM that CTAs can use */
constexpr int kFan = 8;     /* pieces per first-level sum of a long segment */
constexpr unsigned kErrTileTimeout = 16u; /* device error word: a wait for block copies timed out (as the staged kernel) */

/* How an operand is staged. */
struct OperandGeo {
  int ld;     /* doubles between staged columns of A / rows of B */
  int padded; /* 0: whole panels by one bulk copy each, ld = rows; 1: copied by the team in 16-byte units, ld > rows */
  int bytes;  /* of a stage */
};
/* Geometry of a launch, uniform over the grid. */
struct TileGeo {
  int T, nteam;       /* warps per team (one warp tile of C each), teams per CTA */
  OperandGeo a, b;
  int Q;              /* k indices of a DMMA step: Q apart (1, 2, 4) */
  int pk, npan, R;    /* k indices per panel (a multiple of 4 Q unless one panel holds all), panels per entry, stages */
  int region;         /* bytes per team */
};

/* Shared-memory state of a team's ring. */
struct TeamRing {
  uint64_t full[kStages]; /* the stage's copies have landed */
  int odd[kStages];       /* bit 0 / 1: A / B starts 8 bytes into its window */
};

__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
/* This thread's copies so far arrive (one arrival) on the mbarrier when they have landed. */
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(xs_tc::smem_u32(bar)) : "memory");
}

/* Barrier of a team; returns whether any of its threads passed flag. */
__device__ __forceinline__ bool team_any(int id, int threads, bool flag) {
  if (32 == threads) return 0 != __any_sync(0xFFFFFFFFu, flag);
  int r;
  asm volatile(
    "{\n\t.reg .pred p, q;\n\t"
    "setp.ne.s32 p, %3, 0;\n\t"
    "barrier.cta.red.or.pred q, %1, %2, p;\n\t"
    "selp.s32 %0, 1, 0, q;\n\t}"
    : "=r"(r)
    : "r"(id), "r"(threads), "r"(flag ? 1 : 0)
    : "memory");
  return 0 != r;
}

/* First entry of chunk c: the S entries are dealt evenly over the chunks. */
__device__ __forceinline__ int tile_first(const StackTask& tk, int c) { return c * tk.L + min(c, tk.Ls[0]); }

/* Largest count c such that pred(1), ..., pred(c) hold, for a pred that is true up to some point: one
   warp tests 32 candidates per round, at a stride that grows by 32 while all of them hold. */
template <typename Pred>
__device__ __forceinline__ int run_length(Pred pred) {
  const int lane = threadIdx.x & 31;
  int lo = 0, step = 1;
  for (;;) {
    const unsigned m = __ballot_sync(0xFFFFFFFFu, pred(lo + step * (lane + 1)));
    const int cnt = (0xFFFFFFFFu == m) ? 32 : __ffs(~m) - 1;
    lo += step * cnt;
    if (32 == cnt) step *= 32;
    else if (1 == step) return lo;
    else step /= 32;
  }
}

/* The 16-byte-aligned window around `count` doubles at src. */
__device__ __forceinline__ uint32_t window_bytes(const double* src, int count) {
  return (uint32_t)((((uintptr_t)(src + count) + 15) & ~(uintptr_t)15) - ((uintptr_t)src & ~(uintptr_t)15));
}
__device__ __forceinline__ const void* window_start(const double* src) { return (const void*)((uintptr_t)src & ~(uintptr_t)15); }

/* Copies `cols` columns of `rows` contiguous doubles at src into shared memory, columns ld doubles
   apart, in units of U doubles dealt over the threads of a team. */
template <int U>
__device__ __forceinline__ void copy_padded(uint32_t dst, const double* src, int rows, int ld, int cols, int tid, int threads) {
  const int units = rows / U, total = cols * units, dk = threads / units, dr = threads - dk * units;
  const int k0 = tid / units;
  int r = tid - k0 * units;
  uint32_t d = dst + 8u * (uint32_t)(k0 * ld + r * U);
  const uint32_t dd = 8u * (uint32_t)(dk * ld + dr * U), wrap = 8u * (uint32_t)(ld - rows);
  const double* p = src + U * tid;
#pragma unroll 4
  for (int i = tid; i < total; i += threads) {
    if (2 == U) cp_async16(d, p);
    else cp_async8(d, p);
    p += U * threads;
    d += dd;
    r += dr;
    if (r >= units) {
      r -= units;
      d += wrap;
    }
  }
}
__device__ __forceinline__ void copy_operand(const OperandGeo& o, uint32_t dst, const double* src, int rows, int cols, int tid,
  int threads) {
  if (!o.padded) return;
  if (0 == ((uintptr_t)src & 15)) copy_padded<2>(dst, src, rows, o.ld, cols, tid, threads);
  else copy_padded<1>(dst, src, rows, o.ld, cols, tid, threads);
}

template <int REGS>
__device__ __forceinline__ double* piece_at(const StackTask& tk, int slot, int sub) {
  return tk.pieces + ((size_t)slot * tk.nsub + sub) * (REGS * 32) + (threadIdx.x & 31);
}

/* Piece q of the segment that starts in chunk j0: the tail piece of j0, else the head piece of j0 + q. */
__device__ __forceinline__ int piece_slot(int j0, int q) { return (0 == q) ? 2 * j0 + 1 : 2 * (j0 + q); }

/* acc = sum of `count` pieces, piece i at slot_of(i), added in that order by one warp; the loads of
   four pieces are in flight at a time. */
template <int REGS, typename SlotOf>
__device__ __forceinline__ void warp_sum(const StackTask& tk, int sub, int count, SlotOf slot_of, double (&acc)[REGS]) {
  constexpr int F = (REGS > 18) ? 2 : 4, B = (REGS > 18) ? 8 : 6;
#pragma unroll
  for (int r = 0; r < REGS; ++r) acc[r] = 0.0;
  for (int q = 0; q < count; q += F) {
    const double* p[F];
#pragma unroll
    for (int f = 0; f < F; ++f) p[f] = piece_at<REGS>(tk, slot_of(min(q + f, count - 1)), sub);
#pragma unroll
    for (int r0 = 0; r0 < REGS; r0 += B) {
      double v[F][B];
#pragma unroll
      for (int f = 0; f < F; ++f)
#pragma unroll
        for (int r = 0; r < B; ++r)
          if (r0 + r < REGS) v[f][r] = __ldcg(p[f] + (r0 + r) * 32);
#pragma unroll
      for (int f = 0; f < F; ++f)
#pragma unroll
        for (int r = 0; r < B; ++r)
          if (r0 + r < REGS && q + f < count) acc[r0 + r] += v[f][r];
    }
  }
}

/* One warp has stored the pieces of its chunk (head: of a segment that enters the chunk, reaching back
   to chunk j0; tail: of one that leaves it, up to chunk j1; hspans: the head segment also leaves):
   announces them, and sums those of a segment when it was the last to arrive. */
template <int MT, int NT>
__device__ __forceinline__ void finish_pieces(const StackTask& tk, int chunk, int sub, bool head, bool hspans, bool tail, int j0,
  int j1, unsigned kfirst, unsigned klast) {
  constexpr int REGS = MT * NT * 2;
  const int lane = threadIdx.x & 31;
  if (!head && !tail) return;
  /* lane 0: the head piece, lane 1: the tail piece */
  const bool mine = (0 == lane && head) || (1 == lane && tail);
  const int s0 = (0 == lane) ? j0 : chunk, s1 = (0 == lane && !hspans) ? chunk : j1; /* the segment's chunks */
  const int np = s1 - s0 + 1, i1 = (chunk - s0) / kFan;
  const bool two = np > kFan;
  const int target = two ? min(kFan, np - i1 * kFan) : np;
  int done = 0;
  fence_acq_rel_gpu(); /* the pieces are visible device-wide before the arrivals */
  __syncwarp();
  if (mine) {
    int* const c = tk.arrive + (two ? ((size_t)tk.nchunks + piece_slot(s0, i1 * kFan)) * tk.nsub + sub : (size_t)s0 * tk.nsub + sub);
    done = (atomicAdd(c, 1) == target - 1) ? 1 : 0;
  }
  for (int d = 0; d < 2; ++d) {
    if (0 == __shfl_sync(0xFFFFFFFFu, done, d)) continue;
    const int f0 = __shfl_sync(0xFFFFFFFFu, s0, d), fnp = __shfl_sync(0xFFFFFFFFu, np, d), fi = __shfl_sync(0xFFFFFFFFu, i1, d);
    fence_acq_rel_gpu(); /* acquire: the pieces this increment completed are visible */
    double acc[REGS];
    if (fnp > kFan) {
      warp_sum<REGS>(tk, sub, min(kFan, fnp - fi * kFan), [&](int i) { return piece_slot(f0, fi * kFan + i); }, acc);
      double* const dst = piece_at<REGS>(tk, piece_slot(f0, fi * kFan), sub);
#pragma unroll
      for (int r = 0; r < REGS; ++r) __stcg(dst + r * 32, acc[r]);
      const int n1 = (fnp + kFan - 1) / kFan;
      fence_acq_rel_gpu();
      __syncwarp();
      int last = 0;
      if (0 == lane) last = (atomicAdd(tk.arrive + (size_t)f0 * tk.nsub + sub, 1) == n1 - 1) ? 1 : 0;
      if (0 == __shfl_sync(0xFFFFFFFFu, last, 0)) continue;
      fence_acq_rel_gpu();
      warp_sum<REGS>(tk, sub, n1, [&](int i) { return piece_slot(f0, i * kFan); }, acc);
    }
    else warp_sum<REGS>(tk, sub, fnp, [&](int i) { return piece_slot(f0, i); }, acc);
    double tile[MT][NT][2];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        tile[i][j][0] = acc[(i * NT + j) * 2 + 0];
        tile[i][j][1] = acc[(i * NT + j) * 2 + 1];
      }
    Tile<MT, NT> tl;
    tl.init(sub, tk.nsub_n, tk.m, tk.n, lane >> 2);
    commit_tile<MT, NT>(tk.c, (size_t)((0 == d) ? kfirst : klast) - 1, tile, tk.m, tk.n, lane >> 2, lane & 3, tl, tk.alpha);
  }
}

/* Warps per SM that the plan aims for: small tiles need many warps, one of 4 x 4 fragments (64 registers of
   sums) ran best without a spilled register at 8 (64^3, 200000: 4.37 ms; 12 warps of 168 registers
   4.55). The register limit follows from it. */
constexpr int tile_warps(int mt, int nt) { return (mt * nt <= 3) ? 20 : ((mt * nt <= 12) ? 12 : 8); }
constexpr int tile_regs(int mt, int nt) { return (mt * nt <= 3) ? 96 : ((mt * nt <= 12) ? 168 : 255); }

/* One team per chunk of grouped entries, nteam teams per CTA. Per panel: wait (bounded) for its copies,
   team barrier (which also says that everybody has read the other stage), refill the other stage, multiply.
   A wait that runs out sets the grouping error word, which ends the other teams' waits, and a device
   error bit; the team leaves together (the barrier carries the flag) once its copies in flight landed. */
template <int MT, int NT>
__global__ void __maxnreg__(tile_regs(MT, NT)) xs_smm_tile_kernel(const __grid_constant__ StackTask tk, const __grid_constant__ TileGeo geo,
  unsigned* __restrict__ err, unsigned* __restrict__ dev_err, long long wait_limit) {
  constexpr int REGS = MT * NT * 2;
  constexpr unsigned FULL = 0xFFFFFFFFu;
  extern __shared__ __align__(128) unsigned char tsm[];
  __shared__ TeamRing rings[kMaxTeams];
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, warp = threadIdx.x >> 5;
  const int team = warp / geo.T, sub = warp - team * geo.T, threads = 32 * geo.T, tid = threadIdx.x - team * threads;
  TeamRing& rg = rings[team];
  const bool padded = (0 != geo.a.padded) || (0 != geo.b.padded);
  const int R = geo.R;
  if (0 == tid) {
    for (int q = 0; q < R; ++q) xs_tc::mbar_init(&rg.full[q], padded ? threads + 1 : 1);
    xs_tc::fence_barrier_init();
  }
  prefetch_operands(tk);
  pdl_wait();
  pdl_trigger();
  /* the grouping failed (or a wait of a team that started earlier): the team writes nothing. One vote for all its
     threads: the word may change while they read it, and the barriers below count on every warp of a team */
  const bool failed = 0 != *(volatile const unsigned*)err;
  __syncthreads();
  if (team_any(team + 1, threads, failed)) return;
  const int chunk = blockIdx.x * geo.nteam + team;
  if (chunk >= tk.nchunks) return;
  const int m = tk.m, n = tk.n, k = tk.k, npan = geo.npan;
  const unsigned* __restrict__ const keys = tk.keys;
  const unsigned long long* __restrict__ const vals = tk.vals;
  const int p0 = tile_first(tk, chunk), p1 = tile_first(tk, chunk + 1);
  unsigned char* const ring = tsm + (size_t)team * geo.region;
  const uint32_t ring_s = xs_tc::smem_u32(ring);
  const int stage_bytes = geo.a.bytes + geo.b.bytes;
  int wb = p0; /* lane j holds entries wb + j and wb + 32 + j */
  unsigned kc = 0u, kn = 0u;
  unsigned long long vc = 0ull, vn = 0ull;
  if (p0 + lane < p1) {
    kc = keys[p0 + lane];
    vc = vals[p0 + lane];
  }
  if (p0 + 32 + lane < p1) {
    kn = keys[p0 + 32 + lane];
    vn = vals[p0 + 32 + lane];
  }
  auto key_of = [&](int e) -> unsigned {
    const int i = e - wb;
    const unsigned x0 = __shfl_sync(FULL, kc, i & 31), x1 = __shfl_sync(FULL, kn, i & 31);
    return (i < 32) ? x0 : x1;
  };
  int pe = p0, ppan = 0, pst = 0; /* next panel to copy, its stage */
  auto issue = [&]() {
    if (pe >= p1) return;
    if (padded || 0 == sub) {
      const int i = pe - wb;
      const unsigned long long x0 = __shfl_sync(FULL, vc, i & 31), x1 = __shfl_sync(FULL, vn, i & 31);
      const unsigned long long v = (i < 32) ? x0 : x1;
      const int kk = ppan * geo.pk, cols = min(geo.pk, k - kk);
      const double* const srca = tk.a + ((unsigned)v - 1u) + (size_t)kk * m;
      const double* const srcb = tk.b + ((unsigned)(v >> 32) - 1u) + (size_t)kk * n;
      if (0 == tid) {
        unsigned char* const dst = ring + pst * stage_bytes;
        const uint32_t wa = geo.a.padded ? 0u : window_bytes(srca, cols * m), wbb = geo.b.padded ? 0u : window_bytes(srcb, cols * n);
        rg.odd[pst] = (geo.a.padded ? 0 : (int)(((uintptr_t)srca >> 3) & 1u)) | (geo.b.padded ? 0 : (int)(((uintptr_t)srcb >> 2) & 2u));
        xs_tc::mbar_arrive_expect_tx(&rg.full[pst], wa + wbb);
        if (wa) xs_tc::bulk_load(dst, window_start(srca), wa, &rg.full[pst]);
        if (wbb) xs_tc::bulk_load(dst + geo.a.bytes, window_start(srcb), wbb, &rg.full[pst]);
      }
      if (padded) {
        copy_operand(geo.a, ring_s + pst * stage_bytes, srca, m, cols, tid, threads);
        copy_operand(geo.b, ring_s + pst * stage_bytes + geo.a.bytes, srcb, n, cols, tid, threads);
        cp_async_arrive(&rg.full[pst]);
      }
    }
    if (++ppan == npan) {
      ppan = 0;
      ++pe;
    }
    pst = (R - 1 == pst) ? 0 : pst + 1;
  };
  for (int q = 0; q < R - 1; ++q) issue();
  /* the chunk's boundary segments and the range of chunks they span, while the first copies land */
  const unsigned kfirst = key_of(p0), klast = keys[p1 - 1];
  const unsigned kbefore = (0 < p0) ? keys[p0 - 1] : 0u, kafter = (p1 < tk.S) ? keys[p1] : 0u;
  const bool headcross = (0 < p0) && kbefore == kfirst, tailcross = (p1 < tk.S) && kafter == klast;
  int j0 = chunk, j1 = chunk;
  if (headcross) {
    j0 = chunk - 1 - run_length([&](int q) { return chunk - q >= 1 && __ldcg(keys + tile_first(tk, chunk - q) - 1) == kfirst; });
  }
  if (tailcross) {
    j1 = chunk + 1 + run_length([&](int q) { return chunk + 1 + q < tk.nchunks && __ldcg(keys + tile_first(tk, chunk + 1 + q)) == klast; });
  }
  Tile<MT, NT> tl;
  tl.init(sub, tk.nsub_n, m, n, g);
  const int lda = geo.a.ld, ldb = geo.b.ld, Q = geo.Q;
  double acc[MT][NT][2];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  auto step = [&](const double* pa, const double* pb) {
    double fa[MT], fb[NT];
#pragma unroll
    for (int i = 0; i < MT; ++i) fa[i] = pa[8 * i];
#pragma unroll
    for (int j = 0; j < NT; ++j) fb[j] = pb[8 * j];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j) dmma_m8n8k4(acc[i][j][0], acc[i][j][1], fa[i], fb[j]);
  };
  bool head = false, hspans = false, tail = false, bad = false;
  int segstart = p0, pan = 0, st = 0;
  uint32_t phase = 0u;
  unsigned key_cur = kfirst;
  for (int e = p0; e < p1;) {
    bool ok = xs_tc::mbar_test_wait(&rg.full[st], phase);
    if (!ok) ok = xs_tc::mbar_wait(&rg.full[st], phase, err, 2u, wait_limit);
    if (team_any(team + 1, threads, !ok)) { /* the panel is there, and the team has read the one before */
      bad = true;
      break;
    }
    issue();
    {
      const int odd = rg.odd[st], kcur = min(geo.pk, k - pan * geo.pk);
      const double* const sA = (const double*)(ring + st * stage_bytes) + (odd & 1) + tl.r0 + g;
      const double* const sB = (const double*)(ring + st * stage_bytes + geo.a.bytes) + (odd >> 1) + tl.c0 + g;
      const int nfull = kcur / (4 * Q) * Q; /* steps in full groups of 4 Q indices */
      const double* pa = sA + Q * t * lda;
      const double* pb = sB + Q * t * ldb;
#pragma unroll 4
      for (int ks = 0; ks < nfull; ++ks) {
        step(pa, pb);
        const int adv = (Q - 1 == (ks & (Q - 1))) ? 3 * Q + 1 : 1;
        pa += adv * lda;
        pb += adv * ldb;
      }
      pa = sA + (4 * nfull + t) * lda; /* the rest: indices one apart */
      pb = sB + (4 * nfull + t) * ldb;
      const int rem = kcur - 4 * nfull;
      for (int r = rem >> 2; r > 0; --r) {
        step(pa, pb);
        pa += 4 * lda;
        pb += 4 * ldb;
      }
      if (0 != (rem & 3)) { /* fewer than four indices: the lanes beyond them bring zeros */
        const bool kin = t < (rem & 3);
        double fa[MT], fb[NT];
#pragma unroll
        for (int i = 0; i < MT; ++i) fa[i] = kin ? pa[8 * i] : 0.0;
#pragma unroll
        for (int j = 0; j < NT; ++j) fb[j] = kin ? pb[8 * j] : 0.0;
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int j = 0; j < NT; ++j) dmma_m8n8k4(acc[i][j][0], acc[i][j][1], fa[i], fb[j]);
      }
    }
    if (R - 1 == st) {
      st = 0;
      phase ^= 1u;
    }
    else ++st;
    if (++pan < npan) continue;
    pan = 0;
    const bool last = (e + 1 == p1);
    const unsigned key_nxt = key_of(last ? e : e + 1);
    if (last || key_nxt != key_cur) { /* the segment ends with entry e */
      const bool crossl = headcross && (segstart == p0), crossr = tailcross && last;
      if (!crossl && !crossr) commit_tile<MT, NT>(tk.c, (size_t)key_cur - 1, acc, m, n, g, t, tl, tk.alpha);
      else {
        double* const dst = piece_at<REGS>(tk, 2 * chunk + (crossl ? 0 : 1), sub);
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            __stcg(dst + ((i * NT + j) * 2 + 0) * 32, acc[i][j][0]);
            __stcg(dst + ((i * NT + j) * 2 + 1) * 32, acc[i][j][1]);
          }
        if (crossl) {
          head = true;
          hspans = crossr;
        }
        else tail = true;
      }
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
      segstart = e + 1;
    }
    key_cur = key_nxt;
    ++e;
    if (32 == e - wb) {
      wb += 32;
      kc = kn;
      vc = vn;
      kn = 0u;
      vn = 0ull;
      if (wb + 32 + lane < p1) {
        kn = keys[wb + 32 + lane];
        vn = vals[wb + 32 + lane];
      }
    }
  }
  if (bad) { /* wait (bounded) for the copies in flight: the stages from st up to the last one issued */
    if (0 == tid && nullptr != dev_err) atomicOr(dev_err, kErrTileTimeout);
    while (st != pst) {
      const long long t0 = clock64();
      while (!xs_tc::mbar_try_wait(&rg.full[st], phase) && clock64() - t0 < 400000000ll) {
      }
      if (R - 1 == st) phase ^= 1u;
      st = (R - 1 == st) ? 0 : st + 1;
    }
    return;
  }
  finish_pieces<MT, NT>(tk, chunk, sub, head, hspans, tail, j0, j1, kfirst, klast);
}

typedef void (*tile_kernel_t)(const StackTask, const TileGeo, unsigned*, unsigned*, long long);
/* Warp tiles: up to 4 x 4 fragments, and 5 x 2 for blocks of 73..80 (10 fragments a side: ten tiles without
   padding; nine of 4 x 4 pad 44 %). */
#define XS_TILE_ROW(MT) {&xs_smm_tile_kernel<MT, 1>, &xs_smm_tile_kernel<MT, 2>, &xs_smm_tile_kernel<MT, 3>, &xs_smm_tile_kernel<MT, 4>}
const tile_kernel_t tile_table[4][4] = {XS_TILE_ROW(1), XS_TILE_ROW(2), XS_TILE_ROW(3), XS_TILE_ROW(4)};
#undef XS_TILE_ROW
tile_kernel_t tile_kernel(int mt, int nt) { return (5 == mt) ? &xs_smm_tile_kernel<5, 2> : tile_table[mt - 1][nt - 1]; }

/* Wavefronts of a half-warp's fragment read of columns ld doubles apart at k distance Q: 16 lanes, four
   consecutive rows of four columns, 16 banks of 8 bytes. */
int read_conflicts(int ld, int Q) {
  int count[16] = {0}, worst = 0;
  for (int t = 0; t < 4; ++t) {
    for (int g = 0; g < 4; ++g) {
      const int b = (Q * t * ld + g) % 16;
      if (++count[b] > worst) worst = count[b];
    }
  }
  return worst;
}

/* Staging of an operand of `rows` contiguous doubles per k index for k distance Q: as the bulk copies
   bring it, or, when all its columns would start on one bank, in columns padded for distance Q. */
void operand_geo(int rows, int Q, OperandGeo* o) {
  o->padded = (0 == rows % 16 && 4 != Q) ? 1 : 0;
  o->ld = o->padded ? rows + ((1 == Q) ? 4 : 2) : rows;
}

int teams_per_cta(int T) { return (T >= 4) ? 1 : 4 / T; }

struct Choice {
  int mt, nt, T, nteam;
};

/* Warp tiles of an m x n block: the least time of all warps for one entry, 16 cycles per DMMA
   instruction and about 200 for a panel's wait, barrier and addresses. A lone warp with more than nine
   fragments loses to two warps (32^3: 167 us with one 4x4 tile, 135 with two 4x2). Tiles that leave an SM
   fewer than eight warps do not keep its FP64 pipe busy (one team of seven 1x4 tiles, 54x29x73, 9400 entries:
   232 us against the register kernel's 189; now two of 4x4: 150). */
bool choose(int m, int n, int k, Choice* c) {
  const int fm = (m + 7) / 8, fn = (n + 7) / 8, ks = (k - 1) / 4 + 1;
  double best = -1.0;
  for (int mt = 1; mt <= 5; ++mt) {
    for (int nt = 1; nt <= 4; ++nt) {
      if (5 == mt && 2 != nt) continue;
      const long long tiles = (long long)((fm + mt - 1) / mt) * ((fn + nt - 1) / nt);
      if (tiles > kMaxThreads / 32 || 32 * tiles * tile_regs(mt, nt) > 65536) continue;
      const int T = (int)tiles;
      double cost = (double)T * (16.0 * mt * nt * ks + 200.0);
      if (1 == T && 9 < mt * nt) cost *= 1.25;
      const int cta_warps = T * teams_per_cta(T), warps = cta_warps * max(1, tile_warps(mt, nt) / cta_warps);
      if (8 > warps) cost *= 8.0 / warps;
      if (best < 0.0 || cost < best) {
        best = cost;
        c->mt = mt;
        c->nt = nt;
        c->T = T;
      }
    }
  }
  if (best < 0.0) return false;
  c->nteam = teams_per_cta(c->T);
  return true;
}

/* Stage bytes of `cols` k indices, in 64 bits: a whole block may have any k, and the bytes of a panel that does
   not fit must not wrap to a size that does. A bulk-copied window starts up to 8 bytes before the panel. */
long long stage_bytes(const OperandGeo& o, int rows, int cols) {
  return o.padded ? (8ll * o.ld * cols + 15) / 16 * 16 : (8ll * rows * cols + 8 + 15) / 16 * 16;
}

/* The launch geometry of a plan; returns the bytes of a team's ring. The sizes in geo are set only when the ring
   fits an SM. */
long long make_geo(const xs_tile_plan_t* pl, int m, int n, TileGeo* geo) {
  geo->T = pl->T;
  geo->nteam = pl->nteam;
  geo->Q = pl->Q;
  geo->pk = pl->pk;
  geo->npan = pl->npan;
  geo->R = pl->R;
  operand_geo(m, pl->Q, &geo->a);
  operand_geo(n, pl->Q, &geo->b);
  const long long ab = stage_bytes(geo->a, m, pl->pk), bb = stage_bytes(geo->b, n, pl->pk), region = pl->R * (ab + bb);
  if (region <= kSmemMax) {
    geo->a.bytes = (int)ab;
    geo->b.bytes = (int)bb;
    geo->region = (int)region;
  }
  return region;
}

}  // namespace

extern "C" {

int xs_tile_geometry(int m, int n, int k, xs_tile_plan_t* pl) {
  Choice c;
  if (m < 1 || n < 1 || k < 1 || !choose(m, n, k, &c)) return -1;
  /* DMMA steps an entry must have for its staging to pay: few without padded operands, more with one or both
     (200000 entries, register kernel -> this one: 13x22x9 196 -> 172 us, 14^3 157 -> 194; 13x32x22 332 -> 302,
     48x9x9 350 -> 406; 32^3 875 -> 701, 16x32x32 464 -> 517, 48x48x5 557 -> 848) */
  const long long steps = (long long)((m + 7) / 8) * ((n + 7) / 8) * ((k - 1) / 4 + 1);
  const int padded = (0 == m % 16 ? 1 : 0) + (0 == n % 16 ? 1 : 0);
  if (steps < (0 == padded ? 18 : (1 == padded ? 48 : 128))) return -1;
  const int slack = 8 * (8 * (c.mt + c.nt) * 4 + 64); /* reads of padding rows and columns pass the last stage */
  int best = -1;
  for (int Q = 1; Q <= 4; Q *= 2) { /* the k distance with the fewest bank conflicts */
    OperandGeo a, b;
    operand_geo(m, Q, &a);
    operand_geo(n, Q, &b);
    const int cost = c.mt * read_conflicts(a.ld, Q) + c.nt * read_conflicts(b.ld, Q);
    if (best < 0 || cost < best) {
      best = cost;
      pl->Q = Q;
    }
  }
  pl->mt = c.mt;
  pl->nt = c.nt;
  pl->T = c.T;
  pl->nteam = c.nteam;
  pl->nsub_n = ((n + 7) / 8 + c.nt - 1) / c.nt;
  /* as many CTAs per SM as the warps want, or down to 8 warps if that keeps entries in one panel */
  TileGeo geo;
  const int gk = 4 * pl->Q, ngrp = (k - 1) / gk + 1, cta_warps = c.T * c.nteam; /* panels are whole groups of indices */
  const int want = tile_warps(c.mt, c.nt), most = (want / cta_warps > 1) ? want / cta_warps : 1;
  int ctas = most;
  pl->R = kStages;
  bool fits = false;
  auto panels = [&](int npan) { /* whether a ring of entries in npan panels fits ctas times */
    pl->npan = npan;
    pl->pk = (1 == npan) ? k : (ngrp + npan - 1) / npan * gk;
    pl->npan = (k - 1) / pl->pk + 1;
    return make_geo(pl, m, n, &geo) * c.nteam <= (kSmemMax - 1536 * ctas) / ctas - slack;
  };
  for (int q = most; q > 0 && q * cta_warps >= 8 && !fits; --q) {
    ctas = q;
    fits = panels(1);
  }
  if (!fits) { /* as few panels as the longest that fits allows */
    ctas = most;
    if (!panels(ngrp)) return -1;
    const int budget = ((kSmemMax - 1536 * ctas) / ctas - slack) / c.nteam / kStages - 64, one = gk * 8 * (geo.a.ld + geo.b.ld);
    for (int len = max(1, min(ngrp, budget / one)); !fits; --len) fits = panels((ngrp + len - 1) / len);
  }
  pl->ctas = ctas;
  /* DMMA instructions of a warp in a panel: they have to pay for the panel's wait, the team's barrier and, where
     columns are padded, the copies that the team issues itself. Over 1230 stacks (all shapes up to 80, 7e5 to 5e6
     steps) these lines leave out what was up to 1.4 times slower than the register kernel, 5 % in the mean:
     - panels of one or two DMMA steps (k <= 8) with padded columns and fewer than three teams on an SM (32x76x5, 12502
       entries: register kernel 65 us, this one 83), in the only team of an SM, unless it is of ten warps (74x58x6,
       10002: 86, 99; 77x76x4, 8002: 96, 74), and of fewer than 8 (one step) or 18 (two) instructions: 7x72x7, 88890: 153, 178;
       46x13x5, 192109: 228, 256. With one row or column of fragments 8 are enough for two steps (4x78x8);
     - padded columns and a lone warp, unless it copies 32-wide columns or wider ones of one operand for at least eight
       fragments (16x32x64, 6252: 45, 52; 16x9x45, 17710: 47, 55; but 13x32x45, 52085: 0.93 of the time). */
  const int psteps = (min(pl->pk, k) - 1) / 4 + 1, instr = c.mt * c.nt * psteps;
  if (2 >= psteps) {
    if (0 < padded && 3 > ctas * c.nteam) return -1;
    if (1 == ctas * c.nteam && 10 > c.T) return -1;
    if (instr < (1 == psteps || 8 >= m || 8 >= n ? 8 : (10 > c.T ? 18 : 0))) return -1;
  }
  if (0 < padded && 1 == c.T) {
    const int side = (0 == m % 16) ? m : n;
    if (2 == padded || (10 > c.mt * c.nt && (8 > c.mt * c.nt || 16 == side))) return -1;
  }
  pl->smem = (size_t)geo.region * c.nteam + slack;
  return 0;
}

int xs_tile_plan(int S, int m, int n, int k, xs_tile_plan_t* pl) {
  if (S < 1 || 0 != xs_tile_geometry(m, n, k, pl)) return -1;
  const void* const fn = (const void*)tile_kernel(pl->mt, pl->nt);
  int occ = 0;
  if (0 != xs_func_smem(fn, pl->smem)) return -1;
  if (cudaSuccess != cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, 32 * pl->T * pl->nteam, pl->smem) || occ < 1) return -1;
  if (occ > pl->ctas) occ = pl->ctas;
  const long resident = (long)occ * xs_sm_count() * pl->nteam;
  pl->nchunks = (int)((S < resident) ? S : resident);
  pl->L = S / pl->nchunks;
  pl->rem = S - pl->L * pl->nchunks;
  return 0;
}

int xs_tile_launch(const xs_tile_plan_t* pl, const xs_stack::StackTask* task, unsigned* err, void* stream) {
  StackTask tk = *task;
  TileGeo geo;
  tk.L = pl->L;
  tk.Ls[0] = pl->rem;
  tk.nchunks = tk.ngroups = pl->nchunks;
  tk.nsub_n = pl->nsub_n;
  tk.nsub = pl->T;
  make_geo(pl, tk.m, tk.n, &geo);
  const int grid = (pl->nchunks + pl->nteam - 1) / pl->nteam;
  void* prof = xs_profile_begin(stream);
  const cudaError_t r = pdl_launch(tile_kernel(pl->mt, pl->nt), grid, 32 * pl->T * pl->nteam, pl->smem, (cudaStream_t)stream,
    tk, geo, err, xs_device_error_ptr(), xs_wait_limit());
  const double m = tk.m, n = tk.n, k = tk.k;
  xs_profile_end(prof, "smm", 2.0 * m * n * k * (double)tk.S, 8.0 * tk.S * (m * k + k * n + 2.0 * m * n), stream);
  return (int)r;
}

}  // extern "C"
