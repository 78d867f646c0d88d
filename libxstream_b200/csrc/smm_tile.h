/*
 * The tile stack kernel (smm_tile.cu) as the stack path's launcher uses it.
 */
#pragma once

#include "smm_stack.cuh"

extern "C" {

/** How one stack runs on the tile kernel. */
typedef struct xs_tile_plan_t {
  int mt, nt;       /* warp tile of C in 8 x 8 fragments */
  int T, nteam;     /* warps (tiles of one C block) per team, teams per CTA */
  int nsub_n;       /* warp tiles per row of the block */
  int Q;            /* distance of the k indices of a DMMA step */
  int pk, npan, R;  /* k indices per panel, panels per entry, stages of the ring */
  int ctas;         /* CTAs per SM that the shared memory is cut for */
  int nchunks, L, rem; /* the first rem chunks hold L + 1 entries, the others L */
  size_t smem;
} xs_tile_plan_t;

/** The shape's part of a plan (all fields but nchunks, L, rem): host arithmetic only; nonzero when the tile
    kernel does not take the shape. */
int xs_tile_geometry(int m, int n, int k, xs_tile_plan_t* plan);
/** Plans S entries of m x n x k; nonzero when the tile kernel does not take the shape. */
int xs_tile_plan(int S, int m, int n, int k, xs_tile_plan_t* plan);
/** Enqueues the kernel: task with operands, grouped entries, pieces (2 * nchunks * T tiles) and
    zeroed arrival counters (3 * nchunks * T); returns a cudaError_t value. */
int xs_tile_launch(const xs_tile_plan_t* plan, const xs_stack::StackTask* task, unsigned* err, void* stream);

}  // extern "C"
