// te_mma.cuh — interface between the tensor-core histogram path (te_mma.cu) and
// the launch driver of the TE entry points (te_pair.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace tenex {

enum { kOutPairfree = 0, kOutMatrix = 1, kOutStats = 2 };

// Device state of one launch: sort orders and tiles always, bit planes and column
// tables when the workspace has room for the tensor-core path (cap_rows > 0).
struct TeMma {
  const uint8_t* bins;
  int64_t ld;
  const int32_t* npv;
  int n, N, lag, b_max;
  double inv_unit;   // 1 / N, divided by to_fixed's 2^32
  int64_t row_len;
  int64_t p0, p1;
  int t_first, t_last;
  WsHeader* ws;
  int32_t* order;    // (n,) genes stably sorted by bin count (sources)
  // the rest only when cap_rows > 0
  int64_t cap_rows;  // bit-plane rows there is room for
  int sm_pairs;      // pairs of SMs of the device
  int max_cells;     // most cells of a pair of the tensor cores (a rule on N)
  int words;         // 32-bit words of a plane row (a multiple of 8)
  int32_t* rowoff;   // (n,) by gene: first plane row, -1 without planes
  int32_t* ncols;    // (n,) by gene: occupied target states, 0 = not a tensor-core target
  int32_t* torder;   // (n,) targets sorted by ncols, those with 0 first
  int32_t* tpos;     // (n,) by gene: its position in torder
  int32_t* cut;      // (n,) by gene: source positions [0, cut) are the tensor cores'
  int2* src;         // (n,) by source position: gene, first plane row
  int4* tgt;         // (n,) by position in torder: gene, bins, first column, cut
  int4* stile;       // (n,) source tiles: first position, sources, first row, rows
  int4* ttile;       // (n,) target tiles: first position, targets, first column, columns
  int32_t* nst;      // (n,) source tiles a target tile runs against
  int32_t* blk;      // (n / 16 + 2,) first work item of each block of source tiles
  int32_t* c2a;      // (n, 256) by gene: counts of the target states
  uint32_t* grp;     // (n, 16) by position: c1 | columns << 24 of x_t = j
  float2* colq;      // per column: c1 / c2a, c2a
  int2* colrow;      // per column: plane rows of x_{t+lag} and x_t
  // (words / 8, cap_rows, 8): 256 samples of every row, then the next 256, so that a
  // tile's rows are read as one piece. Bit s of row (g, v) = x_g[s] == v
  uint32_t* P;
  uint32_t* F;       // same, of x_g[s + lag]
  // output
  int out_mode;
  float* out;
  int64_t out_ld;
  const float* obs;
  double* sum;
  double* sumsq;
  int32_t* cnt_ge;
  int32_t* counts_dbg;
  int64_t counts_stride;
};

// Bytes behind the workspace's base part that the tensor-core path would use for
// every gene (0: it does not apply to such series, or is not the faster even for all
// pairs of them).
int64_t te_mma_bytes(int n, int64_t row_len, int b_max);

// Lays the path's buffers out in `bytes` bytes at `mem` (256-byte aligned): true
// when there is room for it and the launch has enough pairs.
bool te_mma_layout(TeMma* M, unsigned char* mem, int64_t bytes);

// Enqueues validation, source order and, with M.cap_rows > 0, the plan, the bit
// planes and the tensor-core launch. A pair of source position k and target t is
// this launch's when k < cut[t].
int te_mma_launch(const TeMma& M, const DevAttr& A, bool pair_list, cudaStream_t stream);

// Whether the tensor cores take every pair of the launch (no other launch needed).
bool te_mma_takes_all(const TeMma& M);

}  // namespace tenex
