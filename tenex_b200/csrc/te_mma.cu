// te_mma.cu — joint histograms of many (source, target) pairs as one contraction on
// the tensor cores, for pairs whose histogram has few cells.
//
// The counts c3[xt1, xt, y] of a pair are inner products over the samples of two 0/1
// vectors: [x[s+lag] = xt1 and x[s] = xt] of the target and [y[s] = y] of the source.
// So the histograms of all pairs are one matrix product: rows = (source, y), columns
// = (target, occupied state (xt1, xt)), K = samples. It costs one multiply-add per
// cell and sample where counting costs one shared-memory reduction per sample
// (2.2e12 of them per second), so pairs of few cells come here (te_mma_layout) and the
// others stay with te_pair.cu. Measured, all pairs, counting alone -> with this path:
// 10,000 genes x 20,000 samples (b to 16, 5% to 38) 873 -> 634 ms, 2,000 x 5,000
// (b to 16) 10.6 -> 7.4 ms, 3,281 x 458 (b to 7, every pair here) 6.6 -> 1.7 ms.
//
//   * plan (one CTA): sources sorted by bin count and targets by occupied states are
//     cut into tiles of at most 128 rows and 240 columns, whole genes only, so a
//     pair's cells lie in one tile. Which pairs come here depends on the pair alone
//     (columns of the target x bins of the source), not on the tiles.
//   * planes: one bit per (gene, bin, sample), of x and of x shifted by the lag, the
//     shifted one so that the words of a column are an AND of two aligned words.
//   * contraction: eight warps expand 256 samples of a tile's rows and columns at a
//     time from bits to packed E2M1 values in shared memory (four bit positions of a
//     word go to the four words of a 16-byte chunk, as 0.5, 1 or 2, the other operand
//     scaled inversely so every product is 1: no shifting of single bits); a ninth
//     issues tcgen05.mma kind::mxf4 with unit block scales into 240 float32 TMEM
//     columns (whole numbers, exact below 2^24). From HBM and L2 come 1 bit per row
//     and sample, not 4: 1.4 KB per 64 samples and tile instead of 12 KB, which L2
//     could not deliver.
//   * epilogue: a TMEM lane is one (source, y); it walks the columns of each target by
//     xt, so c2b is a sum of its own registers. The xt that have columns come from one
//     list of 8-byte words per half of the warps, without a loop over targets around
//     them (the kernel alone, 3,281 x 458: 1.79 -> 1.66 ms, 2,000 x 5,000: 5.45 -> 5.36).
//     The terms are te_pair.cu's, operation for operation. Those of one xt, 16 at most,
//     are added in float32, their sums over xt and y in 2^-32 fixed point, so no chain is
//     longer than te_pair.cu's and every order gives the same bits. One float32 chain over
//     a target's columns (up to 240 terms) left 300 samples of 15 bins against 3 up to 2.4
//     times (root mean square 1.4 times) as far from the float64 oracle as te_pair.cu does.
//     Whole launch with that chain / float64 / fixed point: 3,281 x 458 1.75 / 1.81 / 1.78
//     ms, 2,000 x 5,000 7.39 / 7.48 / 7.37, 10,000 x 20,000 634.5 / 636 / 632.8 (a
//     compensated float32 sum: 1.85, 7.52, 636.3).
//   * Bound: the shared-memory pipe (about 520 cycles per SM for a 256-sample step of a
//     256 x 240 tile: operands written, read by the MMAs, and the planes' loads; ncu: the
//     load-store part of it 66% of the cycles, the tensor pipe 62%, the logic pipe 55%).
//     The MMAs alone take under 390 (timed with operands left as they were).
//   * Two CTAs share an SM (256 TMEM columns each): one's epilogue runs under the
//     other's contraction. Work items go round the CTA pairs in an order that takes 16
//     source tiles at a time across all target tiles, so the planes in use stay in L2.
//   * Every mbarrier wait is bounded; on expiry the kernel sets the workspace's item
//     word and leaves after freeing its TMEM.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "te_mma.cuh"
#include "tcgen05.cuh"

namespace tenex {
namespace {

constexpr int kMaxTgtBins = 16;   // target bins (at most 16 columns share an xt)
constexpr int kMaxCols = 240;     // columns of a tile
constexpr int kRows = 128;        // rows of a tile (TMEM lanes) per CTA of a pair
constexpr int kMaxSrcBins = 64;   // source bins
constexpr int kBlk = 8;           // pairs of source tiles per block of the item order
constexpr int kStages = 3;
constexpr int kABytes = kRows * 128, kBBytes = kMaxCols / 2 * 128;
constexpr int kStageBytes = kABytes + kBBytes;
constexpr int kProducers = 256;   // threads that expand operands and run the epilogue
constexpr int kThreads = kProducers + 32;
constexpr uint32_t kSfCol = 248;  // TMEM columns of the unit scale factors
constexpr int kTmemCols = 256;
// Partial sums of a tile: one row (slot) of kRows 64-bit sums per target, two for targets of
// kSplitCols columns or more. Of the latter, those of kSplitBins bins or more are summed by
// two warps per lane quarter, one per slot. Neither number implies the other: a target of 16
// bins whose values lie in two of them, or whose series has few samples, has few columns.
constexpr int kSlots = 56, kSplitCols = 7, kSplitBins = 8;
// xt with columns, and one without for a half of a target of kSplitBins bins that has none
constexpr int kMaxGroups = kMaxCols + kSlots;
constexpr int kBlkCache = 128;    // item blocks whose starts sit in shared memory
static_assert(kSlots * kRows * 8 <= kStages * kStageBytes, "partial sums fit the stages");

// ---------------------------------------------------------------------------
// Validation and the target states' counts. One CTA per gene: every bin of gene g
// in [0, row_len) below n_per_var[g] and 1 <= n_per_var[g] <= b_max, else
// ws->bad_data. Targets of few bins also get c2a and the number of occupied states.
__global__ void __launch_bounds__(256) gene_prepass_kernel(TeMma M) {
  __shared__ int h[256];
  const int g = blockIdx.x, tid = threadIdx.x;
  const int b = M.npv[g];
  const uint8_t* row = M.bins + (int64_t)g * M.ld;
  const int64_t nvec = M.row_len >> 4;
  bool bad = b < 1 || b > M.b_max;
  const uint4* rv = reinterpret_cast<const uint4*>(row);
  for (int64_t v = tid; v < nvec; v += blockDim.x) {
    const uint4 q = __ldg(rv + v);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int bb = 0; bb < 4; ++bb) bad |= ((w[k] >> (8 * bb)) & 0xffu) >= (uint32_t)b;
  }
  for (int64_t i = (nvec << 4) + tid; i < M.row_len; i += blockDim.x) bad |= row[i] >= b;
  if (__syncthreads_or(bad)) {
    if (tid == 0) atomicExch(&M.ws->bad_data, 1);
    return;
  }
  if (M.cap_rows == 0) return;
  if (b > kMaxTgtBins || g < M.t_first || g > M.t_last) {
    if (tid == 0) M.ncols[g] = 0;
    return;
  }
  h[tid] = 0;
  __syncthreads();
  // four samples per step: an aligned word of x[s] and the two words around x[s + lag]
  const uint32_t* rw = reinterpret_cast<const uint32_t*>(row);
  const int last = (int)(M.ld >> 2) - 1, sh = (M.lag & 3) * 8;
  for (int s = tid * 4; s < M.N; s += 256 * 4) {
    const uint32_t a = __ldg(rw + (s >> 2));
    const int w1 = (s + M.lag) >> 2;
    const uint32_t c = __funnelshift_r(__ldg(rw + w1), __ldg(rw + min(w1 + 1, last)), sh);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (s + u < M.N)
        atomicAdd(&h[((c >> (8 * u)) & 0xffu) * (uint32_t)b + ((a >> (8 * u)) & 0xffu)], 1);
  }
  __syncthreads();
  const int v = h[tid];
  M.c2a[(int64_t)g * 256 + tid] = v;
  const int occ = __syncthreads_count(v > 0);
  if (tid == 0) M.ncols[g] = occ <= kMaxCols ? occ : 0;
}

// ---------------------------------------------------------------------------
// Plan: one CTA of 1024 threads.
struct PlanShared {
  int cnt[256], base[256], width[256], scan[256];
  int wc[32][256];
  int cls[256], n_cls;                       // classes with members, ascending
  int seg_tile[256], seg_pos[256], seg_per[256], seg_n[256], n_seg;
  int open_tile[256], open_pos[256], open_n[256], n_open;
  int n_tiles, n_src, room;
};

// Exclusive prefix sums of a[0..255] into out (all threads call; one warp works, eight
// values a lane).
__device__ void scan256(const int* a, int* out, int tid) {
  if (tid < 32) {
    int v[8], sum = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[i] = sum;
      sum += a[tid * 8 + i];
    }
    int before = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, before, o);
      if (tid >= o) before += t;
    }
    before -= sum;
#pragma unroll
    for (int i = 0; i < 8; ++i) out[tid * 8 + i] = before + v[i];
  }
  __syncthreads();
}

// Stable counting sort of 0..n-1 by key(g) in 0..255 into `order`; leaves the class
// sizes in S.cnt and the class starts in S.base.
template <class Key>
__device__ void stable_order(PlanShared& S, int n, Key key, int32_t* order, int tid) {
  const int lane = tid & 31, w = tid >> 5;
  if (tid < 256) S.cnt[tid] = 0;
  __syncthreads();
  for (int g = tid; g < n; g += 1024) atomicAdd(&S.cnt[key(g)], 1);
  __syncthreads();
  scan256(S.cnt, S.base, tid);
  if (tid < 256) S.scan[tid] = S.base[tid];  // next free position of each class
  for (int start = 0; start < n; start += 1024) {
    for (int i = tid; i < 32 * 256; i += 1024) (&S.wc[0][0])[i] = 0;
    __syncthreads();
    const int g = start + tid;
    const bool in = g < n;
    const int k = in ? key(g) : -1;
    const unsigned same = __match_any_sync(0xffffffffu, k);
    const int rank = __popc(same & ((1u << lane) - 1u));
    if (in && rank == 0) S.wc[w][k] = __popc(same);
    __syncthreads();
    if (tid < 256) {
      int run = S.scan[tid];
#pragma unroll 8
      for (int ww = 0; ww < 32; ++ww) {
        const int c = S.wc[ww][tid];
        S.wc[ww][tid] = run;
        run += c;
      }
      S.scan[tid] = run;
    }
    __syncthreads();
    if (in) order[S.wc[w][k] + rank] = g;
    __syncthreads();
  }
}

// Cuts the sorted positions of classes [c_lo, c_hi] (class = width of a member) into
// tiles of at most `room` width and `most` members (a member of a class from `dbl` on
// counts twice), positions from `limit` on left out. Full tiles of one class come out as segments (emitted in parallel by
// emit_tiles), those that span classes one by one.
__device__ void pack_tiles(PlanShared& S, int c_lo, int c_hi, int room, int most, int dbl,
                           int limit, int tid) {
  // a serial chain over the classes: one warp, 32 classes at a time in its lanes, all
  // lanes following the chain, quotients of numbers up to `room` by a reciprocal
  // (x + 1/2 is never within rounding of a multiple)
  if (tid < 32) {
    int n_seg = 0, n_open = 0, tile = 0, k = 0, used = 0, weight = 0, pos0 = 0;
    auto close = [&]() {
      if (tid == 0) {
        S.open_tile[n_open] = tile;
        S.open_pos[n_open] = pos0;
        S.open_n[n_open] = k;
      }
      ++n_open;
      ++tile;
      k = 0;
    };
    for (int c0 = 0; c0 < S.n_cls; c0 += 32) {
      const int ci = c0 + tid, mc = ci < S.n_cls ? S.cls[ci] : 0;
      const bool in = mc >= max(c_lo, 1) && mc <= c_hi;
      const int mpos = in ? S.base[mc] : 0, mm = in ? min(S.cnt[mc], limit - mpos) : 0;
      const float minv = 1.f / (float)max(mc, 1);
      const int mper = min((int)(((float)room + 0.5f) * minv), most >> (mc >= dbl ? 1 : 0));
      const float mpinv = 1.f / (float)max(mper, 1);
      // full tiles' worth of members: the quotient by a reciprocal holds below 2^20
      const bool exact = limit >= (1 << 20);
      for (int l = 0; l < min(32, S.n_cls - c0); ++l) {
        const int c = __shfl_sync(0xffffffffu, mc, l);
        int m = __shfl_sync(0xffffffffu, mm, l), pos = __shfl_sync(0xffffffffu, mpos, l);
        const float inv = __shfl_sync(0xffffffffu, minv, l);
        const int per = __shfl_sync(0xffffffffu, mper, l);
        const float pinv = __shfl_sync(0xffffffffu, mpinv, l);
        if (m <= 0) continue;
        const int sh = c >= dbl ? 1 : 0;
        if (k > 0) {
          const int r = min(m, min((int)(((float)(room - used) + 0.5f) * inv),
                                   (most - weight) >> sh));
          k += r;
          used += r * c;
          weight += r << sh;
          pos += r;
          m -= r;
          if (m > 0) close();
        }
        if (m > 0) {
          const int f = exact ? m / per : (int)(((float)m + 0.5f) * pinv);
          if (f > 0) {
            if (tid == 0) {
              S.seg_tile[n_seg] = tile;
              S.seg_pos[n_seg] = pos;
              S.seg_per[n_seg] = per;
              S.seg_n[n_seg] = f;
            }
            ++n_seg;
            tile += f;
            pos += f * per;
            m -= f * per;
          }
          if (m > 0) {
            pos0 = pos;
            k = m;
            used = m * c;
            weight = m << sh;
          }
        }
      }
    }
    if (k > 0) close();
    if (tid == 0) {
      S.n_seg = n_seg;
      S.n_open = n_open;
      S.n_tiles = tile;
    }
  }
  __syncthreads();
}

template <class Emit>
__device__ void emit_tiles(const PlanShared& S, Emit emit, int tid) {
  for (int i = tid; i < S.n_open; i += 1024) emit(S.open_tile[i], S.open_pos[i], S.open_n[i]);
  for (int s = tid >> 5; s < S.n_seg; s += 32)
    for (int i = tid & 31; i < S.seg_n[s]; i += 32)
      emit(S.seg_tile[s] + i, S.seg_pos[s] + i * S.seg_per[s], S.seg_per[s]);
  __syncthreads();
}

__device__ void list_classes(PlanShared& S, int tid) {
  if (tid < 256) S.width[tid] = S.cnt[tid] > 0;
  __syncthreads();
  scan256(S.width, S.cls, tid);
  const int at = tid < 256 ? S.cls[tid] : 0;
  __syncthreads();
  if (tid < 256 && S.width[tid]) S.cls[at] = tid;
  if (tid == 255) S.n_cls = at + S.width[255];
  __syncthreads();
}

__global__ void __launch_bounds__(1024) plan_kernel(TeMma M) {
  __shared__ PlanShared S;
  const int tid = threadIdx.x, n = M.n;
  // bins already found invalid: the launches that follow do nothing. (Counts outside
  // 1..255 stay in bounds here.)
  const bool bad = *(volatile int*)&M.ws->bad_data != 0;
  stable_order(S, n, [&](int g) { return min(max(M.npv[g], 0), 255); }, M.order, tid);
  if (M.cap_rows == 0 || bad) return;
  list_classes(S, tid);
  // plane rows by position: class start + rank x bins, as far as there is room
  if (tid < 256) S.width[tid] = tid <= kMaxSrcBins ? S.cnt[tid] * tid : 0;
  __syncthreads();
  scan256(S.width, S.wc[0], tid);
  if (tid == 0) {
    int pos = 0;
    for (int ci = 0; ci < S.n_cls; ++ci) {
      const int c = S.cls[ci];
      if (c < 1 || c > kMaxSrcBins) break;
      const int64_t fit = (M.cap_rows - S.wc[0][c]) / c;
      if (fit <= 0) break;
      pos = S.base[c] + (int)(fit < S.cnt[c] ? fit : S.cnt[c]);
      if (fit < S.cnt[c]) break;
    }
    S.n_src = pos;
  }
  __syncthreads();
  const int n_src = S.n_src;
  for (int pos = tid; pos < n; pos += 1024) {
    const int g = M.order[pos], c = M.npv[g];
    const int row = pos < n_src ? S.wc[0][c] + (pos - S.base[c]) * c : -1;
    M.rowoff[g] = row;
    M.src[pos] = make_int2(g, row);
  }
  pack_tiles(S, 1, kMaxSrcBins, kRows, kRows, 256, n_src, tid);
  emit_tiles(S, [&](int t, int pos, int m) {
    const int2 a = M.src[pos], b = M.src[pos + m - 1];
    M.stile[t] = make_int4(pos, m, a.y, b.y + M.npv[b.x] - a.y);
  }, tid);
  const int n_stiles = S.n_tiles;
  // how many source positions each target takes: those with bins x columns within
  // max_cells (S.base still holds the sources' class starts)
  for (int g = tid; g < n; g += 1024) {
    int nc = M.ncols[g], cut = 0;
    if (M.rowoff[g] < 0) nc = 0;
    if (nc > 0) {
      const int c = M.max_cells / nc;
      cut = min(c >= 255 ? n : S.base[c + 1], n_src);
      if (cut == 0) nc = 0;
    }
    M.ncols[g] = nc;
    M.cut[g] = cut;
  }
  __syncthreads();
  stable_order(S, n, [&](int g) { return M.ncols[g]; }, M.torder, tid);
  list_classes(S, tid);
  if (tid < 256) S.width[tid] = S.cnt[tid] * tid;
  __syncthreads();
  scan256(S.width, S.wc[0], tid);
  for (int pos = tid; pos < n; pos += 1024) {
    const int g = M.torder[pos], c = M.ncols[g];
    M.tpos[g] = pos;
    M.tgt[pos] = make_int4(g, M.npv[g], S.wc[0][c] + (pos - S.base[c]) * c, M.cut[g]);
  }
  // Tiles as wide as they can be, except where the items would not give every pair of
  // SMs one: an item's epilogue then sets the launch's time (100 genes x 1,000 samples:
  // 26.8 -> 17 us), so they get narrower, down to 64 columns or the widest target.
  if (tid == 0) {
    int cols = 0, widest = 0;
    for (int i = 0; i < S.n_cls; ++i) {
      cols += S.width[S.cls[i]];
      widest = S.cls[i];
    }
    const int64_t fair = (int64_t)cols * ((n_stiles + 1) / 2) / M.sm_pairs;
    S.room = min(kMaxCols, max(max(64, widest), ((int)min(fair, (int64_t)kMaxCols) + 15) & ~15));
  }
  __syncthreads();
  pack_tiles(S, 1, kMaxCols, S.room, kSlots, kSplitCols, n, tid);
  emit_tiles(S, [&](int t, int pos, int m) { M.ttile[t] = make_int4(pos, m, 0, 0); }, tid);
  for (int t = tid; t < S.n_tiles; t += 1024) {
    const int2 pm = make_int2(M.ttile[t].x, M.ttile[t].y);
    const int4 a = M.tgt[pm.x], b = M.tgt[pm.x + pm.y - 1];
    M.ttile[t] = make_int4(pm.x, pm.y, a.z, b.z + M.ncols[b.x] - a.z);
    // the tile's first target has the fewest columns, so the most sources
    const int cut = a.w;
    int lo = 0, hi = n_stiles;  // source tiles that start below cut
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (M.stile[mid].x < cut) lo = mid + 1;
      else hi = mid;
    }
    M.nst[t] = lo;
  }
  __syncthreads();
  const int n_ttiles = S.n_tiles;
  // items: block by block of kBlk pairs of source tiles, within it target tile by
  // target tile
  const int n_pairs = (n_stiles + 1) / 2, n_blk = (n_pairs + kBlk - 1) / kBlk;
  int run = 0;
  for (int b0 = 0; b0 < n_blk; b0 += 256) {
    const int b = b0 + tid;
    if (tid < 256) {
      int lo = 0, hi = n_ttiles;  // target tiles that reach into the block (nst descends)
      if (b < n_blk)
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (M.nst[mid] > b * kBlk * 2) lo = mid + 1;
          else hi = mid;
        }
      S.width[tid] = b < n_blk ? lo * min(kBlk, n_pairs - b * kBlk) : 0;
    }
    __syncthreads();
    scan256(S.width, S.cls, tid);
    if (tid < 256 && b <= n_blk) M.blk[b] = run + S.cls[tid];
    run += S.cls[255] + S.width[255];
    __syncthreads();
  }
  if (tid == 0) {
    M.blk[n_blk] = run;
    M.ws->mma_blocks = n_blk;
    M.ws->mma_stiles = n_stiles;
    M.ws->mma_items = run;
  }
}

// ---------------------------------------------------------------------------
// Bit planes of a gene (one warp per 256 samples) and a target's column table.
__global__ void __launch_bounds__(256) planes_kernel(TeMma M) {
  if (*(volatile int*)&M.ws->bad_data != 0) return;
  const int g = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row0 = M.rowoff[g];
  if (row0 < 0) return;
  const int b = M.npv[g], nc = M.ncols[g];
  const uint8_t* row = M.bins + (int64_t)g * M.ld;
  const int n_blocks = M.words >> 3;
  for (int kb = blockIdx.y * 8 + warp; kb < n_blocks; kb += gridDim.y * 8) {
    uint32_t x0[8], x1[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int64_t s = (int64_t)kb * 256 + k * 32 + lane;
      x0[k] = s < M.row_len ? row[s] : 255u;
      x1[k] = nc > 0 && s + M.lag < M.row_len ? row[s + M.lag] : 255u;
    }
    for (int v0 = 0; v0 < b; v0 += 32) {
      uint32_t p[8] = {}, f[8] = {};
      const int vn = min(32, b - v0);
      for (int v = 0; v < vn; ++v) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t m = __ballot_sync(0xffffffffu, x0[k] == (uint32_t)(v0 + v));
          if (lane == v) p[k] = m;
        }
        if (nc > 0)
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const uint32_t m = __ballot_sync(0xffffffffu, x1[k] == (uint32_t)(v0 + v));
            if (lane == v) f[k] = m;
          }
      }
      if (lane < vn) {
        const int64_t at = (kb * M.cap_rows + row0 + v0 + lane) * 8;
        uint4* d = reinterpret_cast<uint4*>(M.P + at);
        d[0] = make_uint4(p[0], p[1], p[2], p[3]);
        d[1] = make_uint4(p[4], p[5], p[6], p[7]);
        if (nc > 0) {
          d = reinterpret_cast<uint4*>(M.F + at);
          d[0] = make_uint4(f[0], f[1], f[2], f[3]);
          d[1] = make_uint4(f[4], f[5], f[6], f[7]);
        }
      }
    }
  }
  // columns by x_t = j, then x_{t+lag} = i, occupied states only
  if (nc > 0 && blockIdx.y == 0 && warp == 0) {
    const int32_t* c2a = M.c2a + (int64_t)g * 256;
    int occ = 0, c1 = 0;
    if (lane < b)
      for (int i = 0; i < b; ++i) {
        const int c = c2a[i * b + lane];
        occ += c > 0;
        c1 += c;
      }
    int at = occ;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, at, o);
      if (lane >= o) at += t;
    }
    at -= occ;
    if (lane < b) {
      const int pos = M.tpos[g], c0 = M.tgt[pos].z;
      M.grp[(int64_t)pos * 16 + lane] = (uint32_t)c1 | ((uint32_t)occ << 24);
      for (int i = 0; i < b; ++i) {
        const int c = c2a[i * b + lane];
        if (c == 0) continue;
        M.colq[c0 + at] = make_float2(__fdiv_rn((float)c1, (float)c), (float)c);
        M.colrow[c0 + at] = make_int2(row0 + i, row0 + lane);
        ++at;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// The contraction.
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 32 samples of a row (source) or a column (target) as E2M1 values: bit position
// 4 i + j goes to nibble i of word j, with the values 0.5, 1, 2, 1 (rows) and
// 2, 1, 0.5, 1 (columns) for j = 0..3.
__device__ __forceinline__ uint4 expand_row(uint32_t m) {
  return make_uint4(m & 0x11111111u, m & 0x22222222u, m & 0x44444444u, (m >> 2) & 0x22222222u);
}
__device__ __forceinline__ uint4 expand_col(uint32_t m) {
  const uint32_t d = m >> 2;
  return make_uint4((m << 2) & 0x44444444u, m & 0x22222222u, d & 0x11111111u, d & 0x22222222u);
}

// acc plus the sum over the L states xt1 of one xt (this lane's source bin y) of
// te_pair.cu's terms.
template <int L, int R>
__device__ __forceinline__ float group_terms(float acc, const uint32_t (&r)[R], const float2* q,
                                             float c1) {
  float b = __uint_as_float(r[0]);
#pragma unroll
  for (int u = 1; u < L; ++u) b += __uint_as_float(r[u]);
  const float inv = dev::rcp_count(fmaxf(b, 1.f));
#pragma unroll
  for (int u = 0; u < L; ++u) acc = dev::add_term(acc, __uint_as_float(r[u]), c1, b, inv, q[u]);
  return acc;
}

__device__ __forceinline__ float group_sum(float acc, uint32_t taddr, int len, const float2* q,
                                           float c1) {
  if (len <= 8) {
    uint32_t r[8];
    tmem_ld(taddr, r);
    switch (len) {
      case 0: return acc;
      case 1: return group_terms<1>(acc, r, q, c1);
      case 2: return group_terms<2>(acc, r, q, c1);
      case 3: return group_terms<3>(acc, r, q, c1);
      case 4: return group_terms<4>(acc, r, q, c1);
      case 5: return group_terms<5>(acc, r, q, c1);
      case 6: return group_terms<6>(acc, r, q, c1);
      case 7: return group_terms<7>(acc, r, q, c1);
      default: return group_terms<8>(acc, r, q, c1);
    }
  }
  uint32_t r[16];
  tmem_ld(taddr, r);
  switch (len) {
    case 9: return group_terms<9>(acc, r, q, c1);
    case 10: return group_terms<10>(acc, r, q, c1);
    case 11: return group_terms<11>(acc, r, q, c1);
    case 12: return group_terms<12>(acc, r, q, c1);
    case 13: return group_terms<13>(acc, r, q, c1);
    case 14: return group_terms<14>(acc, r, q, c1);
    case 15: return group_terms<15>(acc, r, q, c1);
    default: return group_terms<16>(acc, r, q, c1);
  }
}

// A work item's tables, copied from global memory while the item before it is in its
// epilogue.
struct Tables {
  int4 st, tt;           // M.stile (of this CTA's half), M.ttile; st.x < 0 ends the launch
  int wide0;             // first target of kSplitCols columns or more (targets ascend)
  float2 q[kMaxCols];    // M.colq
  int2 row[kMaxCols / 2];     // M.colrow of the columns this CTA expands
  // The xt of the tile's targets that have columns (M.grp), in the order in which the
  // epilogue's two groups of warps take them: the first one's from the front on, the
  // second one's from the back. {c1 (float), first column | columns << 8 | slot << 16 |
  // last of its slot << 31}
  uint2 grp[kMaxGroups];
  int n_grp[2];
  int4 tgt[kSlots];      // M.tgt
  int src[kRows];             // genes of the sources
  uint8_t at[kRows + 1];      // their first rows in the tile; then the number of rows
};

struct Shared {
  Tables tab[2];
  int blk[kBlkCache];
  uint64_t full[kStages], empty[kStages], acc;
  uint32_t tmem;
  int abort;
};
constexpr int kSmemBytes = kStages * kStageBytes + 1024 + (int)sizeof(Shared);
static_assert(2 * (kSmemBytes + 1024) <= 228 * 1024, "two CTAs share an SM");

// Four words of bits as four 16-byte chunks (half a step) of an operand row at `row`,
// chunk c at ((c * 16) ^ sw): the 128-byte swizzle.
template <bool ROW>
__device__ __forceinline__ void put_half(unsigned char* row, uint32_t sw, const uint32_t (&m)[4]) {
#pragma unroll
  for (uint32_t c = 0; c < 4; ++c)
    *reinterpret_cast<uint4*>(row + ((c << 4) ^ sw)) = ROW ? expand_row(m[c]) : expand_col(m[c]);
}

// Fills T for the next item with work, from item number q on in steps of the number
// of CTA pairs (one warp). Both CTAs of a pair walk the same numbers.
__device__ void next_item(const TeMma& M, Shared& S, Tables& T, uint32_t* q_io, uint32_t rank,
                          int n_items, int n_blk, int n_stiles, int lane) {
  const int* blk = n_blk <= kBlkCache ? S.blk : M.blk;
  const int n_pairs = (n_stiles + 1) / 2;
  uint32_t q = *q_io;
  int i = -1, j = 0;
  for (; q < (uint32_t)n_items; q += gridDim.x >> 1) {
    int lo = 0, hi = n_blk - 1;  // last block that starts at or below q
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (blk[mid] <= (int)q) lo = mid;
      else hi = mid - 1;
    }
    const int w = min(kBlk, n_pairs - lo * kBlk), rem = (int)q - blk[lo];
    j = rem / w;
    const int i0 = (lo * kBlk + rem - j * w) * 2;
    if (i0 < M.nst[j]) {
      i = i0 + (int)rank;
      q += gridDim.x >> 1;
      break;
    }
  }
  *q_io = q;
  if (i < 0) {
    if (lane == 0) T.st.x = -1;
    return;
  }
  const int4 st = i < n_stiles ? M.stile[i] : make_int4(0, 0, 0, 0), tt = M.ttile[j];
  if (lane == 0) {
    T.st = st;
    T.tt = tt;
    T.at[st.y] = (uint8_t)st.w;
  }
  for (int c = lane; c < tt.w; c += 32) T.q[c] = M.colq[tt.z + c];
  const int n_half = (tt.w + 15) / 16 * 8, c0 = (int)rank * n_half;
  for (int c = lane; c < n_half && c0 + c < tt.w; c += 32) T.row[c] = M.colrow[tt.z + c0 + c];
  int narrow = 0;
  for (int t = lane; t < tt.y; t += 32) {
    const int4 v = M.tgt[tt.x + t];
    T.tgt[t] = v;
    narrow += M.ncols[v.x] < kSplitCols;
  }
  narrow = __reduce_add_sync(0xffffffffu, narrow);
  if (lane == 0) T.wide0 = narrow;
  // two targets at a time, a lane per xt
  const int xt = lane & 15;
  int n0 = 0, n1 = 0;
#pragma unroll 2
  for (int k = lane; k < (tt.y + 1) / 2 * 32; k += 32) {
    const int t = k >> 4;
    const bool in = t < tt.y;
    const int4 v = in ? M.tgt[tt.x + t] : make_int4(0, 0, 0, 0);
    const uint32_t g = xt < v.y ? M.grp[(int64_t)tt.x * 16 + k] : 0u;
    const int len = (int)(g >> 24);
    int at = len;  // columns up to and with this xt
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const int below = __shfl_up_sync(0xffffffffu, at, o, 16);
      if (xt >= o) at += below;
    }
    // targets of many bins and with two slots: half of the xt each; the split depends on
    // the target alone, so a pair's sum does not depend on its tile
    const bool split = v.y >= kSplitBins && t >= narrow;
    const int mid = (v.y + (v.x & 1)) >> 1;
    const int h = split ? xt >= mid : t & 1;
    const uint32_t mine = lane < 16 ? 0xffffu : 0xffff0000u;  // this target's lanes
    const uint32_t some0 = __ballot_sync(0xffffffffu, len > 0 && h == 0) & mine;
    const uint32_t some1 = __ballot_sync(0xffffffffu, len > 0 && h == 1) & mine;
    const uint32_t some = h ? some1 : some0;
    const bool none = in && split && some == 0 && xt == (h ? mid : 0);
    const bool put = len > 0 || none;
    const uint32_t put0 = __ballot_sync(0xffffffffu, put && h == 0);
    const uint32_t put1 = __ballot_sync(0xffffffffu, put && h == 1);
    const uint32_t lt = (1u << lane) - 1;
    const bool last = none || (some >> lane) == 1u;
    if (put) {
      const int i = h ? kMaxGroups - 1 - n1 - __popc(put1 & lt) : n0 + __popc(put0 & lt);
      const int slot = (t < narrow ? t : 2 * t - narrow) + (split ? h : 0);
      T.grp[i] = make_uint2(__float_as_uint((float)(g & 0xffffffu)),
                            (uint32_t)(v.z - tt.z + at - len) | (uint32_t)len << 8 |
                                (uint32_t)slot << 16 | (last ? 0x80000000u : 0u));
    }
    n0 += __popc(put0);
    n1 += __popc(put1);
  }
  if (lane == 0) {
    T.n_grp[0] = n0;
    T.n_grp[1] = n1;
  }
  for (int s = lane; s < st.y; s += 32) {
    const int2 v = M.src[st.x + s];
    T.src[s] = v.x;
    T.at[s] = (uint8_t)(v.y - st.z);
  }
}

// One pair's TE to the launch's output (one thread per pair).
__device__ __forceinline__ void put_pair(const TeMma& M, int src, int tgt, long long tot) {
  const int64_t p = (int64_t)tgt * (M.n - 1) + (src < tgt ? src : src - 1);
  if (src == tgt || p < M.p0 || p >= M.p1) return;
  const float te = (float)((double)tot * M.inv_unit);
  if (M.out_mode == kOutPairfree) {
    M.out[p - M.p0] = te;
  } else if (M.out_mode == kOutMatrix) {
    M.out[(int64_t)src * M.out_ld + tgt] = te;
  } else {
    const int64_t m = (int64_t)src * M.n + tgt;
    const double td = (double)te;
    atomicAdd(M.sum + m, td);
    atomicAdd(M.sumsq + m, td * td);
    if (te >= M.obs[m]) atomicAdd(M.cnt_ge + m, 1);
  }
}

// Raw counts of this lane's (source, y) for target tt (parity checks only).
__device__ void put_counts(const TeMma& M, const Tables& T, int tt, int row, uint32_t lane_base) {
  int s = 0;
  while (s < T.st.y && T.at[s + 1] <= row) ++s;
  const bool mine = s < T.st.y;
  const int4 t = T.tgt[tt];
  const int src = mine ? T.src[s] : 0, tgt = t.x, bt = t.y;
  const int64_t p = (int64_t)tgt * (M.n - 1) + (src < tgt ? src : src - 1);
  const int bs = mine ? T.at[s + 1] - T.at[s] : 1, y = mine ? row - T.at[s] : 0;
  const bool put = mine && src != tgt && p >= M.p0 && p < M.p1;
  int32_t* cd = M.counts_dbg + (put ? (p - M.p0) * M.counts_stride : 0);
  if (put)
    for (int z = 0; z < bt * bt; ++z) cd[z * bs + y] = 0;
  const int r0 = M.rowoff[tgt], c0 = t.z - T.tt.z, nc = M.ncols[tgt];
  for (int c = 0; c < nc; ++c) {
    uint32_t r[8];
    tmem_ld(lane_base + (uint32_t)(c0 + c), r);
    const int2 cr = M.colrow[t.z + c];
    if (put) cd[((cr.x - r0) * bt + cr.y - r0) * bs + y] = (int32_t)__uint_as_float(r[0]);
  }
}

// Two CTAs (a pair of SMs) share an item: 256 rows, each CTA's own 128 in its TMEM;
// each expands half of the columns and the even one issues for both
// (cta_group::2), so a column is expanded once per 256 rows. 10,000 x 20,000: 216 ms
// for two thirds of the pairs. At one limit on cells: 203 ms, 245 before the producers
// were split in two groups, the odd CTA's arrivals lost their cluster-wide release and
// the epilogue its slow reciprocals and float64 sums, 315 with one CTA per 128-row tile.
// Row operands in TMEM instead of shared memory (192 columns, three stages): 407 ms at a
// limit of 1,600 cells against 311 here; the ring is then too short for its round trip of
// about 1,200 cycles.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 2) te_mma_kernel(TeMma M) {
  if (*(volatile int*)&M.ws->bad_data != 0) return;
  const int n_items = M.ws->mma_items, n_blk = M.ws->mma_blocks, n_stiles = M.ws->mma_stiles;
  if (n_items == 0) return;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* stages = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  Shared& S = *reinterpret_cast<Shared*>(stages + kStages * kStageBytes);
  long long* part = reinterpret_cast<long long*>(stages);  // [slot][row], epilogue only
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_rank();
  const int n_steps = (M.N + 255) >> 8;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      // the issuing CTA's: one more arrival for the other CTA's half
      mbar_init(&S.full[s], 2 * kProducers / 64);
      mbar_init(&S.empty[s], 1);
    }
    mbar_init(&S.acc, 1);
    S.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < n_blk && n_blk <= kBlkCache; i += kThreads) S.blk[i] = M.blk[i];
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&S.tmem)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  uint32_t q = blockIdx.x >> 1;  // next item number (last warp)
  if (warp == kProducers / 32)
    next_item(M, S, S.tab[0], &q, rank, n_items, n_blk, n_stiles, lane);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = S.tmem;
  if (warp < 4) tmem_st8(tmem + ((uint32_t)(warp * 32) << 16) + kSfCol, 0x7f7f7f7fu);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();  // both CTAs' barriers and scale factors are in place
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  const bool elected = elect_one();
  const uint32_t desc0 = (uint32_t)smem_desc_sw128(smem_u32(stages));  // low word
  uint32_t stage = 0, parity = 0;  // of the item's first step, in the ring of stages
  for (uint32_t item = 0;; ++item) {
    const Tables& T = S.tab[item & 1];
    if (T.st.x < 0) break;
    const int n_tgts = T.tt.y, n_cols = T.tt.w, n_rows = T.st.w, wide0 = T.wide0;
    const int n_mma = (n_cols + 15) & ~15;  // columns of the MMAs, half from each CTA
    if (tid < kProducers) {
      // ---- producers: warps 0-3 fill the even steps, warps 4-7 the odd ones. A lane
      // pair takes half a step each of rows r and r + 64 of this CTA's and of columns r
      // and r + 64 of its half; a store phase (eight lanes) covers four rows and both
      // halves: all 32 banks once. Words of the next step are loaded before this one's
      // are expanded.
      const int r = (tid & 127) >> 1, half = tid & 1, hc = n_mma >> 1;
      const int nb = min(hc, n_cols - (int)rank * hc);  // columns to expand here
      const bool a0_on = r < n_rows, a1_on = r + 64 < n_rows, b0_on = r < nb, b1_on = r + 64 < nb;
      const int2 c0 = b0_on ? T.row[r] : make_int2(0, 0);
      const int2 c1 = b1_on ? T.row[r + 64] : make_int2(0, 0);
      const uint32_t oa = (uint32_t)(T.st.z + (a0_on ? r : 0)) * 2 + half;
      const uint32_t oa1 = oa + (a1_on ? 128 : 0);
      const uint32_t of0 = (uint32_t)c0.x * 2 + half, oq0 = (uint32_t)c0.y * 2 + half;
      const uint32_t of1 = (uint32_t)c1.x * 2 + half, oq1 = (uint32_t)c1.y * 2 + half;
      const uint32_t sw = (uint32_t)((r & 7) ^ (half << 2)) << 4;  // all four rows'
      const int64_t stride = M.cap_rows * 2;  // 256 samples on
      unsigned char* const op = stages + r * 128;
      int k = warp >> 2;
      uint32_t s = stage + k, ph = parity ^ 1;  // `empty` starts as if just released
      if (s >= kStages) {
        s -= kStages;
        ph ^= 1;
      }
      const uint4* Pk = reinterpret_cast<const uint4*>(M.P) + k * stride;
      const uint4* Fk = reinterpret_cast<const uint4*>(M.F) + k * stride;
      uint4 va0, va1, vf0, vq0, vf1, vq1;
      if (k < n_steps) {
        va0 = __ldg(Pk + oa);
        va1 = __ldg(Pk + oa1);
        vf0 = __ldg(Fk + of0);
        vq0 = __ldg(Pk + oq0);
        vf1 = __ldg(Fk + of1);
        vq1 = __ldg(Pk + oq1);
      }
      for (; k < n_steps; k += 2) {
        const uint32_t a0[4] = {va0.x, va0.y, va0.z, va0.w};
        const uint32_t a1[4] = {va1.x, va1.y, va1.z, va1.w};
        const uint32_t b0[4] = {vf0.x & vq0.x, vf0.y & vq0.y, vf0.z & vq0.z, vf0.w & vq0.w};
        const uint32_t b1[4] = {vf1.x & vq1.x, vf1.y & vq1.y, vf1.z & vq1.z, vf1.w & vq1.w};
        if (k + 2 < n_steps) {
          Pk += 2 * stride;
          Fk += 2 * stride;
          va0 = __ldg(Pk + oa);
          va1 = __ldg(Pk + oa1);
          vf0 = __ldg(Fk + of0);
          vq0 = __ldg(Pk + oq0);
          vf1 = __ldg(Fk + of1);
          vq1 = __ldg(Pk + oq1);
        }
        if (!mbar_wait_warp(&S.empty[s], ph)) {
          *(volatile int*)&S.abort = 1;
          break;
        }
        unsigned char* const row = op + s * kStageBytes;
        if (a0_on) put_half<true>(row, sw, a0);
        if (b0_on) put_half<false>(row + kABytes, sw, b0);
        if (a1_on) put_half<true>(row + 64 * 128, sw, a1);
        if (b1_on) put_half<false>(row + kABytes + 64 * 128, sw, b1);
        fence_proxy_async_smem();
        __syncwarp();
        if (elected) mbar_arrive_cluster(&S.full[s], 0);
        s += 2;
        if (s >= kStages) {
          s -= kStages;
          ph ^= 1;
        }
      }
    } else if (rank == 0) {
      // ---- MMA issue, for both CTAs. The whole warp runs the loop, so that stage
      // numbers and descriptors stay in uniform registers; one lane issues -----------
      const uint32_t idesc = idesc_mxf4(2 * kRows, n_mma);
      const uint32_t last = (uint32_t)(((M.N & 255) + 63) >> 6);  // MMAs of a short last step
      uint32_t s = stage, ph = parity;
      for (int k = 0; k < n_steps; ++k) {
        if (!mbar_wait_warp(&S.full[s], ph)) {
          *(volatile int*)&S.abort = 1;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a = desc0 + s * (kStageBytes >> 4), b = a + (kABytes >> 4);
        const uint32_t n = (k + 1 < n_steps || last == 0) ? 4u : last;  // 64 samples each
        if (elected) {
#pragma unroll
          for (uint32_t kk = 0; kk < 4; ++kk)
            if (kk < n)
              mma_mxf4_pair(tmem, a + 2 * kk, b + 2 * kk, idesc, (k > 0 || kk > 0) ? 1u : 0u,
                            tmem + kSfCol);
          mma_commit_pair(&S.empty[s]);
        }
        __syncwarp();
        if (++s == kStages) {
          s = 0;
          ph ^= 1;
        }
      }
      if (elected) mma_commit_pair(&S.acc);
      __syncwarp();
    }
    // where the next item's steps start in the ring
    stage += (uint32_t)n_steps % kStages;
    parity ^= ((uint32_t)n_steps / kStages) & 1;
    if (stage >= kStages) {
      stage -= kStages;
      parity ^= 1;
    }

    // ---- epilogue: this CTA's rows ---------------------------------------------------
    if (!mbar_wait_sleep(&S.acc, item & 1, 64)) *(volatile int*)&S.abort = 1;
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (*(volatile int*)&S.abort) break;
    if (tid < kProducers) {
      const int half = warp >> 2, row = (warp & 3) * 32 + lane;
      const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
      if ((warp & 3) * 32 < n_rows) {
        const uint2* g = half ? T.grp + kMaxGroups - 1 : T.grp;
        const int step = half ? -1 : 1, n = T.n_grp[half];
        uint2 next = *g;
        long long sum = 0;
        for (int i = 0; i < n; ++i) {
          const float c1 = __uint_as_float(next.x);
          const uint32_t w = next.y;
          g += step;
          if (i + 1 < n) next = *g;
          const uint32_t at = w & 255u;
          sum += dev::to_fixed(group_sum(0.f, lane_base + at, (int)(w >> 8 & 31u), T.q + at, c1));
          if ((int32_t)w < 0) {
            part[(w >> 16 & 127u) * kRows + row] = sum;
            sum = 0;
          }
        }
        if (M.counts_dbg != nullptr && half == 0)
          for (int t = 0; t < n_tgts; ++t) put_counts(M, T, t, row, lane_base);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    } else {
      next_item(M, S, S.tab[(item + 1) & 1], &q, rank, n_items, n_blk, n_stiles, lane);
    }
    __syncthreads();
    const int n_src = T.st.y;
    for (int i = tid; i < n_src * n_tgts; i += kThreads) {
      const int tt = i / n_src, s = i - tt * n_src;
      const int4 t = T.tgt[tt];
      if (T.st.x + s >= t.w) continue;  // te_pair.cu's pair
      const long long* a = part + (tt < wide0 ? tt : 2 * tt - wide0) * kRows;
      long long tot = 0;
      const int y1 = T.at[s + 1];
      if (t.y >= kSplitBins && tt >= wide0)
        for (int y = T.at[s]; y < y1; ++y) tot += a[y] + a[y + kRows];
      else
        for (int y = T.at[s]; y < y1; ++y) tot += a[y];
      put_pair(M, T.src[s], t.x, tot);
    }
    __syncthreads();
  }
  // a wait ran out: nothing more is issued; what was issued before completes by itself
  __syncthreads();
  if (tid == 0 && S.abort) atomicExch(&M.ws->bad_item, 2);
  __syncwarp();
  cluster_sync();  // neither CTA's shared memory or TMEM goes while the other runs
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTmemCols)
                 : "memory");
  }
}

// Buffers behind the base workspace, each 256-byte aligned.
int64_t tables_bytes(int n) {
  const int64_t i = round_up((int64_t)n * 4, 256);
  return 6 * i + 2 * round_up((int64_t)n * 8, 256) /* src, blk */ +
         3 * round_up((int64_t)n * 16, 256) /* tgt, stile, ttile */ +
         round_up((int64_t)n * 1024, 256) /* c2a */ + round_up((int64_t)n * 64, 256) /* grp */;
}

// Most columns the targets can have: b_max^2 each, at most kMaxCols.
int64_t col_bound(int n, int b_max) {
  const int b = std::min(b_max, kMaxTgtBins);
  return (int64_t)n * std::min(b * b, kMaxCols);
}

// A pair's cells (occupied target states x source bins) up to which the tensor cores are
// the faster: their time goes with cells x samples, the counting kernel's with samples
// plus, per cell, its own entropy pass. Measured, ms of both kernels with 900 / 1,050 /
// 1,200 / 1,400 for the 1,200 below: 10,000 genes x 20,000 samples 637 / 637 / 634 / 638;
// 2,000 x 5,000 7.10 / 7.14 / 7.22 / 7.34; 1,000 x 2,500 1.39 / 1.38 / 1.35 / 1.30; 301 x
// 101,003 2.35 / 2.17 / 2.12 / 2.21. Short series: 2,000 x 600 (b to 16) at a limit of
// 1,000 / 1,600 / 2,600 cells 4.82 / 4.19 / 3.76.
int max_cells(double N) { return N <= 2078.0 ? 4096 : (int)(1200.0 * N / (N - 1470.0)); }

// Whether a pair of b_max bins each is the tensor cores': then every pair is.
bool takes_every_pair(int b_max, int N) {
  const int64_t b = b_max;
  return b * b <= kMaxCols && b * b * b <= max_cells(N);
}

// Whether a launch over `pairs` pairs is faster with the tensor-core path than in the
// counting kernel alone, with room for its planes. The path adds two launches and the plan's
// serial chain (25 us at the least), the planes of all n genes however few the pairs, and an
// item's chain of N / 256 steps; where only some pairs are its own the counting kernel runs after it, with
// its own last round of items. The counting kernel takes pairs x (N + about 2,000) / 2.1e12
// s where its items (32 sources of one target at the least) fill the SMs; up to 17 genes
// the two chains are about equally long. Measured, us with the path / without, b_max 6 | b_max 16:
//   genes x samples  100 x 300 46 / 36 | 86 / 64   200 x 300 68 / 67 | 129 / 125
//   100 x 2,000 54 / 46 | 119 / 74   200 x 2,000 71 / 84 | 184 / 146
//   300 x 2,000 87 / 150 | 271 / 261   140 x 20,000 102 / 189 | 323 / 263
//   300 x 20,000 148 / 671 | 856 / 973   20 x 100,000 189 / 248 | 507 / 334
//   10 x 1,000,000 1,320 / 1,140 | 3,570 / 2,020   20 x 1,000,000 1,530 / 2,200 | 5,230 / 3,460
//   10,000 x 20,000, b_max 16, one target's pairs 1,010 / 204, 16 targets' 1,960 / 1,750,
//   32 targets' 2,900 / 3,180; 2,000 x 20,000, b_max 6, 1 target 182 / 79, 8: 197 / 221.
// Above 16 bins most genes usually have fewer (a bin count of 38 after coarsening comes from a
// few), so the path takes most pairs there and is worth it sooner: 283 genes x 5,516 samples
// of 3 bins, 3% of 38, 246 / 377; 311 x 3,714, 4 bins and 8% of 38, 322 / 454.
// Over 2,700 sizes about the line (12 to 1,000 genes, 200 to 120,000 samples, with and without
// genes of 38 bins) the choice is on average within 1.2% of the better one, and at most 28%
// slower than the path always taken (one in ninety over 10%).
bool worth_it(int n, int N, int b_max, int64_t pairs) {
  const double work = (double)pairs * (N + 2000.0), planes = (double)n * N;
  if (!takes_every_pair(b_max, N)) {
    const double more = b_max > kMaxTgtBins ? std::min(2e4 * N, 7e8) : std::min(1.5e5 * N, 5e8);
    return work >= 1e8 + more + 25.0 * planes;
  }
  const double items = ((double)pairs / (n - 1) + 1) * ((n + 31) / 32), sms = 148;
  return pairs >= 300 && work * std::max(1.0, sms / items) >= 1e8 + 5.0 * planes;
}

// The same where the workspace has room for a part of the plane rows only: `room` is that
// part of the most rows the genes can have. Genes have about half of the most bins, and the
// counting kernel still runs after the path, so about min(1, 2 room)^2 of the pairs have to
// be worth what the path adds. Measured, us without / with room for 0.07, 0.15, 0.25, 0.4,
// 0.75 of the rows:
//   100 x 20,000 (b to 6)   130 / 188, 196, 193, 164, 105   200 x 2,000 (6)  90 / 122, 119, 115, 105, 87
//   300 x 5,000 (6)         238 / 276, 265, 244, 213, 106   400 x 3,000 (16) 497 / 518, 499, 473, 433, 408
//   600 x 2,000 (6)         480 / 506, 475, 438, 357, 161   1,000 x 5,000 (16) 3,209 / 3,130, 2,898, 2,643, ...
// Up to a twentieth short (tables moved to an aligned address) counts as all.
bool worth_it_with(double room, int N, int64_t pairs) {
  const double share = std::min(1.0, 2.0 * room);
  return room >= 0.95 || (double)pairs * (N + 2000.0) * share * share >= 2.5e8;
}

}  // namespace

// Plane rows for every gene up to 16 bins; sources of more bins use what those leave.
// 8 GiB of planes at most (22,000 genes of 16 bins x 100,000 cells).
int64_t te_mma_bytes(int n, int64_t row_len, int b_max) {
  if (row_len >= ((int64_t)1 << 24)) return 0;  // float32 counts are exact below 2^24
  if (!worth_it(n, (int)row_len - 1, b_max, (int64_t)n * (n - 1))) return 0;
  const int64_t plane = round_up(row_len, 256) / 8 * 2;
  int64_t rows = (int64_t)n * std::min(b_max, kMaxTgtBins);
  rows = std::min(rows, ((int64_t)8 << 30) / plane);
  return tables_bytes(n) + round_up(col_bound(n, b_max) * 16, 256) + 256 + rows * plane;
}

bool te_mma_layout(TeMma* M, unsigned char* mem, int64_t bytes) {
  M->cap_rows = 0;
  if (M->row_len >= ((int64_t)1 << 24) || !worth_it(M->n, M->N, M->b_max, M->p1 - M->p0))
    return false;
  const int n = M->n;
  // work items are counted in 32 bits: at most one per target and pair of source tiles (a
  // full tile has over kRows - bins rows). Beyond 170,000 genes of 16 bins.
  const int64_t c = std::min(M->b_max, kMaxSrcBins);
  const int64_t tile_pairs = ((int64_t)n * c / (kRows + 1 - c) + 2) / 2;
  if ((int64_t)(M->t_last - M->t_first + 1) * tile_pairs > 0x7fffffff) return false;
  M->words = (int)(round_up(M->row_len, 256) / 32);
  const int64_t cols = col_bound(n, M->b_max);
  const int64_t fixed = tables_bytes(n) + round_up(cols * 16, 256) + 256;
  const int64_t rows = (bytes - fixed) / ((int64_t)M->words * 8);
  if (bytes < fixed || rows < 2) return false;
  const double most = (double)n * std::min(M->b_max, kMaxTgtBins);
  if (!worth_it_with((double)rows / most, M->N, M->p1 - M->p0)) return false;
  unsigned char* at = mem;
  auto take = [&](int64_t b) {
    unsigned char* p = at;
    at += round_up(b, 256);
    return p;
  };
  M->rowoff = reinterpret_cast<int32_t*>(take((int64_t)n * 4));
  M->ncols = reinterpret_cast<int32_t*>(take((int64_t)n * 4));
  M->torder = reinterpret_cast<int32_t*>(take((int64_t)n * 4));
  M->tpos = reinterpret_cast<int32_t*>(take((int64_t)n * 4));
  M->cut = reinterpret_cast<int32_t*>(take((int64_t)n * 4));
  M->nst = reinterpret_cast<int32_t*>(take((int64_t)n * 4));
  M->src = reinterpret_cast<int2*>(take((int64_t)n * 8));
  M->blk = reinterpret_cast<int32_t*>(take((int64_t)n * 8));
  M->tgt = reinterpret_cast<int4*>(take((int64_t)n * 16));
  M->stile = reinterpret_cast<int4*>(take((int64_t)n * 16));
  M->ttile = reinterpret_cast<int4*>(take((int64_t)n * 16));
  M->c2a = reinterpret_cast<int32_t*>(take((int64_t)n * 1024));
  M->grp = reinterpret_cast<uint32_t*>(take((int64_t)n * 64));
  M->colq = reinterpret_cast<float2*>(take(cols * 16));
  M->colrow = reinterpret_cast<int2*>(M->colq + cols);
  M->max_cells = max_cells(M->N);
  M->cap_rows = std::min<int64_t>(rows, (int64_t)1 << 29);
  M->P = reinterpret_cast<uint32_t*>(at);
  M->F = M->P + M->cap_rows * M->words;
  return true;
}

bool te_mma_takes_all(const TeMma& M) {
  return takes_every_pair(M.b_max, M.N) && (int64_t)M.n * M.b_max <= M.cap_rows;
}

int te_mma_launch(const TeMma& M, const DevAttr& A, bool pair_list, cudaStream_t stream) {
  gene_prepass_kernel<<<M.n, 256, 0, stream>>>(M);
  int st = check_launch("gene_prepass_kernel");
  if (st || pair_list) return st;
  plan_kernel<<<1, 1024, 0, stream>>>(M);
  if ((st = check_launch("plan_kernel")) || M.cap_rows == 0) return st;
  // about four 256-sample blocks per warp
  const int blocks = M.words / 8;
  planes_kernel<<<dim3((unsigned)M.n, (unsigned)std::max(1, std::min(64, blocks / 32))), 256, 0,
                  stream>>>(M);
  if ((st = check_launch("planes_kernel"))) return st;
  cudaError_t e = cudaFuncSetAttribute(te_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kSmemBytes);
  if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute");
  te_mma_kernel<<<A.sm_count / 2 * 4, kThreads, kSmemBytes, stream>>>(M);
  return check_launch("te_mma_kernel");
}

}  // namespace tenex
