// Batched personalised PageRank: B teleport vectors solved together as a
// sparse matrix times dense matrix iteration (SpMM). Each column is the
// reference's PageRank with that personalization vector
// (crates/engine/src/metrics/spectral.rs:211-281): it has its own
// normalisation, dangling mass and L1 change, and it stops at its own first
// sweep with change <= tol, keeping that iterate while the others go on.
//
// Layout: the iterate is node-major, Y[i * B + c], so the gather of a source
// node's B values is one contiguous run (coalesced across the warp: lane l
// holds columns l, l + 32, ...). Rows are split over warps in ranges of
// about equal arc counts; rows with more than LONG_ROW arcs are cut into
// chunks whose partial sums a second kernel adds in chunk order. Per-column
// sums are kept per lane, joined per CTA in warp order and per sweep in CTA
// order, so the results do not change from run to run.
//
// A sweep costs what its width costs, and columns stop at very different sweeps
// (most of 100 seed sets on R-MAT 20 after 17 to 43, one that reaches a closed
// class after 125), so the columns still running are packed into a narrower
// iterate whenever a quarter of the width has stopped; the others leave with
// their result. On that batch only 23% of the column-sweeps of full-width
// sweeps did anything (380 ms a solve at full width, 125 ms packed). Up to 16 columns a warp takes several rows at once (spmm_rows with
// W < 32 lanes per row).
//
// Precision: FP64, or mixed (FP32 sweeps until every column's change is below
// max(tol * switch_factor, switch_floor), then, on the same trajectories, one
// FP64 anchor sweep and refinement sweeps gathering the FP32 correction (or
// plain FP64 sweeps) until each column meets tol).
#include <algorithm>
#include <cfloat>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <vector>

#include "batch.cuh"
#include "pagerank.cuh"

namespace knb {

constexpr int BT = 256;          // threads per CTA
constexpr int BW = BT / 32;      // warps per CTA
constexpr int MAXVW = 8;         // columns per lane (B <= 256 per launch)
constexpr uint32_t LONG_ROW = 512;
// A warp's share of rows: an arc costs one gathered iterate row, a row about
// ROW_COST of them (its iterates read and written, and a chain of waits). With
// 256 per range and rows at 1 a third of the sweep's time went by with SMs
// idle: ranges of empty rows took longest.
constexpr uint32_t RANGE_ARCS = 128;
constexpr uint32_t ROW_COST = 6;

struct RowRange {
  uint32_t lo, hi;
};
struct Chunk {
  uint32_t row, a0, a1;
};

// Per-column state of a batch phase.
struct ColState {
  double inv_total;       // 1 / sum of the column's current iterate
  double dterm;           // its dangling mass, normalised
  double prev_inv_total;
  double total, change;
  int32_t frozen;         // converged (or finished) columns keep their iterate
  int32_t iter;           // sweeps this column took
  int32_t converged;
  int32_t buf;            // the buffer its last sweep wrote
};

// A sweep's columns: `B` of them, the iterate's row length. Column c of the
// sweep is column cmap[c] of the `Bo` columns the batch began with, which the
// teleport columns and the refinement's FP64 arrays keep; inv is the inverse
// (NO_COL for a column that has stopped and left).
constexpr uint32_t NO_COL = 0xFFFFFFFFu;
struct BatchScalars {
  double d;
  double pu;    // 1 / n
  uint32_t n, B, Bo;
  int jump_uniform;
  double tol;
  int32_t max_iter;
  const uint32_t* cmap;
  const uint32_t* inv;
};

// Arcs whose gathers one warp keeps in flight together (U): 1, 2 or 4,
// picked per operator by timing (tune_arcs_in_flight). The products are
// added in arc order whatever U is, so the choice never changes a result.
constexpr int U_CANDIDATES[] = {1, 2, 4};

// The normalised teleport columns: dense node-major P[i * B + c], or, when
// few entries are nonzero, each row's nonzero (column, value) pairs in
// column order (rowptr over n + 1 rows).
struct PersView {
  const double* dense;
  const uint32_t* rowptr;
  const uint32_t* cols;
  const double* vals;
};

// Row sum of arcs [a0, a1) of A times Z for this lane's columns, taking every
// P-th arc from a0. U arcs at a time: their indices, then all their gathers,
// then the products added in arc order (so each sum keeps the order of a
// one-arc loop).
template <class VT, class MT, int VW, int U, int P>
__device__ __forceinline__ void row_product(const OpView<MT>& op, const VT* __restrict__ Z,
                                            uint32_t B, uint32_t a0, uint32_t a1, int lane,
                                            VT (&acc)[VW]) {
#pragma unroll
  for (int v = 0; v < VW; ++v) acc[v] = VT(0);
  uint32_t k = a0;
  for (; k + (U - 1) * P < a1; k += U * P) {
    uint32_t j[U];
    VT w[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      j[u] = __ldg(op.cols + k + u * P);
      w[u] = op.vals ? (VT)__ldg(op.vals + k + u * P) : VT(1);
    }
    VT z[U][VW];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const VT* zr = Z + (size_t)j[u] * B;
#pragma unroll
      for (int v = 0; v < VW; ++v) {
        const uint32_t c = lane + 32 * v;
        z[u][v] = c < B ? __ldg(zr + c) : VT(0);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int v = 0; v < VW; ++v)
        if (lane + 32 * v < B) acc[v] += w[u] * z[u][v];
  }
  for (; k < a1; k += P) {
    const uint32_t j = __ldg(op.cols + k);
    const VT w = op.vals ? (VT)__ldg(op.vals + k) : VT(1);
    const VT* zr = Z + (size_t)j * B;
#pragma unroll
    for (int v = 0; v < VW; ++v) {
      const uint32_t c = lane + 32 * v;
      if (c < B) acc[v] += w * __ldg(zr + c);
    }
  }
}

// Epilogue modes: the plain update (VT iterate), the anchor sweep and the
// refinement sweeps of the mixed path's FP64 phase. As in the single-vector
// path (RefineEpi, pagerank.cu) each column's iterate is held from the
// anchor on as y = y_ref + e with e in FP32: the anchor sweep gathers the
// FP64 z_ref = y_ref / out and keeps s_ref = A z_ref; a refinement sweep
// gathers z_e = e / out in FP32 and forms s = s_ref + A z_e, the update, the
// sums and the change in FP64. A refinement sweep gathers B FP32 values per
// arc where an FP64 sweep gathers B FP64 values.
enum { EPI_PLAIN = 0, EPI_ANCHOR = 1, EPI_REFINE = 2 };
struct RefineBufs {
  const double* yref;  // n x B: the iterate the anchor sweep starts from
  double* sref;        // n x B: A z_ref, written by the anchor sweep
  const float* eold;   // refinement sweeps: e of the input iterate
  float* enew;         // e of the new iterate
  float* zenew;        // enew / out
  const float* io32;   // 1 / out in FP32 (0 for dangling nodes)
};

// What row i's update reads besides the product, loaded before the product so
// that the waits overlap (the FP64 arrays of the refinement after it: with
// them the sweep needs 80 registers, a CTA per SM less).
template <class VT, int VW>
struct RowIn {
  VT yo[VW];         // plain: the old iterate; refinement: e of the old iterate
  VT io;
  uint32_t e0, e1;   // the row's sparse teleport entries
};

template <class VT, int VW, int MODE>
__device__ __forceinline__ RowIn<VT, VW> row_fetch(uint32_t i, int lane,
                                                         const BatchScalars& bs,
                                                         const VT* __restrict__ Yold,
                                                         const VT* __restrict__ inv_out,
                                                         const PersView& pv,
                                                         const RefineBufs& rb) {
  RowIn<VT, VW> in;
  in.e0 = in.e1 = 0;
  if (!pv.dense) {
    in.e0 = pv.rowptr[i];
    in.e1 = pv.rowptr[i + 1];
  }
  in.io = MODE == EPI_PLAIN ? inv_out[i] : (VT)rb.io32[i];
#pragma unroll
  for (int v = 0; v < VW; ++v) {
    const uint32_t c = lane + 32 * v;
    in.yo[v] = VT(0);
    if (c >= bs.B) continue;
    if constexpr (MODE == EPI_PLAIN) in.yo[v] = Yold[(size_t)i * bs.B + c];
    if constexpr (MODE == EPI_REFINE) in.yo[v] = (VT)rb.eold[(size_t)i * bs.B + c];
  }
  return in;
}

// The PageRank update of row i for this lane's columns, and its per-column
// sums (mass, dangling mass, L1 change) into the group's slice red[3][B] of
// shared memory (every slot has one writer, which takes its rows in order).
template <class VT, int VW, int MODE>
__device__ __forceinline__ void row_update(uint32_t i, const VT (&s)[VW], int lane,
                                           const BatchScalars& bs, const ColState* cs,
                                           const RowIn<VT, VW>& in, VT* __restrict__ Ynew,
                                           VT* __restrict__ Znew, const PersView& pv,
                                           const RefineBufs& rb, double* red) {
  using PT = std::conditional_t<MODE == EPI_PLAIN, VT, double>;
  PT psp[VW];  // this lane's teleport values of row i (sparse teleport)
#pragma unroll
  for (int v = 0; v < VW; ++v) psp[v] = PT(0);
  for (uint32_t e = in.e0; e < in.e1; ++e) {
    const uint32_t c = __ldg(bs.inv + pv.cols[e]);
    if (c == NO_COL || (c & 31u) != (uint32_t)lane) continue;
    const PT x = (PT)pv.vals[e];
#pragma unroll
    for (int v = 0; v < VW; ++v)
      if ((c >> 5) == (uint32_t)v) psp[v] = x;
  }
#pragma unroll
  for (int v = 0; v < VW; ++v) {
    const uint32_t c = lane + 32 * v;
    if (c >= bs.B || cs[c].frozen) continue;
    const size_t q = (size_t)i * bs.B + c;
    if constexpr (MODE == EPI_PLAIN) {
      const VT io = in.io;
      const VT it = (VT)cs[c].inv_total, dt = (VT)cs[c].dterm;
      const VT pg = pv.dense ? (VT)pv.dense[(size_t)i * bs.Bo + __ldg(bs.cmap + c)] : psp[v];
      const VT jg = bs.jump_uniform ? (VT)bs.pu : pg;
      const VT u = (VT)bs.d * (s[v] * it + dt * jg) + (VT)(1.0 - bs.d) * pg;
      const VT xo = in.yo[v] * it;
      Ynew[q] = u;
      Znew[q] = u * io;
      red[c] += (double)u;
      if (io == VT(0)) red[bs.B + c] += (double)u;
      red[2 * bs.B + c] += fabs((double)u - (double)xo);
    } else {
      const float io = (float)in.io;
      const double it = cs[c].inv_total, dt = cs[c].dterm;
      const size_t r = (size_t)i * bs.Bo + __ldg(bs.cmap + c);
      double sum;
      if constexpr (MODE == EPI_ANCHOR) {
        sum = (double)s[v];
        rb.sref[r] = sum;
      } else {
        sum = rb.sref[r] + (double)s[v];
      }
      const double pg = pv.dense ? pv.dense[r] : psp[v];
      const double jg = bs.jump_uniform ? bs.pu : pg;
      const double u = bs.d * (sum * it + dt * jg) + (1.0 - bs.d) * pg;
      const double yr = rb.yref[r];
      const double yo = MODE == EPI_ANCHOR ? yr : yr + (double)in.yo[v];
      const float en = (float)(u - yr);
      const double us = yr + (double)en;  // the iterate as stored
      rb.enew[q] = en;
      rb.zenew[q] = en * io;
      red[c] += us;
      if (io == 0.0f) red[bs.B + c] += us;
      red[2 * bs.B + c] += fabs(us - yo * it);
    }
  }
}

// Lanes of a row: a whole warp for more than 16 columns (lane l holds columns
// l, l + 32, ...). Up to 16 columns W lanes hold them, the power of two that
// does, and a row takes S = max(W, 8) lanes, which share its arcs out by
// S / W: a warp then has 32 / S rows under way, and a row of 512 arcs does not
// hold up its neighbours (one column on R-MAT 20: 200 us a sweep with one lane
// per row, 95 us with 8).
template <int W>
struct Lanes {
  static constexpr int S = W < 8 ? 8 : W;
  static constexpr int G = 32 / S;  // rows a warp takes at once
  static constexpr int P = S / W;   // arcs of a row under way at once
  int col, group, arc;
  __device__ __forceinline__ Lanes() {
    const int lane = threadIdx.x & 31;
    col = lane % W;
    arc = lane % S / W;
    group = lane / S;
  }
  // The sum over the lanes that share a row's arcs, in a fixed order, in
  // every one of them.
  template <class VT, int VW>
  __device__ __forceinline__ void join(VT (&acc)[VW]) const {
    if constexpr (P > 1) {
      const unsigned mask = ((1u << S) - 1u) << (group * S);
#pragma unroll
      for (int o = W; o < S; o <<= 1)
#pragma unroll
        for (int v = 0; v < VW; ++v) acc[v] += __shfl_xor_sync(mask, acc[v], o);
    }
  }
};

// Zeroes this group's slice [3][B] of the CTA's column sums in smem
// ([BW][G][3][B]) and returns it.
template <int W>
__device__ __forceinline__ double* group_sums(double* smem, uint32_t B) {
  const Lanes<W> l;
  double* red = smem + (size_t)((threadIdx.x >> 5) * Lanes<W>::G + l.group) * 3 * B;
  for (uint32_t q = l.arc * W + l.col; q < 3 * B; q += Lanes<W>::S) red[q] = 0.0;
  __syncwarp();
  return red;
}

// Joins the groups' column sums of a CTA in order into part[cta][3][B].
template <int W>
__device__ __forceinline__ void cta_column_sums(uint32_t B, double* __restrict__ part,
                                                const double* smem) {
  __syncthreads();
  for (uint32_t q = threadIdx.x; q < 3 * B; q += BT) {
    double a = 0;
    for (int g = 0; g < BW * Lanes<W>::G; ++g) a += smem[(size_t)g * 3 * B + q];
    part[(size_t)blockIdx.x * 3 * B + q] = a;
  }
}

// The rows of at most LONG_ROW arcs: their products and updates. Bound by the
// gathers, one iterate row (B values) per arc: 100 columns on R-MAT 20 (6.2 GB
// of gathers a sweep) 2.35 ms with ranges by arcs, late loads and 4 CTAs per
// SM whatever the kernel's registers, 1.00 ms since (refinement 3.05 and
// 1.60).
template <class VT, class MT, int W, int VW, int U, int MODE>
__global__ void __launch_bounds__(BT, VW * sizeof(VT) <= 16 ? 4 : 2)
spmm_rows(OpView<MT> op, const VT* __restrict__ Z, const RowRange* __restrict__ ranges,
          uint32_t nranges, BatchScalars bs, const ColState* __restrict__ cs,
          const VT* __restrict__ Yold, VT* __restrict__ Ynew, VT* __restrict__ Znew,
          const VT* __restrict__ inv_out, PersView P, RefineBufs rb,
          double* __restrict__ part, const int32_t* __restrict__ all_frozen) {
  if (*all_frozen) return;
  extern __shared__ double smem_b[];
  const Lanes<W> l;
  double* red = group_sums<W>(smem_b, bs.B);
  const uint32_t gw = blockIdx.x * BW + (threadIdx.x >> 5), nw = gridDim.x * BW;
  for (uint32_t r = gw; r < nranges; r += nw) {
    const RowRange rr = ranges[r];
    for (uint32_t i = rr.lo + l.group; i < rr.hi; i += Lanes<W>::G) {
      const uint32_t a0 = op.off[i], a1 = op.off[i + 1];
      if (a1 - a0 > LONG_ROW) continue;  // long rows: spmm_chunks / spmm_long
      const auto in = row_fetch<VT, VW, MODE>(i, l.col, bs, Yold, inv_out, P, rb);
      VT acc[VW];
      row_product<VT, MT, VW, U, Lanes<W>::P>(op, Z, bs.B, a0 + l.arc, a1, l.col, acc);
      l.join(acc);
      if (l.arc == 0)
        row_update<VT, VW, MODE>(i, acc, l.col, bs, cs, in, Ynew, Znew, P, rb, red);
    }
  }
  cta_column_sums<W>(bs.B, part, smem_b);
}

// Partial products of the chunks of long rows: a warp per chunk, whose lanes
// share its arcs out by 32 / W.
template <class VT, class MT, int W, int VW, int U>
__global__ void __launch_bounds__(BT)
spmm_chunks(OpView<MT> op, const VT* __restrict__ Z, const Chunk* __restrict__ chunks,
            uint32_t nchunks, uint32_t B, VT* __restrict__ scratch,
            const int32_t* __restrict__ all_frozen) {
  if (*all_frozen) return;
  constexpr int P = 32 / W;
  const int lane = threadIdx.x & 31, col = lane % W, arc = lane / W;
  const uint32_t gw = blockIdx.x * BW + (threadIdx.x >> 5), nw = gridDim.x * BW;
  for (uint32_t q = gw; q < nchunks; q += nw) {
    const Chunk ch = chunks[q];
    VT acc[VW];
    row_product<VT, MT, VW, U, P>(op, Z, B, ch.a0 + arc, ch.a1, col, acc);
#pragma unroll
    for (int o = W; o < 32; o <<= 1)
#pragma unroll
      for (int v = 0; v < VW; ++v) acc[v] += __shfl_xor_sync(0xffffffffu, acc[v], o);
#pragma unroll
    for (int v = 0; v < VW; ++v) {
      const uint32_t c = col + 32 * v;
      if (arc == 0 && c < B) scratch[(size_t)q * B + c] = acc[v];
    }
  }
}

// Long rows: chunk partials added in chunk order, then the update.
template <class VT, int W, int VW, int MODE>
__global__ void __launch_bounds__(BT)
spmm_long(const uint32_t* __restrict__ lrow, const uint32_t* __restrict__ lfirst, uint32_t nlong,
          const VT* __restrict__ scratch, BatchScalars bs, const ColState* __restrict__ cs,
          const VT* __restrict__ Yold, VT* __restrict__ Ynew, VT* __restrict__ Znew,
          const VT* __restrict__ inv_out, PersView P, RefineBufs rb,
          double* __restrict__ part, const int32_t* __restrict__ all_frozen) {
  if (*all_frozen) return;
  extern __shared__ double smem_b[];
  const Lanes<W> l;
  double* red = group_sums<W>(smem_b, bs.B);
  const uint32_t gw = (blockIdx.x * BW + (threadIdx.x >> 5)) * Lanes<W>::G + l.group;
  const uint32_t nw = gridDim.x * BW * Lanes<W>::G;
  for (uint32_t q = gw; q < nlong; q += nw) {
    const auto in = row_fetch<VT, VW, MODE>(lrow[q], l.col, bs, Yold, inv_out, P, rb);
    VT acc[VW];
#pragma unroll
    for (int v = 0; v < VW; ++v) acc[v] = VT(0);
#pragma unroll 4
    for (uint32_t k = lfirst[q]; k < lfirst[q + 1]; ++k)
#pragma unroll
      for (int v = 0; v < VW; ++v) {
        const uint32_t c = l.col + 32 * v;
        if (c < bs.B) acc[v] += scratch[(size_t)k * bs.B + c];
      }
    if (l.arc == 0)
      row_update<VT, VW, MODE>(lrow[q], acc, l.col, bs, cs, in, Ynew, Znew, P, rb, red);
  }
  cta_column_sums<W>(bs.B, part, smem_b);
}

// tot[q] = sum over p of part[p][q], q < count: CTA j takes 32 values, its
// warps every 32nd partial in order, then the warps' sums in order. One CTA
// for all of them (a thread per column, 1,184 partials one after the other)
// took 0.9 ms a sweep, as long as half of the products (10 us since).
constexpr int SP_T = 1024;
__device__ __forceinline__ void sum_parts_tile(const double* __restrict__ part, uint32_t nparts,
                                               uint32_t count, double* __restrict__ tot) {
  __shared__ double sh[32][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t q = blockIdx.x * 32 + lane;
  double a = 0.0;
  if (q < count) {
#pragma unroll 4
    for (uint32_t p = w; p < nparts; p += 32) a += part[(size_t)p * count + q];
  }
  sh[w][lane] = a;
  __syncthreads();
  if (w == 0 && q < count) {
    double t = 0.0;
    for (int k = 0; k < 32; ++k) t += sh[k][lane];
    tot[q] = t;
  }
}

__global__ void __launch_bounds__(SP_T)
sum_parts(const double* __restrict__ part, uint32_t nparts, uint32_t count,
          double* __restrict__ tot) {
  sum_parts_tile(part, nparts, count, tot);
}

// The sweep's column sums, then (last CTA) per column the stopping rule and
// the scalars of the next sweep, and whether every column is frozen.
// flags: 0 all frozen, 1 ticket.
__global__ void __launch_bounds__(SP_T)
spmm_finish(const double* __restrict__ part, uint32_t nparts, BatchScalars bs, ColState* cs,
            double* __restrict__ tot, int32_t* flags, int32_t newbuf) {
  __shared__ int any_active;
  __shared__ bool last;
  if (flags[0]) return;
  sum_parts_tile(part, nparts, 3 * bs.B, tot);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    any_active = 0;
    last = atomicAdd((unsigned int*)flags + 1, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (uint32_t c = threadIdx.x; c < bs.B; c += blockDim.x) {
    ColState s = cs[c];
    if (!s.frozen) {
      const double T = __ldcg(tot + c), D = __ldcg(tot + bs.B + c), ch = __ldcg(tot + 2 * bs.B + c);
      s.prev_inv_total = s.inv_total;
      s.total = T;
      s.inv_total = 1.0 / T;
      s.dterm = D / T;
      s.change = ch;
      s.iter += 1;
      s.buf = newbuf;
      if (ch <= bs.tol) {
        s.converged = 1;
        s.frozen = 1;
      } else if (s.iter >= bs.max_iter) {
        s.frozen = 1;
      }
      cs[c] = s;
    }
    if (!s.frozen) atomicOr(&any_active, 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    flags[1] = 0;
    if (!any_active) flags[0] = 1;
  }
}

// Start: Y = 1/n, Z = Y / out.
template <class VT>
__global__ void spmm_init(VT* __restrict__ Y, VT* __restrict__ Zb, const VT* __restrict__ inv_out,
                          uint32_t n, uint32_t B) {
  const VT x0 = (VT)(1.0 / (double)n);
  const uint64_t total = (uint64_t)n * B;
  for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < total;
       q += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t i = (uint32_t)(q / B);
    Y[q] = x0;
    Zb[q] = x0 * inv_out[i];
  }
}

// Dangling count (same for every column at the start): D0 = n_dangling / n.
__global__ void spmm_set_state(ColState* cs, uint32_t B, double dterm0) {
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < B; c += gridDim.x * blockDim.x) {
    ColState s{};
    s.inv_total = 1.0;
    s.prev_inv_total = 1.0;
    s.dterm = dterm0;
    s.total = 1.0;
    cs[c] = s;
  }
}

// The columns sel[0, count) of a sweep's iterate (row length B), packed.
template <class VT>
__global__ void spmm_pack(const VT* __restrict__ Y, const VT* __restrict__ Z, uint32_t n,
                          uint32_t B, const uint32_t* __restrict__ sel, uint32_t count,
                          VT* __restrict__ Yp, VT* __restrict__ Zp) {
  const uint64_t total = (uint64_t)n * count;
  for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < total;
       q += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t i = (uint32_t)(q / count), c = sel[q % count];
    Yp[q] = Y[(size_t)i * B + c];
    Zp[q] = Z[(size_t)i * B + c];
  }
}

// FP32 -> FP64 hand-over of the columns sel[0, count) of a sweep that have
// stopped: Y64 = Y32 / T, read from the buffer the column stopped in; Z64 =
// Y64 / out, in the batch's own column order.
__global__ void spmm_switch(const float* __restrict__ Y0, const float* __restrict__ Y1,
                            const ColState* __restrict__ cs32, const uint32_t* __restrict__ sel,
                            uint32_t count, const uint32_t* __restrict__ cmap, uint32_t B,
                            uint32_t Bo, double* __restrict__ Y64, double* __restrict__ Z64,
                            const double* __restrict__ inv_out, uint32_t n) {
  const uint64_t total = (uint64_t)n * count;
  for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < total;
       q += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t i = (uint32_t)(q / count), c = sel[q % count];
    const float* Y = cs32[c].buf ? Y1 : Y0;
    const double y = (double)Y[(size_t)i * B + c] * cs32[c].inv_total;
    const size_t r = (size_t)i * Bo + cmap[c];
    Y64[r] = y;
    Z64[r] = y * inv_out[i];
  }
}

// Column sums (and dangling sums) of a node-major n x B matrix: CTA b adds
// rows b, b + G, ... per column (thread c owns column c), then one CTA adds
// the CTA partials in order and writes the column states.
__global__ void column_sums_part(const double* __restrict__ Y, const double* __restrict__ inv_out,
                                 uint32_t n, uint32_t B, double* __restrict__ part) {
  const uint32_t c = threadIdx.x;
  if (c >= B) return;
  double T = 0, D = 0;
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
    const double y = Y[(size_t)i * B + c];
    T += y;
    if (inv_out[i] == 0.0) D += y;
  }
  part[(size_t)blockIdx.x * 2 * B + c] = T;
  part[(size_t)blockIdx.x * 2 * B + B + c] = D;
}

__global__ void column_sums_finish(const double* __restrict__ tot, uint32_t B, ColState* cs) {
  const uint32_t c = threadIdx.x;
  if (c >= B) return;
  ColState s{};
  s.total = tot[c];
  s.inv_total = 1.0 / s.total;
  s.prev_inv_total = s.inv_total;
  s.dterm = tot[B + c] / s.total;
  cs[c] = s;
}

// Personalization: column-major input (p[c * n + i]) checked, and its sum per
// column in a fixed order: PERS_CTAS CTAs a column (one warp a column took
// 3.8 ms for 100 columns of 2^20 values, 0.13 ms since), then one warp.
constexpr uint32_t PERS_CTAS = 32;
__global__ void __launch_bounds__(BT)
pers_columns(const double* __restrict__ pin, uint32_t n, double* __restrict__ part,
             int32_t* __restrict__ bad) {
  __shared__ double sh[BT / 32];
  const uint32_t c = blockIdx.y;
  const double* p = pin + (size_t)c * n;
  double a = 0;
  int b = 0;
  for (uint32_t i = blockIdx.x * BT + threadIdx.x; i < n; i += PERS_CTAS * BT) {
    const double v = p[i];
    if (!isfinite(v) || v < 0.0) b = 1;
    else a += v;
  }
  a = block_sum(a, sh);
  if (__syncthreads_or(b) && threadIdx.x == 0) atomicOr(bad, 1);
  if (threadIdx.x == 0) part[c * PERS_CTAS + blockIdx.x] = a;
}

__global__ void pers_sums(const double* __restrict__ part, uint32_t B, double* __restrict__ sums,
                          int32_t* __restrict__ bad) {
  static_assert(PERS_CTAS == 32, "one lane per CTA's sum");
  const uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (c >= B) return;
  const double a = warp_sum(part[c * PERS_CTAS + lane]);
  if (lane == 0) {
    sums[c] = a;
    if (!(a > 0.0)) atomicOr(bad, 2);
  }
}

__global__ void pers_scatter(const double* __restrict__ pin, const double* __restrict__ sums,
                             uint32_t n, uint32_t B, double* __restrict__ pnm) {
  const uint64_t total = (uint64_t)n * B;
  for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < total;
       q += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t i = (uint32_t)(q / B), c = (uint32_t)(q % B);
    pnm[q] = pin[(size_t)c * n + i] / sums[c];
  }
}

// Nonzero teleport entries per node of a column group (column-major input).
__global__ void pers_row_counts(const double* __restrict__ pin, uint32_t n, uint32_t B,
                                uint32_t* __restrict__ cnt) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t k = 0;
    for (uint32_t c = 0; c < B; ++c) k += pin[(size_t)c * n + i] != 0.0 ? 1u : 0u;
    cnt[i] = k;
  }
}

// Each node's nonzero entries, normalised as pers_scatter does, in column order.
__global__ void pers_row_fill(const double* __restrict__ pin, const double* __restrict__ sums,
                              uint32_t n, uint32_t B, const uint32_t* __restrict__ rowptr,
                              uint32_t* __restrict__ cols, double* __restrict__ vals) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t e = rowptr[i];
    for (uint32_t c = 0; c < B; ++c) {
      const double v = pin[(size_t)c * n + i];
      if (v != 0.0) {
        cols[e] = c;
        vals[e] = v / sums[c];
        ++e;
      }
    }
  }
}

// Scores of the columns sel[0, count) of a sweep that have stopped, into
// column-major out (column cmap[c]): Y / T from the buffer the column stopped
// in, or with Yref (row length Bo) (y_ref + e) / T. A CTA transposes tiles of
// 32 rows by 32 columns through shared memory, so that both sides are read and
// written in runs (100 columns of 2^20: 4.1 ms without, 1.1 ms in the four
// calls of a solve).
template <class VT>
__global__ void __launch_bounds__(256)
spmm_output(const VT* __restrict__ Y0, const VT* __restrict__ Y1, const double* __restrict__ Yref,
            const ColState* __restrict__ cs, const uint32_t* __restrict__ sel, uint32_t count,
            const uint32_t* __restrict__ cmap, uint32_t B, uint32_t Bo, uint32_t n,
            double* __restrict__ out) {
  __shared__ double tile[32][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const uint32_t k0 = blockIdx.y * 32;
  const bool live = k0 + x < count;
  const uint32_t c = live ? sel[k0 + x] : 0u, co = live ? cmap[c] : 0u;
  const VT* Y = live && cs[c].buf ? Y1 : Y0;
  const double total = live ? cs[c].total : 1.0;
  const uint32_t nt = (n + 31) / 32;
  for (uint32_t t = blockIdx.x; t < nt; t += gridDim.x) {
    for (int r = y; r < 32; r += 8) {
      const uint32_t i = t * 32 + r;
      if (!live || i >= n) continue;
      double v = (double)Y[(size_t)i * B + c];
      if (Yref) v = Yref[(size_t)i * Bo + co] + v;
      tile[r][x] = v / total;
    }
    __syncthreads();
    for (int k = y; k < 32; k += 8) {
      const uint32_t i = t * 32 + x;
      if (k0 + k < count && i < n) out[(size_t)cmap[sel[k0 + k]] * n + i] = tile[x][k];
    }
    __syncthreads();
  }
}

// ----------------------------------------------------------------------- host
struct BatchPlan {
  std::vector<RowRange> ranges;
  std::vector<Chunk> chunks;
  std::vector<uint32_t> lrow, lfirst;
};

static BatchPlan make_plan(const std::vector<uint32_t>& off, uint32_t n) {
  BatchPlan p;
  uint32_t lo = 0;
  uint64_t acc = 0;
  for (uint32_t i = 0; i < n; ++i) {
    uint32_t deg = off[i + 1] - off[i];
    if (deg > LONG_ROW) {
      p.lrow.push_back(i);
      p.lfirst.push_back((uint32_t)p.chunks.size());
      for (uint32_t a = off[i]; a < off[i + 1]; a += LONG_ROW)
        p.chunks.push_back({i, a, std::min(off[i + 1], a + LONG_ROW)});
    } else {
      acc += deg + ROW_COST;
    }
    if (acc >= RANGE_ARCS) {
      p.ranges.push_back({lo, i + 1});
      lo = i + 1;
      acc = 0;
    }
  }
  if (lo < n) p.ranges.push_back({lo, n});
  p.lfirst.push_back((uint32_t)p.chunks.size());
  return p;
}

template <class T>
static void upload(DevBuf<T>& d, const std::vector<T>& h, cudaStream_t s) {
  d.alloc(std::max<size_t>(h.size(), 1));
  if (!h.empty()) KNB_CUDA(cudaMemcpyAsync(d.get(), h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, s));
}

// What the sweeps of one operator share: its row plan, and the scratch.
struct SweepPlan {
  const RowRange* ranges;
  const Chunk* chunks;
  const uint32_t *lrow, *lfirst;
  uint32_t nranges, nchunks, nlong;
  double* part;
  double* tot;
  int32_t* flags;  // all frozen, ticket
};

// CTAs of a sweep kernel that fit on the GPU at once, at most MAX_CTAS.
constexpr unsigned MAX_CTAS = 148 * 8;
static unsigned resident_ctas(const void* fn, size_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<int, const void*, size_t>, unsigned> known;
  int dev = 0;
  KNB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  unsigned& g = known[{dev, fn, smem}];
  if (!g) {
    int per_sm = 0, sms = 0;
    KNB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, BT, smem));
    KNB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    g = std::min(MAX_CTAS, (unsigned)std::max(1, per_sm) * (unsigned)sms);
  }
  return g;
}

// One sweep from buffers (Yold, Zold) to (Ynew, Znew) = buffer newbuf: the
// row products and updates, then (finish) the per-column sums, stopping rule
// and next sweep's scalars. Without finish the sweep only rewrites Ynew, Znew,
// the chunk scratch and the partials.
template <class VT, class MT, int W, int VW, int U, int MODE>
static int batch_sweep(const OpView<MT>& op, const SweepPlan& sp, const BatchScalars& bs,
                       ColState* cs, const VT* Yold, VT* Ynew, const VT* Zold, VT* Znew,
                       const VT* inv_out, const PersView& P, const RefineBufs& rb, VT* scratch,
                       int newbuf, bool finish, cudaStream_t s) {
  const size_t smem = (size_t)BW * Lanes<W>::G * 3 * bs.B * sizeof(double);
  if (W == 32) {
    set_func_attr((const void*)spmm_rows<VT, MT, W, VW, U, MODE>,
                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                  (int)(BW * 3 * 256 * sizeof(double)));
    set_func_attr((const void*)spmm_long<VT, W, VW, MODE>,
                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                  (int)(BW * 3 * 256 * sizeof(double)));
  }
  // the CTAs that fit at once, at most what the partials hold
  const unsigned grid = resident_ctas((const void*)spmm_rows<VT, MT, W, VW, U, MODE>, smem);
  int launches = 1;
  if (sp.nchunks) {
    spmm_chunks<VT, MT, W, VW, U><<<148 * 8, BT, 0, s>>>(op, Zold, sp.chunks, sp.nchunks, bs.B,
                                                       scratch, sp.flags);
    ++launches;
  }
  spmm_rows<VT, MT, W, VW, U, MODE><<<grid, BT, smem, s>>>(op, Zold, sp.ranges, sp.nranges, bs,
                                                           cs, Yold, Ynew, Znew, inv_out, P, rb,
                                                           sp.part, sp.flags);
  unsigned parts = grid;
  if (sp.nlong) {
    const unsigned gl = std::min(grid, (sp.nlong + BW - 1) / BW);
    spmm_long<VT, W, VW, MODE><<<gl, BT, smem, s>>>(sp.lrow, sp.lfirst, sp.nlong, scratch, bs, cs,
                                                    Yold, Ynew, Znew, inv_out, P, rb,
                                                    sp.part + (size_t)grid * 3 * bs.B, sp.flags);
    parts += gl;
    ++launches;
  }
  if (finish) {
    spmm_finish<<<(3 * bs.B + 31) / 32, SP_T, 0, s>>>(sp.part, parts, bs, cs, sp.tot, sp.flags,
                                                      newbuf);
    ++launches;
  }
  KNB_LAUNCH("batch sweep");
  return launches;
}

// u: arcs in flight per lane of a whole-warp row (1, 2 or 4; lanes of narrow
// rows, which hold one column, keep 4).
template <class VT, class MT, int MODE = EPI_PLAIN>
static int batch_sweep_vw(int u, const OpView<MT>& op, const SweepPlan& sp, const BatchScalars& bs,
                          ColState* cs, const VT* Yold, VT* Ynew, const VT* Zold, VT* Znew,
                          const VT* inv_out, const PersView& P, const RefineBufs& rb, VT* scratch,
                          int newbuf, cudaStream_t s, bool finish = true) {
#define KNB_SW(WW, V, UU)                                                                          \
  return batch_sweep<VT, MT, WW, V, UU, MODE>(op, sp, bs, cs, Yold, Ynew, Zold, Znew, inv_out, P,  \
                                              rb, scratch, newbuf, finish, s)
#define KNB_SWU(V)                       \
  switch (u) {                           \
    case 1: KNB_SW(32, V, 1);            \
    case 2: KNB_SW(32, V, 2);            \
    default: KNB_SW(32, V, 4);           \
  }
  if (bs.B <= 1) KNB_SW(1, 1, 4);
  if (bs.B <= 2) KNB_SW(2, 1, 4);
  if (bs.B <= 4) KNB_SW(4, 1, 4);
  if (bs.B <= 8) KNB_SW(8, 1, 4);
  if (bs.B <= 16) KNB_SW(16, 1, 4);
  if (bs.B <= 32) KNB_SWU(1);
  if (bs.B <= 64) KNB_SWU(2);
  if (bs.B <= 128) KNB_SWU(4);
  KNB_SWU(8);
#undef KNB_SWU
#undef KNB_SW
}

// Times one sweep of each arcs-in-flight candidate on the phase's starting
// state (without the finish, so nothing but buffers the first real sweep
// rewrites is touched) and returns the fastest.
template <class VT, class MT>
static int tune_arcs_in_flight(const OpView<MT>& op, const SweepPlan& sp, const BatchScalars& bs,
                               ColState* cs, const VT* Yold, VT* Ynew, const VT* Zold, VT* Znew,
                               const VT* inv_out, const PersView& P, VT* scratch, cudaStream_t s) {
  cudaEvent_t e0, e1;
  KNB_CUDA(cudaEventCreate(&e0));
  KNB_CUDA(cudaEventCreate(&e1));
  int best = U_CANDIDATES[0];
  float best_ms = 0;
  for (int u : U_CANDIDATES) {
    KNB_CUDA(cudaEventRecord(e0, s));
    batch_sweep_vw<VT, MT>(u, op, sp, bs, cs, Yold, Ynew, Zold, Znew, inv_out, P, RefineBufs{},
                           scratch, 1, s, false);
    KNB_CUDA(cudaEventRecord(e1, s));
    KNB_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    KNB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    if (u == U_CANDIDATES[0] || ms < best_ms) {
      best = u;
      best_ms = ms;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return best;
}

static int vw_for(uint32_t B) {
  if (B <= 32) return 1;
  if (B <= 64) return 2;
  if (B <= 128) return 4;
  return 8;
}

// What batched solves on one operator keep between calls: the row ranges
// and chunks, and every buffer (grown when a call needs more, never shrunk;
// freeing the tens of GB a large batch holds costs as much as a quarter of a
// solve). A solve holds `mu` while it runs, so concurrent calls on one
// operator take turns.
struct BatchWorkspace : Workspace {
  std::mutex mu;
  bool planned = false;
  uint32_t nranges = 0, nchunks = 0, nlong = 0;
  DevBuf<RowRange> d_ranges;
  DevBuf<Chunk> d_chunks;
  DevBuf<uint32_t> d_lrow, d_lfirst, prow, pcols;
  DevBuf<double> pin, dout, Pd, sums, pvals, part, Y64[2], Z64[2], sc64;
  DevBuf<float> Y32[2], Z32[2], sc32;
  DevBuf<ColState> cs;
  DevBuf<int32_t> flags, all_frozen;
  DevBuf<double> tot, pparts;
  DevBuf<uint32_t> maps;  // cmap, inv and the columns selected, 256 each
};

template <class T>
static void grow(DevBuf<T>& b, size_t count) {
  if (b.n < count) b.alloc(count);
}

void pagerank_batch(GraphHandleImpl& g, const BatchParams& prm, const double* pers_colmajor,
                    double* out_colmajor, BatchInfo* info, cudaStream_t s) {
  const uint32_t n = g.n;
  if (n == 0 || prm.B == 0) return;
  const int which = (g.directed && prm.directed) ? 1 : (g.directed ? 2 : 0);
  const double lfac = prm.loops == 2 ? 0.0 : (which == 1 ? 1.0 : (prm.loops == 0 ? 2.0 : 1.0));
  Operator& op = g.op(which, prm.weighted, lfac, s);
  // arcs in flight per (column width, value types), tuned on first use
  auto tuned_u = [&](int key) {
    std::lock_guard<std::mutex> lock(op.mu);
    auto it = op.batch_u.find(key);
    return it == op.batch_u.end() ? 0 : it->second;
  };
  auto keep_u = [&](int key, int u) {
    std::lock_guard<std::mutex> lock(op.mu);
    op.batch_u[key] = u;
  };
  BatchWorkspace* wsp = nullptr;
  {
    std::lock_guard<std::mutex> lock(op.mu);
    if (!op.batch_ws) op.batch_ws = std::make_unique<BatchWorkspace>();
    wsp = static_cast<BatchWorkspace*>(op.batch_ws.get());
  }
  BatchWorkspace& ws = *wsp;
  std::lock_guard<std::mutex> ws_lock(ws.mu);
  if (!ws.planned) {
    std::vector<uint32_t> hoff(n + 1);
    KNB_CUDA(cudaMemcpyAsync(hoff.data(), op.rows->off.get(), ((size_t)n + 1) * 4,
                             cudaMemcpyDeviceToHost, s));
    KNB_CUDA(cudaStreamSynchronize(s));
    BatchPlan plan = make_plan(hoff, n);
    upload(ws.d_ranges, plan.ranges, s);
    upload(ws.d_chunks, plan.chunks, s);
    upload(ws.d_lrow, plan.lrow, s);
    upload(ws.d_lfirst, plan.lfirst, s);
    ws.nranges = (uint32_t)plan.ranges.size();
    ws.nchunks = (uint32_t)plan.chunks.size();
    ws.nlong = (uint32_t)plan.lrow.size();
    KNB_CUDA(cudaStreamSynchronize(s));
    ws.planned = true;
  }
  const uint32_t nchunks = ws.nchunks;

  cudaEvent_t t0, t1, l0, l1;
  KNB_CUDA(cudaEventCreate(&t0));
  KNB_CUDA(cudaEventCreate(&t1));
  KNB_CUDA(cudaEventCreate(&l0));
  KNB_CUDA(cudaEventCreate(&l1));
  KNB_CUDA(cudaEventRecord(t0, s));
  double sweep_ms = 0.0;  // device time of the sweep loops alone
  auto loop_end = [&] {
    KNB_CUDA(cudaEventRecord(l1, s));
    KNB_CUDA(cudaEventSynchronize(l1));
    float lm = 0;
    KNB_CUDA(cudaEventElapsedTime(&lm, l0, l1));
    sweep_ms += lm;
  };
  int launches = 0;
  int64_t sweeps32 = 0, sweeps64 = 0, colits32 = 0;
  const bool mixed = prm.precision == PREC_MIXED;
  // mixed: the FP64 phase as one anchor sweep and refinement sweeps (tuning
  // key 9 at 0: plain FP64 sweeps)
  const bool refine = mixed && tuning().refine != 0;
  const uint32_t Btot = prm.B;
  DevBuf<double>& pin = ws.pin;
  grow(pin, (size_t)n * Btot);
  KNB_CUDA(cudaMemcpyAsync(pin.get(), pers_colmajor, (size_t)n * Btot * 8,
                           prm.on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, s));
  double* outp = out_colmajor;
  if (!prm.on_device) {
    grow(ws.dout, (size_t)n * Btot);
    outp = ws.dout.get();
  }
  std::vector<int32_t> col_iters(Btot, 0);
  // column groups of at most 256
  for (uint32_t c0 = 0; c0 < Btot; c0 += 256) {
    const uint32_t B = std::min<uint32_t>(256, Btot - c0);
    const int vw = vw_for(B);
    DevBuf<double>& Pd = ws.Pd;
    DevBuf<double>& sums = ws.sums;
    DevBuf<double>& pvals = ws.pvals;
    DevBuf<uint32_t>& prow = ws.prow;
    DevBuf<uint32_t>& pcols = ws.pcols;
    DevBuf<int32_t>& flags = ws.flags;
    grow(sums, B);
    grow(prow, (size_t)n + 1);
    grow(flags, 2);
    KNB_CUDA(cudaMemsetAsync(flags.get(), 0, 8, s));
    grow(ws.pparts, (size_t)PERS_CTAS * 256);
    pers_columns<<<dim3(PERS_CTAS, B), BT, 0, s>>>(pin.get() + (size_t)c0 * n, n, ws.pparts.get(),
                                                   flags.get());
    pers_sums<<<(B + BW - 1) / BW, BT, 0, s>>>(ws.pparts.get(), B, sums.get(), flags.get());
    int32_t hf[2];
    KNB_CUDA(cudaMemcpyAsync(hf, flags.get(), 8, cudaMemcpyDeviceToHost, s));
    KNB_CUDA(cudaStreamSynchronize(s));
    if (hf[0] & 1) throw Error("the personalization vector must hold finite, nonnegative values");
    if (hf[0] & 2) throw Error("the personalization vector must have a positive sum");
    // Teleport columns: the nonzero entries per node when at most 1/16 of
    // them are nonzero (seed-set personalisation), else dense; a sweep then
    // reads only the rows that hold seeds.
    KNB_CUDA(cudaMemsetAsync(prow.get(), 0, ((size_t)n + 1) * 4, s));
    pers_row_counts<<<grid_for(n, 256), 256, 0, s>>>(pin.get() + (size_t)c0 * n, n, B, prow.get());
    const uint32_t pnnz = exclusive_scan<uint32_t>(prow.get(), prow.get(), (size_t)n + 1, s);
    PersView P{nullptr, nullptr, nullptr, nullptr};
    if ((uint64_t)pnnz * 16 <= (uint64_t)n * B) {
      grow(pcols, std::max<uint32_t>(pnnz, 1));
      grow(pvals, std::max<uint32_t>(pnnz, 1));
      pers_row_fill<<<grid_for(n, 256), 256, 0, s>>>(pin.get() + (size_t)c0 * n, sums.get(), n, B,
                                                     prow.get(), pcols.get(), pvals.get());
      P = PersView{nullptr, prow.get(), pcols.get(), pvals.get()};
    } else {
      grow(Pd, (size_t)n * B);
      pers_scatter<<<grid_for((uint64_t)n * B, 256), 256, 0, s>>>(pin.get() + (size_t)c0 * n,
                                                                   sums.get(), n, B, Pd.get());
      P = PersView{Pd.get(), nullptr, nullptr, nullptr};
    }
    KNB_LAUNCH("teleport columns");
    launches += 4;
    grow(ws.cs, 256);
    grow(ws.all_frozen, 2);
    grow(ws.maps, 3 * 256);
    grow(ws.tot, 3 * 256);
    grow(ws.part, (size_t)2 * MAX_CTAS * 3 * std::max<uint32_t>(B, 16));  // rows, long rows
    uint32_t* const cmap = ws.maps.get();
    uint32_t* const inv = cmap + 256;
    uint32_t* const sel = inv + 256;
    ColState* const cs = ws.cs.get();
    double* const part = ws.part.get();
    const SweepPlan sp{ws.d_ranges.get(), ws.d_chunks.get(), ws.d_lrow.get(), ws.d_lfirst.get(),
                       ws.nranges, ws.nchunks, ws.nlong, part, ws.tot.get(), ws.all_frozen.get()};
    BatchScalars bs{prm.damping, 1.0 / n, n, B, B, prm.dangling == 1 ? 1 : 0, 0.0,
                    (int32_t)std::min<int64_t>(prm.max_iter, INT32_MAX), cmap, inv};
    const double dterm0 = (double)op.n_dangling / (double)n;
    const size_t nb = (size_t)n * B;
    float* Y32[2] = {nullptr, nullptr};
    float* Z32[2] = {nullptr, nullptr};
    double* Y64[2];
    double* Z64[2];
    for (int k = 0; k < 2; ++k) {
      if (mixed) {
        grow(ws.Y32[k], nb);
        grow(ws.Z32[k], nb);
        Y32[k] = ws.Y32[k].get();
        Z32[k] = ws.Z32[k].get();
      }
      grow(ws.Y64[k], nb);
      grow(ws.Z64[k], nb);
      Y64[k] = ws.Y64[k].get();
      Z64[k] = ws.Z64[k].get();
    }
    grow(ws.sc64, std::max<size_t>((size_t)nchunks * B, 1));
    if (mixed) grow(ws.sc32, std::max<size_t>((size_t)nchunks * B, 1));
    float* const sc32 = ws.sc32.get();
    double* const sc64 = ws.sc64.get();

    // The sweep's columns, by their number in the batch; all of them at the
    // start of a phase.
    std::vector<uint32_t> cols;
    auto set_columns = [&](std::vector<uint32_t> c) {
      cols = std::move(c);
      std::vector<uint32_t> m(512, NO_COL);
      for (uint32_t k = 0; k < cols.size(); ++k) {
        m[k] = cols[k];
        m[256 + cols[k]] = k;
      }
      KNB_CUDA(cudaMemcpyAsync(cmap, m.data(), m.size() * 4, cudaMemcpyHostToDevice, s));
      bs.B = (uint32_t)cols.size();
    };
    auto all_columns = [&] {
      std::vector<uint32_t> c(B);
      for (uint32_t k = 0; k < B; ++k) c[k] = k;
      set_columns(std::move(c));
    };
    auto select = [&](const std::vector<uint32_t>& k) {
      KNB_CUDA(cudaMemcpyAsync(sel, k.data(), k.size() * 4, cudaMemcpyHostToDevice, s));
      return (uint32_t)k.size();
    };
    // Runs sweeps (from, to = buffer indices) until every column has stopped.
    // Every 4 sweeps the host looks at the columns' states; once a quarter of
    // the width has stopped, the stopped columns leave (leave(count): sel's
    // columns, in their last buffers) and the others are packed, which costs
    // about as much as half a sweep. Returns the sweeps run.
    auto run = [&](int cur, int64_t k, auto sweep, auto leave, auto Y, auto Z) -> int64_t {
      std::vector<ColState> h;
      for (;;) {
        sweep(cur, 1 - cur);
        cur = 1 - cur;
        ++k;
        if (k % 4 != 0) continue;
        h.resize(bs.B);
        KNB_CUDA(cudaMemcpyAsync(h.data(), cs, bs.B * sizeof(ColState), cudaMemcpyDeviceToHost, s));
        KNB_CUDA(cudaStreamSynchronize(s));
        std::vector<uint32_t> gone, left, names;
        for (uint32_t c = 0; c < bs.B; ++c) (h[c].frozen ? gone : left).push_back(c);
        if (!left.empty() && left.size() * 4 > (size_t)bs.B * 3) continue;
        for (uint32_t c : gone) {
          if (!h[c].converged)
            throw Error("PageRank did not converge to tolerance " + std::to_string(prm.tol) +
                        " within " + std::to_string(prm.max_iter) + " iterations");
          col_iters[c0 + cols[c]] += h[c].iter;
        }
        if (!gone.empty()) launches += leave(select(gone));
        if (left.empty()) return k;
        const uint32_t count = select(left);
        spmm_pack<<<grid_for((uint64_t)n * count, 256), 256, 0, s>>>(
            Y[cur], Z[cur], n, bs.B, sel, count, Y[1 - cur], Z[1 - cur]);
        KNB_LAUNCH("spmm_pack");
        ++launches;
        cur = 1 - cur;
        std::vector<ColState> hs;
        for (uint32_t c : left) {
          names.push_back(cols[c]);
          hs.push_back(h[c]);
        }
        set_columns(std::move(names));
        KNB_CUDA(cudaMemcpyAsync(cs, hs.data(), hs.size() * sizeof(ColState),
                                 cudaMemcpyHostToDevice, s));
      }
    };
    all_columns();
    KNB_CUDA(cudaMemsetAsync(ws.all_frozen.get(), 0, 8, s));
    int u32 = 4;
    if (mixed) {
      spmm_init<float><<<grid_for(nb, 256), 256, 0, s>>>(Y32[0], Z32[0], op.inv_out32.get(), n, B);
      spmm_set_state<<<1, 256, 0, s>>>(cs, B, dterm0);
      bs.tol = std::max(prm.tol * prm.switch_factor, prm.switch_floor);
      launches += 2;
      if (B > 16 && !(u32 = tuned_u(vw * 4 + 0))) {
        u32 = tune_arcs_in_flight<float, float>(op.view32(), sp, bs, cs, Y32[0], Y32[1], Z32[0],
                                                Z32[1], op.inv_out32.get(), P, sc32, s);
        keep_u(vw * 4 + 0, u32);
      }
      KNB_CUDA(cudaEventRecord(l0, s));
      sweeps32 += run(
          0, 0,
          [&](int a, int b) {
            launches += batch_sweep_vw<float, float>(u32, op.view32(), sp, bs, cs, Y32[a], Y32[b],
                                                     Z32[a], Z32[b], op.inv_out32.get(), P,
                                                     RefineBufs{}, sc32, b, s);
          },
          [&](uint32_t count) {
            spmm_switch<<<grid_for((uint64_t)n * count, 256), 256, 0, s>>>(
                Y32[0], Y32[1], cs, sel, count, cmap, bs.B, B, Y64[0], Z64[0],
                op.inv_out64.get(), n);
            KNB_LAUNCH("batch hand-over");
            return 1;
          },
          Y32, Z32);
      loop_end();
      for (uint32_t c = 0; c < B; ++c) colits32 += col_iters[c0 + c];
      all_columns();
      column_sums_part<<<1184, 256, 0, s>>>(Y64[0], op.inv_out64.get(), n, B, part);
      sum_parts<<<(2 * B + 31) / 32, SP_T, 0, s>>>(part, 1184, 2 * B, ws.tot.get());
      column_sums_finish<<<1, 256, 0, s>>>(ws.tot.get(), B, cs);
      KNB_LAUNCH("batch hand-over");
      launches += 3;
    } else {
      spmm_init<double><<<grid_for(nb, 256), 256, 0, s>>>(Y64[0], Z64[0], op.inv_out64.get(), n,
                                                           B);
      spmm_set_state<<<1, 256, 0, s>>>(cs, B, dterm0);
      launches += 2;
    }
    // FP64 phase
    KNB_CUDA(cudaMemsetAsync(ws.all_frozen.get(), 0, 8, s));
    bs.tol = prm.tol;
    const bool use32v = op.has_vals && op.vals32_exact;
    const int key64 = vw * 4 + (use32v ? 1 : 2);
    int u64 = 4;
    if (B > 16 && !(u64 = tuned_u(key64))) {
      u64 = use32v ? tune_arcs_in_flight<double, float>(op.view32(), sp, bs, cs, Y64[0], Y64[1],
                                                        Z64[0], Z64[1], op.inv_out64.get(), P,
                                                        sc64, s)
                   : tune_arcs_in_flight<double, double>(op.view64(), sp, bs, cs, Y64[0], Y64[1],
                                                         Z64[0], Z64[1], op.inv_out64.get(), P,
                                                         sc64, s);
      keep_u(key64, u64);
    }
    auto out_grid = [&](uint32_t count) {
      return dim3(std::min<uint32_t>((n + 31) / 32, 148 * 16), (count + 31) / 32);
    };
    double* const outc = outp + (size_t)c0 * n;
    KNB_CUDA(cudaEventRecord(l0, s));
    if (refine) {
      // the anchor sweep: FP64 gathers of z_ref = Y64[0] / out; s_ref into
      // Y64[1], the correction e and z_e into Y32[1] and Z32[1]
      const RefineBufs rb0{Y64[0], Y64[1], nullptr, Y32[1], Z32[1], op.inv_out32.get()};
      if (use32v)
        launches += batch_sweep_vw<double, float, EPI_ANCHOR>(
            u64, op.view32(), sp, bs, cs, Y64[0], Y64[1], Z64[0], Z64[1], op.inv_out64.get(), P,
            rb0, sc64, 1, s);
      else
        launches += batch_sweep_vw<double, double, EPI_ANCHOR>(
            u64, op.view64(), sp, bs, cs, Y64[0], Y64[1], Z64[0], Z64[1], op.inv_out64.get(), P,
            rb0, sc64, 1, s);
      // refinement sweeps: FP32 gathers of z_e, FP32 arc values (the FP32
      // phase's arcs in flight)
      sweeps64 += run(
          1, 1,
          [&](int a, int b) {
            const RefineBufs rb{Y64[0], Y64[1], Y32[a], Y32[b], Z32[b], op.inv_out32.get()};
            launches += batch_sweep_vw<float, float, EPI_REFINE>(
                u32, op.view32(), sp, bs, cs, Y32[a], Y32[b], Z32[a], Z32[b], op.inv_out32.get(),
                P, rb, sc32, b, s);
          },
          [&](uint32_t count) {
            spmm_output<float><<<out_grid(count), 256, 0, s>>>(Y32[0], Y32[1], Y64[0], cs, sel,
                                                               count, cmap, bs.B, B, n, outc);
            KNB_LAUNCH("spmm_output");
            return 1;
          },
          Y32, Z32);
    } else {
      sweeps64 += run(
          0, 0,
          [&](int a, int b) {
            if (use32v)
              launches += batch_sweep_vw<double, float>(u64, op.view32(), sp, bs, cs, Y64[a],
                                                        Y64[b], Z64[a], Z64[b],
                                                        op.inv_out64.get(), P, RefineBufs{}, sc64,
                                                        b, s);
            else
              launches += batch_sweep_vw<double, double>(u64, op.view64(), sp, bs, cs, Y64[a],
                                                         Y64[b], Z64[a], Z64[b],
                                                         op.inv_out64.get(), P, RefineBufs{},
                                                         sc64, b, s);
          },
          [&](uint32_t count) {
            spmm_output<double><<<out_grid(count), 256, 0, s>>>(Y64[0], Y64[1], nullptr, cs, sel,
                                                                count, cmap, bs.B, B, n, outc);
            KNB_LAUNCH("spmm_output");
            return 1;
          },
          Y64, Z64);
    }
    loop_end();
  }
  if (!prm.on_device)
    KNB_CUDA(cudaMemcpyAsync(out_colmajor, outp, (size_t)n * Btot * 8, cudaMemcpyDeviceToHost, s));
  KNB_CUDA(cudaEventRecord(t1, s));
  KNB_CUDA(cudaStreamSynchronize(s));
  float ms = 0;
  KNB_CUDA(cudaEventElapsedTime(&ms, t0, t1));
  cudaEventDestroy(t0);
  cudaEventDestroy(t1);
  cudaEventDestroy(l0);
  cudaEventDestroy(l1);
  if (info) {
    info->seconds = ms * 1e-3;
    info->sweep_seconds = sweep_ms * 1e-3;
    info->sweeps = sweeps32 + sweeps64;
    info->sweeps_fp32 = sweeps32;
    int64_t tot = 0, mx = 0;
    for (uint32_t c = 0; c < Btot; ++c) {
      tot += col_iters[c];
      mx = std::max<int64_t>(mx, col_iters[c]);
    }
    info->column_iterations = tot;
    info->column_iterations_fp32 = colits32;
    info->max_column_iterations = mx;
    info->refined = refine ? 1 : 0;
    info->kernel_launches = launches;
  }
}

}  // namespace knb
