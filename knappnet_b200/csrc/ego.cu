// Many small graphs at once: PageRank on every block of a block-diagonal
// graph (ego networks, layers, subgraphs packed into one handle), in one
// persistent launch.
//
// Graphs are taken off queues largest first (so the last graphs to start are
// the small ones) and each runs the reference's iteration on its own
// (crates/engine/src/metrics/spectral.rs:247-280), every sum in a fixed order.
// Scores are those of a separate net_pagerank call on the graph up to rounding
// (sums are associated in another way and the division by the total comes a
// sweep later), and the sweep a graph stops on is that of the iteration which
// divides by the total in every sweep (ego_normalising): it decides where
// rounding could. A large graph would keep one CTA busy long after the rest of
// the batch is done, so the launch runs in thread-block clusters: each cluster
// first splits the large graphs over its CTAs, then every CTA takes small
// graphs alone. A single small graph's solve runs here too, as a batch of one.
//
// What bounds an iteration of a graph this small is latency: the chain from a
// row's offsets over its columns to the gathered values, the sums, and the
// barriers. So a graph is brought into shared memory once (16-bit columns,
// values, out-strengths, and z = x / out in two buffers of which an iteration
// reads one and writes the other), and an iteration has one reduction and one
// barrier: the division by the total is left to the next iteration's scalars,
// as in the sweeps (pagerank.cu). CTAs of a cluster each keep all of z and write
// every value they compute into all of the copies. Graphs whose arcs do not
// fit keep those in global memory, graphs whose vectors do not fit keep
// everything there.
// With the graph in global memory and two reductions an iteration of a graph
// of 500 nodes took 8.0 us, now 1.8 us; 10,000 nodes and 100,000 arcs, on a
// cluster of 8 then, of 16 and still in global memory now, 13.6 us and 6.5 us;
// R-MAT graphs of 30,000 nodes, whose hub rows each waited for one thread, 235 us
// and 25 us.
#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <numeric>
#include <tuple>
#include <type_traits>
#include <vector>

#include <cooperative_groups.h>

#include "ego.cuh"

namespace cg = cooperative_groups;

namespace knb {

struct EgoParams {
  double d;
  double tol;
  int32_t max_iter;
  int32_t jump_uniform;  // dangling nodes jump uniformly (1) or by p (0)
};

// How the normalising iteration associates its sums, whatever the launch's
// shape: `threads` partial sums (of every threads-th row) joined warp by warp,
// for a graph of at least `split` nodes over each of EGO_SHARES equal shares of
// its rows.
constexpr int EGO_SHARES = 8;
struct EgoOrder {
  uint32_t threads;
  uint32_t split;
};

// Fixed-order sums of three values over the threads of a graph's CTAs: warp
// butterflies, the warps of each CTA, and with C > 1 the CTAs of the cluster
// in rank order, each CTA writing its sums into all CTAs' slots, so that all
// hold the same bits. The barrier in it (the CTA's, or the cluster's) also
// publishes everything written before it. sh (2 x 3 x 32 doubles) and slots
// (2 x C x 4) are taken by turns: whoever writes one again has passed the
// next barrier, so everybody has read it.
template <int C>
__device__ __forceinline__ void ego_sums(double (&v)[3], double* sh, double* slots, int turn) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double* s = sh + (turn & 1) * 96;
  const double m = warp_sum_scatter<3>(v, lane);
  if ((lane & 7) == 0 && lane < 24) s[(lane >> 3) * 32 + w] = m;
  __syncthreads();
  if (C == 1 || w == 0) {
    double a[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) a[k] = lane < nw ? s[k * 32 + lane] : 0.0;
    const double t = warp_sum_scatter<3>(a, lane);
    if constexpr (C == 1) {
#pragma unroll
      for (int k = 0; k < 3; ++k) v[k] = __shfl_sync(0xffffffffu, t, 8 * k);
    } else {
      cg::cluster_group cl = cg::this_cluster();
      const int k = lane >> 3;
      if (k < 3)
        for (int r = lane & 7; r < C; r += 8)
          cl.map_shared_rank(slots, (unsigned)r)[((turn & 1) * C + cl.block_rank()) * 4 + k] = t;
    }
  }
  if constexpr (C > 1) {
    cg::this_cluster().sync();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      double t = 0;
#pragma unroll
      for (int r = 0; r < C; ++r) t += slots[((turn & 1) * C + r) * 4 + k];
      v[k] = t;
    }
  }
}

// A graph and this CTA's rows of it.
struct EgoGraph {
  OpView<double> op;
  const float* vals32;   // the values in FP32 where all are exact there, else null
  const double* inv_out; // 1 / out-strength, 0 for dangling nodes
  const double* outstr;  // out-strength
  uint32_t g_lo, nk;     // its nodes [g_lo, g_lo + nk)
  uint32_t lo, hi;       // this CTA's rows
  uint32_t rmax;         // most rows of any CTA of the cluster
  const double* pers;    // null: uniform
  double ps;             // sum of the graph's pers
  double *y, *z;         // global iterates, each in two buffers n apart
  uint32_t n;
  double* out;
};

// Rows of more arcs than this are summed by a whole warp, before the others
// and spread over the warps (the hubs of a skewed graph tend to be neighbours).
constexpr uint32_t EGO_LONG = 32;

// How a graph's solve ended: at the iteration cap, at the tolerance, or open.
enum { EGO_CAPPED = 0, EGO_DONE = 1, EGO_OPEN = 2 };

// Where a graph lives: everything in shared memory, all but its arcs, nothing.
enum { EGO_SMEM = 1, EGO_ARCS_GLOBAL = 2, EGO_GLOBAL = 3 };

__host__ __device__ constexpr size_t ego_vector_bytes(size_t nk, size_t rows, bool pers) {
  return 16 * nk + rows * (16 + 8 + (pers ? 8 : 0)) + 4 * ((rows + 2) & ~size_t(1));
}
__host__ __device__ constexpr size_t ego_arc_bytes(size_t arcs, size_t value_bytes) {
  return ((arcs * value_bytes + 7) & ~size_t(7)) + arcs * 2;
}

// How far rounding may part the L1 change of this iteration from that of the
// normalising one: a row of m arcs is off by about sqrt(m) units of its value,
// `rows` = sum x sqrt(m) over the rows. Measured between the two iterations at
// the same sweep, 16,000 solves of 20 to 20,000 nodes, with and without hub rows
// and weights: mean 5e-17, at most 7.6e-16; a graph of 12 arcs a node gets
// 2e-15 here.
__device__ __forceinline__ double ego_rounding(double rows, double change) {
  return DBL_EPSILON * (2.0 + 2.0 * rows + 64.0 * change);
}

// One graph's iteration. y holds the unnormalised iterate (x = y / T), z =
// y / out; a sweep forms u = d (s / T + (D / T) jump) + (1 - d) p with D the
// dangling mass of y. MT: the arc values' type (void: every entry is 1).
// False, with nothing written to the outputs, where the change comes so near to
// the tolerance that rounding decides (in all CTAs of a cluster alike).
template <int C, int TIER, class MT>
__device__ __forceinline__ bool ego_iterate(const EgoGraph& g, const EgoParams& prm, double* sh,
                                            double* slots, int32_t* it_out, int32_t* done_out,
                                            double* change_out) {
  extern __shared__ __align__(16) unsigned char ego_smem[];
  constexpr bool VALS = !std::is_void<MT>::value;
  using V = std::conditional_t<VALS, MT, double>;
  const uint32_t R = g.hi - g.lo, first = g.lo - g.g_lo;
  const uint32_t lane = threadIdx.x & 31, T = blockDim.x;
  const double inv_n = 1.0 / (double)g.nk;
  const uint32_t a0 = g.op.off[g.lo], na = g.op.off[g.hi] - a0;
  const float root = sqrtf((float)(g.op.off[g.g_lo + g.nk] - g.op.off[g.g_lo]));
  // z and y in two buffers each: b zs, b ys apart
  double* z;
  double* y;
  const double* io;
  const double* p;
  const uint32_t* off;
  const V* vals = nullptr;
  const uint16_t* c16 = nullptr;
  uint32_t zs = g.n, ys = g.n, off0 = a0;  // off[r] - off0: position in the CTA's arcs
  const uint32_t* c32 = g.op.cols + a0;
  if constexpr (VALS) {
    if constexpr (sizeof(V) == 4) vals = g.vals32 + a0;
    else vals = g.op.vals + a0;
  }
  if constexpr (TIER != EGO_GLOBAL) {
    z = reinterpret_cast<double*>(ego_smem);
    zs = g.nk;
    y = z + 2 * zs;
    ys = g.rmax;
    double* sio = y + 2 * ys;
    double* sp = sio + g.rmax;
    uint32_t* soff = reinterpret_cast<uint32_t*>(sp + (g.pers ? g.rmax : 0));
    for (uint32_t r = threadIdx.x; r < R; r += T) {
      sio[r] = g.inv_out[g.lo + r];
      if (g.pers) sp[r] = g.pers[g.lo + r] / g.ps;
    }
    for (uint32_t r = threadIdx.x; r <= R; r += T) soff[r] = g.op.off[g.lo + r] - a0;
    if constexpr (TIER == EGO_SMEM) {
      V* sv = reinterpret_cast<V*>(soff + ((g.rmax + 2) & ~1u));
      uint16_t* sc = reinterpret_cast<uint16_t*>(sv);
      if constexpr (VALS) sc = reinterpret_cast<uint16_t*>(sv + (sizeof(V) == 4 ? (na + 1) & ~1u : na));
      for (uint32_t k = threadIdx.x; k < na; k += T) {
        sc[k] = (uint16_t)(c32[k] - g.g_lo);
        if constexpr (VALS) sv[k] = vals[k];
      }
      c16 = sc;
      if constexpr (VALS) vals = sv;
    }
    io = sio;
    p = sp;
    off = soff;
    off0 = 0;
    __syncthreads();
  } else {
    z = g.z + g.g_lo;
    y = g.y + g.lo;
    io = g.inv_out + g.lo;
    p = g.pers + g.lo;
    off = g.op.off + g.lo;
  }
  const bool pers = g.pers != nullptr;
  // z value of row r into every copy of buffer b
  auto put_z = [&](int b, uint32_t r, double v) {
    if constexpr (C == 1 || TIER == EGO_GLOBAL) {
      z[b * zs + first + r] = v;
    } else {
      cg::cluster_group cl = cg::this_cluster();
#pragma unroll
      for (int q = 0; q < C; ++q) cl.map_shared_rank(z, (unsigned)q)[b * zs + first + r] = v;
    }
  };
  auto column = [&](uint32_t k) {
    if constexpr (TIER == EGO_SMEM) return (uint32_t)c16[k];
    else return c32[k] - g.g_lo;
  };
  auto value = [&](uint32_t k) {
    if constexpr (VALS) return vals[k];
    else return 1.0;
  };
  auto term = [&](V w, double zv) {
    if constexpr (VALS) return (double)w * zv;
    else return zv;
  };
  int turn = 0;
  double v3[3] = {0.0, 0.0, 0.0};
  bool any_long = false;
  for (uint32_t r = threadIdx.x; r < R; r += T) {
    any_long |= off[r + 1] - off[r] > EGO_LONG;
    y[r] = inv_n;
    const double i = io[r];
    put_z(0, r, inv_n * i);
    if (i == 0.0) v3[1] += inv_n;
  }
  any_long = __syncthreads_or(any_long);
  ego_sums<C>(v3, sh, slots, turn++);
  double c_it = 1.0, c_dt = v3[1], total = 1.0, change = 0.0;
  int32_t it = 0, done = 0;
  int b = 0;
  while (it < prm.max_iter) {
    const double* zb = z + b * zs;
    const double* yo = y + b * ys;
    double* yn = y + (b ^ 1) * ys;
    double acc[3] = {0.0, 0.0, 0.0};
    if (any_long) {  // their sums, left in yn
      const uint32_t w = threadIdx.x >> 5, nw = T >> 5;
      for (uint32_t r0 = 0; r0 < R; r0 += T) {
        const uint32_t r = r0 + lane * nw + w;
        const uint32_t k = r < R ? off[r] - off0 : 0u, ke = r < R ? off[r + 1] - off0 : 0u;
        for (uint32_t m = __ballot_sync(0xffffffffu, ke - k > EGO_LONG); m; m &= m - 1) {
          const int src = __ffs(m) - 1;
          const uint32_t kb = __shfl_sync(0xffffffffu, k, src);
          const uint32_t kx = __shfl_sync(0xffffffffu, ke, src);
          double t = 0.0;
#pragma unroll 4
          for (uint32_t q = kb + lane; q < kx; q += 32) t += term(value(q), zb[column(q)]);
          t = warp_sum(t);
          if ((int)lane == src) yn[r] = t;
        }
      }
      __syncthreads();
    }
    for (uint32_t r = threadIdx.x; r < R; r += T) {
      uint32_t k = off[r] - off0;
      const uint32_t ke = off[r + 1] - off0;
      double s = 0.0;
      // arcs in CSR order, four under way at a time
      if (ke - k > EGO_LONG) {
        s = yn[r];
      } else {
        for (; k < ke; k += 4) {
          uint32_t c[4];
          V w[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint32_t q = min(k + u, ke - 1);
            c[u] = column(q);
            w[u] = value(q);
          }
          double t[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) t[u] = zb[c[u]];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (k + u < ke) s += term(w[u], t[u]);
        }
      }
      const double pr = !pers ? inv_n : TIER != EGO_GLOBAL ? p[r] : p[r] / g.ps;
      const double u = prm.d * (s * c_it + c_dt * (prm.jump_uniform ? inv_n : pr)) +
                       (1.0 - prm.d) * pr;
      const double i = io[r];
      yn[r] = u;
      put_z(b ^ 1, r, u * i);
      acc[0] += u;
      if (i == 0.0) acc[1] += u;
      acc[2] += fabs(u - yo[r] * c_it);
    }
    ego_sums<C>(acc, sh, slots, turn++);
    // sum |u - x| differs from the change sum |u / T - x| by at most |1 - T|;
    // where that or rounding could decide otherwise (the rows' errors are at
    // most sqrt(all arcs) of their units), the change itself and its rounding
    total = acc[0];
    change = acc[2];
    if (fabs(change - prm.tol) <=
        2.0 * fabs(1.0 - total) + ego_rounding(root, fmax(change, prm.tol))) {
      double ex[3] = {0.0, 0.0, 0.0};
      for (uint32_t r = threadIdx.x; r < R; r += T) {
        const double x = yn[r] / total;
        ex[0] += fabs(x - yo[r] * c_it);
        ex[1] += x * sqrtf((float)(off[r + 1] - off[r]));
      }
      ego_sums<C>(ex, sh, slots, turn++);
      change = ex[0];
      if (fabs(change - prm.tol) <= ego_rounding(ex[1], fmax(change, prm.tol))) return false;
    }
    c_it = 1.0 / total;
    c_dt = acc[1] * c_it;
    b ^= 1;
    ++it;
    if (change <= prm.tol) {  // the same bits in every CTA of a cluster
      done = EGO_DONE;
      break;
    }
  }
  // a tolerance that rounding keeps this iteration above may be met by the other
  if (!done && change <= prm.tol + 32.0 * ego_rounding(root, prm.tol)) return false;
  for (uint32_t r = threadIdx.x; r < R; r += T) g.out[g.lo + r] = y[b * ys + r] / total;
  *it_out = it;
  *done_out = done;
  *change_out = change;
  return true;
}

// K sums over the rows [g.g_lo, g_hi) of a graph in the order `o` states:
// row(i, a) adds row i's terms to a[0, K). The CTAs of a cluster take the
// shares by turns, each in the launch's own threads, and every CTA adds the
// shares' sums in order (slots: 2 turns x EGO_SHARES x 2; sh: 2 turns x 2 x 32).
// The barrier in it publishes everything written before it. Warps of `o` that
// have no rows add nothing: for 60 nodes two warps' sums are joined, not 32.
template <int C, int K, class F>
__device__ __forceinline__ void ego_ordered_sums(const EgoGraph& g, uint32_t g_hi,
                                                 const EgoOrder& o, double (&out)[K], double* sh,
                                                 double* slots, int turn, F row) {
  const uint32_t shares = g.nk >= o.split ? EGO_SHARES : 1;
  const uint32_t per = (g.nk + shares - 1) / shares;
  const uint32_t lane = threadIdx.x & 31;
  double* mine = slots + (turn & 1) * EGO_SHARES * 2;
  sh += (turn & 1) * 64;
  unsigned rank = 0;
  if constexpr (C > 1) rank = cg::this_cluster().block_rank();
  for (uint32_t r = rank; r < shares; r += C) {
    const uint32_t lo = min(g_hi, g.g_lo + r * per), hi = min(g_hi, lo + per);
    const uint32_t used = min(o.threads, (hi - lo + 31u) & ~31u);
    for (uint32_t t = threadIdx.x; t < used; t += blockDim.x) {
      double a[K];
#pragma unroll
      for (int j = 0; j < K; ++j) a[j] = 0.0;
      for (uint32_t i = lo + t; i < hi; i += o.threads) row(i, a);
#pragma unroll
      for (int j = 0; j < K; ++j) {
        a[j] = warp_sum(a[j]);
        if (lane == 0) sh[32 * j + (t >> 5)] = a[j];
      }
    }
    __syncthreads();
    if (C == 1 && shares == 1) {
#pragma unroll
      for (int j = 0; j < K; ++j) {
        double t = 0.0;
#pragma unroll 4
        for (uint32_t k = 0; k < used / 32; ++k) t += sh[32 * j + k];
        out[j] = t;
      }
      return;
    }
    if (threadIdx.x < K) {
      double t = 0.0;
#pragma unroll 4
      for (uint32_t k = 0; k < used / 32; ++k) t += sh[32 * threadIdx.x + k];
      if constexpr (C == 1) {
        mine[r * 2 + threadIdx.x] = t;
      } else {
        cg::cluster_group cl = cg::this_cluster();
        for (int q = 0; q < C; ++q)
          cl.map_shared_rank(mine, (unsigned)q)[r * 2 + threadIdx.x] = t;
      }
    }
    __syncthreads();  // sh is read
  }
  if constexpr (C > 1) cg::this_cluster().sync();
#pragma unroll
  for (int j = 0; j < K; ++j) {
    double t = 0.0;
    for (uint32_t r = 0; r < shares; ++r) t += mine[r * 2 + j];
    out[j] = t;
  }
}

// The reference's iteration step by step (z = x / out with the dangling mass,
// A z, the update, the division by the total, the L1 change), with two
// reductions an iteration and every row's sum in CSR order. It runs, with its
// three vectors in shared memory where one CTA's holds them, for a graph whose
// other iteration comes so near to the tolerance that rounding would decide the
// sweep it stops on: about one in a hundred at 1e-12. 2,000 graphs take 2.04 ms a
// call without it and 2.06 with; a small batch whose longest graph is such a one
// up to twice as long (60 graphs of up to 1,000 nodes 0.27 and 0.53 ms, one batch
// of sixteen). In batches of 300 and 2,000 graphs at 60 tolerances each, 25 of 1.7
// million solves stopped a sweep earlier or later than here without it.
struct EgoEnd {
  int32_t it, done;
  double change;
};
template <int C>
__device__ __noinline__ EgoEnd ego_normalising(const EgoGraph g, const uint32_t g_hi,
                                               const EgoParams prm, const EgoOrder o,
                                               const uint32_t sm_bytes, double* sh,
                                               double* slots) {
  extern __shared__ __align__(16) unsigned char ego_smem[];
  const double inv_n = 1.0 / (double)g.nk;
  // (copies: what a store might change would be loaded again after each)
  const uint32_t* __restrict__ off = g.op.off;
  const uint32_t* __restrict__ cols = g.op.cols;
  const double* __restrict__ vals = g.op.vals;
  const double* __restrict__ outstr = g.outstr;
  const double* __restrict__ pers = g.pers;
  const double d = prm.d, ps = g.ps;
  const bool jump_uniform = prm.jump_uniform;
  double* x = g.y;
  double* y = g.y + g.n;
  double* z = g.z;
  if (C == 1 && (size_t)24 * g.nk <= sm_bytes) {  // row i at its place in the graph
    x = reinterpret_cast<double*>(ego_smem) - g.g_lo;
    y = x + g.nk;
    z = y + g.nk;
  }
  int turn = 0;
  double st[1];
  ego_ordered_sums<C, 1>(g, g_hi, o, st, sh, slots, turn++, [=](uint32_t i, double* a) {
    x[i] = inv_n;
    const double out = outstr[i];
    if (out > 0.0) {
      z[i] = inv_n / out;
    } else {
      z[i] = 0.0;
      a[0] += inv_n;
    }
  });
  double stuck = st[0];
  int32_t it = 0, done = 0;
  double change = 0.0;
  while (it < prm.max_iter) {
    double tot[1];
    ego_ordered_sums<C, 1>(g, g_hi, o, tot, sh, slots, turn++, [=](uint32_t i, double* a) {
      // arcs in CSR order; four gathers in flight before their products
      // are added in that order
      double s = 0;
      uint32_t k = off[i];
      const uint32_t ke = off[i + 1];
      for (; k + 4 <= ke; k += 4) {
        double zk[4], wk[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          zk[u] = z[cols[k + u]];
          wk[u] = vals ? vals[k + u] : 1.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) s += wk[u] * zk[u];
      }
      for (; k < ke; ++k) {
        const double w = vals ? vals[k] : 1.0;
        s += w * z[cols[k]];
      }
      const double p = pers ? pers[i] / ps : inv_n;
      const double jmp = jump_uniform ? inv_n : p;
      const double v = d * (s + stuck * jmp) + (1.0 - d) * p;
      y[i] = v;
      a[0] += v;
    });
    const double total = tot[0];
    // the division, the change, and the next z and dangling mass
    double cs[2];
    ego_ordered_sums<C, 2>(g, g_hi, o, cs, sh, slots, turn++, [=](uint32_t i, double* a) {
      const double v = y[i] / total;
      y[i] = v;
      a[0] += fabs(v - x[i]);
      const double out = outstr[i];
      if (out > 0.0) {
        z[i] = v / out;
      } else {
        z[i] = 0.0;
        a[1] += v;
      }
    });
    change = cs[0];
    stuck = cs[1];
    double* t = x;
    x = y;
    y = t;
    ++it;
    if (change <= prm.tol) {  // the same bits in every CTA of a cluster
      done = EGO_DONE;
      break;
    }
  }
  double none[1];
  double* const out = g.out;
  ego_ordered_sums<C, 1>(g, g_hi, o, none, sh, slots, turn,
                         [=](uint32_t i, double*) { out[i] = x[i]; });
  return {it, done, change};
}

// Row boundary k of C of a graph: the first row i with i + off[i] (from the
// graph's start) at least k / C of its rows plus arcs.
__device__ __forceinline__ uint32_t ego_bound(const uint32_t* off, uint32_t g_lo, uint32_t g_hi,
                                              uint32_t k, uint32_t C) {
  const uint64_t all = (uint64_t)(g_hi - g_lo) + (off[g_hi] - off[g_lo]);
  const uint64_t want = all * k / C;
  uint32_t lo = g_lo, hi = g_hi;
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if ((uint64_t)(mid - g_lo) + (off[mid] - off[g_lo]) >= want) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// A graph's solve; EGO_OPEN in *done where rounding decides and the launch is
// not to run the normalising iteration itself.
template <int C, class MT, bool BOTH>
__device__ __forceinline__ void ego_solve(EgoGraph g, uint32_t g_hi, const EgoParams& prm,
                          const EgoOrder& order, uint32_t sm_bytes, uint32_t* bounds, double* sh,
                          double* slots, int32_t* it, int32_t* done, double* ch) {
  uint32_t amax;
  if constexpr (C == 1) {
    g.lo = g.g_lo;
    g.hi = g_hi;
    g.rmax = g.nk;
    amax = g.op.off[g_hi] - g.op.off[g.g_lo];
  } else {
    if (threadIdx.x <= C)
      bounds[threadIdx.x] = ego_bound(g.op.off, g.g_lo, g_hi, threadIdx.x, C);
    __syncthreads();
    const unsigned rank = cg::this_cluster().block_rank();
    g.lo = bounds[rank];
    g.hi = bounds[rank + 1];
    g.rmax = 0;
    amax = 0;
    for (int k = 0; k < C; ++k) {  // the same in every CTA: all take the same tier
      g.rmax = max(g.rmax, bounds[k + 1] - bounds[k]);
      amax = max(amax, g.op.off[bounds[k + 1]] - g.op.off[bounds[k]]);
    }
  }
  const size_t vec = ego_vector_bytes(g.nk, g.rmax, g.pers != nullptr);
  size_t value_bytes = 0;
  if constexpr (!std::is_void<MT>::value) value_bytes = sizeof(MT);
  const size_t arcs = ego_arc_bytes(amax, value_bytes);
  bool decided = false;
  if (prm.tol <= 16.0 * DBL_EPSILON) {  // rounding decides in any case
  } else if (vec + arcs <= sm_bytes && g.nk <= 65536u) {
    decided = ego_iterate<C, EGO_SMEM, MT>(g, prm, sh, slots, it, done, ch);
  } else if (vec <= sm_bytes) {
    decided = ego_iterate<C, EGO_ARCS_GLOBAL, MT>(g, prm, sh, slots, it, done, ch);
  } else {
    decided = ego_iterate<C, EGO_GLOBAL, MT>(g, prm, sh, slots, it, done, ch);
  }
  if (decided) return;
  if constexpr (BOTH) {
    // every CTA has read the last sums before their places are used anew
    if constexpr (C > 1) cg::this_cluster().sync();
    else __syncthreads();
    const EgoEnd e = ego_normalising<C>(g, g_hi, prm, order, sm_bytes, sh, slots);
    *it = e.it;
    *done = e.done;
    *ch = e.change;
  } else {
    *done = EGO_OPEN;
  }
}

// What a launch reports of a graph: 0 stopped at the tolerance, 1 at the cap, 2 open.
__device__ __forceinline__ int32_t ego_status(int32_t done) {
  return done == EGO_DONE ? 0 : done == EGO_CAPPED ? 1 : 2;
}

// The persistent launch. With clusters of C > 1 CTAs, each cluster first
// takes the large graphs (order[0, nbig), largest first) off queue[0], its
// CTAs splitting each graph's rows; once those are gone every CTA takes the
// other graphs (order[nbig, count)) off queue[1] alone. Cluster barriers
// are hardware barriers every CTA of the cluster executes the same number of
// times: the graph index comes from rank 0's shared memory, and every CTA
// stops a graph's iteration on the same bits. BOTH: the launch runs the
// normalising iteration itself where rounding decides; a single graph's launch
// leaves that to the host (ego_one), since the call of it costs registers that
// the other iteration then spills (500 nodes: 175.6 against 177.1 us a call,
// 10,000 nodes 272 against 278). A large batch nearly always has such graphs.
template <int C, class MT, bool BOTH>
__global__ void __launch_bounds__(1024, 1)
ego_pagerank(EgoGraph g, const uint32_t* __restrict__ node_off,
             const uint32_t* __restrict__ order, uint32_t count, uint32_t nbig,
             unsigned int* __restrict__ queue, EgoParams prm, EgoOrder sums,
             const double* __restrict__ psum, uint32_t sm_bytes, int32_t* __restrict__ iters,
             int32_t* __restrict__ status, double* __restrict__ changes) {
  __shared__ double sh[2 * 3 * 32];
  __shared__ double slots[2 * (C > EGO_SHARES / 2 ? C : EGO_SHARES / 2) * 4];
  __shared__ uint32_t bounds[C + 1];
  __shared__ uint32_t g_sh;
  auto take = [&](uint32_t graph) {
    g.g_lo = node_off[graph];
    const uint32_t g_hi = node_off[graph + 1];
    g.nk = g_hi - g.g_lo;
    if (g.pers) g.ps = psum[graph];
    return g_hi;
  };
  if constexpr (C > 1) {
    cg::cluster_group cl = cg::this_cluster();
    const unsigned rank = cl.block_rank();
    for (;;) {
      if (rank == 0 && threadIdx.x == 0) g_sh = atomicAdd(queue, 1u);
      cl.sync();  // rank 0's pick is visible
      const uint32_t gi = *cl.map_shared_rank(&g_sh, 0u);
      cl.sync();  // every CTA has read it before rank 0 picks again or leaves
      if (gi >= nbig) break;
      const uint32_t graph = order[gi];
      const uint32_t g_hi = take(graph);
      int32_t it = 0, done = 0;
      double ch = 0.0;
      ego_solve<C, MT, BOTH>(g, g_hi, prm, sums, sm_bytes, bounds, sh, slots, &it, &done, &ch);
      if (rank == 0 && threadIdx.x == 0) {
        iters[graph] = it;
        status[graph] = ego_status(done);
        changes[graph] = ch;
      }
    }
  }
  for (;;) {
    if (threadIdx.x == 0) g_sh = atomicAdd(queue + 1, 1u);
    __syncthreads();
    const uint32_t gi = nbig + g_sh;
    __syncthreads();
    if (gi >= count) return;
    const uint32_t graph = order[gi];
    const uint32_t g_hi = take(graph);
    int32_t it = 0, done = 0;
    double ch = 0.0;
    if (g.nk == 0) done = EGO_DONE;
    else ego_solve<1, MT, BOTH>(g, g_hi, prm, sums, sm_bytes, bounds, sh, slots, &it, &done, &ch);
    if (threadIdx.x == 0) {
      iters[graph] = it;
      status[graph] = ego_status(done);
      changes[graph] = ch;
    }
    __syncthreads();
  }
}

// The normalising iteration of a single graph (nodes [0, g.nk)) on one cluster.
template <int C>
__global__ void __launch_bounds__(1024, 1)
ego_one(EgoGraph g, EgoParams prm, EgoOrder sums, uint32_t sm_bytes, int32_t* __restrict__ iters,
        int32_t* __restrict__ status, double* __restrict__ changes) {
  __shared__ double sh[2 * 2 * 32];
  __shared__ double slots[2 * EGO_SHARES * 2];
  // (the first sums write into every CTA's slots: all have to be there)
  if constexpr (C > 1) cg::this_cluster().sync();
  const EgoEnd e = ego_normalising<C>(g, g.nk, prm, sums, sm_bytes, sh, slots);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *iters = e.it;
    *status = ego_status(e.done);
    *changes = e.change;
  }
}

// Edges must stay inside their graph: the first crossing edge, if any.
__global__ void ego_check_blocks(const uint32_t* __restrict__ src, const uint32_t* __restrict__ tgt,
                                 uint64_t m, const uint32_t* __restrict__ node_off, uint32_t count,
                                 unsigned long long* __restrict__ bad) {
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m;
       e += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t a = src[e], b = tgt[e];
    // graph of a: largest k with node_off[k] <= a
    uint32_t lo = 0, hi = count;
    while (hi - lo > 1) {
      uint32_t mid = (lo + hi) >> 1;
      if (node_off[mid] <= a) lo = mid; else hi = mid;
    }
    if (b < node_off[lo] || b >= node_off[lo + 1]) atomicMin(bad, (unsigned long long)e);
  }
}

// Process-wide settings (net_set_tuning keys 6, 16, 15), read by solves that
// may run on other threads.
static std::atomic<int> g_ego_threads{0};  // 0: chosen per batch (tuned for large batches)
static std::atomic<int> g_ego_cluster{0};  // CTAs per cluster for the large graphs; 0: chosen
static std::atomic<int64_t> g_ego_big{0};  // nodes from which a graph is large; 0: automatic

void set_ego_threads(int t) { g_ego_threads = t; }
void set_ego_cluster(int c) { g_ego_cluster = c; }
void set_ego_big_nodes(int64_t v) { g_ego_big = v; }

// The most dynamic shared memory a CTA can get (4 KB cover the static arrays
// and what the driver takes).
static uint32_t ego_most_smem() {
  int dev = 0, optin = 0;
  KNB_CUDA(cudaGetDevice(&dev));
  KNB_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  return (uint32_t)optin - 4096;
}

// Shape of a launch.
struct EgoShape {
  int threads = 256;
  int cluster = 1;    // CTAs that split a large graph: 1, 4, 8 or 16
  uint32_t smem = 0;  // dynamic shared memory per CTA
  bool operator==(const EgoShape& o) const {
    return threads == o.threads && cluster == o.cluster && smem == o.smem;
  }
};

// In a batch, shared memory for the small graphs (about 600 nodes of 12 arcs,
// in 1,200 vectors only) and the rest of the SM's 256 KB to L1, which serves the
// gathers of the graphs that do not fit: 2,000 graphs of up to 50,000 nodes
// take 1.24 ms with 32 KB a CTA, 2.3 ms with all there is.
constexpr uint32_t EGO_BATCH_SMEM = 32768;

// CTAs (C == 1) or clusters of C CTAs of `threads` that fit on the device at
// once with their shared memory (0 if none), per device and shape.
template <int C, class MT, bool BOTH>
static int ego_resident(int threads, uint32_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<int, int, uint32_t>, int> cache;
  int dev = 0;
  KNB_CUDA(cudaGetDevice(&dev));
  if (C > 8)
    set_func_attr((const void*)ego_pagerank<C, MT, BOTH>,
                  cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  set_func_attr((const void*)ego_pagerank<C, MT, BOTH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                (int)ego_most_smem());
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find({dev, threads, smem});
  if (it != cache.end()) return it->second;
  int fit = 0;
  if constexpr (C == 1) {
    int per_sm = 0, sms = 0;
    KNB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ego_pagerank<1, MT, BOTH>,
                                                           threads, smem));
    KNB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    fit = std::max(1, per_sm) * sms;
  } else {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&fit, (const void*)ego_pagerank<C, MT, BOTH>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      fit = 0;
    }
  }
  cache[{dev, threads, smem}] = fit;
  return fit;
}

// A packed batch kept per operator between calls: the graph offsets and the
// largest-first order, every buffer, and the launch (queue reset and kernel)
// instantiated as a CUDA graph, which later calls with the same offsets,
// parameters and threads replay instead of capturing it again. Teleport
// values are copied in on every call. A call with other offsets rebuilds
// the plan; solves on one operator take turns on its mutex.
struct EgoPlan : Workspace {
  std::mutex mu;
  std::vector<uint32_t> hoff;  // the batch the buffers are laid out for
  bool pers = false;
  EgoParams prm{};
  std::vector<uint32_t> sizes;  // node counts of the graphs, largest first
  bool tuned = false;          // this batch's shape is chosen, with these pinned:
  int pin_t = 0, pin_c = 0;
  EgoShape pick;
  EgoShape shape;              // of the instantiated launch
  int64_t pin_big = 0;         // the large-graph threshold it was pinned to
  uint32_t nbig = 0;           // graphs it gives to clusters
  DevBuf<uint32_t> doff, dorder;
  DevBuf<double> dpers, y, z;
  DevBuf<double> result;  // scores (n), changes (count), iterations and statuses (2 count int32)
  DevBuf<unsigned int> queue;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaEvent_t t0 = nullptr, t1 = nullptr;
  int instantiations = 0;
  ~EgoPlan() override {
    drop_graph();
    if (t0) cudaEventDestroy(t0);
    if (t1) cudaEventDestroy(t1);
  }
  void drop_graph() {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    exec = nullptr;
    graph = nullptr;
  }
};

template <class T>
struct TypeIs {
  using type = T;
};

static bool same_params(const EgoParams& a, const EgoParams& b) {
  return a.d == b.d && a.tol == b.tol && a.max_iter == b.max_iter &&
         a.jump_uniform == b.jump_uniform;
}

void pagerank_graphs(GraphHandleImpl& g, const EgoInput& in, double* out, EgoResult* res,
                     cudaStream_t s) {
  const uint32_t n = g.n;
  const uint32_t count = in.count;
  // node offsets: nondecreasing, from 0 to n
  if (in.node_offsets[0] != 0 || (uint64_t)in.node_offsets[count] != n)
    throw Error("graph offsets must start at 0 and end at the node count");
  for (uint32_t k = 0; k < count; ++k)
    if (in.node_offsets[k + 1] < in.node_offsets[k])
      throw Error("graph offsets must be nondecreasing");
  std::vector<uint32_t> hoff(count + 1);
  for (uint32_t k = 0; k <= count; ++k) hoff[k] = (uint32_t)in.node_offsets[k];
  // personalization: per-graph sums (host, in node order within each graph)
  std::vector<double> ps;
  if (in.personalization) {
    ps.assign(count, 0.0);
    for (uint32_t k = 0; k < count; ++k) {
      double t = 0;
      for (uint32_t i = hoff[k]; i < hoff[k + 1]; ++i) {
        double v = in.personalization[i];
        if (!std::isfinite(v) || v < 0.0)
          throw Error("the personalization vector must hold finite, nonnegative values");
        t += v;
      }
      if (hoff[k + 1] > hoff[k] && !(t > 0.0))
        throw Error("the personalization vector must have a positive sum");
      ps[k] = t;
    }
  }
  const int which = (g.directed && in.directed) ? 1 : (g.directed ? 2 : 0);
  const double lfac = in.loops == 2 ? 0.0 : (which == 1 ? 1.0 : (in.loops == 0 ? 2.0 : 1.0));
  Operator& op = g.op(which, in.weighted, lfac, s);
  EgoPlan* pp = nullptr;
  {
    std::lock_guard<std::mutex> lock(op.mu);
    if (!op.ego_ws) op.ego_ws = std::make_unique<EgoPlan>();
    pp = static_cast<EgoPlan*>(op.ego_ws.get());
  }
  EgoPlan& P = *pp;
  std::lock_guard<std::mutex> plan_lock(P.mu);
  const bool pers = in.personalization != nullptr;
  if (P.hoff != hoff) {
    // a new batch: check that no edge joins two graphs, order, buffers
    P.drop_graph();
    P.hoff.clear();
    P.doff.alloc(count + 1);
    P.dorder.alloc(std::max<uint32_t>(count, 1));
    KNB_CUDA(cudaMemcpyAsync(P.doff.get(), hoff.data(), (count + 1) * 4, cudaMemcpyHostToDevice, s));
    if (g.m) {
      DevBuf<unsigned long long> bad(1);
      KNB_CUDA(cudaMemsetAsync(bad.get(), 0xFF, 8, s));
      ego_check_blocks<<<grid_for(g.m, 256), 256, 0, s>>>(g.src.get(), g.tgt.get(), g.m,
                                                          P.doff.get(), count, bad.get());
      KNB_LAUNCH("ego_check_blocks");
      unsigned long long hb = 0;
      KNB_CUDA(cudaMemcpyAsync(&hb, bad.get(), 8, cudaMemcpyDeviceToHost, s));
      KNB_CUDA(cudaStreamSynchronize(s));
      if (hb != ~0ull)
        throw Error("edge " + std::to_string(hb) + " joins two different graphs of the batch");
    }
    // largest graphs first
    std::vector<uint32_t> order(count);
    std::iota(order.begin(), order.end(), 0u);
    std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) {
      return hoff[a + 1] - hoff[a] > hoff[b + 1] - hoff[b];
    });
    KNB_CUDA(cudaMemcpyAsync(P.dorder.get(), order.data(), (size_t)count * 4,
                             cudaMemcpyHostToDevice, s));
    P.tuned = false;
    P.sizes.resize(count);
    for (uint32_t k = 0; k < count; ++k) P.sizes[k] = hoff[order[k] + 1] - hoff[order[k]];
    P.y.alloc((size_t)2 * n);
    P.z.alloc((size_t)2 * n);
    P.result.alloc((size_t)n + 2 * (size_t)count);
    P.queue.alloc(2);
    P.dpers.release();
    KNB_CUDA(cudaStreamSynchronize(s));
    P.hoff = hoff;
  }
  double* const scores = P.result.get();
  double* const changes = scores + n;
  int32_t* const iters = reinterpret_cast<int32_t*>(changes + count);
  int32_t* const status = iters + count;
  const HostStaging staging;
  unsigned char* const stage = staging.p;
  if (pers) {  // the vectors, then their sums
    if (!P.dpers.get()) P.dpers.alloc((size_t)n + count);
    if (stage && ((size_t)n + count) * 8 <= STAGING_HALF) {
      memcpy(stage, in.personalization, (size_t)n * 8);
      memcpy(stage + (size_t)n * 8, ps.data(), (size_t)count * 8);
      KNB_CUDA(cudaMemcpyAsync(P.dpers.get(), stage, ((size_t)n + count) * 8,
                               cudaMemcpyHostToDevice, s));
    } else {
      KNB_CUDA(cudaMemcpyAsync(P.dpers.get(), in.personalization, (size_t)n * 8,
                               cudaMemcpyHostToDevice, s));
      KNB_CUDA(cudaMemcpyAsync(P.dpers.get() + n, ps.data(), (size_t)count * 8,
                               cudaMemcpyHostToDevice, s));
    }
  }
  const EgoParams prm{in.damping, in.tol, (int32_t)std::min<int64_t>(in.max_iter, INT32_MAX),
                      in.dangling == 1 ? 1 : 0};
  int dev = 0, sms = 148;
  KNB_CUDA(cudaGetDevice(&dev));
  KNB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // The launch: with clusters of C > 1 CTAs the graphs of at least `big`
  // nodes (by default max(4096, n / CTAs of the grid), so no graph holds
  // much more than a CTA's share of the batch) are each split over a
  // cluster; the others go one per CTA. Returns the graphs given to clusters.
  const int64_t pin_big = g_ego_big.load();
  auto big_count = [&](uint64_t ctas) {
    const uint64_t big =
        pin_big > 0 ? (uint64_t)pin_big
        : count == 1 ? 1  // the shape chosen for it says whether it is split
                     : std::max<uint64_t>(4096, (uint64_t)n / std::max<uint64_t>(ctas, 1));
    uint32_t nb = 0;
    while (nb < count && P.sizes[nb] >= big) ++nb;
    return nb;
  };
  EgoGraph base{};
  base.op = op.view64();
  base.vals32 = op.has_vals && op.vals32_exact ? op.vals32.get() : nullptr;
  base.inv_out = op.inv_out64.get();
  base.outstr = op.colsum.get();
  base.pers = pers ? P.dpers.get() : nullptr;
  base.ps = 1.0;
  base.y = P.y.get();
  base.z = P.z.get();
  base.n = n;
  base.out = scores;
  // The order of the normalising iteration's sums: that of a launch of clusters
  // of 8 with the threads that were fastest for such a batch where every solve
  // took it.
  const bool many = op.nnz >= (1u << 20);
  EgoOrder sums;
  sums.threads = !many ? (count < (uint32_t)sms ? 1024 : 256)
                 : !count || P.sizes[0] < 4096 ? 256 : n <= (1u << 18) ? 1024 : 512;
  sums.split = std::max<uint32_t>(4096, n / ((uint32_t)sms * (2048 / sums.threads)));
  auto launch_as = [&](auto mt, auto both, const EgoShape& shape, cudaStream_t st) -> uint32_t {
    using MT = typename decltype(mt)::type;
    constexpr bool BOTH = decltype(both)::value;
    KNB_CUDA(cudaMemsetAsync(P.queue.get(), 0, 8, st));
    const int threads = shape.threads, C = shape.cluster;
    const uint32_t smem = shape.smem;
    int clusters = 0;
    if (C == 4) clusters = ego_resident<4, MT, BOTH>(threads, smem);
    if (C == 8) clusters = ego_resident<8, MT, BOTH>(threads, smem);
    if (C == 16) clusters = ego_resident<16, MT, BOTH>(threads, smem);
    const uint32_t nbig = clusters > 0 ? big_count((uint64_t)clusters * C) : 0;
    const double* psum = pers ? P.dpers.get() + n : nullptr;
    if (nbig == 0) {
      const unsigned grid =
          (unsigned)std::min<uint64_t>(count, (uint64_t)ego_resident<1, MT, BOTH>(threads, smem));
      ego_pagerank<1, MT, BOTH><<<grid, threads, smem, st>>>(
          base, P.doff.get(), P.dorder.get(), count, 0u, P.queue.get(), prm, sums, psum, smem,
          iters, status, changes);
      KNB_LAUNCH("ego_pagerank");
      return 0;
    }
    // no more clusters than there is work for
    if (nbig == count) clusters = (int)std::min<uint32_t>((uint32_t)clusters, nbig);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * C));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto args = [&](auto fn) {
      KNB_CUDA(cudaLaunchKernelEx(&cfg, fn, base, (const uint32_t*)P.doff.get(),
                                  (const uint32_t*)P.dorder.get(), count, nbig, P.queue.get(), prm,
                                  sums, psum, smem, iters, status, changes));
    };
    if (C == 4) args(ego_pagerank<4, MT, BOTH>);
    else if (C == 8) args(ego_pagerank<8, MT, BOTH>);
    else args(ego_pagerank<16, MT, BOTH>);
    KNB_LAUNCH("ego_pagerank");
    return nbig;
  };
  auto launch = [&](const EgoShape& shape, cudaStream_t st) -> uint32_t {
    auto with = [&](auto mt) {
      return count > 1 ? launch_as(mt, std::true_type{}, shape, st)
                       : launch_as(mt, std::false_type{}, shape, st);
    };
    if (!op.has_vals) return with(TypeIs<void>{});
    if (base.vals32) return with(TypeIs<float>{});
    return with(TypeIs<double>{});
  };
  // The normalising iteration of a single graph, as wide as its sums' shares.
  auto launch_one = [&] {
    EgoGraph g1 = base;
    g1.nk = n;
    g1.ps = pers ? ps[0] : 1.0;
    if (n < sums.split) {
      const uint32_t most = ego_most_smem();
      set_func_attr((const void*)ego_one<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                    (int)most);
      const uint32_t smem = (size_t)24 * n <= most ? 24 * n : 0;
      ego_one<1><<<1, sums.threads, smem, s>>>(g1, prm, sums, smem, iters, status, changes);
    } else {
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = EGO_SHARES;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(EGO_SHARES);
      cfg.blockDim = dim3(sums.threads);
      cfg.stream = s;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      KNB_CUDA(cudaLaunchKernelEx(&cfg, ego_one<EGO_SHARES>, g1, prm, sums, 0u, iters, status,
                                  changes));
    }
    KNB_LAUNCH("ego_one");
  };
  if (!P.t0) {
    KNB_CUDA(cudaEventCreate(&P.t0));
    KNB_CUDA(cudaEventCreate(&P.t1));
  }
  // The launch's shape, unless pinned (tuning keys 6 and 16). Results do not
  // depend on it beyond the association of a split graph's sums.
  // - One graph: from 400 nodes on a cluster of 8 (500 nodes: 270 us a call
  //   against 292 on one CTA, 200 nodes: 258 against 208), as many threads as
  //   its CTAs have rows, and all the shared memory; a graph too large for
  //   that takes a cluster of 16 and leaves the memory to L1.
  // - A batch of at least 2^20 arcs: timed once per batch layout on the batch
  //   itself.
  // - Smaller batches: 1,024 threads and clusters of 16 when a graph is large
  //   enough to be split (100 graphs up to 20,000 nodes: 390 us against 626
  //   with 256 threads), else 256 threads.
  const int pin_t = g_ego_threads.load(), pin_c = g_ego_cluster.load();
  // (a single graph's depends on whether it has a teleport vector to hold)
  if (!P.tuned || count == 1 || P.pin_t != pin_t || P.pin_c != pin_c) {
    EgoShape pick;
    const uint32_t most = ego_most_smem();
    if (count == 1) {
      const size_t vb = !op.has_vals ? 0 : base.vals32 ? 4 : 8;
      const bool fits = ego_vector_bytes(n, n / 8 + n / 16, pers) +
                            ego_arc_bytes(op.nnz / 8 + op.nnz / 32, vb) <= most;
      const uint32_t rows = fits ? n / 8 : n / 16;
      pick.cluster = n < 400 ? 1 : fits ? 8 : 16;
      pick.threads = n < 400 || rows <= 256 ? 256 : rows <= 512 ? 512 : 1024;
      pick.smem = fits ? most : 4096;
    } else {
      const bool split = P.sizes[0] >= 4096;
      pick = {split ? 1024 : 256, split ? 16 : 8, EGO_BATCH_SMEM};
      if ((pin_t == 0 || pin_c == 0) && op.nnz >= (1u << 20)) {
        float best = 1e30f;
        for (EgoShape c : {EgoShape{256, 8, EGO_BATCH_SMEM}, EgoShape{256, 16, EGO_BATCH_SMEM},
                           EgoShape{512, 16, EGO_BATCH_SMEM}, EgoShape{1024, 16, EGO_BATCH_SMEM}}) {
          if (pin_t) c.threads = pin_t;
          if (pin_c) c.cluster = pin_c;
          if (c.cluster == 16 && c.threads == 256 && !split) continue;
          KNB_CUDA(cudaEventRecord(P.t0, s));
          launch(c, s);
          KNB_CUDA(cudaEventRecord(P.t1, s));
          KNB_CUDA(cudaEventSynchronize(P.t1));
          float ms = 0;
          KNB_CUDA(cudaEventElapsedTime(&ms, P.t0, P.t1));
          if (ms < best) {
            best = ms;
            pick = c;
          }
        }
      }
    }
    P.pick = pick;
    P.tuned = true;
    P.pin_t = pin_t;
    P.pin_c = pin_c;
  }
  EgoShape shape = P.pick;
  if (pin_t) shape.threads = pin_t;
  if (pin_c) shape.cluster = pin_c;
  if (!P.exec || !(P.shape == shape) || P.pin_big != pin_big || P.pers != pers ||
      !same_params(P.prm, prm)) {
    P.drop_graph();
    cudaStream_t cs;
    KNB_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    KNB_CUDA(cudaStreamSynchronize(s));
    KNB_CUDA(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
    P.nbig = launch(shape, cs);
    KNB_CUDA(cudaStreamEndCapture(cs, &P.graph));
    KNB_CUDA(cudaGraphInstantiate(&P.exec, P.graph, 0));
    KNB_CUDA(cudaStreamDestroy(cs));
    P.shape = shape;
    P.pin_big = pin_big;
    P.pers = pers;
    P.prm = prm;
    ++P.instantiations;
  }
  KNB_CUDA(cudaEventRecord(P.t0, s));
  KNB_CUDA(cudaGraphLaunch(P.exec, s));
  KNB_CUDA(cudaEventRecord(P.t1, s));
  // what the launch reports, and with it, where both are small, the scores:
  // one copy through page-locked memory
  const size_t meta = (size_t)count * 16, all = (size_t)n * 8 + meta;
  const bool together = stage && !in.out_on_device && all <= STAGING_HALF;
  std::vector<unsigned char> own;
  unsigned char* back = stage + STAGING_HALF;
  if (!stage || meta > STAGING_HALF) {
    own.resize(meta);
    back = own.data();
  }
  auto fetch = [&] {
    KNB_CUDA(cudaMemcpyAsync(back, together ? scores : changes, together ? all : meta,
                             cudaMemcpyDeviceToHost, s));
    KNB_CUDA(cudaStreamSynchronize(s));
  };
  fetch();
  const double* hscores = reinterpret_cast<const double*>(back);
  const double* hchange = together ? hscores + n : hscores;
  const int32_t* hit = reinterpret_cast<const int32_t*>(hchange + count);
  const int32_t* hst = hit + count;
  if (count == 1 && hst[0] == 2) {
    launch_one();
    KNB_CUDA(cudaEventRecord(P.t1, s));
    fetch();
  }
  float ms = 0;
  KNB_CUDA(cudaEventElapsedTime(&ms, P.t0, P.t1));
  for (uint32_t k = 0; k < count; ++k)
    if (hst[k])
      throw Error("PageRank did not converge to tolerance " + std::to_string(in.tol) +
                  " within " + std::to_string(in.max_iter) + " iterations" +
                  (count > 1 ? " (graph " + std::to_string(k) + " of the batch)" : ""));
  if (together) {
    memcpy(out, hscores, (size_t)n * 8);
  } else {
    KNB_CUDA(cudaMemcpyAsync(out, scores, (size_t)n * 8,
                             in.out_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                             s));
    KNB_CUDA(cudaStreamSynchronize(s));
  }
  if (res) {
    res->seconds = ms * 1e-3;
    res->threads = shape.threads;
    res->cluster = P.nbig ? shape.cluster : 1;
    res->split_graphs = (int32_t)P.nbig;
    res->instantiations = P.instantiations;
    int64_t tot = 0, mx = 0;
    for (uint32_t k = 0; k < count; ++k) {
      tot += hit[k];
      mx = std::max<int64_t>(mx, hit[k]);
    }
    res->total_iterations = tot;
    res->change = count == 1 ? hchange[0] : 0.0;
    res->max_iterations = mx;
    if (in.iterations_out)
      for (uint32_t k = 0; k < count; ++k) in.iterations_out[k] = hit[k];
  }
}

}  // namespace knb
