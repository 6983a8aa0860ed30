// Differentiable PageRank: PageRank of caller-supplied edge weights, and the
// gradient of a loss L(x) with respect to those weights.
//
// At the fixed point, x = d (M x + jump 1_D^T x) + (1 - d) p with 1^T x = 1,
// where M_ij = sum of f_e w_e over arcs e = (j -> i), divided by the
// out-strength s_j, f_e the self-loop factor, and D the dangling nodes
// (s_j = 0). With A = I - d M - d jump 1_D^T (invertible for d < 1: the
// matrix d (M + jump 1_D^T) is d times a column-stochastic matrix) and
// g = dL/dx, the adjoint lambda solves A^T lambda = g, i.e.
//     lambda = g + d M^T lambda + d 1_D (jump^T lambda),
// a fixed-point iteration lambda <- g + d G lambda that contracts by d in the
// max norm. G is the walk itself (row-stochastic), so what each closed class
// of nodes holds on average shrinks by no more than d per sweep, where
// PageRank's own change dies out much faster; the span of the last sweeps
// gives that part's limit (adj_extrapolate). The sweep pulls along out-arcs,
// (M^T lambda)_j = sum over arcs (j -> i) of f_e w_e lambda_i / s_j, on the
// merge-path sweep over the out-adjacency. Then, since
// dM_kj/dw_e = f_e (delta_ki - M_kj) / s_j for e = (j -> i),
//     dL/dw_e = d f_e (x_j / s_j) (lambda_i - (M^T lambda)_j),
// the second term being the derivative of the row (out-strength)
// normalisation. An undirected edge adds the terms of its two arcs. Dangling
// nodes stay dangling for positive weights, so D does not move.
#include <cfloat>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "adjoint.cuh"
#include "pagerank.cuh"

namespace knb {

// One adjoint sweep: the update, its L1 change and jump^T lambda'. A solve
// ends when the change meets the tolerance. Once an extrapolation has been
// taken (st->ambiguous) it goes on to SETTLED times the tolerance, so that the
// faster parts end about as small as the sweeps left out would have made
// them, or to the sweep at which the plain iteration would have ended
// (st->prev_inv_total), whichever is first.
constexpr double SETTLED = 1e-2;
__device__ __forceinline__ void adj_decide(IterState* st) {
  const bool enough = st->ambiguous ? st->change <= SETTLED * st->tol ||
                                          (st->change <= st->tol && st->iter >= st->prev_inv_total)
                                    : st->change <= st->tol;
  if (enough) st->converged = 1;
  else if (st->iter >= st->max_iter) st->stopped = 1;
}

struct AdjointEpi {
  static constexpr int NACC = 2;
  static constexpr bool SUMS = true;
  const double* g;
  const double* lam_old;
  double* lam_new;
  const double* inv_out;
  const double* jump;  // null: uniform
  double d, pu;
  double jdot = 0;

  __device__ __forceinline__ void prepare(const IterState* st) { jdot = st->dterm; }
  static __device__ __forceinline__ void init(double* a) { a[0] = a[1] = 0.0; }
  static __device__ __forceinline__ double identity(int) { return 0.0; }
  static __device__ __forceinline__ double combine(int, double a, double b) { return a + b; }
  static __device__ __forceinline__ double warp_combine(int, double v) { return warp_sum(v); }
  struct In {
    double io, gj, lo, jj;
  };
  __device__ __forceinline__ In fetch(uint32_t j) const {
    return {inv_out[j], g[j], lam_old[j], jump ? jump[j] : pu};
  }
  __device__ __forceinline__ void row_in(uint32_t j, double r, const In& in, double* a) const {
    const double v = in.gj + d * (in.io > 0.0 ? r * in.io : jdot);
    lam_new[j] = v;
    a[0] += fabs(v - in.lo);
    a[1] += in.jj * v;
  }
  __device__ __forceinline__ void row(uint32_t j, double r, double* a) const {
    row_in(j, r, fetch(j), a);
  }
  __device__ void finish(IterState* st, const double* tot) const {
    st->change = tot[0];
    st->dterm = tot[1];
    st->iter += 1;
    adj_decide(st);
  }
};

// Row sums r_j = sum of f_e w_e lambda_i (final lambda), stored.
struct RowSumEpi {
  static constexpr int NACC = 0;
  double* r;
  __device__ __forceinline__ void prepare(const IterState*) {}
  static __device__ __forceinline__ void init(double*) {}
  static __device__ __forceinline__ double identity(int) { return 0.0; }
  static __device__ __forceinline__ double combine(int, double a, double b) { return a + b; }
  static __device__ __forceinline__ double warp_combine(int, double v) { return v; }
  __device__ __forceinline__ void row(uint32_t j, double s, double*) const { r[j] = s; }
  __device__ void finish(IterState*, const double*) const {}
};

// Sums of v[0..N-1] over the grid in CTA order, in the CTA that comes last.
template <int N>
__device__ __forceinline__ bool last_sums(double (&v)[N], double* __restrict__ part,
                                          uint32_t* ticket, double* sh) {
  __shared__ bool last;
  if (threadIdx.x == 0)
    for (int k = 0; k < N; ++k) part[N * blockIdx.x + k] = v[k];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    double x = 0;
    for (uint32_t q = threadIdx.x; q < gridDim.x; q += blockDim.x) x += __ldcg(part + N * q + k);
    v[k] = block_sum(x, sh);
  }
  return true;
}

// lambda = g; jump^T g; the tolerance, scaled by max(1, ||g||_1).
__global__ void __launch_bounds__(256)
adj_init(const double* __restrict__ g, const double* __restrict__ jump, uint32_t n, double tol,
         double* __restrict__ lam, double* __restrict__ part, IterState* st) {
  __shared__ double sh[8];
  double a = 0, b = 0;
  const double pu = 1.0 / n;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double v = g[i];
    lam[i] = v;
    a += (jump ? jump[i] : pu) * v;
    b += fabs(v);
  }
  double v[2] = {block_sum(a, sh), block_sum(b, sh)};
  if (!last_sums(v, part, &st->ticket, sh) || threadIdx.x != 0) return;
  st->dterm = v[0];
  st->tol = tol * fmax(1.0, v[1]);
  st->ticket = 0;
}

// Extrapolation over the last SPAN sweeps. The part of lambda's error that G
// keeps (the average over each closed class of nodes: G^SPAN leaves it as it
// is, also where a class is a cycle of SPAN's divisors 2, 3 or 6) shrinks by
// d^SPAN over SPAN sweeps, so E = b + c (b - a), c = d^SPAN / (1 - d^SPAN),
// has none of it, where a is the iterate SPAN sweeps before b. Sweeping is
// affine: had lambda been extrapolated one sweep earlier (from a0 and b0, the
// iterates before a and b), this sweep would have turned it into E with the
// change (1 + c) (b - b0) - c (a - a0). So E's place in the iteration, its
// change and the same stopping rule come from one pass over four vectors, and
// E is taken only where that change is below half of the plain one: a graph
// whose error has no such part keeps the plain iteration.
//
// The plain iteration's last sweeps move every node the same way, by d of the
// sweep before, until all of them round to what they were. E is past that: what
// is left of its error changes sign and may stay at one unit in the last place
// of every node, back and forth, for good. So E is not taken where the tolerance
// is below ROUNDED of lambda's size (n nodes at one unit each come to at most
// 2^-52 of it), and a solve whose change, above the tolerance, has not come down
// to `stall` of that a cycle before is stopped; the caller then iterates plainly
// from the start.
constexpr int SPAN = 6;
constexpr int CYCLE = 24;  // an extrapolation is tried every CYCLE sweeps
constexpr double ROUNDED = 4.0 * DBL_EPSILON;

__global__ void __launch_bounds__(256)
adj_extrapolate(const double* __restrict__ a0, const double* __restrict__ a,
                const double* __restrict__ b0, const double* __restrict__ b, double c, double d,
                double stall, const double* __restrict__ jump, uint32_t n,
                double* __restrict__ part, IterState* st) {
  if (iteration_done(st)) return;
  __shared__ double sh[8];
  double ch = 0, jd = 0, size = 0;
  const double pu = 1.0 / n;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double av = a[i], bv = b[i];
    size += fabs(bv);
    ch += fabs((1.0 + c) * (bv - b0[i]) - c * (av - a0[i]));
    jd += (jump ? jump[i] : pu) * (bv + c * (bv - av));
  }
  double v[3] = {block_sum(ch, sh), block_sum(jd, sh), block_sum(size, sh)};
  if (!last_sums(v, part, &st->ticket, sh) || threadIdx.x != 0) return;
  st->ticket = 0;
  const double before = st->slack;  // the change a cycle ago
  if (v[0] < 0.5 * st->change && st->tol >= ROUNDED * v[2]) {
    if (!st->ambiguous) {
      st->ambiguous = 1;
      st->prev_inv_total = st->iter + ceil(log(st->tol / st->change) / log(d));
      st->slack = INFINITY;
    }
    st->top = 1.0;  // adj_take replaces b by E
    st->change = v[0];
    st->dterm = v[1];
    adj_decide(st);
  }
  if (st->ambiguous) {
    if (st->slack == before && st->change > st->tol && !(st->change <= stall * before))
      st->stopped = 1;
    st->slack = st->change;
  }
}

__global__ void adj_take(const double* __restrict__ a, double* __restrict__ b, double c,
                         uint32_t n, IterState* st) {
  if (st->top == 0.0) return;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    b[i] = b[i] + c * (b[i] - a[i]);
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&st->ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (last && threadIdx.x == 0) {
    st->top = 0.0;
    st->ticket = 0;
  }
}

// Per node j, what the gradients of its out-arcs share: d x_j / s_j and
// (M^T lambda)_j (both 0 for a node without out-strength: nothing depends on
// its arcs).
__global__ void adj_node_terms(const double* __restrict__ x, const double* __restrict__ inv_out,
                               const double* __restrict__ r, uint32_t n, double d,
                               double2* __restrict__ t) {
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const double io = inv_out[j];
    t[j] = io > 0.0 ? make_double2(d * (x[j] * io), r[j] * io) : make_double2(0.0, 0.0);
  }
}

// dL/dw_e, one thread per edge e = (u, v) in input order: the term of arc
// u -> v, plus that of v -> u where the edge is walked both ways (`both`; a
// loop is one arc). Edges are balanced whatever the degrees and the gradient
// is written in order; bound by the three or six gathered node values per
// edge. R-MAT 20 (16.8M edges): 10.4 ms with one thread per row of the
// out-adjacency, which waited for the hubs; 0.074 ms over the edges.
__global__ void adj_grad(const uint32_t* __restrict__ src, const uint32_t* __restrict__ tgt,
                         uint64_t m, double lf, const double2* __restrict__ t,
                         const double* __restrict__ lam, int both, double* __restrict__ grad) {
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m;
       e += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t u = src[e], v = tgt[e];
    const double2 a = t[u];
    double g = a.x * (lam[v] - a.y);
    if (u == v) {
      g *= lf;
    } else if (both) {
      const double2 b = t[v];
      g += b.x * (lam[u] - b.y);
    }
    grad[e] = g;
  }
}

// Buffers, pinned state and events of adjoint solves, kept with the weight
// slot of the forward operator (whose mutex a solve holds) between calls.
struct AdjointWorkspace : Workspace {
  DevBuf<double> lam[4], r, carry, head, part1, part2, part3, jump;
  DevBuf<double2> terms;
  DevBuf<IterState> st;
  IterState* hst = nullptr;  // pinned, 2 slots
  cudaEvent_t t0 = nullptr, t1 = nullptr, done[2] = {nullptr, nullptr};
  ~AdjointWorkspace() override {
    if (hst) cudaFreeHost(hst);
    for (cudaEvent_t e : {t0, t1, done[0], done[1]})
      if (e) cudaEventDestroy(e);
  }
  void ensure(uint32_t n, uint32_t ntiles) {
    if (hst) return;  // a slot's sizes never change
    for (auto& l : lam) l.alloc(n);
    r.alloc(n);
    terms.alloc(n);
    carry.alloc(ntiles + 1);
    head.alloc(ntiles + 1);
    part1.alloc((size_t)ntiles * AdjointEpi::NACC + 4);
    part2.alloc((size_t)SPLIT_CTAS * AdjointEpi::NACC + 4);
    part3.alloc(3 * 1184 + 2);
    st.alloc(1);
    KNB_CUDA(cudaEventCreate(&t0));
    KNB_CUDA(cudaEventCreate(&t1));
    for (auto& e : done) KNB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    KNB_CUDA(cudaMallocHost(&hst, 2 * sizeof(IterState)));
  }
};

void pagerank_weights(GraphHandleImpl& g, const double* d_w, const PagerankParams& prm,
                      double* d_out, PagerankInfo* info, cudaStream_t s) {
  if (g.n == 0) return;
  const int which = pagerank_rows(g, prm.directed);
  const double lf = pagerank_loop_factor(which, prm.loops);
  GraphHandleImpl::WeightSlot& slot = g.weight_slot(which, lf, s);
  std::lock_guard<std::mutex> lock(slot.mu);
  g.fill_weights(*slot.op, d_w, lf, true, true, s);
  PagerankParams p = prm;
  p.weighted = true;
  p.relabel = false;  // values change every call: no renumbered copy
  pagerank_op(*slot.op, p, d_out, true, info, s);
}

void pagerank_grad(GraphHandleImpl& g, const double* d_w, const double* d_x, const double* d_gx,
                   const AdjointParams& prm, double* d_gw, double* d_lambda, AdjointInfo* info,
                   cudaStream_t s) {
  const uint32_t n = g.n;
  if (n == 0) return;
  const int which = pagerank_rows(g, prm.directed);
  const double lf = pagerank_loop_factor(which, prm.loops);
  // fwd: its column sums are the out-strengths; tr: pull along out-arcs
  const int twhich = which == 1 ? 0 : which;
  GraphHandleImpl::WeightSlot& fslot = g.weight_slot(which, lf, s);
  GraphHandleImpl::WeightSlot& tslot = g.weight_slot(twhich, lf, s);
  std::unique_lock<std::mutex> flock(fslot.mu, std::defer_lock), tlock(tslot.mu, std::defer_lock);
  if (&fslot == &tslot) flock.lock();
  else std::lock(flock, tlock);
  Operator* fwd = fslot.op.get();
  Operator* tr = tslot.op.get();
  // the sweeps pull over tr's values; of fwd only the out-strengths are read
  g.fill_weights(*tr, d_w, lf, true, tr == fwd, s);
  if (tr != fwd) g.fill_weights(*fwd, d_w, lf, false, true, s);
  constexpr int IPT = 4, WPB = 16;
  const Partition& P = tr->partition(32 * IPT, s);
  if (!fslot.adj_ws) fslot.adj_ws = std::make_unique<AdjointWorkspace>();
  AdjointWorkspace& W = *static_cast<AdjointWorkspace*>(fslot.adj_ws.get());
  W.ensure(n, P.ntiles);
  const double* jump = nullptr;
  if (prm.personalization && prm.dangling == 0) {
    if (!W.jump.p) W.jump.alloc(n);
    KNB_CUDA(cudaMemcpyAsync(W.jump.get(), prm.personalization, (size_t)n * 8,
                             cudaMemcpyDeviceToDevice, s));
    normalize_personalization_device(W.jump.get(), n, s);
    jump = W.jump.get();
  }
  IterState* st = W.st.get();
  KNB_CUDA(cudaEventRecord(W.t0, s));
  const unsigned gv = grid_for(n, 256, 1184);
  int launches = 0;
  // one CTA of 16 warps takes tiles until none is left; as many CTAs as fit
  // at once (against one tile per warp and 4 warps per CTA: 104 -> 79 us a
  // sweep on R-MAT 20)
  constexpr size_t smem = warp_smem_bytes<double, IPT, WPB>();
  const unsigned grid =
      std::min((P.ntiles + WPB - 1) / WPB, 148u * (unsigned)warp_min_blocks<double, IPT, WPB>());
  const OpView<double> v = tr->view64();
  fit_warp_carveout<double, double, AdjointEpi, IPT, WPB>();
  fit_warp_carveout<double, double, RowSumEpi, IPT, WPB>();
  const double dspan = std::pow(prm.damping, SPAN), c = dspan / (1.0 - dspan);
  const double stall = std::pow(prm.damping, CYCLE / 2);
  // Sweep k turns iterate k into iterate k + 1. Iterates alternate between
  // two buffers, but the two that an extrapolation looks back on (SPAN + 1
  // and SPAN sweeps before the end of a cycle) have buffers of their own.
  auto buffer = [&](int k) -> double* {
    const int at = k == 0 ? 0 : (k - 1) % CYCLE + 1;  // place in its cycle, 1..CYCLE
    return W.lam[at == CYCLE - SPAN - 1 ? 2 : at == CYCLE - SPAN ? 3 : k & 1].get();
  };
  int k = 0;
  auto enqueue = [&](int slot, bool extrapolate) {
    for (int q = 0; q < 8; ++q, ++k) {
      AdjointEpi e;
      e.g = d_gx;
      e.lam_old = buffer(k);
      e.lam_new = buffer(k + 1);
      e.inv_out = fwd->inv_out64.get();
      e.jump = jump;
      e.d = prm.damping;
      e.pu = 1.0 / n;
      launch_chained(warp_spmv<double, double, AdjointEpi, IPT, WPB>, grid, WPB * 32, smem, s, v,
                     buffer(k), e, P.coords.get(), P.ntiles, W.carry.get(), W.head.get(),
                     W.part1.get(), st, 0xFFFFFFFFu);
      launch_chained(split_rows<double, AdjointEpi>, split_grid(P.nsplit, P.nshort, grid),
                     SPMV_THREADS, 0, s, P.split.get(), P.nsplit, P.nshort, W.carry.get(),
                     W.head.get(), e, W.part1.get(), grid, W.part2.get(), st);
      launches += 2;
      if (extrapolate && (k + 1) % CYCLE == 0) {
        adj_extrapolate<<<gv, 256, 0, s>>>(W.lam[2].get(), W.lam[3].get(), buffer(k),
                                           buffer(k + 1), c, prm.damping, stall, jump, n,
                                           W.part3.get(), st);
        adj_take<<<gv, 256, 0, s>>>(W.lam[3].get(), buffer(k + 1), c, n, st);
        launches += 2;
      }
    }
    KNB_LAUNCH("adjoint sweep");
    KNB_CUDA(cudaMemcpyAsync(&W.hst[slot], st, sizeof(IterState), cudaMemcpyDeviceToHost, s));
    KNB_CUDA(cudaEventRecord(W.done[slot], s));
  };
  // one batch of sweeps in flight ahead of the state the host looks at;
  // sweeps after the end exit at once
  auto solve = [&](bool extrapolate) -> IterState {
    W.hst[0] = IterState{};
    W.hst[0].max_iter = (int32_t)std::min<int64_t>(prm.max_iter, INT32_MAX);
    KNB_CUDA(cudaMemcpyAsync(st, &W.hst[0], sizeof(IterState), cudaMemcpyHostToDevice, s));
    adj_init<<<gv, 256, 0, s>>>(d_gx, jump, n, prm.tol, W.lam[0].get(), W.part3.get(), st);
    KNB_LAUNCH("adj_init");
    ++launches;
    k = 0;
    enqueue(0, extrapolate);
    for (int slot = 0;; slot ^= 1) {
      enqueue(slot ^ 1, extrapolate);
      KNB_CUDA(cudaEventSynchronize(W.done[slot]));
      if (W.hst[slot].converged || W.hst[slot].stopped) {
        KNB_CUDA(cudaEventSynchronize(W.done[slot ^ 1]));
        break;
      }
    }
    return W.hst[0].iter > W.hst[1].iter ? W.hst[0] : W.hst[1];
  };
  IterState h = solve(true);
  // The cap counts the sweeps of the plain iteration, which st->prev_inv_total
  // foretells: only a solve that is clearly within it stands.
  if (h.ambiguous && !(h.converged && h.prev_inv_total + CYCLE <= (double)prm.max_iter))
    h = solve(false);
  if (!h.converged)
    throw Error("the PageRank adjoint did not converge within " + std::to_string(prm.max_iter) +
                " iterations");
  const double* lam_final = buffer(h.iter);
  // (M^T lambda)_j numerators with the final lambda, then the edge gradients
  {
    RowSumEpi e{W.r.get()};
    launch_chained(warp_spmv<double, double, RowSumEpi, IPT, WPB>, grid, WPB * 32, smem, s, v,
                   lam_final, e, P.coords.get(), P.ntiles, W.carry.get(), W.head.get(),
                   W.part1.get(), nullptr, 0xFFFFFFFFu);
    launch_chained(split_rows<double, RowSumEpi>, split_grid(P.nsplit, P.nshort, grid),
                   SPMV_THREADS, 0, s, P.split.get(), P.nsplit, P.nshort, W.carry.get(),
                   W.head.get(), e, W.part1.get(), grid, W.part2.get(), nullptr);
    adj_node_terms<<<grid_for(n, 256), 256, 0, s>>>(d_x, fwd->inv_out64.get(), W.r.get(), n,
                                                    prm.damping, W.terms.get());
    if (g.m)
      adj_grad<<<grid_for(g.m, 256), 256, 0, s>>>(g.src.get(), g.tgt.get(), g.m, lf,
                                                  W.terms.get(), lam_final, which != 1 ? 1 : 0,
                                                  d_gw);
    launches += 4;
    KNB_LAUNCH("adjoint gradient");
  }
  if (d_lambda)
    KNB_CUDA(cudaMemcpyAsync(d_lambda, lam_final, (size_t)n * 8, cudaMemcpyDeviceToDevice, s));
  KNB_CUDA(cudaEventRecord(W.t1, s));
  KNB_CUDA(cudaStreamSynchronize(s));
  float ms = 0;
  KNB_CUDA(cudaEventElapsedTime(&ms, W.t0, W.t1));
  if (info) {
    info->iterations = h.iter;
    info->change = h.change;
    info->seconds = ms * 1e-3;
    info->kernel_launches = launches;
  }
}

}  // namespace knb
