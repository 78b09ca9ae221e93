// Control kernels of the device-driven KKT solve.  One refined solve (condense, reduced solve
// with inner refinement against the unshifted Schur complement, recover, outer refinement against
// the original operator: kkt/condensed/kkt.rs:275-318 with kkt/refinement.rs:118-191) runs as ONE
// CUDA graph whose two refinement loops are WHILE conditional nodes.  After each straight run of
// the graph one kernel reduces the run's norms and one thread of its last block applies the
// reference's stopping rule (tolerance abstol + reltol |b|, stop when the residual ratio falls below stop_ratio,
// keep the candidate only when it improved, at most max_iter steps) and sets the loop's
// condition.  Every loop also stops once `guard` body executions have run, so no condition can
// stay set.  The arithmetic is the host driver's, operation for operation, so the graph's
// results equal the host-driven refinement's bit for bit.
#include "common.cuh"

__device__ __forceinline__ void ctl_set(cudaGraphConditionalHandle h, bool go) {
  cudaGraphSetConditional(h, go ? 1u : 0u);
}

// Start of a reduced solve: |r|max, |e|max, finite(x) of the first pass (and, at the head of a KKT
// solve, finite(bx), finite(bz)).  reset != 0 starts a new KKT solve.
__device__ void refine_head(const double* v, int rows, int reset, RefineCtl* c, const RefineParams& p,
                            cudaGraphConditionalHandle h) {
  if (reset) {
    RefineCtl z{};
    z.ok = 1;
    *c = z;
  }
  bool ok = c->ok != 0;
  for (int k = 3; k < rows; ++k)
    if (v[k] != 1.0) ok = false;
  if (v[2] != 1.0 || !isfinite(v[1])) ok = false;
  c->ok = ok ? 1 : 0;
  c->normb = v[0];
  c->norme = v[1];
  c->tol = p.abstol + p.reltol * c->normb;
  c->it = 0;
  c->accept = c->cont = 0;
  ctl_set(h, ok && !(c->norme <= c->tol) && p.max_iter > 0);
}

// After one inner step: |e2|max of the candidate's reduced residual.
__device__ void refine_step(double e, RefineCtl* c, const RefineParams& p, cudaGraphConditionalHandle h) {
  c->inner_steps++;
  c->guard++;
  bool go = false;
  int acc = 0;
  if (!isfinite(e)) {
    c->ok = 0;
  } else {
    const double ratio = c->norme / e;
    if (ratio < p.stop_ratio) {
      acc = ratio > 1.0;
    } else {
      acc = 1;
      c->norme = e;
      c->it++;
      go = !(e <= c->tol) && c->it < p.max_iter;
    }
  }
  if (c->guard >= p.guard_max) {
    go = false;
    c->ok = 0;
  }
  c->accept = acc;
  c->cont = go;
  ctl_set(h, go);
}

// After recover + full residual: |bx|, |bz|, |ex|, |ez|.
__device__ void refine_outer_init(const double* v, RefineCtl* c, const RefineParams& p,
                                  cudaGraphConditionalHandle h) {
  c->onormb = max_nan(v[0], v[1]);
  const double e = max_nan(v[2], v[3]);
  c->onorme = e;
  c->oit = 0;
  c->oaccept = c->ocont = 0;
  bool go = false;
  if (!isfinite(e)) {
    c->ok = 0;
  } else if (c->ok) {
    c->otol = p.abstol + p.reltol * c->onormb;
    go = !(e <= c->otol) && p.max_iter > 0;
  }
  ctl_set(h, go);
}

// After one outer correction: |ex2|, |ez2| of the candidate's full residual.
__device__ void refine_outer_step(const double* v, RefineCtl* c, const RefineParams& p,
                                  cudaGraphConditionalHandle h) {
  c->outer_steps++;
  c->guard++;
  bool go = false;
  int acc = 0;
  if (c->ok) {  // the correction's own solve passed its checks
    const double e = max_nan(v[0], v[1]);
    if (!isfinite(e)) {
      c->ok = 0;
    } else {
      const double ratio = c->onorme / e;
      if (ratio < p.stop_ratio) {
        acc = ratio > 1.0;
      } else {
        acc = 1;
        c->onorme = e;
        c->oit++;
        go = !(e <= c->otol) && c->oit < p.max_iter;
      }
    }
  }
  if (c->guard >= p.guard_max) {
    go = false;
    c->ok = 0;
  }
  c->oaccept = acc;
  c->ocont = go;
  ctl_set(h, go);
}

// The norms of one control point and the control itself in one launch: grid row r is request r
// (largest magnitude, NaN kept, or all finite, both independent of the order of combination), the block that
// arrives last folds every row, one thread of it applies the stopping rule and sets the loop's
// condition, and after an inner step the block keeps the candidate and its residual (n entries).
// A graph node costs about 3 us here whatever it computes, and a refined solve of a small system is
// little else: norms, control and copy were three nodes each time.
// Both kinds of request are a maximum of unsigned integers: a magnitude's bits (max_nan), or 1 for an entry
// that is not finite.  The copy has eight loads of each vector in flight a thread: 2048 entries a memory round
// trip, so that one block is enough beside the matrix products of a step.
extern "C" __global__ void __launch_bounds__(256)
k_refine(RedBatch b, double* __restrict__ partial, unsigned* __restrict__ ticket, int pitch, RefineOp op,
         RefineCtl* c, RefineParams p, cudaGraphConditionalHandle h) {
  typedef unsigned long long u64;
  __shared__ u64 red[8];
  __shared__ double val[kRedBatchMax];
  __shared__ int last, keep[2];
  const RedReq q = b.r[blockIdx.y];
  const bool fin = q.op == 3;  // RED_FINITE, else RED_MAXABS
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  u64* part = reinterpret_cast<u64*>(partial);
  u64 acc = 0;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < q.n; i += (long)gridDim.x * blockDim.x) {
    const u64 v = (u64)__double_as_longlong(q.x[i]) & ~(1ull << 63);
    acc = max(acc, fin ? (u64)(v >= 0x7ff0000000000000ull) : v);
  }
  for (int o = 16; o > 0; o >>= 1) acc = max(acc, __shfl_xor_sync(0xffffffffu, acc, o));
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) acc = max(acc, red[w]);
    part[blockIdx.y * pitch + blockIdx.x] = acc;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x * gridDim.y - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int r = warp; r < op.rows; r += 8) {
    u64 v = 0;
    for (int k = lane; k < (int)gridDim.x; k += 32) v = max(v, __ldcg(part + r * pitch + k));
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) val[r] = b.r[r].op == 3 ? (v ? 0.0 : 1.0) : __longlong_as_double((long long)v);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *ticket = 0u;
    if (op.kind == REFINE_HEAD) refine_head(val, op.rows, op.reset, c, p, h);
    else if (op.kind == REFINE_STEP) refine_step(val[0], c, p, h);
    else if (op.kind == REFINE_OUTER_INIT) refine_outer_init(val, c, p, h);
    else refine_outer_step(val, c, p, h);
    keep[0] = op.kind == REFINE_STEP && c->accept;
    keep[1] = op.kind == REFINE_STEP && c->cont;
  }
  __syncthreads();
  const bool k0 = keep[0], k1 = keep[1];
  if (!k0 && !k1) return;
  for (long i0 = threadIdx.x; i0 < op.n; i0 += 8 * 256) {
    double y[8], f[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const bool in = i0 + 256 * u < op.n;
      y[u] = in && k0 ? op.cand[i0 + 256 * u] : 0.0;
      f[u] = in && k1 ? op.e2[i0 + 256 * u] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const bool in = i0 + 256 * u < op.n;
      if (in && k0) op.x[i0 + 256 * u] = y[u];
      if (in && k1) op.e[i0 + 256 * u] = f[u];
    }
  }
}

// After an outer step: x1 <- y1 (n entries) and x2 <- y2 (m) when the candidate is kept, e1 <- f1 and
// e2 <- f2 when the loop goes on.
extern "C" __global__ void k_refine_keep(const RefineCtl* c, long n, double* x1, const double* y1, double* e1,
                                         const double* f1, long m, double* x2, const double* y2, double* e2,
                                         const double* f2) {
  const bool a = c->oaccept != 0, b = c->ocont != 0;
  if (!a && !b) return;
  const long stride = (long)gridDim.x * blockDim.x;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n + m; i += stride) {
    if (i < n) {
      if (a) x1[i] = y1[i];
      if (b) e1[i] = f1[i];
    } else {
      if (a) x2[i - n] = y2[i - n];
      if (b) e2[i - n] = f2[i - n];
    }
  }
}
