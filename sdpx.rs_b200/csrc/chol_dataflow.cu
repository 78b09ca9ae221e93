// Persistent dataflow Cholesky of the dense Schur complement, H = U'U (upper, 64 x 64 tiles).
//
// The reference factors the reduced KKT matrix with a right-looking tiled Cholesky
// (dense_block.rs:515-594: potrf on the diagonal tile, trsm on the tile row, syrk/gemm on the
// trailing tiles, dynamic pivot rule potrf_dynamic 334-365).  At the sizes of the condensed
// system (m of a few thousand) that chain is latency-bound: every diagonal tile waits for the
// previous step's trailing update.  Here the whole factorization is ONE launch:
//
//  * the critical path -- POTRF(k), TRSM(k, k+1) and the last update of tile (k+1, k+1) for every
//    k -- is ONE work item, the chain (ticket 0): a single CTA keeps the diagonal tile, U_kk^-T
//    and U(k, k+1) in shared memory from one step to the next;
//  * every other tile is one item, taken by an atomic ticket: its whole sum over the earlier tile
//    rows, left-looking, in registers (the tile is read and written once, its operands stream
//    through a two-stage shared-memory ring), then FULL(i, j > i+1): U(i, j) = U_ii^-T (...), or
//    PRE(i, i) and PRE(i, i+1): the sum up to what the chain adds itself;
//  * the inverse of the factor, X = U^-1, is part of the same launch: INV(i, j) forms
//    X(i, j) = -(sum_{i <= s < j} X(i, s) U(s, j)) X(j, j) (INV(j, j) copies X(j, j)), a few tile rows
//    behind the factorization, on SMs that would wait for the chain.  A launch pair per level of a
//    recursive inverse after the factorization took 390 us at m = 2000 and 1450 at m = 4000;
//  * progress words in global memory (acquire/release at GPU scope): prog[j] counts the final
//    tiles of tile column j of U from the top (a tile is final only after the one above it),
//    xprog[i] those of tile row i of X up to the column, one flag per PRE tile.  Every item's inputs
//    come from earlier tickets or from chain steps whose own inputs do, and a ticket is only taken by
//    a running CTA, so the schedule cannot deadlock;
//  * every wait is bounded: past the limit the CTA sets SDPXG_ST_SYNC_TIMEOUT and the shared
//    error word, and every CTA leaves at its next wait;
//  * ten warps: eight work on the FP64 tensor cores (mma.sync m8n8k4 f64), warp 8 polls the
//    progress words and streams operands (cp.async, completion on an mbarrier), warp 9 publishes the
//    chain's results (a GPU-scope fence takes about a microsecond that the chain does not wait).
//
// What bounds it: below m of about 3000 the chain (15 us a step: POTRF 9, TRSM 2, the update of the
// next diagonal tile 2.2, stores 1), above it the tensor-pipe time of the tile sums (one 64^3
// product is 2.1 us of an SM's FP64 pipe).  Right-looking with every tile task reloaded from L2 and
// the inverse of the diagonal tiles formed after the panels the factor alone took 27 us a step:
// m = 1024 457 us, 2000 864, 4000 3206; so 242, 486 and 1274, and with the whole inverse 248, 533 and
// 2115.  Holding U_kk^-T back to copy it out by one warp was slower (627 at m = 2000): the tiles of
// row k wait for it.
#include "chol_publish.cuh"
#include "common.cuh"

#define DF_NB 64
#define DF_LD 68          // 68 = 4 mod 16: the fragment reads of a half-warp hit distinct banks
#define DF_MMA 256        // 8 warps: one 8-column block of a 64 x 64 output tile each
#define DF_THREADS 320
#define DF_TILE (DF_NB * DF_LD)
#define DF_SPIN_LIMIT (1 << 22)
#define DF_WAIT_NS 20000000000ull
#define DFS(A, i, j) (A)[(i) + (j) * DF_LD]

enum : unsigned { DF_INV = 0u, DF_FULL = 1u, DF_PRE = 2u, DF_CHAIN = 3u };

namespace {

struct DfShared {
  uint64_t full[2], empty[2];  // ring stages (chain: 0 the tile (k, k+1), 1 the tile (k+1, k+1))
  uint64_t pub[chol_publish::kSlots];  // chain: the eight warps' stores of a publication are issued
  int item, abort, fail;
};

__device__ __forceinline__ int df_ld_acquire(const int* p) {
  int v;
  asm volatile("ld.global.acquire.gpu.b32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void df_st_release(int* p, int v) {
  asm volatile("st.global.release.gpu.b32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}

// One thread: poll *flag until it reaches target; its value, or -1 when another CTA raised the
// error word or the poll limit was reached (then the error word and the status are set).
__device__ int df_wait(const int* flag, int target, int* err, uint32_t* status) {
  for (int it = 0; it < DF_SPIN_LIMIT; ++it) {
    const int v = df_ld_acquire(flag);
    if (v >= target) return v;
    if ((it & 15) == 15 && df_ld_acquire(err) != 0) return -1;  // each load is a round trip to L2
    __nanosleep(it < 64 ? 20 : 100);
  }
  atomicOr(status, SDPXG_ST_SYNC_TIMEOUT);
  atomicExch(err, 1);
  return -1;
}

// ---- CTA-level synchronisation ----
__device__ __forceinline__ uint32_t df_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void df_bar_init(uint64_t* b, int count) {
  asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"(df_smem(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void df_bar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared.b64 _, [%0];" ::"r"(df_smem(b)) : "memory");
}
__device__ __forceinline__ unsigned long long df_time() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// Wait for the phase of parity `par`; false once the CTA aborts (the side that would complete the
// phase has given up) or past the time limit.
__device__ bool df_bar_wait(uint64_t* b, uint32_t par, DfShared* sh) {
  unsigned long long t0 = 0;
  for (uint32_t it = 0;; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(df_smem(b)), "r"(par)
        : "memory");
    if (ok) return *(volatile int*)&sh->abort == 0;
    if (*(volatile int*)&sh->abort) return false;
    if ((it & 1023u) == 1023u) {
      const unsigned long long t = df_time();
      if (t0 == 0) t0 = t;
      if (t - t0 > DF_WAIT_NS) {
        *(volatile int*)&sh->abort = 2;
        return false;
      }
    }
  }
}
template <int ID, int N>
__device__ __forceinline__ void df_sync() {
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(N) : "memory");
}
template <int ID, int N>
__device__ __forceinline__ void df_arrive() {
  asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"(N) : "memory");
}
enum { BAR_MMA = 1, BAR_PANEL = 2, BAR_ROW = 3, BAR_REST = 4 };
// BAR_MMA with a vote: true when every MMA thread says so (one decision for all eight warps).
__device__ __forceinline__ bool df_all(bool ok) {
  uint32_t v;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(v)
      : "r"(ok ? 1u : 0u), "n"((int)BAR_MMA), "n"((int)DF_MMA)
      : "memory");
  return v != 0;
}

// One warp: 64 x 64 tile from global (column-major, leading dimension ld, even, so every column of
// a tile starts on 16 bytes) into shared memory through L2 (other SMs wrote it); 16-byte pieces of
// columns >= nc or starting at rows >= nr are zeroed.  Completion arrives on `full`, once per lane.
__device__ __forceinline__ void df_stream_tile(double* S, const double* __restrict__ G, long ld, int nr, int nc) {
  const int lane = threadIdx.x & 31;
#pragma unroll 8
  for (int c = 0; c < DF_NB; ++c) {
    const bool in = c < nc && 2 * lane < nr;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(df_smem(&DFS(S, 2 * lane, c))),
                 "l"(in ? G + (long)c * ld + 2 * lane : G), "r"(in ? 16 : 0)
                 : "memory");
  }
}
__device__ __forceinline__ void df_stream_done(uint64_t* full) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(df_smem(full)) : "memory");
}

// ---- tile products ----
// acc (this warp's 8-column block w of a 64 x 64 output) -= A' B over K = 64.
// Fragments (m8n8k4 f64): lane l holds A[l/4][l%4], B[l%4][l/4], C[l/4][2(l%4) + {0,1}].
__device__ __forceinline__ void df_sub_atb(const double* As, const double* Bs, double (&acc)[8][2]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int q = lane & 3, r = lane >> 2;
#pragma unroll 4
  for (int ks = 0; ks < DF_NB / 4; ++ks) {
    const int kk = ks * 4 + q;
    const double b = -DFS(Bs, kk, 8 * w + r);
#pragma unroll
    for (int R = 0; R < 8; ++R) dmma_m8n8k4(acc[R][0], acc[R][1], DFS(As, kk, 8 * R + r), b);
  }
}

// acc (this warp's 8-column block w) -= A B over K = 64.
__device__ __forceinline__ void df_sub_ab(const double* As, const double* Bs, double (&acc)[8][2]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int q = lane & 3, r = lane >> 2;
#pragma unroll 4
  for (int ks = 0; ks < DF_NB / 4; ++ks) {
    const int kk = ks * 4 + q;
    const double b = -DFS(Bs, kk, 8 * w + r);
#pragma unroll
    for (int R = 0; R < 8; ++R) dmma_m8n8k4(acc[R][0], acc[R][1], DFS(As, 8 * R + r, kk), b);
  }
}

// The packed upper triangle u of an 8 x 8 block factored in place, v <- U^-T v.  Returns false (u
// and v then unusable) when a pivot does not lie in (floor, 2^1000].
__device__ __forceinline__ bool df_factor8(double (&u)[36], double (&v)[8], double floor) {
  bool ok = true;
#pragma unroll
  for (int kk = 0; kk < 8; ++kk) {
    const double d = u[kk * (kk + 3) / 2];
    ok = ok && d > floor && d <= 0x1p1000;
    const double ri = rsqrt_mid(d);
    u[kk * (kk + 3) / 2] = d * ri;
#pragma unroll
    for (int j = kk + 1; j < 8; ++j) u[j * (j + 1) / 2 + kk] *= ri;  // row kk of U
    v[kk] *= ri;
#pragma unroll
    for (int j = kk + 1; j < 8; ++j)
#pragma unroll
      for (int i = kk + 1; i <= j; ++i)
        u[j * (j + 1) / 2 + i] -= u[i * (i + 1) / 2 + kk] * u[j * (j + 1) / 2 + kk];
#pragma unroll
    for (int i = kk + 1; i < 8; ++i) v[i] -= u[i * (i + 1) / 2 + kk] * v[kk];
  }
  return ok;
}

// The same block under the dynamic pivot rule, off the common path: a pivot within eps of zero
// becomes delta unless it is clearly negative; non-finite or non-positive pivots fail.
__device__ __noinline__ void df_factor8_rule(const double* A, int p, int c, double* u, double* v, int nb,
                                             const double* diag, double eps, double delta, int dynamic, bool* fail) {
  for (int j = 0; j < 8; ++j) {
    v[j] = (j == c) ? 1.0 : 0.0;
    for (int i = 0; i <= j; ++i) u[j * (j + 1) / 2 + i] = DFS(A, 8 * p + i, 8 * p + j);
  }
  for (int kk = 0; kk < 8; ++kk) {
    double d = u[kk * (kk + 3) / 2];
    if (8 * p + kk < nb) {
      if (!isfinite(d)) {
        *fail = true;
        d = 1.0;
      } else if (dynamic && d <= eps) {
        if (d < -64.0 * 2.220446049250313e-16 * nb * fabs(diag[8 * p + kk])) *fail = true;
        else d = delta;
      }
      if (!(d > 0.0)) {
        *fail = true;
        d = 1.0;
      }
    }
    const double ri = rsqrt(d);
    u[kk * (kk + 3) / 2] = d * ri;
    for (int j = kk + 1; j < 8; ++j) u[j * (j + 1) / 2 + kk] *= ri;
    v[kk] *= ri;
    for (int j = kk + 1; j < 8; ++j)
      for (int i = kk + 1; i <= j; ++i) u[j * (j + 1) / 2 + i] -= u[i * (i + 1) / 2 + kk] * u[j * (j + 1) / 2 + kk];
    for (int i = kk + 1; i < 8; ++i) v[i] -= u[i * (i + 1) / 2 + kk] * v[kk];
  }
}

// Warp 0: factor the 8 x 8 diagonal block of panel p in registers.  Every lane factors the whole
// block (packed upper triangle, static indices, no shuffles and no branches on the pivot chain; a
// pivot that needs the rule takes the block through df_factor8_rule) and lane c < 8 carries column
// c of the identity through the same elimination, which leaves column c of U_pp^-T: the inverse
// costs the chain nothing.  One reciprocal root per pivot: sqrt(d) = d / sqrt(d).
// Wd[kk + 8 r] = U_pp^-1(kk, r).
__device__ __forceinline__ void df_panel_factor(double* A, double* Wd, int p, int nb, const double* diag, double eps,
                                                double delta, int dynamic, int* s_fail) {
  const int lane = threadIdx.x & 31, c = lane & 7;
  double u[36], v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i <= j; ++i) u[j * (j + 1) / 2 + i] = DFS(A, 8 * p + i, 8 * p + j);
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = (i == c) ? 1.0 : 0.0;
  if (!df_factor8(u, v, dynamic ? fmax(eps, 0x1p-1000) : 0x1p-1000)) {
    double su[36], sv[8];
    bool fail = false;
    df_factor8_rule(A, p, c, su, sv, nb, diag, eps, delta, dynamic, &fail);
    if (fail && lane == 0) *s_fail = 1;
#pragma unroll
    for (int i = 0; i < 36; ++i) u[i] = su[i];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = sv[i];
    __syncwarp();
  }
  if (lane == 0) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int i = 0; i <= j; ++i) DFS(A, 8 * p + i, 8 * p + j) = u[j * (j + 1) / 2 + i];
  }
  if (lane < 8) {
#pragma unroll
    for (int i = 0; i < 8; ++i) Wd[c + 8 * i] = v[i];  // U^-T(i, c) = U^-1(c, i)
  }
}

// One 8 x 8 block (one warp): M[P, J] = W' M[P, J].
__device__ __forceinline__ void df_block_row(double* M, const double* Wd, int p, int J) {
  const int lane = threadIdx.x & 31, q = lane & 3, r = lane >> 2;
  double c0 = 0.0, c1 = 0.0, d0 = 0.0, d1 = 0.0;  // two chains: a dependent DMMA waits 59 cycles
  dmma_m8n8k4(c0, c1, Wd[q + 8 * r], DFS(M, 8 * p + q, 8 * J + r));
  dmma_m8n8k4(d0, d1, Wd[q + 4 + 8 * r], DFS(M, 8 * p + q + 4, 8 * J + r));
  __syncwarp();
  DFS(M, 8 * p + r, 8 * J + 2 * q) = c0 + d0;
  DFS(M, 8 * p + r, 8 * J + 2 * q + 1) = c1 + d1;
}
// One 8 x 8 block (one warp): A[I, I] -= A[P, I]' A[P, I].
__device__ __forceinline__ void df_block_diag(double* A, int p, int I) {
  const int lane = threadIdx.x & 31, q = lane & 3, r = lane >> 2;
  double c0 = DFS(A, 8 * I + r, 8 * I + 2 * q), c1 = DFS(A, 8 * I + r, 8 * I + 2 * q + 1), d0 = 0.0, d1 = 0.0;
  const double a = DFS(A, 8 * p + q, 8 * I + r), b = DFS(A, 8 * p + q + 4, 8 * I + r);
  dmma_m8n8k4(c0, c1, -a, a);
  dmma_m8n8k4(d0, d1, -b, b);
  DFS(A, 8 * I + r, 8 * I + 2 * q) = c0 + d0;
  DFS(A, 8 * I + r, 8 * I + 2 * q + 1) = c1 + d1;
}

// The trailing blocks of panel p that warps 1..7 update, five at most each: A[I, J], p < I <= J, but
// (p+1, p+1) (warp 0's), then Y[I, C], I > p, C <= p.  Entry: I | J << 3, 64 for Y, 128 for a block
// that starts from zero (C = p).
struct DfTrail {
  unsigned char n[7], e[7][35];
};
constexpr DfTrail df_trail() {
  DfTrail t{};
  for (int p = 0; p < 7; ++p) {
    int n = 0;
    for (int I = p + 1; I < 8; ++I)
      for (int J = I; J < 8; ++J)
        if (I != p + 1 || J != p + 1) t.e[p][n++] = (unsigned char)(I | J << 3);
    for (int I = p + 1; I < 8; ++I)
      for (int C = 0; C <= p; ++C) t.e[p][n++] = (unsigned char)(I | C << 3 | 64 | (C == p ? 128 : 0));
    t.n[p] = (unsigned char)n;
  }
  return t;
}
__constant__ DfTrail kDfTrail = df_trail();

// One warp of seven (index g): its blocks -= U[P, I]' M[P, J], all five at once so that the
// operand loads and the tensor-pipe latency overlap.
__device__ __forceinline__ void df_trailing(double* A, double* Y, int p, int g) {
  const int lane = threadIdx.x & 31, q = lane & 3, r = lane >> 2, n = kDfTrail.n[p];
  double c0[5], c1[5], a[5][2], b[5][2];
  double* out[5];
#pragma unroll
  for (int u = 0; u < 5; ++u) {
    const int t = g + 7 * u;
    if (t < n) {
      const int e = kDfTrail.e[p][t], I = e & 7, J = (e >> 3) & 7;
      double* M = (e & 64) ? Y : A;
      out[u] = &DFS(M, 8 * I + r, 8 * J + 2 * q);
      c0[u] = (e & 128) ? 0.0 : out[u][0];
      c1[u] = (e & 128) ? 0.0 : out[u][DF_LD];
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) {
        a[u][ks] = -DFS(A, 8 * p + 4 * ks + q, 8 * I + r);
        b[u][ks] = DFS(M, 8 * p + 4 * ks + q, 8 * J + r);
      }
    }
  }
#pragma unroll
  for (int ks = 0; ks < 2; ++ks)
#pragma unroll
    for (int u = 0; u < 5; ++u)
      if (g + 7 * u < n) dmma_m8n8k4(c0[u], c1[u], a[u][ks], b[u][ks]);
#pragma unroll
  for (int u = 0; u < 5; ++u)
    if (g + 7 * u < n) {
      out[u][0] = c0[u];
      out[u][DF_LD] = c1[u];
    }
}

// Factor the diagonal tile in A (upper triangle valid) in place, A <- U, and Y <- U^-T (lower
// triangle of 8 x 8 blocks, zeros above the diagonal inside the diagonal blocks), by the 8 MMA
// warps.  Panels of 8 columns.  Warp 0 is the chain: it factors panel p's diagonal block, forms
// U(p, p+1), updates diagonal block p+1 with it and goes on to panel p+1; the other seven warps
// follow one panel behind (the rest of row p, row p of Y, then the trailing blocks of both), and
// warp 0 waits for them only before it touches row p+1.  Wd: two 8 x 8 buffers.
__device__ void df_potrf_tile(double* A, double* Y, double* Wd, int nb, const double* diag, double eps, double delta,
                              int dynamic, int* s_fail) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (w == 0) {
    for (int p = 0; p < 8; ++p) {
      double* W = Wd + (p & 1) * 64;
      df_panel_factor(A, W, p, nb, diag, eps, delta, dynamic, s_fail);
      __syncwarp();
      if (p > 0) df_sync<BAR_REST, DF_MMA>();  // panel p-1 is applied to the blocks below row p
      if (p < 7) {
        df_block_row(A, W, p, p + 1);
        __syncwarp();
        df_block_diag(A, p, p + 1);
        __syncwarp();
      }
      df_arrive<BAR_PANEL, DF_MMA>();
    }
  } else {
    for (int p = 0; p < 8; ++p) {
      const double* W = Wd + (p & 1) * 64;
      df_sync<BAR_PANEL, DF_MMA>();
      const int na = p < 6 ? 6 - p : 0;
      for (int t = w - 1; t < na + p + 1; t += 7) {
        if (t < na) {
          df_block_row(A, W, p, p + 2 + t);
        } else if (t - na < p) {
          df_block_row(Y, W, p, t - na);
        } else {  // Y[P, P] = U_pp^-T
          for (int e = lane; e < 64; e += 32) DFS(Y, 8 * p + (e & 7), 8 * p + (e >> 3)) = W[(e >> 3) + 8 * (e & 7)];
        }
      }
      if (p == 7) break;
      df_sync<BAR_ROW, DF_MMA - 32>();
      df_trailing(A, Y, p, w - 1);
      df_arrive<BAR_REST, DF_MMA>();
    }
  }
}

// The critical path of the factorization, step k = 0 .. nt-1, in one CTA:
//   POTRF: factor the diagonal tile in T0, U_kk^-T in T1, which is stored (U_kk itself is read by
//   nobody: the solves go through the inverse);
//   TRSM(k, k+1): U(k, k+1) = U_kk^-T H(k, k+1) over the tile that warp 8 brought into T2 while
//   POTRF ran (sums of steps < k done by PRE(k, k+1)); warp 9 publishes it;
//   the next diagonal tile = (tile (k+1, k+1) in T3, sums of steps < k) - U(k, k+1)' U(k, k+1),
//   upper blocks only, into T0.
// Products with the triangular U_kk^-T skip its zero blocks.
__device__ void df_chain(double* __restrict__ F, long ld, int m, int nt, int* prog, int* pre_d, int* pre_o, int* err,
                         double eps, double delta, int dynamic, const double* __restrict__ diag0,
                         double* __restrict__ Dinv, uint32_t* __restrict__ status, double* T, double* Wd,
                         DfShared* sh) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *As = T, *Ys = T + DF_TILE, *Bs = T + 2 * DF_TILE, *Cs = T + 3 * DF_TILE;
  if (warp == 8) {  // brings the next tiles
    for (int k = 0; k + 1 < nt; ++k) {
      const int k0 = k * DF_NB, j0 = k0 + DF_NB, nc = min(DF_NB, m - j0);
      for (int x = 0; x < 2; ++x) {
        int ok = 1;
        if (lane == 0) {
          const int* flag = x == 0 ? pre_o + k : pre_d + k + 1;
          if (k >= 1 && df_wait(flag, 1, err, status) < 0) ok = 0;
          if (!ok) *(volatile int*)&sh->abort = 1;
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        __syncwarp();
        if (!ok || !df_bar_wait(&sh->empty[x], (k & 1) ^ 1, sh)) return;
        if (x == 0) df_stream_tile(Bs, F + k0 + (long)j0 * ld, ld, DF_NB, nc);
        else df_stream_tile(Cs, F + j0 + (long)j0 * ld, ld, nc, nc);
        df_stream_done(&sh->full[x]);
      }
    }
    return;
  }
  if (warp == 9) {  // publishes what the MMA warps stored
    if (lane != 0) return;
    for (int t = 0; t + 1 < 2 * nt; ++t) {
      const int k = t >> 1;
      if (!df_bar_wait(&sh->pub[chol_publish::slot(t)], chol_publish::parity(t), sh)) return;
      __threadfence();
      if (t & 1) df_st_release(prog + k + 1, k + 1);
      else df_st_release(prog + k, k + 1);
    }
    return;
  }
  const int w = warp, q = lane & 3, r = lane >> 2;
  for (int e = threadIdx.x; e < DF_NB * DF_NB; e += DF_MMA) {  // the first diagonal tile
    const int row = e & 63, col = e >> 6, nb = min(DF_NB, m);
    DFS(As, row, col) = (row < nb && col < nb) ? __ldcg(F + row + (long)col * ld) : (row == col ? 1.0 : 0.0);
  }
  df_sync<BAR_MMA, DF_MMA>();
  for (int k = 0; k < nt; ++k) {
    const int k0 = k * DF_NB, nb = min(DF_NB, m - k0);
    df_potrf_tile(As, Ys, Wd, nb, diag0 + k0, eps, delta, dynamic, &sh->fail);
    df_sync<BAR_MMA, DF_MMA>();
    if (*(volatile int*)&sh->fail) {  // the dependants leave at their next wait
      if (threadIdx.x == 0) {
        atomicOr(status, SDPXG_ST_PIVOT_FAIL);
        atomicExch(err, 1);
        *(volatile int*)&sh->abort = 1;
      }
      return;
    }
    {  // U_kk^-T, zero above the diagonal: the tiles of row k wait for it
      double2* D = reinterpret_cast<double2*>(Dinv + (long)k * DF_NB * DF_NB);
      const int row = 2 * lane;
#pragma unroll
      for (int c = w; c < DF_NB; c += 8) {
        double2 v = *reinterpret_cast<const double2*>(&DFS(Ys, row, c));
        if (row < c || row >= nb) v.x = 0.0;
        if (row + 1 < c || row + 1 >= nb) v.y = 0.0;
        D[c * (DF_NB / 2) + lane] = v;
      }
    }
    __syncwarp();
    if (lane == 0) df_bar_arrive(&sh->pub[chol_publish::slot(2 * k)]);
    if (k + 1 >= nt) return;
    const int j0 = k0 + DF_NB, nc = min(DF_NB, m - j0);
    if (!df_all(df_bar_wait(&sh->full[0], k & 1, sh))) return;
    double t[8][2] = {};
#pragma unroll
    for (int ks = 0; ks < DF_NB / 4; ++ks) {
      const int kk = ks * 4 + q;
      const double b = DFS(Bs, kk, 8 * w + r);
#pragma unroll
      for (int R = 0; R < 8; ++R)
        if (R >= ks / 2) dmma_m8n8k4(t[R][0], t[R][1], DFS(Ys, 8 * R + r, kk), b);
    }
    __syncwarp();  // this warp's columns of T2 are read by this warp alone
#pragma unroll
    for (int R = 0; R < 8; ++R)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int row = 8 * R + r, col = 8 * w + 2 * q + e;
        const double v = (col < nc) ? t[R][e] : 0.0;
        DFS(Bs, row, col) = v;
        if (col < nc) F[(k0 + row) + (long)(j0 + col) * ld] = v;
      }
    __syncwarp();
    if (lane == 0) df_bar_arrive(&sh->pub[chol_publish::slot(2 * k + 1)]);
    df_sync<BAR_MMA, DF_MMA>();
    if (!df_all(df_bar_wait(&sh->full[1], k & 1, sh))) return;
    {  // upper 8 x 8 blocks (R, J), numbers w, w + 8, ... of 36: up to five at once
      double c0[5], c1[5];
      int Rb[5], Jb[5];
      const int nblk = w < 4 ? 5 : 4;
#pragma unroll
      for (int u = 0; u < 5; ++u) {
        int J = 0, R = w + 8 * u;
        while (R > J) {
          R -= J + 1;
          ++J;
        }
        Rb[u] = R;
        Jb[u] = J;
        const int row = 8 * R + r, col = 8 * J + 2 * q;
        const bool on = u < nblk && row < nc;
        c0[u] = on && col < nc ? DFS(Cs, row, col) : 0.0;
        c1[u] = on && col + 1 < nc ? DFS(Cs, row, col + 1) : 0.0;
      }
#pragma unroll 4
      for (int ks = 0; ks < DF_NB / 4; ++ks) {
        const int kk = ks * 4 + q;
#pragma unroll
        for (int u = 0; u < 5; ++u)
          if (u < nblk) dmma_m8n8k4(c0[u], c1[u], -DFS(Bs, kk, 8 * Rb[u] + r), DFS(Bs, kk, 8 * Jb[u] + r));
      }
#pragma unroll
      for (int u = 0; u < 5; ++u)
        if (u < nblk) {
          const int row = 8 * Rb[u] + r, col = 8 * Jb[u] + 2 * q;
          DFS(As, row, col) = (row == col && row >= nc) ? 1.0 : c0[u];
          DFS(As, row, col + 1) = (row == col + 1 && row >= nc) ? 1.0 : c1[u];
        }
    }
    df_sync<BAR_MMA, DF_MMA>();
    if (threadIdx.x == 0) {
      df_bar_arrive(&sh->empty[0]);
      df_bar_arrive(&sh->empty[1]);
    }
  }
}

}  // namespace

// items[t] = type << 30 | k << 20 | i << 10 | j (topological order, built on the host):
//   FULL (k = i): U(i, j) = U_ii^-T (H(i, j) - sum_{s < i} U(s, i)' U(s, j));
//   PRE: H(i, j) -= sum_{s < k} U(s, i)' U(s, j), for j = i (k = i - 1) and j = i + 1 (k = i);
//   INV: X(i, j) into Uinv and, transposed, UinvT (n x n, leading dimension m), and into Xr, from
//   which later INV items read it.
// F and Xr: even leading dimensions ld and ldx (Xr may be Uinv when m is even).
// sync = {ticket, error, prog[nt], pre_o[nt], pre_d[nt], xprog[nt]}, zero at launch.
extern "C" __global__ void __launch_bounds__(DF_THREADS, 1)
k_chol_dataflow(double* __restrict__ F, long ld, int m, int nt, const unsigned* __restrict__ items, int nitems,
                int* __restrict__ sync, double eps, double delta, int dynamic, const double* __restrict__ diag0,
                double* __restrict__ Dinv, double* Xr, long ldx, double* Uinv, double* UinvT,
                uint32_t* __restrict__ status) {
  extern __shared__ __align__(16) double df_sm[];
  __shared__ DfShared sh;
  double* T = df_sm;                  // four tiles: two ring stages of two operands
  double* Wd = df_sm + 4 * DF_TILE;
  int* ticket = sync;
  int* err = sync + 1;
  int* prog = sync + 2;
  int* pre_o = prog + nt;
  int* pre_d = pre_o + nt;
  int* xprog = pre_d + nt;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, q = lane & 3, r = lane >> 2;
  unsigned cnt = 0;  // ring stages used so far
  bool ring = false;

  for (;;) {
    if (threadIdx.x == 0) sh.item = atomicAdd(ticket, 1);
    __syncthreads();
    const int t = sh.item;
    if (t >= nitems) break;
    const unsigned code = items[t];
    const int type = (int)(code >> 30);
    const int i = (int)((code >> 10) & 1023u), j = (int)(code & 1023u);
    if (!ring) {  // the chain's tiles are released by one thread, the ring's by the eight warps
      if (threadIdx.x == 0) {
        for (int x = 0; x < 2; ++x) {
          df_bar_init(&sh.full[x], 32);
          df_bar_init(&sh.empty[x], type == (int)DF_CHAIN ? 1 : 8);
        }
        for (int x = 0; x < chol_publish::kSlots; ++x) df_bar_init(&sh.pub[x], 8);
        sh.abort = sh.fail = 0;
      }
      __syncthreads();
      ring = true;
    }
    if (type == (int)DF_CHAIN) {
      df_chain(F, ld, m, nt, prog, pre_d, pre_o, err, eps, delta, dynamic, diag0, Dinv, status, T, Wd, &sh);
      __syncthreads();
      if (threadIdx.x == 0 && sh.abort == 2) {
        atomicOr(status, SDPXG_ST_SYNC_TIMEOUT);
        atomicExch(err, 1);
      }
      break;  // this CTA's barriers belong to the chain
    }
    const int i0 = i * DF_NB, j0 = j * DF_NB;
    const int ni = min(DF_NB, m - i0), nc = min(DF_NB, m - j0);
    const bool full = type == (int)DF_FULL, inv = type == (int)DF_INV;
    // tile rows s0 .. s1-1 of the sum, then one more stage with the tile U_dd^-T (d = i or j)
    const int s0 = inv ? i : 0, s1 = inv ? j : (int)((code >> 20) & 1023u);
    const bool close = full || inv;
    const int d = full ? i : j;
    if (w == 8) {  // operands
      int pa = 0, pj = 0;
      for (int s = s0; s < s1 + (close ? 1 : 0); ++s) {
        int ok = 1;
        if (lane == 0) {
          if (s < s1) {
            if (pa <= s) pa = df_wait(inv ? xprog + i : prog + i, s + 1, err, status);
            if (pa > 0 && pj <= s) pj = df_wait(prog + j, s + 1, err, status);
            ok = pa > 0 && pj > 0;
          } else {
            ok = df_wait(prog + d, d + 1, err, status) > 0;
          }
          if (!ok) *(volatile int*)&sh.abort = 1;
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        __syncwarp();
        const unsigned x = cnt & 1;
        if (!ok || !df_bar_wait(&sh.empty[x], ((cnt >> 1) & 1) ^ 1, &sh)) break;
        double* As = T + 2 * x * DF_TILE;
        if (s == s1) {
          df_stream_tile(As, Dinv + (long)d * DF_NB * DF_NB, DF_NB, DF_NB, DF_NB);
        } else {
          if (inv) df_stream_tile(As, Xr + i0 + (long)s * DF_NB * ldx, ldx, DF_NB, DF_NB);
          else df_stream_tile(As, F + s * DF_NB + (long)i0 * ld, ld, DF_NB, ni);
          if (inv || i != j) df_stream_tile(As + DF_TILE, F + s * DF_NB + (long)j0 * ld, ld, DF_NB, nc);
        }
        df_stream_done(&sh.full[x]);
        ++cnt;
      }
    } else if (w < 8) {
      double acc[8][2];
#pragma unroll
      for (int R = 0; R < 8; ++R)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int row = 8 * R + r, col = 8 * w + 2 * q + e;
          acc[R][e] = (!inv && row < ni && col < nc) ? __ldcg(F + (i0 + row) + (long)(j0 + col) * ld) : 0.0;
        }
      bool ok = true;
      for (int s = s0; s < s1; ++s) {
        const unsigned x = cnt & 1;
        ok = df_bar_wait(&sh.full[x], (cnt >> 1) & 1, &sh);
        if (!ok) break;
        const double* As = T + 2 * x * DF_TILE;
        if (inv) df_sub_ab(As, As + DF_TILE, acc);
        else df_sub_atb(As, i == j ? As : As + DF_TILE, acc);
        __syncwarp();
        if (lane == 0) df_bar_arrive(&sh.empty[x]);
        ++cnt;
      }
      if (close) {
        const unsigned x = cnt & 1;
        const double* Ys = T + 2 * x * DF_TILE;  // U_dd^-T
        double* Bs = T + (2 * x + 1) * DF_TILE;
        ok = df_all(ok && df_bar_wait(&sh.full[x], (cnt >> 1) & 1, &sh));
        if (ok && (full || i != j)) {
#pragma unroll
          for (int R = 0; R < 8; ++R)
#pragma unroll
            for (int e = 0; e < 2; ++e) DFS(Bs, 8 * R + r, 8 * w + 2 * q + e) = acc[R][e];
#pragma unroll
          for (int R = 0; R < 8; ++R) acc[R][0] = acc[R][1] = 0.0;
        }
        if (ok && full) {  // U(i, j) = U_ii^-T acc: this warp's columns alone
          __syncwarp();
#pragma unroll
          for (int ks = 0; ks < DF_NB / 4; ++ks) {
            const int kk = ks * 4 + q;
            const double b = DFS(Bs, kk, 8 * w + r);
#pragma unroll
            for (int R = 0; R < 8; ++R)
              if (R >= ks / 2) dmma_m8n8k4(acc[R][0], acc[R][1], DFS(Ys, 8 * R + r, kk), b);
          }
        } else if (ok && i != j) {  // X(i, j) = acc X(j, j), X(j, j)(k, c) = U_jj^-T(c, k)
          df_sync<BAR_MMA, DF_MMA>();
          for (int ks = 0; ks < 2 * w + 2; ++ks) {
            const int kk = ks * 4 + q;
            const double b = DFS(Ys, 8 * w + r, kk);
#pragma unroll
            for (int R = 0; R < 8; ++R) dmma_m8n8k4(acc[R][0], acc[R][1], DFS(Bs, 8 * R + r, kk), b);
          }
        } else if (ok) {  // X(j, j)
#pragma unroll
          for (int R = 0; R < 8; ++R)
#pragma unroll
            for (int e = 0; e < 2; ++e) acc[R][e] = DFS(Ys, 8 * w + 2 * q + e, 8 * R + r);
        }
        __syncwarp();
        if (ok && lane == 0) df_bar_arrive(&sh.empty[x]);
        ++cnt;
      }
      if (ok) {
#pragma unroll
        for (int R = 0; R < 8; ++R)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int row = 8 * R + r, col = 8 * w + 2 * q + e;
            if (row >= ni || col >= nc) continue;
            if (inv) {
              Uinv[(i0 + row) + (long)(j0 + col) * m] = acc[R][e];
              UinvT[(j0 + col) + (long)(i0 + row) * m] = acc[R][e];
              if (Xr != Uinv) Xr[(i0 + row) + (long)(j0 + col) * ldx] = acc[R][e];
            } else {
              F[(i0 + row) + (long)(j0 + col) * ld] = acc[R][e];
            }
          }
      }
      df_sync<BAR_MMA, DF_MMA>();
      if (threadIdx.x == 0 && ok) {
        __threadfence();
        if (inv) df_st_release(xprog + i, j + 1);
        else if (full) df_st_release(prog + j, i + 1);
        else df_st_release((i == j ? pre_d : pre_o) + i, 1);
      }
    }
    __syncthreads();
    if (sh.abort) {
      if (threadIdx.x == 0 && sh.abort == 2) {
        atomicOr(status, SDPXG_ST_SYNC_TIMEOUT);
        atomicExch(err, 1);
      }
      break;
    }
  }
  if (w == 8) asm volatile("cp.async.wait_all;\n" ::: "memory");  // copies of an item that was given up
}
