// Shared definitions for the sm_100a SDPX hot-path kernels.
//
// Layout conventions (all device buffers in HBM, float64):
//  * PSD vectors use the reference's triangle convention: upper triangle, column order,
//    off-diagonal entries scaled by sqrt(2); entry (i, j), i <= j, sits at j(j+1)/2 + i
//    (include/sdpx.h:32-33 of the reference).
//  * Per-block n x n matrices (R, Rinv, Ginv, ...) are column-major with leading dimension n,
//    packed one after another at BlockDesc::mat_off.
//  * The Schur complement and its factor are dense column-major m x m.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define SDPXG_NMAX 64               // largest PSD block order handled by the CTA kernels
// Shared-memory leading dimension: 68 = 4 (mod 16), so the 16 lanes of a half-warp reading an
// m8n8k4 f64 fragment (rows r + 4-column k, or 4-row k + columns r) hit 16 distinct 8-byte
// bank pairs, and a column read is conflict-free.
#define SDPXG_LD 68
#define SDPXG_THREADS 256         // dense tile kernels (their thread maps assume 256)
#define SDPXG_CONE_THREADS 1024   // one CTA per PSD block
#define SDPXG_NT_SVD_THREADS 256  // the NT scaling's Jacobi launch (4 warps iterate)
constexpr size_t kSchurSmem = 2 * 2 * 32 * 36 * sizeof(double);  // the chunk ring of k_schur_block_gemm
constexpr int kSchurGatherTile = 8;                              // rows and columns of a CTA of k_schur_gather
#define SDPXG_EIG_THREADS 256     // step length and margins (tridiagonalisation in 4 warps' registers)
#define SDPXG_TRIDIAG_WORK 544    // doubles of shared scratch for cta_tridiagonalize
#define SDPXG_STURM_WORK (2 * SDPXG_NMAX)  // and for cta_eig_min / cta_eig_all
#define SDPXG_RSQRT2 0.70710678118654752440
#define SDPXG_SQRT2 1.41421356237309504880

// Device status bits reported by the kernels (read back by the host after each phase).
enum SdpxgStatus : uint32_t {
  SDPXG_ST_OK = 0,
  SDPXG_ST_CHOL_FAIL = 1u,        // Cholesky of s or z failed (not interior)
  SDPXG_ST_SVD_UNCONVERGED = 2u,  // Jacobi sweeps hit their bound
  SDPXG_ST_NONFINITE = 4u,        // a non-finite value was produced
  SDPXG_ST_PIVOT_FAIL = 8u,       // clearly negative or non-finite Schur pivot
  SDPXG_ST_EIG_FAIL = 16u,        // eigenvalue bisection did not converge
  SDPXG_ST_SYNC_TIMEOUT = 32u,    // a bounded inter-CTA wait gave up (no progress)
  SDPXG_ST_EXACT_SPREAD = 64u,    // an exact dot's terms spread beyond the device accumulator
};

// Device-resident control of one refined KKT solve: the stopping rules of the two-level
// stationary refinement (kkt/refinement.rs:118-191) evaluated by one-thread control kernels that
// drive the WHILE nodes of the solve's CUDA graph; the host reads it once per solve.
struct RefineCtl {
  double normb, norme, tol;      // reduced-system level (inner)
  double onormb, onorme, otol;   // original-operator level (outer)
  int it, oit;                   // accepted steps at each level
  int ok;                        // cleared by the first failed check
  int accept, oaccept;           // the last candidate is kept
  int cont, ocont;               // the loop goes on (its residual is carried over)
  int inner_steps, outer_steps;  // refinement steps run (trace counters)
  int guard;                     // loop-body executions: a hard bound on every loop
};
struct RefineParams {
  double abstol, reltol, stop_ratio;
  int max_iter, guard_max;
};

// What a fused norm-and-control kernel of the refined solve does (k_refine).
enum RefineKind { REFINE_HEAD = 0, REFINE_STEP = 1, REFINE_OUTER_INIT = 2, REFINE_OUTER_STEP = 3 };
struct RefineOp {
  int kind, rows, reset;    // reset: HEAD starts a new KKT solve
  long n;                   // STEP: entries of the two copies below
  double* x;                // STEP: x <- cand when the candidate is kept
  const double* cand;
  double* e;                // STEP: e <- e2 when the loop goes on
  const double* e2;
};

// One reduction of a batched launch (k_reduce_batch): op over x (and y) of length n.
struct RedReq {
  int op;
  long n;
  const double* x;
  const double* y;
};
constexpr int kRedBatchMax = 12;
struct RedBatch {
  RedReq r[kRedBatchMax];
};

// One vector update of a batched launch (k_lincomb_batch): out = a x + b y + c w over n entries
// (a null operand is left out), with the arithmetic of k_lincomb.
struct LinReq {
  long n;
  double a, b, c;
  const double* x;
  const double* y;
  const double* w;
  double* out;
};
constexpr int kLinBatchMax = 6;
struct LinBatch {
  LinReq r[kLinBatchMax];
};

struct BlockDesc {
  int n;         // block order
  int svec_off;  // first row of the block in the stacked cone vector
  int mat_off;   // offset of the block's n*n matrices
  int vec_off;   // offset of the block's length-n vectors (lambda, Lambda^-1/2)
};

// A matrix-valued sampled block (dim D > 1): its PSD block j, D, basis rows h, basis columns c,
// and the offsets of its basis Q (h x c), of V = R^-1 U (n x Dc) and of K = V'V (Dc x Dc).
struct MsDesc {
  int j, D, h, c;
  long q_off, v_off, k_off;
};

__device__ __forceinline__ int tri_idx(int i, int j) {  // i <= j
  return j * (j + 1) / 2 + i;
}

// The larger of two magnitudes, NaN when either is one (fmax and std::max lose one): a residual of NaNs is
// no small residual.  Magnitudes order like their bits as unsigned integers, NaNs of either sign (fabs
// may leave one negative) above infinity.
__host__ __device__ __forceinline__ double max_nan(double a, double b) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)max((unsigned long long)__double_as_longlong(a),
                                             (unsigned long long)__double_as_longlong(b)));
#else
  return (b <= a || a != a) ? a : b;
#endif
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ double warp_min(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ------------------------------------------------------------------------------------
// CTA-level helpers on n x n shared-memory matrices with leading dimension SDPXG_LD.
// Callers place __syncthreads() between dependent calls.
// ------------------------------------------------------------------------------------
#define SM(A, i, j) (A)[(i) + (j) * SDPXG_LD]

// Shared matrices are 64 x 64 (leading dimension SDPXG_LD) whatever the block order n; the entries outside
// n x n up to the next multiple of eight are zero, so that the tensor-core products below can run on whole
// 8 x 8 x 4 fragments.  Loads write that padding (`pad`: to another size); products of padded inputs keep
// it.  What lies beyond is not read into a result.
__device__ __forceinline__ int pad8(int n) { return (n + 7) & ~7; }

// M = smat(v): symmetric matrix from an svec.  Column j of the upper triangle is contiguous in the svec
// (v[j(j+1)/2 + i], i <= j): one warp per column reads it coalesced, the loads of U columns in flight, and
// writes both triangles.  U = 64 / warps, at most 4.
template <int U = 4>
__device__ __forceinline__ void cta_load_smat(double* M, const double* __restrict__ v, int n,
                                              int pad = SDPXG_NMAX) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  for (int j0 = warp; j0 < pad; j0 += U * nwarps) {
    double x[U][2];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = j0 + u * nwarps;
      const double* col = v + j * (j + 1) / 2;
#pragma unroll
      for (int h = 0; h < 2; ++h) x[u][h] = (j < n && lane + 32 * h <= j) ? col[lane + 32 * h] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = j0 + u * nwarps;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = lane + 32 * h;
        if (j < pad && i <= j) {
          const double y = i != j ? x[u][h] * SDPXG_RSQRT2 : x[u][h];
          SM(M, i, j) = y;
          SM(M, j, i) = y;
        }
      }
    }
  }
}

// v = svec(sym(M)): off-diagonal (M_ij + M_ji) / sqrt(2).
__device__ __forceinline__ void cta_store_svec(double* __restrict__ v, const double* M, int n) {
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    int i = e % n, j = e / n;
    if (i > j) continue;
    v[tri_idx(i, j)] = (i == j) ? SM(M, i, j) : (SM(M, i, j) + SM(M, j, i)) * SDPXG_RSQRT2;
  }
}

// M = the n x n matrix at g, one warp a column, the loads of U columns in flight.
template <int U = 4>
__device__ __forceinline__ void cta_load_mat(double* M, const double* __restrict__ g, int n,
                                             int pad = SDPXG_NMAX) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  for (int j0 = warp; j0 < pad; j0 += U * nwarps) {
    double x[U][2];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = lane + 32 * h, j = j0 + u * nwarps;
        x[u][h] = (i < n && j < n) ? g[i + j * n] : 0.0;
      }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = lane + 32 * h, j = j0 + u * nwarps;
        if (i < pad && j < pad) SM(M, i, j) = x[u][h];
      }
  }
}

__device__ __forceinline__ void cta_store_mat(double* __restrict__ g, const double* M, int n) {
  const int lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  for (int j = threadIdx.x >> 5; j < n; j += nwarps)
    for (int i = lane; i < n; i += 32) g[i + j * n] = SM(M, i, j);
}

// One FP64 tensor-core MMA: D(8x8) = A(8x4) B(4x8) + C.  Fragments (PTX mma.m8n8k4 .f64):
// lane l holds A[l/4][l%4], B[l%4][l/4] and C/D[l/4][2(l%4) + {0,1}].
__device__ __forceinline__ void dmma_m8n8k4(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// What is known of a product: nothing; A'B of two lower triangular matrices (only k >= max(i, j)
// counts); op(B) is upper triangular (k <= j); the result is symmetric (tiles i <= j, mirrored).
enum GemmForm { GEMM_FULL, GEMM_LOWER_TN, GEMM_UPPER_B, GEMM_SYMMETRIC };

// C = op(A) op(B) on zero-padded shared matrices.  A warp takes 8 x 8 tiles of one tile row (NJ of them:
// 8 with 8 warps, 2 with 32), so that one fragment of A serves NJ MMAs: with a fragment of each operand
// per MMA the shared-memory reads take as long as the tensor pipe (16 cycles an MMA and quarter).  Warps
// w and w + 4 of an SM quarter take tile rows w and 7 - w, equal work for every form.
// K runs to n rounded up to 4, never further: C is written only up to n rounded up to 8, and
// a later product that reads C as an operand must not reach its unwritten columns (another
// kernel's leftovers there, NaN included, would enter through 0 x NaN).  C must not alias A or B.
// blockDim.x is 2048 / NJ.
template <bool TA, bool TB, int NJ, GemmForm F = GEMM_FULL>
__device__ __forceinline__ void cta_gemm(double* C, const double* A, const double* B, int n) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tiles = (n + 7) >> 3, ksteps = (n + 3) >> 2;
  const int r = lane >> 2, q = lane & 3;
  const int I = (warp & 4) ? 7 - (warp & 3) : (warp & 3), J0 = warp >> 3;  // tile columns J0, J0 + 8 / NJ, ...
  if (I >= tiles) return;
  double d[NJ][2];
#pragma unroll
  for (int u = 0; u < NJ; ++u) d[u][0] = d[u][1] = 0.0;
  for (int ks = F == GEMM_LOWER_TN ? 2 * I : 0; ks < ksteps; ++ks) {
    const int k = (ks << 2) + q;
    const double a = TA ? SM(A, k, 8 * I + r) : SM(A, 8 * I + r, k);
    double b[NJ];
#pragma unroll
    for (int u = 0; u < NJ; ++u) {
      const int J = J0 + u * (8 / NJ);
      b[u] = TB ? SM(B, 8 * J + r, k) : SM(B, k, 8 * J + r);
    }
#pragma unroll
    for (int u = 0; u < NJ; ++u) {
      const int J = J0 + u * (8 / NJ);
      if (J < tiles && (F != GEMM_LOWER_TN || ks >= 2 * J) && (F != GEMM_UPPER_B || ks < 2 * J + 2) &&
          (F != GEMM_SYMMETRIC || J >= I))
        dmma_m8n8k4(d[u][0], d[u][1], a, b[u]);
    }
  }
#pragma unroll
  for (int u = 0; u < NJ; ++u) {
    const int J = J0 + u * (8 / NJ);
    if (J >= tiles || (F == GEMM_SYMMETRIC && J < I)) continue;
    SM(C, 8 * I + r, 8 * J + 2 * q) = d[u][0];
    SM(C, 8 * I + r, 8 * J + 2 * q + 1) = d[u][1];
    if (F == GEMM_SYMMETRIC && J != I) {
      SM(C, 8 * J + 2 * q, 8 * I + r) = d[u][0];
      SM(C, 8 * J + 2 * q + 1, 8 * I + r) = d[u][1];
    }
  }
}

// v in [2^-1000, 2^1000): an integer test on the exponent (a double comparison takes part of the FP64
// pipe and three times as long).
__device__ __forceinline__ bool mid_range(double v) {
  return (unsigned)__double2hiint(v) - 0x01700000u < 0x7d000000u;
}

// 1/v for v in the mid range: the hardware approximation refined by two Newton-Raphson steps
// y <- y + y (1 - v y) (each doubles the correct bits; the error left is the last step's rounding, 2^-53
// relative).
__device__ __forceinline__ double recip_mid(double v) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
  double e = fma(-v, y, 1.0);
  y = fma(y, e, y);
  e = fma(-v, y, 1.0);
  return fma(y, e, y);
}

// 1/sqrt(v) for v in the mid range (and 2^1000): the hardware approximation y (about 22 bits) and one
// Householder step of third order, y (1 + e/2 + 3 e^2 / 8) with e = 1 - v y^2.  The step leaves e^3; the rounding
// of v y moves the result by half of 2^-53, that of the last operation by 2^-53.
__device__ __forceinline__ double rsqrt_mid(double v) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
  const double e = fma(-v * y, y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

// One 8-column panel of cta_cholesky_lower in one warp, columns kb .. kb+w-1, any pivot: lane l holds the
// panel's rows kb + l and kb + 32 + l, pivots and the updating rows' entries come by shuffles.  False at
// a pivot that is not positive and finite.
static __device__ __noinline__ bool cholesky_panel_any(double* A, int n, int kb, int w) {
  const int lane = threadIdx.x & 31, r0 = kb + lane, r1 = kb + 32 + lane;
  double P0[8], P1[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    P0[c] = (c < w && r0 < n) ? SM(A, r0, kb + c) : 0.0;
    P1[c] = (c < w && r1 < n) ? SM(A, r1, kb + c) : 0.0;
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    if (c < w) {
      const double piv = __shfl_sync(0xffffffffu, P0[c], c);
      if (!(piv > 0.0 && isfinite(piv))) return false;
      const double d = sqrt(piv), rd = 1.0 / d;
      P0[c] = lane < c ? 0.0 : (lane == c ? d : P0[c] * rd);
      P1[c] *= rd;
#pragma unroll
      for (int c2 = c + 1; c2 < 8; ++c2) {
        const double l = __shfl_sync(0xffffffffu, P0[c], c2);  // L(kb + c2, kb + c)
        P0[c2] = fma(-P0[c], l, P0[c2]);
        P1[c2] = fma(-P1[c], l, P1[c2]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    if (c < w && r0 < n) SM(A, r0, kb + c) = P0[c];
    if (c < w && r1 < n) SM(A, r1, kb + c) = P1[c];
  }
  return true;
}

// In-place lower Cholesky A = L L' (lower triangle of A used, zero padded; 256 threads): panels of 8
// columns, right-looking.  Warp 0 factors the panel: every lane has the 8 x 8 diagonal block to itself
// and eliminates it next to its own two rows, so that the chain of a column is root -> scale -> update
// (about 70 cycles) without a shuffle; L(r,c) = a(r,c) rd, rd = pivot^-1/2, and L(c,c) = pivot rd with
// the residual of its square corrected.  A pivot out of [2^-1000, 2^1000) repeats the panel the slow way.
// Then A22 -= L21 L21' on the lower 8 x 8 tiles on the FP64 tensor cores (two m8n8k4 steps), one warp a
// tile row, rows w and 7 - w in the same quarter of the SM.  Two barriers a panel.  False when a pivot
// is not positive and finite.  Entries above the diagonal end as zeros.
// Order 64: 19200 cycles; with a shuffle per updating entry, a root and a reciprocal a column and the
// tiles dealt to 32 warps, two matrices at once, 31900.
__device__ inline bool cta_cholesky_lower(double* A, int n) {
  __shared__ int live;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ti = (warp & 4) ? 7 - (warp & 3) : (warp & 3), r = lane >> 2, q = lane & 3;
  if (threadIdx.x == 0) live = 1;
  __syncthreads();
  for (int kb = 0; kb < n; kb += 8) {
    const int w = min(8, n - kb);
    if (warp == 0) {
      const int r0 = kb + lane, r1 = kb + 32 + lane;
      double D[36], P0[8], P1[8], dg[8];  // D: the block's lower triangle by columns
#pragma unroll
      for (int c = 0, e = 0; c < 8; ++c)
#pragma unroll
        for (int i = c; i < 8; ++i, ++e) D[e] = i < w ? SM(A, kb + i, kb + c) : (i == c ? 1.0 : 0.0);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        P0[c] = (c < w && r0 < n) ? SM(A, r0, kb + c) : 0.0;
        P1[c] = (c < w && r1 < n) ? SM(A, r1, kb + c) : 0.0;
      }
      bool mid = true;
#pragma unroll
      for (int c = 0, e = 0; c < 8; e += 8 - c, ++c) {
        const double piv = D[e], rd = rsqrt_mid(piv), d0 = piv * rd;
        mid = mid && mid_range(piv);
        dg[c] = fma(0.5 * rd, fma(-d0, d0, piv), d0);
#pragma unroll
        for (int i = c + 1; i < 8; ++i) D[e + i - c] *= rd;
        P0[c] *= rd;
        P1[c] *= rd;
#pragma unroll
        for (int j = c + 1, f = e + 8 - c; j < 8; f += 8 - j, ++j) {
          const double l = D[e + j - c];
#pragma unroll
          for (int i = j; i < 8; ++i) D[f + i - j] = fma(-D[e + i - c], l, D[f + i - j]);
          P0[j] = fma(-P0[c], l, P0[j]);
          P1[j] = fma(-P1[c], l, P1[j]);
        }
      }
      bool ok = true;
      if (mid) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const double v = lane < c ? 0.0 : (lane == c ? dg[c] : P0[c]);
          if (c < w && r0 < n) SM(A, r0, kb + c) = v;
          if (c < w && r1 < n) SM(A, r1, kb + c) = P1[c];
        }
      } else {
        ok = cholesky_panel_any(A, n, kb, w);
      }
      if (!ok && lane == 0) live = 0;
    }
    __syncthreads();
    if (!live) return false;
    const int t0 = kb + 8, nt = (n - t0 + 7) >> 3;
    if (ti < nt) {
      const double a0 = -SM(A, t0 + 8 * ti + r, kb + q), a1 = -SM(A, t0 + 8 * ti + r, kb + 4 + q);
#pragma unroll
      for (int tj = 0; tj < 7; ++tj) {
        if (tj <= ti) {
          double* C = &SM(A, t0 + 8 * ti + r, t0 + 8 * tj + 2 * q);
          double d0 = C[0], d1 = C[SDPXG_LD];
          dmma_m8n8k4(d0, d1, a0, SM(A, t0 + 8 * tj + r, kb + q));
          dmma_m8n8k4(d0, d1, a1, SM(A, t0 + 8 * tj + r, kb + 4 + q));
          C[0] = d0;
          C[SDPXG_LD] = d1;
        }
      }
    }
    __syncthreads();
  }
  for (int j = warp; j < n; j += 8)
    for (int i = lane; i < j; i += 32) SM(A, i, j) = 0.0;
  __syncthreads();
  return true;
}

// B := L^-T B for the lower triangular L (n x n, n <= 64, both zero padded), back substitution by blocks
// of 8 rows from the bottom, left-looking: warp w has the 8 columns from 8w on to itself, so no barrier
// of the CTA is needed between blocks.  B(I, w) -= sum_{K > I} L(K, I)' X(K, w) on the FP64 tensor cores,
// then the 8 x 8 diagonal block, one lane a column with its eight entries in registers (x_i = (b_i -
// sum_k L(k,i) x_k) / L(i,i), the reciprocals formed first).
// blockDim.x >= 256; `rd` is n doubles of shared memory.
__device__ __forceinline__ void cta_trsm_lower_t_blocked(const double* L, double* B, int n, double* rd) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) rd[i] = 1.0 / SM(L, i, i);
  __syncthreads();
  const int lane = threadIdx.x & 31, J = threadIdx.x >> 5, r = lane >> 2, q = lane & 3, nt = (n + 7) >> 3;
  for (int I = nt - 1; J < nt && I >= 0; --I) {
    const int ib = 8 * I;
    if (I < nt - 1) {
      double d[2][2];
      d[0][0] = SM(B, ib + r, 8 * J + 2 * q);
      d[0][1] = SM(B, ib + r, 8 * J + 2 * q + 1);
      d[1][0] = d[1][1] = 0.0;
      for (int K = ib + 8; K < 8 * nt; K += 8) {
#pragma unroll
        for (int u = 0; u < 2; ++u)
          dmma_m8n8k4(d[u][0], d[u][1], -SM(L, K + 4 * u + q, ib + r), SM(B, K + 4 * u + q, 8 * J + r));
      }
      SM(B, ib + r, 8 * J + 2 * q) = d[0][0] + d[1][0];
      SM(B, ib + r, 8 * J + 2 * q + 1) = d[0][1] + d[1][1];
      __syncwarp();
    }
    if (lane < 8) {
      const int j = 8 * J + lane;
      double x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = ib + i < n ? SM(B, ib + i, j) : 0.0;
#pragma unroll
      for (int i = 7; i >= 0; --i) {
        if (ib + i < n) {
          x[i] *= rd[ib + i];
          SM(B, ib + i, j) = x[i];
#pragma unroll
          for (int k = 0; k < i; ++k) x[k] = fma(-SM(L, ib + i, ib + k), x[i], x[k]);
        }
      }
    }
    __syncwarp();
  }
  __syncthreads();
}
