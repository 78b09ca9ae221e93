// PSD-cone kernels: Nesterov-Todd scaling, W congruences, Jordan products, step lengths
// and interior margins.  One CTA per PSD block (and per right-hand side or side of the
// step); every block of order <= SDPXG_NMAX lives in shared memory for the whole kernel.
//
// Reference functions restated (crates/solver/src/solver/cones/psdtrianglecone.rs):
//   update_scaling 311-439, mul_Wx_scratch 860-917, circ_op 927-938,
//   lambda_inv_circ_op 757-780, affine_ds 455-460, step_length_psd_component 1180-1231,
//   admits 1168-1178, margins ~590-606; and the binary64 factored Hs / Hs^-1 application
//   of kkt/condensed/psd.rs:1968-2002.
#include <cooperative_groups.h>

#include "eig.cuh"

namespace {

constexpr int kMat = SDPXG_LD * SDPXG_NMAX;  // doubles per shared matrix

}  // namespace

// ---------------------------------------------------------------------------------------
// NT scaling.  L1 = chol(S), L2 = chol(Z), L2'L1 = U diag(lam) V' (psdtrianglecone.rs:311-439).
// The reference forms R = L1 V lam^-1/2 and Rinv = lam^1/2 V' L1^-1.  With M = L2'L1 and
// M V = U lam, the same matrices are
//   R = L2^-T U lam^1/2,   Rinv = lam^-1/2 U' L2'
// (L1 V = L1 M^-1 U lam = L2^-T U lam), which needs only the LEFT singular vectors: the
// normalised columns that one-sided Jacobi leaves in M, so the rotations are not accumulated
// into V.  Both forms have the same
// normwise accuracy (a triangular solve with L1 or with L2 each).  Ginv = Rinv' Rinv.
// Two launches: k_nt_factor, one CTA per block and matrix, leaves L1 in R's slot and L2 in Rinv's slot
// of each block; k_nt_svd reads them back and writes R, Rinv, Ginv, lam and lam^-1/2.  A failed
// factorisation sets SDPXG_ST_CHOL_FAIL, which the second launch reads to leave every block alone (the
// scaling is rejected as a whole).
// Shared memory of k_nt_factor: 1 matrix; of k_nt_svd: 5 matrices + 5n doubles + n ints + 1 int.
// At n = 64, k_nt_factor 31 us with both factors and M in one CTA of 1024 threads, now 22; k_nt_svd (12
// sweeps) 357 us with eight warps on the Jacobi rounds, scalar loops over the columns and a back
// substitution with two barriers a block of rows, now 257.
// ---------------------------------------------------------------------------------------
extern "C" __global__ void __launch_bounds__(SDPXG_EIG_THREADS)
k_nt_factor(const BlockDesc* __restrict__ blocks, const double* __restrict__ s,
            const double* __restrict__ z, double* __restrict__ R, double* __restrict__ Rinv,
            uint32_t* __restrict__ status) {
  extern __shared__ double smem[];
  const BlockDesc bd = blocks[blockIdx.x];
  const int n = bd.n;
  double* L = smem;
  cta_load_smat(L, (blockIdx.y == 0 ? s : z) + bd.svec_off, n, pad8(n));
  if (!cta_cholesky_lower(L, n)) {
    if (threadIdx.x == 0) atomicOr(status, SDPXG_ST_CHOL_FAIL);
    return;
  }
  cta_store_mat((blockIdx.y == 0 ? R : Rinv) + bd.mat_off, L, n);
}

// a / b from y = 1 / b rounded: one residual step (a b that is no denominator of an ordinary quotient
// divides).
__device__ __forceinline__ double quotient(double a, double b, double y) {
  const double q = a * y;
  const double q1 = fma(fma(-q, b, a), y, q);
  return mid_range(b) && isfinite(q1) ? q1 : a / b;
}

extern "C" __global__ void __launch_bounds__(SDPXG_NT_SVD_THREADS)
k_nt_svd(const BlockDesc* __restrict__ blocks, double* __restrict__ R, double* __restrict__ Rinv,
         double* __restrict__ Ginv, double* __restrict__ lam, double* __restrict__ lisqrt,
         uint32_t* __restrict__ status) {
  extern __shared__ double smem[];
  if (*status & SDPXG_ST_CHOL_FAIL) return;
  const BlockDesc bd = blocks[blockIdx.x];
  const int n = bd.n;
  double* L1 = smem;
  double* L2 = L1 + kMat;
  double* M = L2 + kMat;
  double* V = M + kMat;
  double* X = V + kMat;
  double* sig = X + kMat;
  double* lsort = sig + SDPXG_NMAX;
  double* root = lsort + SDPXG_NMAX;
  double* iroot = root + SDPXG_NMAX;
  double* isig = iroot + SDPXG_NMAX;
  int* rank = reinterpret_cast<int*>(isig + SDPXG_NMAX);
  int* flag = rank + SDPXG_NMAX;

  for (int j = threadIdx.x >> 5; j < pad8(n); j += SDPXG_NT_SVD_THREADS / 32)  // V and X are written n x n
    for (int i = threadIdx.x & 31; i < pad8(n); i += 32)                       // only: zeros for the MMAs
      if (i >= n || j >= n) SM(V, i, j) = SM(X, i, j) = 0.0;
  cta_load_mat(L1, R + bd.mat_off, n, pad8(n));
  cta_load_mat(L2, Rinv + bd.mat_off, n, pad8(n));
  __syncthreads();
  cta_gemm<true, false, 8, GEMM_LOWER_TN>(M, L2, L1, n);  // M = L2' L1
  __syncthreads();
  int sweeps = cta_jacobi_left(M, n, L1, flag);  // M -> U diag(lam); L1 as scratch
  if (sweeps < 0) {
    if (threadIdx.x == 0) atomicOr(status, SDPXG_ST_SVD_UNCONVERGED);
    return;
  }
  // singular values and their ranks, eight threads a column
  const int g8 = threadIdx.x >> 3, u8 = threadIdx.x & 7;
  for (int j0 = 0; j0 < n; j0 += SDPXG_NT_SVD_THREADS / 8) {
    const int j = j0 + g8;
    double acc = 0.0;
    for (int k = u8; k < n; k += 8) acc = j < n ? fma(SM(M, k, j), SM(M, k, j), acc) : 0.0;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (u8 == 0 && j < n) sig[j] = sqrt(acc);
  }
  __syncthreads();
  bool good = true;
  for (int j0 = 0; j0 < n; j0 += SDPXG_NT_SVD_THREADS / 8) {
    const int j = j0 + g8;
    int r = 0;
    if (j < n)
      for (int k = u8; k < n; k += 8) r += (sig[k] > sig[j]) || (sig[k] == sig[j] && k < j);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    if (u8 == 0 && j < n) {
      rank[j] = r;
      lsort[r] = sig[j];
      root[r] = sqrt(sig[j]);
      iroot[r] = 1.0 / sqrt(sig[j]);
      isig[j] = 1.0 / sig[j];
      good = sig[j] > 0.0 && isfinite(sig[j]);
    }
  }
  if (!__syncthreads_and(good)) {
    if (threadIdx.x == 0) atomicOr(status, SDPXG_ST_CHOL_FAIL);
    return;
  }
  // X = U with columns in descending singular-value order; V = X as the right-hand side
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  for (int j = warp; j < n; j += nwarps) {
    const int c = rank[j];
    for (int i = lane; i < n; i += 32) {
      const double u = quotient(SM(M, i, j), sig[j], isig[j]);
      SM(X, i, c) = u;
      SM(V, i, c) = u;
    }
  }
  __syncthreads();
  cta_trsm_lower_t_blocked(L2, V, n, sig);  // V = L2^-T U (sig is free: lsort holds lambda)
  double* Rg = R + bd.mat_off;
  for (int j = warp; j < n; j += nwarps)
    for (int i = lane; i < n; i += 32) Rg[i + j * n] = SM(V, i, j) * root[j];
  cta_gemm<true, true, 8, GEMM_UPPER_B>(L1, X, L2, n);  // L1 = U' L2'
  __syncthreads();
  double* Rig = Rinv + bd.mat_off;
  bool fin = true;
  for (int j = warp; j < n; j += nwarps)
    for (int i = lane; i < n; i += 32) {
      const double v = quotient(SM(L1, i, j), root[i], iroot[i]);  // Rinv = lam^-1/2 U' L2'
      SM(L1, i, j) = v;
      Rig[i + j * n] = v;
      fin = fin && isfinite(v);
    }
  __syncthreads();
  cta_gemm<true, false, 8, GEMM_SYMMETRIC>(M, L1, L1, n);  // Ginv = Rinv' Rinv
  __syncthreads();
  double* Gg = Ginv + bd.mat_off;
  for (int j = warp; j < n; j += nwarps)
    for (int i = lane; i < n; i += 32) {
      const double v = SM(M, i, j);
      Gg[i + j * n] = v;
      fin = fin && isfinite(v);
    }
  if (!fin) atomicOr(status, SDPXG_ST_NONFINITE);
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    lam[bd.vec_off + j] = lsort[j];
    lisqrt[bd.vec_off + j] = iroot[j];
  }
}

// Identity scaling: R = Rinv = Ginv = I, lam = 1 (the default start, core/solver.rs:1212).
extern "C" __global__ void k_identity_scaling(const BlockDesc* __restrict__ blocks,
                                              double* R, double* Rinv, double* Ginv, double* lam,
                                              double* lisqrt) {
  const BlockDesc bd = blocks[blockIdx.x];
  const int n = bd.n;
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    double v = (e % n == e / n) ? 1.0 : 0.0;
    R[bd.mat_off + e] = v;
    Rinv[bd.mat_off + e] = v;
    Ginv[bd.mat_off + e] = v;
  }
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    lam[bd.vec_off + j] = 1.0;
    lisqrt[bd.vec_off + j] = 1.0;
  }
}

// G^-1 = R^-T R^-1 per block from a given R^-1 (column-major n x n): G^-1(a, b) =
// sum_r R^-1(r, a) R^-1(r, b), summed in r order (exactly symmetric).
extern "C" __global__ void k_ginv_from_rinv(const BlockDesc* __restrict__ blocks, const double* __restrict__ Rinv,
                                            double* __restrict__ Ginv) {
  const BlockDesc bd = blocks[blockIdx.x];
  const int n = bd.n;
  const double* X = Rinv + bd.mat_off;
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int a = e % n, b = e / n;
    const int lo = a < b ? a : b, hi = a < b ? b : a;
    double acc = 0.0;
    for (int r = 0; r < n; ++r) acc = fma(X[r + lo * n], X[r + hi * n], acc);
    Ginv[bd.mat_off + e] = acc;
  }
}

// Y = B X B' (outer_t) or B' X B for a symmetric X, 256 threads.
__device__ void cta_congruence(double* Y, double* T, const double* X, const double* B,
                               bool outer_t, int n) {
  if (outer_t) {
    cta_gemm<false, true, 8>(T, X, B, n);  // T = X B'
    __syncthreads();
    cta_gemm<false, false, 8, GEMM_SYMMETRIC>(Y, B, T, n);  // Y = B T
  } else {
    cta_gemm<false, false, 8>(T, X, B, n);  // T = X B
    __syncthreads();
    cta_gemm<true, false, 8, GEMM_SYMMETRIC>(Y, B, T, n);  // Y = B' T
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------------------
// Congruences on svec vectors.  mode:
//   0  W x     = svec(R' X R)          1  W' x     = svec(R X R')
//   2  Winv x  = svec(Rinv' X Rinv)    3  Winv' x  = svec(Rinv X Rinv')
//   4  Hs x    = W'(W x)  (two congruences through R, never the squared G)
//   5  Hs^-1 x = Winv(Winv' x)
// plus `base` when it is given (y = op(x) + base).  grid.y: columns; column c of x / y / base
// starts at c * ld.
//
// One cluster of four CTAs per block.  A 64^3 product is 2.1 us of one SM's FP64 pipe and an
// operator of two congruences has four of them, so one CTA per block was bound by its own pipe
// (about 10 us at n = 60); the 8-wide tile columns J and 7 - J go to CTA J (equal work on the upper
// triangle), which forms T = X op(B) for its columns and the upper tiles of op(B)' T.  Between the
// two congruences each CTA reads the others' columns through distributed shared memory.
// ---------------------------------------------------------------------------------------
namespace {

constexpr int kCongCtas = 4;
constexpr int kCongThreads = 256;

// T (16 columns: tile columns J0 and J1 of CTA `rank`) = X op(B), op(B) = B' (outer_t) or B: warp w
// forms row tile w of both tile columns, its four accumulation chains in flight together.
__device__ __forceinline__ void slab_times(double* T, const double* X, const double* B, bool outer_t, int n, int J0,
                                           int J1) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r = lane >> 2, q = lane & 3;
  const int nt = (n + 7) >> 3, ks = (n + 3) >> 2;
  if (w >= nt || J0 >= nt) return;
  const bool two = J1 < nt;
  double c[4][2] = {};
  for (int k0 = 0; k0 < ks; k0 += 2) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int k = ((k0 + u) << 2) + q;
      if (k0 + u < ks) {
        const double a = SM(X, 8 * w + r, k);
        dmma_m8n8k4(c[u][0], c[u][1], a, outer_t ? SM(B, 8 * J0 + r, k) : SM(B, k, 8 * J0 + r));
        if (two) dmma_m8n8k4(c[2 + u][0], c[2 + u][1], a, outer_t ? SM(B, 8 * J1 + r, k) : SM(B, k, 8 * J1 + r));
      }
    }
  }
  SM(T, 8 * w + r, 2 * q) = c[0][0] + c[1][0];
  SM(T, 8 * w + r, 2 * q + 1) = c[0][1] + c[1][1];
  SM(T, 8 * w + r, 8 + 2 * q) = c[2][0] + c[3][0];
  SM(T, 8 * w + r, 8 + 2 * q + 1) = c[2][1] + c[3][1];
}

// Y (the same 16 columns, upper tiles only) = op(B)' T, op(B)' = B (outer_t) or B'.
__device__ __forceinline__ void slab_close(double* Y, const double* T, const double* B, bool outer_t, int n, int J0,
                                           int J1) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r = lane >> 2, q = lane & 3;
  const int nt = (n + 7) >> 3, ks = (n + 3) >> 2;
  const int n1 = J1 < nt ? J1 + 1 : 0, n0 = J0 < nt ? J0 + 1 : 0;
  for (int t = w; t < n1 + n0; t += kCongThreads / 32) {
    const int I = t < n1 ? t : t - n1, s = t < n1 ? 8 : 0;
    double c[4][2] = {};
    for (int k0 = 0; k0 < ks; k0 += 4) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = ((k0 + u) << 2) + q;
        if (k0 + u < ks)
          dmma_m8n8k4(c[u][0], c[u][1], outer_t ? SM(B, 8 * I + r, k) : SM(B, k, 8 * I + r), SM(T, k, s + r));
      }
    }
    SM(Y, 8 * I + r, s + 2 * q) = (c[0][0] + c[1][0]) + (c[2][0] + c[3][0]);
    SM(Y, 8 * I + r, s + 2 * q + 1) = (c[0][1] + c[1][1]) + (c[2][1] + c[3][1]);
  }
}

}  // namespace

extern "C" __global__ void __cluster_dims__(kCongCtas, 1, 1) __launch_bounds__(kCongThreads)
k_congruence(const BlockDesc* __restrict__ blocks, int mode, const double* __restrict__ R,
             const double* __restrict__ Rinv, const double* __restrict__ x, const double* __restrict__ base,
             double* __restrict__ y, long ld) {
  namespace cg = cooperative_groups;
  extern __shared__ double smem[];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), J0 = rank, J1 = 7 - rank;
  const BlockDesc bd = blocks[blockIdx.x / kCongCtas];
  const int n = bd.n;
  const long off = (long)blockIdx.y * ld + bd.svec_off;
  double* B = smem;
  double* X = B + kMat;
  double* T = X + kMat;
  double* Y = T + 16 * SDPXG_LD;
  const bool use_r = (mode == 0 || mode == 1 || mode == 4);
  cta_load_mat(B, (use_r ? R : Rinv) + bd.mat_off, n, pad8(n));
  cta_load_smat(X, x + off, n, pad8(n));
  __syncthreads();
  // W x (R' X R) first for Hs, Winv' x (Rinv X Rinv') first for Hs^-1
  bool outer_t = mode == 1 || mode == 3 || mode == 5;
  slab_times(T, X, B, outer_t, n, J0, J1);
  __syncthreads();
  slab_close(Y, T, B, outer_t, n, J0, J1);
  if (mode >= 4) {
    cluster.sync();  // every CTA's columns are in its Y, and nobody reads X any more
    for (int e = threadIdx.x; e < SDPXG_NMAX * SDPXG_NMAX; e += kCongThreads) {
      const int i = e & 63, j = e >> 6, J = j >> 3;
      if (i > j || j >= n) continue;
      const double* Yr = cluster.map_shared_rank(Y, J < kCongCtas ? J : 7 - J);
      const double v = SM(Yr, i, (J < kCongCtas ? 0 : 8) + (j & 7));
      SM(X, i, j) = v;
      SM(X, j, i) = v;
    }
    cluster.sync();  // everyone has read Y
    outer_t = !outer_t;
    slab_times(T, X, B, outer_t, n, J0, J1);
    __syncthreads();
    slab_close(Y, T, B, outer_t, n, J0, J1);
  }
  __syncthreads();
  for (int c = threadIdx.x >> 5; c < 16; c += kCongThreads / 32) {  // svec: one warp a column
    const int j = (c < 8 ? J0 : J1) * 8 + (c & 7);
    if (j >= n) continue;
    for (int i = threadIdx.x & 31; i <= j; i += 32) {
      const double v = (i == j) ? SM(Y, i, c) : SM(Y, i, c) * SDPXG_SQRT2;
      const long o = off + tri_idx(i, j);
      y[o] = base ? v + base[o] : v;
    }
  }
}

// The same operators with one CTA a block, for problems of small blocks or of many: four CTAs a block load
// the operands four times, and past one wave of clusters that is what takes the time.  The same chains of
// products, so the same bits.  Shared memory: four matrices of `cols` columns, the largest order rounded up to
// eight.
extern "C" __global__ void __launch_bounds__(1024)
k_congruence_one(const BlockDesc* __restrict__ blocks, int mode, const double* __restrict__ R,
                 const double* __restrict__ Rinv, const double* __restrict__ x, const double* __restrict__ base,
                 double* __restrict__ y, long ld, int cols) {
  extern __shared__ double smem[];
  const BlockDesc bd = blocks[blockIdx.x];
  const int n = bd.n, nt = (n + 7) >> 3, ks = (n + 3) >> 2;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5, r = lane >> 2, q = lane & 3;
  const long off = (long)blockIdx.y * ld + bd.svec_off;
  double* B = smem;
  double* X = B + cols * SDPXG_LD;
  double* T = X + cols * SDPXG_LD;
  double* Y = T + cols * SDPXG_LD;
  const bool use_r = (mode == 0 || mode == 1 || mode == 4);
  cta_load_mat(B, (use_r ? R : Rinv) + bd.mat_off, n, 8 * nt);
  cta_load_smat(X, x + off, n, 8 * nt);
  __syncthreads();
  auto products = [&](auto a, auto b, auto c) {  // fragments of four steps of the inner index at once
    int k0 = 0;
    for (; k0 + 4 <= ks; k0 += 4) {
      double x[4], y4[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        x[u] = a(((k0 + u) << 2) + q);
        y4[u] = b(((k0 + u) << 2) + q);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) dmma_m8n8k4(c(u)[0], c(u)[1], x[u], y4[u]);
    }
#pragma unroll
    for (int u = 0; u < 3; ++u)
      if (k0 + u < ks) dmma_m8n8k4(c(u)[0], c(u)[1], a(((k0 + u) << 2) + q), b(((k0 + u) << 2) + q));
  };
  auto congruence = [&](bool outer_t) {  // Y (upper tiles) = op(B)' X op(B), as slab_times and slab_close
    for (int t = w; t < nt * nt; t += warps) {
      const int I = t % nt, J = t / nt;
      double c[2][2] = {};
      products([&](int k) { return SM(X, 8 * I + r, k); },
               [&](int k) { return outer_t ? SM(B, 8 * J + r, k) : SM(B, k, 8 * J + r); },
               [&](int u) -> double(&)[2] { return c[u & 1]; });
      SM(T, 8 * I + r, 8 * J + 2 * q) = c[0][0] + c[1][0];
      SM(T, 8 * I + r, 8 * J + 2 * q + 1) = c[0][1] + c[1][1];
    }
    __syncthreads();
    for (int t = w; t < nt * (nt + 1) / 2; t += warps) {
      int I = t, J = 0;
      while (I > J) I -= ++J;
      double c[4][2] = {};
      products([&](int k) { return outer_t ? SM(B, 8 * I + r, k) : SM(B, k, 8 * I + r); },
               [&](int k) { return SM(T, k, 8 * J + r); }, [&](int u) -> double(&)[2] { return c[u]; });
      SM(Y, 8 * I + r, 8 * J + 2 * q) = (c[0][0] + c[1][0]) + (c[2][0] + c[3][0]);
      SM(Y, 8 * I + r, 8 * J + 2 * q + 1) = (c[0][1] + c[1][1]) + (c[2][1] + c[3][1]);
    }
    __syncthreads();
  };
  const bool outer_t = mode == 1 || mode == 3 || mode == 5;
  congruence(outer_t);
  if (mode >= 4) {
    for (int j = w; j < n; j += warps)
      for (int i = lane; i <= j; i += 32) SM(X, i, j) = SM(X, j, i) = SM(Y, i, j);
    __syncthreads();
    congruence(!outer_t);
  }
  for (int j = w; j < n; j += warps)
    for (int i = lane; i <= j; i += 32) {
      const double v = (i == j) ? SM(Y, i, j) : SM(Y, i, j) * SDPXG_SQRT2;
      const long o = off + tri_idx(i, j);
      y[o] = base ? v + base[o] : v;
    }
}

// x = svec((Y Z + Z Y) / 2) per block.
extern "C" __global__ void __launch_bounds__(SDPXG_CONE_THREADS)
k_circ_op(const BlockDesc* __restrict__ blocks, const double* __restrict__ yv,
          const double* __restrict__ zv, double* __restrict__ xv) {
  extern __shared__ double smem[];
  const BlockDesc bd = blocks[blockIdx.x];
  const int n = bd.n;
  double* Y = smem;
  double* Z = Y + kMat;
  cta_load_smat<2>(Y, yv + bd.svec_off, n, n);
  cta_load_smat<2>(Z, zv + bd.svec_off, n, n);
  __syncthreads();
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    int i = e % n, j = e / n;
    if (i > j) continue;
    double a = 0.0, b = 0.0;
    for (int k = 0; k < n; ++k) {
      a = fma(SM(Y, i, k), SM(Z, k, j), a);
      b = fma(SM(Z, i, k), SM(Y, k, j), b);
    }
    double v = 0.5 * (a + b);
    xv[bd.svec_off + tri_idx(i, j)] = (i == j) ? v : v * SDPXG_SQRT2;
  }
}

// x = lambda \ z: X_ij = 2 Z_ij / (lam_i + lam_j) (svec scaling commutes).
extern "C" __global__ void k_lam_inv_circ(const BlockDesc* __restrict__ blocks,
                                          const double* __restrict__ lam,
                                          const double* __restrict__ zv, double* __restrict__ xv) {
  const BlockDesc bd = blocks[blockIdx.x];
  const int n = bd.n;
  for (int e = threadIdx.x; e < n * (n + 1) / 2; e += blockDim.x) {
    int j = (int)((sqrt(8.0 * e + 1.0) - 1.0) * 0.5);
    while (j * (j + 1) / 2 > e) --j;
    while ((j + 1) * (j + 2) / 2 <= e) ++j;
    int i = e - j * (j + 1) / 2;
    xv[bd.svec_off + e] = 2.0 * zv[bd.svec_off + e] / (lam[bd.vec_off + i] + lam[bd.vec_off + j]);
  }
}

// ds = svec(diag(lam^2)), plus a multiple of the identity: ds += a * I.
extern "C" __global__ void k_affine_ds(const BlockDesc* __restrict__ blocks,
                                       const double* __restrict__ lam, double* __restrict__ ds) {
  const BlockDesc bd = blocks[blockIdx.x];
  const int n = bd.n;
  for (int e = threadIdx.x; e < n * (n + 1) / 2; e += blockDim.x) ds[bd.svec_off + e] = 0.0;
  __syncthreads();
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    double l = lam[bd.vec_off + k];
    ds[bd.svec_off + tri_idx(k, k)] = l * l;
  }
}

// v[diag] += a  (scaled_unit_shift, psdtrianglecone.rs:260-266)
extern "C" __global__ void k_shift_unit(const BlockDesc* __restrict__ blocks, double* v, double a) {
  const BlockDesc bd = blocks[blockIdx.x];
  for (int k = threadIdx.x; k < bd.n; k += blockDim.x) v[bd.svec_off + tri_idx(k, k)] += a;
}

// ---------------------------------------------------------------------------------------
// Step length per (block, side).  side 0: dual, Delta = lam^-1/2 (R' dZ R) lam^-1/2;
// side 1: primal, Delta = lam^-1/2 (Rinv dS Rinv') lam^-1/2.
// mode 0: bound  alpha = amax if chol(I + amax Delta) succeeds, else min(-1/lmin, amax);
// mode 1: admission only (out = amax if admitted else 0).
// out[2*block + side].
// ---------------------------------------------------------------------------------------
extern "C" __global__ void __launch_bounds__(SDPXG_EIG_THREADS)
k_step_length(const BlockDesc* __restrict__ blocks, const double* __restrict__ R,
              const double* __restrict__ Rinv, const double* __restrict__ lisqrt,
              const double* __restrict__ dz, const double* __restrict__ ds, double amax, int mode,
              double* __restrict__ out, uint32_t* __restrict__ status) {
  extern __shared__ double smem[];
  const int b = blockIdx.x, side = blockIdx.y;
  const BlockDesc bd = blocks[b];
  const int n = bd.n;
  double* B = smem;
  double* X = B + kMat;
  double* T = X + kMat;
  double* D = T + kMat;
  double* dd = D + kMat;  // d[n], e[n], one int
  double* ee = dd + SDPXG_NMAX;
  int* best = reinterpret_cast<int*>(ee + SDPXG_NMAX);
  cta_load_mat(B, (side == 0 ? R : Rinv) + bd.mat_off, n, pad8(n));
  cta_load_smat(X, (side == 0 ? dz : ds) + bd.svec_off, n, pad8(n));
  __syncthreads();
  cta_congruence(D, T, X, B, side == 1, n);
  const double* ls = lisqrt + bd.vec_off;
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    int i = e % n, j = e / n;
    double v = 0.5 * (SM(D, i, j) + SM(D, j, i));
    SM(X, i, j) = ls[i] * v * ls[j];  // Delta (symmetric)
  }
  __syncthreads();
  double res = amax;
  // admission: chol(I + amax Delta)
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    int i = e % n, j = e / n;
    SM(T, i, j) = amax * SM(X, i, j) + (i == j ? 1.0 : 0.0);
  }
  __syncthreads();
  bool admitted = (n <= 3 && mode == 0) ? false : cta_cholesky_lower(T, n);
  if (mode == 1) {
    if (threadIdx.x == 0) out[2 * b + side] = admitted ? amax : 0.0;
    return;
  }
  if (!admitted) {
    cta_tridiagonalize(X, n, dd, ee, T);
    bool ok = true;
    double g = cta_eig_min(dd, ee, n, reinterpret_cast<double2*>(B), best, &ok);
    if (!ok || !isfinite(g)) {
      if (threadIdx.x == 0) atomicOr(status, SDPXG_ST_EIG_FAIL);
      res = 0.0;
    } else {
      res = (g < 0.0) ? fmin(-1.0 / g, amax) : amax;
    }
  }
  if (threadIdx.x == 0) out[2 * b + side] = res;
}

// Eigenvalue summary of smat(v) per block: out[2b] = lambda_min, out[2b+1] = sum of positive
// eigenvalues.  (margins, psdtrianglecone.rs; also the cone distance of the original-
// coordinate acceptance test, default/original_check.rs:306-340.)
// min_only != 0 (the acceptance test, which reads only max(0, -lambda_min)): out[2b] =
// min(lambda_min, 0) and out[2b+1] = 0.  A block whose Cholesky factorisation succeeds is
// positive definite to working accuracy and gives 0 without an eigensolve; the others take the
// tridiagonal reduction and the multisection for lambda_min alone.
extern "C" __global__ void __launch_bounds__(SDPXG_EIG_THREADS)
k_margins(const BlockDesc* __restrict__ blocks, const double* __restrict__ v, long ld,
          double* __restrict__ out, uint32_t* __restrict__ status, int min_only) {
  extern __shared__ double smem[];
  const int b = blockIdx.x;
  const BlockDesc bd = blocks[b];
  const int n = bd.n;
  double* X = smem;
  double* dd = X + kMat;
  double* ee = dd + SDPXG_NMAX;
  double* work = ee + SDPXG_NMAX;
  double* eig = work + SDPXG_TRIDIAG_WORK;
  int* best = reinterpret_cast<int*>(eig + SDPXG_NMAX);
  const double* vb = v + (long)blockIdx.y * ld + bd.svec_off;
  const long o = 2L * ((long)blockIdx.y * gridDim.x + b);
  cta_load_smat(X, vb, n, pad8(n));
  __syncthreads();
  if (min_only) {
    if (cta_cholesky_lower(X, n)) {
      if (threadIdx.x == 0) out[o] = out[o + 1] = 0.0;
      return;
    }
    cta_load_smat(X, vb, n, pad8(n));
    __syncthreads();
    cta_tridiagonalize(X, n, dd, ee, work);
    bool ok = true;
    const double g = cta_eig_min(dd, ee, n, reinterpret_cast<double2*>(work), best, &ok);
    if (threadIdx.x == 0) {
      if (!ok || !isfinite(g)) atomicOr(status, SDPXG_ST_EIG_FAIL);
      out[o] = fmin(g, 0.0);
      out[o + 1] = 0.0;
    }
    return;
  }
  cta_tridiagonalize(X, n, dd, ee, work);
  cta_eig_all(dd, ee, n, reinterpret_cast<double2*>(work), eig, status);
  __syncthreads();
  if (threadIdx.x == 0) {
    double mn = eig[0], pos = 0.0;
    for (int k = 0; k < n; ++k) {
      mn = fmin(mn, eig[k]);
      pos += fmax(eig[k], 0.0);
    }
    out[o] = mn;
    out[o + 1] = pos;
  }
}
