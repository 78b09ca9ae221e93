// Condensed Schur complement of the PSD rows and the constraint-operator products.
//
// Data layout (uploaded once per problem):
//   For PSD block j the columns of A that touch it are stored densely, column-major,
//   as Acol[acol_off[j] + t * tri(n_j) + r], t < k_j, with their global indices
//   col_idx[col_ptr[j] + t].  The transpose map lists, per constraint i, its (block, t)
//   pairs in cone order: c2b_ptr[i] .. c2b_ptr[i+1] into c2b_blk / c2b_loc.
//
// Schur entry (kkt/condensed/psd.rs:1120-1570, scaling.rs:7-81):
//   H_ab = sum_j < A_aj , Ginv_j A_bj Ginv_j >  (+ P_ab)
// computed as T = svec(Ginv A Ginv) per column (k_schur_transform), one grouped GEMM
// S_j = Acol_j' T_j per block (k_schur_block_gemm), and a deterministic cone-order gather
// into the dense m x m matrix (k_schur_gather).
#include <cooperative_groups.h>

#include "common.cuh"

namespace {
constexpr int kMat = SDPXG_LD * SDPXG_NMAX;
}

// One CTA per (block, column) work item: item w -> block wblk[w], local column wloc[w].
extern "C" __global__ void __launch_bounds__(SDPXG_CONE_THREADS)
k_schur_transform(const BlockDesc* __restrict__ blocks, const int* __restrict__ wblk,
                  const int* __restrict__ wloc, const long* __restrict__ acol_off,
                  const double* __restrict__ Ginv, const double* __restrict__ Acol,
                  double* __restrict__ Tcol) {
  extern __shared__ double smem[];
  const int j = wblk[blockIdx.x], t = wloc[blockIdx.x];
  const BlockDesc bd = blocks[j];
  const int n = bd.n;
  const int tn = n * (n + 1) / 2;
  double* G = smem;
  double* X = G + kMat;
  double* Y = X + kMat;
  cta_load_mat<2>(G, Ginv + bd.mat_off, n, pad8(n));
  const long off = acol_off[j] + (long)t * tn;
  cta_load_smat<2>(X, Acol + off, n, pad8(n));
  __syncthreads();
  cta_gemm<false, false, 2>(Y, G, X, n);  // Y = Ginv A
  __syncthreads();
  cta_gemm<false, false, 2, GEMM_SYMMETRIC>(X, Y, G, n);  // X = Ginv A Ginv
  __syncthreads();
  cta_store_svec(Tcol + off, X, n);
}

// Grouped GEMM S_j = Acol_j' * Tcol_j (k_j x k_j, inner tri(n_j)) on the FP64 tensor cores.
// Tile list entries (block, tile row, tile col) of 32 x 32 output tiles; the inner rows of a tile are dealt
// in 32-row chunks to the CTAs of one cluster (its size is the launch's), whose sums meet through
// distributed shared memory in rank order.  A two-stage ring of chunks (cp.async, 8 bytes: a column
// starts anywhere) feeds the 8 warps, each with two 8 x 8 output subtiles accumulated by mma.sync m8n8k4
// (lane (r, q): A fragment A'(row r, k q), B fragment T(k q, column r); results C(r, 2q) and C(r, 2q + 1)).
// Chunk columns are 36 doubles apart (4 mod 16: the fragment reads of a half-warp hit distinct banks).
// Bound by the latency of the chunks while the tiles are few: 49 tiles of 1275 inner rows (order 50, 200
// constraints) took 117 us with one CTA a tile and plain loads, 27.5 with a ring, 17 with it in clusters.  Two
// stages leave room for six CTAs an SM; with four stages and three CTAs an SM 16.3 us against 14.4 here, 59.6
// against 57.5 (256 tiles of 2080 rows), 720 against 654 (4000 tiles of 2080 rows), 611 against 444 (50000 tiles of
// 36 rows).
#define SCHUR_TILE 32
#define SCHUR_KC 32
#define SCHUR_LD 36
#define SCHUR_STAGES 2
static_assert(kSchurSmem == SCHUR_STAGES * 2 * SCHUR_TILE * SCHUR_LD * sizeof(double), "ring");

namespace {

__device__ __forceinline__ void schur_copy8(double* dst, const double* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 8 : 0)
               : "memory");
}

}  // namespace

extern "C" __global__ void __launch_bounds__(SDPXG_THREADS)
k_schur_block_gemm(const BlockDesc* __restrict__ blocks, const int* __restrict__ tiles,
                   const int* __restrict__ kcount, const long* __restrict__ acol_off,
                   const long* __restrict__ s_off, const double* __restrict__ Acol,
                   const double* __restrict__ Tcol, double* __restrict__ S) {
  namespace cg = cooperative_groups;
  extern __shared__ double smem[];
  cg::cluster_group cluster = cg::this_cluster();
  const int split = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int* tile = tiles + 3 * (blockIdx.x / split);
  const int j = tile[0], ti = tile[1], tj = tile[2];
  const int n = blocks[j].n;
  const int tn = n * (n + 1) / 2;
  const int k = kcount[j];
  const double* A = Acol + acol_off[j];
  const double* T = Tcol + acol_off[j];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r = lane >> 2, q = lane & 3;
  const int chunks = (tn + SCHUR_KC - 1) / SCHUR_KC, c_end = (int)((long)chunks * (rank + 1) / split);
  int next = (int)((long)chunks * rank / split);
  auto load = [&](int c, int stage) {  // a lane: one row; a warp: columns w, w + 8, ...
    if (c < c_end) {
      double* As = smem + stage * 2 * SCHUR_TILE * SCHUR_LD;
      double* Ts = As + SCHUR_TILE * SCHUR_LD;
      const int row = c * SCHUR_KC + lane;
#pragma unroll
      for (int u = 0; u < SCHUR_TILE / 8; ++u) {
        const int cc = w + 8 * u, ca = ti * SCHUR_TILE + cc, cb = tj * SCHUR_TILE + cc;
        const bool ia = row < tn && ca < k, ib = row < tn && cb < k;
        schur_copy8(As + cc * SCHUR_LD + lane, ia ? A + (long)ca * tn + row : A, ia);
        schur_copy8(Ts + cc * SCHUR_LD + lane, ib ? T + (long)cb * tn + row : T, ib);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  // subtiles w and w + 8 of the 4 x 4 grid of 8 x 8 subtiles
  const int I0 = w >> 2, J = w & 3, I1 = I0 + 2;
  double c[2][2] = {};
  const int first = next;
  for (int s = 0; s < SCHUR_STAGES - 1; ++s) load(next + s, s);
  for (; next < c_end; ++next) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(SCHUR_STAGES - 2) : "memory");
    __syncthreads();
    load(next + SCHUR_STAGES - 1, (next - first + SCHUR_STAGES - 1) % SCHUR_STAGES);
    const double* As = smem + (next - first) % SCHUR_STAGES * 2 * SCHUR_TILE * SCHUR_LD;
    const double* Ts = As + SCHUR_TILE * SCHUR_LD;
#pragma unroll
    for (int ks = 0; ks < SCHUR_KC / 4; ++ks) {
      const int kk = 4 * ks + q;
      const double b = Ts[(8 * J + r) * SCHUR_LD + kk];
      dmma_m8n8k4(c[0][0], c[0][1], As[(8 * I0 + r) * SCHUR_LD + kk], b);
      dmma_m8n8k4(c[1][0], c[1][1], As[(8 * I1 + r) * SCHUR_LD + kk], b);
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  double* sum = smem;  // 32 x 32, columns SCHUR_LD apart
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    double* o = sum + 8 * (I0 + 2 * h) + r + (8 * J + 2 * q) * SCHUR_LD;
    o[0] = c[h][0];
    o[SCHUR_LD] = c[h][1];
  }
  cluster.sync();
  double* out = S + s_off[j];
  for (int e = threadIdx.x + rank * blockDim.x; e < SCHUR_TILE * SCHUR_TILE; e += split * blockDim.x) {
    const int i = e & 31, cc = e >> 5, a0 = ti * SCHUR_TILE + i, b0 = tj * SCHUR_TILE + cc;
    if (a0 >= k || b0 >= k) continue;
    double v = 0.0;
    for (int p = 0; p < split; ++p) v += cluster.map_shared_rank(sum, p)[i + cc * SCHUR_LD];
    out[a0 + (long)b0 * k] = v;
  }
  cluster.sync();  // nobody leaves while its sums are read
}

// H (m x m, full, column-major) = sum over shared blocks of S_j[la, lb], in cone order.
// One CTA per 8 x 8 tile on or above the diagonal (grid.x numbers them by columns); both triangles are
// written (symmetrised by construction), the mirrored tile through shared memory so that its stores are
// whole sectors too.  A non-finite entry sets SDPXG_ST_NONFINITE (`status`), which saves another pass over H
// (74 us at m = 4000).  A thread's chain of loads bounds it, so small CTAs on all SMs: m = 4000, four of 64
// blocks a row, 129 us (131 with 16 x 16, 145 with 32 x 32 tiles; 164 with one thread an entry and stores a
// column apart); m = 100, all of 200 blocks a row, 76 us (80, 174); m = 1500, 40 blocks 184 (209, 264).
#define SCHUR_GT kSchurGatherTile
extern "C" __global__ void __launch_bounds__(SCHUR_GT * SCHUR_GT)
k_schur_gather(int m, const int* __restrict__ c2b_ptr, const int* __restrict__ c2b_blk,
               const int* __restrict__ c2b_loc, const int* __restrict__ kcount,
               const long* __restrict__ s_off, const double* __restrict__ S, double* __restrict__ H,
               uint32_t* __restrict__ status) {
  __shared__ double mirror[SCHUR_GT][SCHUR_GT + 1];
  int tj = (int)((sqrtf(8.0f * blockIdx.x + 1.0f) - 1.0f) * 0.5f);
  while ((long)tj * (tj + 1) / 2 > blockIdx.x) --tj;
  while ((long)(tj + 1) * (tj + 2) / 2 <= blockIdx.x) ++tj;
  const int ti = (int)(blockIdx.x - (long)tj * (tj + 1) / 2);
  const int lane = threadIdx.x % SCHUR_GT, w = threadIdx.x / SCHUR_GT;
  const int a = SCHUR_GT * ti + lane;
  bool bad = false;
  {
    const int b = SCHUR_GT * tj + w;
    if (a <= b && b < m) {
      int pa = c2b_ptr[a], pb = c2b_ptr[b];
      const int ea = c2b_ptr[a + 1], eb = c2b_ptr[b + 1];
      double acc = 0.0;
      while (pa < ea && pb < eb) {
        int ja = c2b_blk[pa], jb = c2b_blk[pb];
        if (ja < jb) {
          ++pa;
        } else if (jb < ja) {
          ++pb;
        } else {
          const int k = kcount[ja];
          const double* Sj = S + s_off[ja];
          int la = c2b_loc[pa], lb = c2b_loc[pb];
          // symmetric in exact arithmetic: average the two computed halves
          acc += 0.5 * (Sj[la + (long)lb * k] + Sj[lb + (long)la * k]);
          ++pa;
          ++pb;
        }
      }
      H[a + (long)b * m] = acc;
      mirror[lane][w] = acc;
      bad = !isfinite(acc);
    }
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(status, SDPXG_ST_NONFINITE);
  const int b = SCHUR_GT * tj + lane;
  const int col = SCHUR_GT * ti + w;
  if (col < b && b < m) H[b + (long)col * m] = mirror[w][lane];
}

// H += sym(P) for P given as an upper-triangular CSC (n x n).
extern "C" __global__ void k_add_upper_csc(int n, const int* __restrict__ colptr,
                                           const int* __restrict__ rowval,
                                           const double* __restrict__ val, double* __restrict__ H) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  for (int p = colptr[j]; p < colptr[j + 1]; ++p) {
    int i = rowval[p];
    if (i > j) continue;
    H[i + (long)j * n] += val[p];
    if (i != j) H[j + (long)i * n] += val[p];
  }
}

// y[rows of block j] = alpha * Acol_j x[cols_j] + beta * base.  One CTA per 32-row tile of a block
// (tile list ftile_blk / ftile_r0): one row a lane, the columns dealt to GROUPS warps; the partial sums are
// combined in a fixed order (deterministic).  Bound by the memory round trips of a thread's columns while the
// tiles are few (then sixteen warps and eight loads in flight a thread), by the warps themselves when they are
// many (four).
namespace {

template <int GROUPS>
__global__ void __launch_bounds__(32 * GROUPS)
k_op_forward(const BlockDesc* __restrict__ blocks, const int* __restrict__ kcount,
             const int* __restrict__ col_ptr, const int* __restrict__ col_idx,
             const long* __restrict__ acol_off, const double* __restrict__ Acol,
             const int* __restrict__ ftile_blk, const int* __restrict__ ftile_r0,
             const double* __restrict__ x, double alpha, double beta, const double* base, double* y) {
  __shared__ double part[GROUPS][32];
  const int j = ftile_blk[blockIdx.x], r0 = ftile_r0[blockIdx.x];
  const BlockDesc bd = blocks[j];
  const int tn = bd.n * (bd.n + 1) / 2;
  const int k = kcount[j];
  const double* A = Acol + acol_off[j];
  const int* cols = col_idx + col_ptr[j];
  const int rr = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int r = r0 + rr;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  if (r < tn) {
    if (GROUPS == 4) {
      for (int t = g; t < k; t += GROUPS) acc[0] = fma(A[(long)t * tn + r], x[cols[t]], acc[0]);
    } else {  // steps t, t + GROUPS, ...: whole fours into the four sums, the rest into the first
      int t = g;
      for (; t + 7 * GROUPS < k; t += 8 * GROUPS) {
        int c[8];
        double a[8], v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          c[u] = __ldg(cols + t + u * GROUPS);
          a[u] = __ldg(A + (long)(t + u * GROUPS) * tn + r);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = __ldg(x + c[u]);
#pragma unroll
        for (int u = 0; u < 8; ++u) acc[u & 3] = fma(a[u], v[u], acc[u & 3]);
      }
      if (t < k) {  // the last ones at once too
        int c[7];
        double a[7], v[7];
#pragma unroll
        for (int u = 0; u < 7; ++u) {
          const bool in = t + u * GROUPS < k;
          c[u] = in ? __ldg(cols + t + u * GROUPS) : -1;
          a[u] = in ? __ldg(A + (long)(t + u * GROUPS) * tn + r) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 7; ++u) v[u] = c[u] >= 0 ? __ldg(x + c[u]) : 0.0;
        const bool four = t + 3 * GROUPS < k;
#pragma unroll
        for (int u = 0; u < 7; ++u) {
          if (t + u * GROUPS >= k) continue;
          if (u > 0 && u < 4 && four) acc[u] = fma(a[u], v[u], acc[u]);
          else acc[0] = fma(a[u], v[u], acc[0]);
        }
      }
    }
  }
  part[g][rr] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
  __syncthreads();
  if (g == 0 && r < tn) {
    double s = 0.0;
#pragma unroll
    for (int u = 0; u < GROUPS; ++u) s += part[u][rr];
    const long o = bd.svec_off + r;
    y[o] = alpha * s + ((beta == 0.0) ? 0.0 : beta * base[o]);
  }
}

}  // namespace

namespace sdpxg {

// Sixteen warps a tile up to four CTAs an SM, four above.  Sixteen / four, us: 40 tiles of 200 columns 5.7 / 9.2, 150
// of 3000 37 / 190, 65 of 500 6.2 / 16.4; 1000 of 300 16.4 / 12.3, 3500 of 10 22.6 / 6.2, 13000 of 50 141 / 45.
void launch_op_forward(int tiles, const BlockDesc* blocks, const int* kcount, const int* col_ptr, const int* col_idx,
                       const long* acol_off, const double* Acol, const int* ftile_blk, const int* ftile_r0,
                       const double* x, double alpha, double beta, const double* base, double* y, cudaStream_t st) {
  auto go = [&](auto kernel, int groups) {
    kernel<<<tiles, 32 * groups, 0, st>>>(blocks, kcount, col_ptr, col_idx, acol_off, Acol, ftile_blk, ftile_r0, x,
                                          alpha, beta, base, y);
  };
  if (tiles <= 4 * 148) go(k_op_forward<16>, 16);
  else go(k_op_forward<4>, 4);
}

}  // namespace sdpxg

// Per-block partial adjoint p[acol column] = Acol_j[:, t] . z_j  (one warp per column, eight loads
// in flight a lane)
extern "C" __global__ void k_op_adjoint_partial(const BlockDesc* __restrict__ blocks,
                                                const int* __restrict__ wblk,
                                                const int* __restrict__ wloc,
                                                const int* __restrict__ col_ptr,
                                                const long* __restrict__ acol_off,
                                                const double* __restrict__ Acol,
                                                const double* __restrict__ z, long ldz,
                                                double* __restrict__ p, long ldp, int nwork) {
  const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= nwork) return;
  const int j = wblk[w], t = wloc[w];
  const BlockDesc bd = blocks[j];
  const int tn = bd.n * (bd.n + 1) / 2;
  const double* A = Acol + acol_off[j] + (long)t * tn;
  const double* zc = z + (long)blockIdx.y * ldz + bd.svec_off;
  double a8[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  int r = lane;
  for (; r + 7 * 32 < tn; r += 8 * 32)
#pragma unroll
    for (int u = 0; u < 8; ++u) a8[u] = fma(A[r + 32 * u], zc[r + 32 * u], a8[u]);
  if (tn - (r - lane) > 64) {
#pragma unroll
    for (int u = 0; u < 7; ++u)
      if (r + 32 * u < tn) a8[u] = fma(A[r + 32 * u], zc[r + 32 * u], a8[u]);
  } else {  // a short column, or a long one's end
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (r + 32 * u < tn) a8[u] = fma(A[r + 32 * u], zc[r + 32 * u], a8[u]);
  }
  double acc = ((a8[0] + a8[1]) + (a8[2] + a8[3])) + ((a8[4] + a8[5]) + (a8[6] + a8[7]));
  acc = warp_sum(acc);
  if (lane == 0) p[(long)blockIdx.y * ldp + col_ptr[j] + t] = acc;
}

// y[i] = alpha * sum over (block, t) of constraint i of p[...] + beta * base[i]  (cone order)
extern "C" __global__ void k_op_adjoint_gather(int n, const int* __restrict__ c2b_ptr,
                                               const int* __restrict__ c2b_blk,
                                               const int* __restrict__ c2b_loc,
                                               const int* __restrict__ col_ptr,
                                               const double* __restrict__ p, long ldp,
                                               double alpha, double beta, const double* base, double* y,
                                               long ldy) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* pc = p + (long)blockIdx.y * ldp;
  double acc = 0.0;
  for (int q = c2b_ptr[i]; q < c2b_ptr[i + 1]; ++q) acc += pc[col_ptr[c2b_blk[q]] + c2b_loc[q]];
  const long o = (long)blockIdx.y * ldy + i;
  y[o] = alpha * acc + ((beta == 0.0) ? 0.0 : beta * base[o]);
}
