// MPFR dense LDL' kernels on MpFloat<N> arrays (see mp_ldl.cuh and mp.cuh).
#include <cooperative_groups.h>

#include <stdexcept>

#include "device.cuh"
#include "mp.cuh"
#include "mp_ldl.cuh"

namespace sdpxg {
namespace {

using mpd::Val;

template <int N>
__device__ __forceinline__ unsigned char* el(unsigned char* A, long i, long j, long ld) {
  return A + (i + j * ld) * (8L * N + 8);
}
template <int N>
__device__ __forceinline__ const unsigned char* el(const unsigned char* A, long i, long j, long ld) {
  return A + (i + j * ld) * (8L * N + 8);
}

// arrow.rs:156-242 ldl_dots on one block: columns in order; the pivot
// d_j = a_jj - dot(r_j, w_j) (the exact difference rounded once when that rounds to zero), the
// pivot rule, D^-1; then every later row i: r_ij = (a_ij - dot(r_i, w_j)) * d_j^-1,
// w_ij = r_ij d_j.  Dots are exact and rounded once; the other operations round once each.
// One cluster of four CTAs, bound by the chain of its columns: the pivot (dot, difference, reciprocal)
// and the column's dots are independent once the column before is done, so warp 0 of every CTA forms
// the pivot (the same one: cheaper than handing it round) while the other warps take the dots of the
// CTA's rows (i mod 4), 16 lanes a row; then one thread a row finishes its two products.  A barrier of the
// cluster closes a column.  The block's lower triangle is copied into a row-major scratch R (W is row-major
// too), w_j is staged in shared memory.
// Up to 4 limbs 512 threads leave 128 registers for the accumulator, operands and product of a
// dot; above, 256 threads and 8 lanes a row.  LDL' of order 1000 at 256 bits (eight leaves of 125): 217 ms
// with a warp a row and run-time limb loops in local memory, 26 ms with one CTA (33000 cycles a column: dots
// 28000, or dot 9100, reciprocal 13900 of the pivot; 8300 for the products, on four warps), 19.1 with four and the long division; a
// leaf 1348 us with R in global memory, 1211 with the CTAs' rows and the pivot's in shared memory.
// Scratch: 2 size^2 elements (W, then R).
constexpr int kLeafCtas = 4;
// The rows of a CTA stay in shared memory, where they fit next to the rest (32 rows of 128 entries).
template <int N>
constexpr bool kLeafRows = N <= 5;
template <int N>
constexpr int kLeafThreads = N <= 4 ? 512 : 256;
template <int N>
__global__ void __cluster_dims__(kLeafCtas, 1, 1) __launch_bounds__(kLeafThreads<N>)
    k_mp_ldl_dots(unsigned char* A, long lda, int off, int size, unsigned char* Wsc, unsigned char* dinv,
                  const unsigned char* reg, uint32_t* status) {
  namespace cg = cooperative_groups;
  constexpr int esz = 8 * N + 8, G = N <= 4 ? 16 : 8, C = kLeafCtas;
  constexpr bool kRows = kLeafRows<N>;
  extern __shared__ __align__(8) unsigned char sr[];             // the CTA's rows of R (kRows)
  __shared__ __align__(8) unsigned char srow[kMpRecBase * esz];  // w_j
  __shared__ __align__(8) unsigned char sprow[kMpRecBase * esz]; // r_j
  __shared__ __align__(8) unsigned char sdot[kMpRecBase * esz];  // dot(r_i, w_j), i > j
  __shared__ __align__(8) unsigned char sd[2 * esz];             // d_j, d_j^-1
  __shared__ int s_fail;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), tid = rank * (int)blockDim.x + (int)threadIdx.x;
  unsigned char* B = A + ((long)off + (long)off * lda) * esz;
  unsigned char* W = Wsc;                            // row-major: (i, c) at i * size + c
  unsigned char* R = Wsc + (long)size * size * esz;  // row-major copy of the lower triangle
  auto rm = [&](unsigned char* M, int i, int c) { return M + ((long)i * size + c) * esz; };
  auto own = [&](int i, int c) { return kRows ? sr + ((i / C) * size + c) * esz : rm(R, i, c); };  // i mod C = rank
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) s_fail = 0;
  for (long wd = threadIdx.x; kRows && wd < (long)(size + C - 1) / C * size * (N + 1); wd += blockDim.x) {
    const long e = wd / (N + 1), o = wd % (N + 1) * 8;
    const int i = (int)(e / size) * C + rank, c = (int)(e % size);
    if (i < size && c <= i)
      *reinterpret_cast<unsigned long long*>(own(i, c) + o) =
          *reinterpret_cast<const unsigned long long*>(el<N>(B, i, c, lda) + o);
  }
  for (long wd = tid; !kRows && wd < (long)size * size * (N + 1); wd += C * blockDim.x) {  // R(i, c) = B(i, c)
    const long e = wd / (N + 1), o = wd % (N + 1) * 8;
    const int i = (int)(e / size), c = (int)(e % size);
    if (c <= i)
      *reinterpret_cast<unsigned long long*>(rm(R, i, c) + o) =
          *reinterpret_cast<const unsigned long long*>(el<N>(B, i, c, lda) + o);
  }
  cluster.sync();
  for (int j = 0; j < size; ++j) {
    for (int wd = threadIdx.x; wd < j * (N + 1); wd += blockDim.x) {
      reinterpret_cast<unsigned long long*>(srow)[wd] = reinterpret_cast<const unsigned long long*>(rm(W, j, 0))[wd];
      reinterpret_cast<unsigned long long*>(sprow)[wd] = reinterpret_cast<const unsigned long long*>(rm(R, j, 0))[wd];
    }
    __syncthreads();
    bool ok = true;
    if (warp == 0) {  // the pivot: the dot over the lanes, the rest on lane 0
      const Val<N> a = mpd::load<N>(el<N>(B, j, j, lda));  // B is written after the last column
      const Val<N> dot = mpd::dot<N, 32>(nullptr, sprow, 1, srow, 1, j, &ok);
      Val<N> d = mpd::addsub<N>(a, dot, -1);
      if (d.zero && j > 0) d = mpd::dot<N, 32>(&a, sprow, 1, srow, 1, j, &ok);
      if (lane == 0) {
        if (reg) {  // DenseLeaf::pivot (arrow.rs:618-632), sign +1
          const Val<N> eps = mpd::load<N>(reg), delta = mpd::load<N>(reg + esz);
          if (mpd::cmp<N>(d, eps) < 0) d = delta;
        }
        if (d.zero) {
          atomicOr(status, SDPXG_ST_PIVOT_FAIL);
          s_fail = 1;
        } else {
          const Val<N> di = mpd::recip<N>(d);
          mpd::store<N>(sd, d, status);
          mpd::store<N>(sd + esz, di, status);
          if (rank == 0) mpd::store<N>(dinv + (long)j * esz, di, status);
        }
      }
    } else {
      const int sub = lane & (G - 1);
      // the rows i > j with i mod C = rank, group-uniform
      for (int i = j + 1 + ((rank - j - 1) & (C - 1)) + C * ((threadIdx.x - 32) / G); i < size;
           i += C * ((blockDim.x - 32) / G)) {
        const Val<N> dot = mpd::dot<N, G>(nullptr, own(i, 0), 1, srow, 1, j, &ok);
        if (sub == 0) mpd::stage<N>(sdot + i * esz, dot);
      }
    }
    if (!ok) atomicOr(status, SDPXG_ST_EXACT_SPREAD);
    __syncthreads();
    if (s_fail) return;  // in every CTA: the pivots are the same
    for (int i = j + 1 + ((rank - j - 1) & (C - 1)) + C * (int)threadIdx.x; i < size; i += C * blockDim.x) {
      const Val<N> d = mpd::load<N>(sd), di = mpd::load<N>(sd + esz);
      const Val<N> t = mpd::addsub<N>(mpd::load<N>(own(i, j)), mpd::unstage<N>(sdot + i * esz), -1);
      const Val<N> v = mpd::mul<N>(t, di);
      mpd::store<N>(rm(R, i, j), v, status);
      if (kRows) mpd::store<N>(own(i, j), v, status);
      mpd::store<N>(rm(W, i, j), mpd::mul<N>(v, d), status);
    }
    cluster.sync();  // row j + 1 of R and W is there for every CTA
  }
  for (long wd = tid; wd < (long)size * size * (N + 1); wd += C * blockDim.x) {  // B(i, c) = R(i, c), c < i
    const long e = wd / (N + 1), o = wd % (N + 1) * 8;
    const int i = (int)(e / size), c = (int)(e % size);
    if (c < i)
      *reinterpret_cast<unsigned long long*>(el<N>(B, i, c, lda) + o) =
          *reinterpret_cast<const unsigned long long*>(rm(R, i, c) + o);
  }
  for (int j = tid; j < size; j += C * blockDim.x)  // unit diagonal
    mpd::store<N>(el<N>(B, j, j, lda), mpd::one_val<N>(), status);
}

// arrow.rs:437-447: each row of B solves x L' = b by exact dots, x_j = b_j - dot(x_<j, L(j, <j)).
// One warp per row, four rows per CTA: bound by the chain of the row's k dots, each over the 32
// lanes with the row's solved entries and the row of L in shared memory (the next one on its way in
// registers meanwhile): k = 125 at 256 bits 473 us, 597 with L read from global memory by every dot.
constexpr int kSolveRows = 4;
template <int N>
__global__ void __launch_bounds__(32 * kSolveRows) k_mp_solve_lt(const unsigned char* L, long ldl, int k,
                                                                 unsigned char* B, long ldb, int m,
                                                                 uint32_t* status) {
  constexpr int esz = 8 * N + 8;
  static_assert(32 * kSolveRows == kMpRecBase, "a thread has N + 1 words of a row of L");
  __shared__ __align__(8) unsigned char sx[kSolveRows][kMpRecBase * esz];
  __shared__ __align__(8) unsigned char sl[kMpRecBase * esz];  // L(j, c), c < j
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * kSolveRows + warp;
  for (int j = 0; j < k; ++j) {
    unsigned long long next[N + 1];  // words threadIdx.x + 128 u of L(j + 1, 0 .. j)
#pragma unroll
    for (int u = 0; u <= N; ++u) {
      const int wd = (int)threadIdx.x + 32 * kSolveRows * u, c = wd / (N + 1);
      next[u] = j + 1 < k && c <= j
                    ? reinterpret_cast<const unsigned long long*>(el<N>(L, j + 1, c, ldl))[wd % (N + 1)]
                    : 0ull;
    }
    if (i < m) {  // warp-uniform
      bool ok = true;
      const Val<N> b = mpd::load<N>(el<N>(B, i, j, ldb));
      const Val<N> dot = mpd::dot<N, 32>(nullptr, sx[warp], 1, sl, 1, j, &ok);
      const Val<N> x = mpd::addsub<N>(b, dot, -1);
      if (lane == 0) {
        if (!ok) atomicOr(status, SDPXG_ST_EXACT_SPREAD);
        mpd::store<N>(sx[warp] + j * esz, x, status);
        mpd::store<N>(el<N>(B, i, j, ldb), x, status);
      }
    }
    __syncthreads();  // x_j visible to the lanes' next dot, nobody reads row j of L any more
#pragma unroll
    for (int u = 0; u <= N; ++u)
      reinterpret_cast<unsigned long long*>(sl)[threadIdx.x + 32 * kSolveRows * u] = next[u];
    __syncthreads();
  }
}

template <int N>
__global__ void k_mp_sub_block(unsigned char* B, long ldb, const unsigned char* P, long ldp, int m, int n,
                               uint32_t* status) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long)m * n) return;
  const int i = (int)(idx % m), j = (int)(idx / m);
  unsigned char* b = el<N>(B, i, j, ldb);
  mpd::store<N>(b, mpd::addsub<N>(mpd::load<N>(b), mpd::load<N>(el<N>(P, i, j, ldp)), -1), status);
}

template <int N>
__global__ void k_mp_copy_scale_cols(unsigned char* A, long lda, unsigned char* W, const unsigned char* d, int m,
                                     int n, uint32_t* status) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long)m * n) return;
  const int i = (int)(idx % m), j = (int)(idx / m);
  unsigned char* src = el<N>(A, i, j, lda);
  const Val<N> a = mpd::load<N>(src);
  unsigned long long* w = reinterpret_cast<unsigned long long*>(el<N>(W, i, j, m));
#pragma unroll
  for (int q = 0; q <= N; ++q) w[q] = reinterpret_cast<const unsigned long long*>(src)[q];
  mpd::store<N>(src, mpd::mul<N>(a, mpd::load<N>(el<N>(d, j, 0, 0))), status);
}

template <int N>
__global__ void k_mp_sub_upper_t(unsigned char* A, long lda, const unsigned char* C, long ldc, int n,
                                 uint32_t* status) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long)n * n) return;
  const int b = (int)(idx % n), a = (int)(idx / n);  // entry (b, a) of the lower triangle
  if (b < a) return;
  unsigned char* x = el<N>(A, b, a, lda);
  mpd::store<N>(x, mpd::addsub<N>(mpd::load<N>(x), mpd::load<N>(el<N>(C, a, b, ldc)), -1), status);
}

// XpotrfScalar::xpotrf for MpFloat (algebra/dense/blas/mpfr.rs:726-789): left-looking Cholesky
// of the stored triangle, entry (i, k), i >= k, at i * si + k * sk (lower: si = 1, sk = ld;
// upper: si = ld, sk = 1).  Per column j: d = a_jj - dot(l_j, l_j) (the dot exact and rounded
// once, the difference rounded), failure when d <= 0 (info = j + 1), l_jj = sqrt(d) rounded; then
// every later row i: l_ij = (a_ij - dot(l_i, l_j)) / l_jj, each operation rounded once.  The rows'
// dots take eight lanes each.
constexpr int kPotrfThreads = 256;
template <int N>
__global__ void __launch_bounds__(kPotrfThreads) k_mp_potrf(unsigned char* A, long si, long sk, int n, int* info,
                                                            uint32_t* status) {
  constexpr int esz = 8 * N + 8, G = 8;
  __shared__ __align__(8) unsigned char sd[esz];
  __shared__ int s_fail;
  auto at = [&](long i, long k) { return A + (i * si + k * sk) * esz; };
  if (threadIdx.x == 0) {
    s_fail = 0;
    *info = 0;
  }
  __syncthreads();
  for (int j = 0; j < n; ++j) {
    bool ok = true;
    if (threadIdx.x < 32) {  // warp 0 forms the pivot's dot, its lane 0 the rest
      const Val<N> dot = mpd::dot<N, 32>(nullptr, at(j, 0), sk, at(j, 0), sk, j, &ok);
      if (threadIdx.x == 0) {
        const Val<N> d = mpd::addsub<N>(mpd::load<N>(at(j, j)), dot, -1);
        if (d.zero || d.neg) {
          mpd::store<N>(at(j, j), d, status);
          *info = j + 1;
          s_fail = 1;
        } else {
          const Val<N> r = mpd::root<N>(d);
          mpd::store<N>(at(j, j), r, status);
          mpd::store<N>(sd, r, status);
        }
      }
    }
    __syncthreads();
    if (s_fail) {
      if (!ok) atomicOr(status, SDPXG_ST_EXACT_SPREAD);
      return;
    }
    const Val<N> r = mpd::load<N>(sd);
    for (long i = j + 1 + threadIdx.x / G; i < n; i += kPotrfThreads / G) {  // group-uniform
      const Val<N> dot = mpd::dot<N, G>(nullptr, at(i, 0), sk, at(j, 0), sk, j, &ok);
      if ((threadIdx.x & (G - 1)) == 0) {
        unsigned char* p = at(i, j);
        mpd::store<N>(p, mpd::divide<N>(mpd::addsub<N>(mpd::load<N>(p), dot, -1), r), status);
      }
    }
    if (!ok) atomicOr(status, SDPXG_ST_EXACT_SPREAD);
    __syncthreads();
  }
}

void check_limbs(int N) {
  if (N < 1 || N > mpd::kMaxN) throw std::invalid_argument("MPFR LDL: limbs must be in 1..8");
}

}  // namespace

void mp_launch_ldl_dots(unsigned char* A, long lda, int off, int size, int N, unsigned char* W, unsigned char* dinv,
                        const unsigned char* reg, uint32_t* status, cudaStream_t st) {
  check_limbs(N);
  if (size <= 0) return;
  if (size > kMpRecBase) throw std::invalid_argument("MPFR LDL: leaf above the recursion base");
  mpd::by_limbs(N, [&](auto n) {
    constexpr size_t esz = 8 * n() + 8;
    const size_t rows = kLeafRows<n()> ? (size + kLeafCtas - 1) / kLeafCtas * size * esz : 0;
    if (rows)  // per device
      check(cudaFuncSetAttribute(k_mp_ldl_dots<n()>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rows),
            "LDL leaf smem attribute");
    ++g_launches, k_mp_ldl_dots<n()><<<kLeafCtas, kLeafThreads<n()>, rows, st>>>(A, lda, off, size, W, dinv, reg,
                                                                                status);
  });
  check(cudaGetLastError(), "k_mp_ldl_dots");
}

// The stacked operands of the block product sum (rns_blas.rs:2656-2923 gemm_blocks_upper): block
// b's w_b x q_b factor y_b (column-major) fills rows [r0_b, r0_b + w_b) of the W x m matrices Y
// and Z at its global columns cols, Y = y_b and Z = d_b[r] * y_b (each product rounded once); every
// other entry is zero.  One thread per stacked entry (W x m): the block of a row by binary search
// over the row offsets, the column by a search of the block's sorted column list.
template <int N>
__global__ void k_mp_stack_blocks(int nb, const long* __restrict__ r0, const long* __restrict__ yoff,
                                  const long* __restrict__ coff, const int* __restrict__ qn,
                                  const unsigned char* __restrict__ y, const unsigned char* __restrict__ d,
                                  const unsigned long long* __restrict__ cols, long W, int m,
                                  unsigned char* __restrict__ Z, unsigned char* __restrict__ Y,
                                  uint32_t* __restrict__ status) {
  const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= W * m) return;
  const long row = e % W;
  const int col = (int)(e / W);
  constexpr size_t esz = 8 * (size_t)N + 8;
  int lo = 0, hi = nb - 1;  // last block with r0 <= row
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (r0[mid] <= row) lo = mid; else hi = mid - 1;
  }
  const int b = lo;
  const long r = row - r0[b], w = r0[b + 1] - r0[b];
  const unsigned long long* cb = cols + coff[b];
  int a = 0, z = qn[b] - 1, c = -1;
  while (a <= z) {
    const int mid = (a + z) / 2;
    if (cb[mid] == (unsigned long long)col) { c = mid; break; }
    if (cb[mid] < (unsigned long long)col) a = mid + 1; else z = mid - 1;
  }
  Val<N> vy = mpd::zero_val<N>(), vz = vy;
  if (c >= 0) {
    vy = mpd::load<N>(y + (size_t)(yoff[b] + r + (long)c * w) * esz);
    vz = mpd::mul<N>(mpd::load<N>(d + (size_t)(r0[b] + r) * esz), vy);
  }
  mpd::store<N>(Y + (size_t)e * esz, vy, status);
  mpd::store<N>(Z + (size_t)e * esz, vz, status);
}

void mp_launch_potrf(unsigned char* A, long lda, int n, bool lower, int N, int* info, uint32_t* status,
                     cudaStream_t st) {
  check_limbs(N);
  if (n <= 0) return;
  mpd::by_limbs(N, [&](auto l) {
    ++g_launches, k_mp_potrf<l()><<<1, kPotrfThreads, 0, st>>>(A, lower ? 1 : lda, lower ? lda : 1, n, info, status);
  });
  check(cudaGetLastError(), "k_mp_potrf");
}

void mp_launch_solve_lt(const unsigned char* L, long ldl, int k, unsigned char* B, long ldb, int m, int N,
                        uint32_t* status, cudaStream_t st) {
  check_limbs(N);
  if (m <= 0 || k <= 0) return;
  if (k > kMpRecBase) throw std::invalid_argument("MPFR LDL: triangular solve above the recursion base");
  mpd::by_limbs(N, [&](auto n) {
    ++g_launches, k_mp_solve_lt<n()><<<(m + kSolveRows - 1) / kSolveRows, 32 * kSolveRows, 0, st>>>(L, ldl, k, B, ldb,
                                                                                                    m, status);
  });
  check(cudaGetLastError(), "k_mp_solve_lt");
}

void mp_launch_sub_block(unsigned char* B, long ldb, const unsigned char* P, long ldp, int m, int n, int N,
                         uint32_t* status, cudaStream_t st) {
  if (m <= 0 || n <= 0) return;
  mpd::by_limbs(N, [&](auto l) {
    ++g_launches, k_mp_sub_block<l()><<<(unsigned)(((long)m * n + 127) / 128), 128, 0, st>>>(B, ldb, P, ldp, m, n,
                                                                                            status);
  });
  check(cudaGetLastError(), "k_mp_sub_block");
}

void mp_launch_copy_scale_cols(unsigned char* A, long lda, unsigned char* W, const unsigned char* d, int m, int n,
                               int N, uint32_t* status, cudaStream_t st) {
  if (m <= 0 || n <= 0) return;
  mpd::by_limbs(N, [&](auto l) {
    ++g_launches, k_mp_copy_scale_cols<l()><<<(unsigned)(((long)m * n + 127) / 128), 128, 0, st>>>(A, lda, W, d, m, n,
                                                                                                  status);
  });
  check(cudaGetLastError(), "k_mp_copy_scale_cols");
}

void mp_launch_sub_upper_t(unsigned char* A, long lda, const unsigned char* C, long ldc, int n, int N,
                           uint32_t* status, cudaStream_t st) {
  if (n <= 0) return;
  mpd::by_limbs(N, [&](auto l) {
    ++g_launches, k_mp_sub_upper_t<l()><<<(unsigned)(((long)n * n + 127) / 128), 128, 0, st>>>(A, lda, C, ldc, n,
                                                                                              status);
  });
  check(cudaGetLastError(), "k_mp_sub_upper_t");
}

void mp_launch_stack_blocks(int nb, const long* r0, const long* yoff, const long* coff, const int* qn,
                            const unsigned char* y, const unsigned char* d, const unsigned long long* cols, long W,
                            int m, int N, unsigned char* Z, unsigned char* Y, uint32_t* status, cudaStream_t st) {
  check_limbs(N);
  if (W <= 0 || m <= 0) return;
  mpd::by_limbs(N, [&](auto l) {
    ++g_launches, k_mp_stack_blocks<l()><<<(unsigned)((W * m + 127) / 128), 128, 0, st>>>(nb, r0, yoff, coff, qn, y, d,
                                                                                         cols, W, m, Z, Y, status);
  });
  check(cudaGetLastError(), "k_mp_stack_blocks");
}

}  // namespace sdpxg
