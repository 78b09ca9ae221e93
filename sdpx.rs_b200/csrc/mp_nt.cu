// NT scaling of PSD blocks at MPFR width on the GPU: the reference's
// PSDTriangleCone::update_scaling (crates/solver/src/solver/cones/psdtrianglecone.rs:311-439) for
// MpFloat<N> (N <= 8), one CTA per block of order n <= 64:
//   S = mat(s), Z = mat(z) (off-diagonals times the working-precision 1/sqrt 2, matrix_math.rs:156-180)
//   L1 = chol(S), L2 = chol(Z)         exact-dot left-looking Cholesky (the reference's xpotrf,
//                                      algebra/dense/blas/mpfr.rs:726-789), the two factored
//                                      concurrently by the two halves of the CTA
//   M = L2' L1                          every entry an exact dot rounded once
//   M V = U Sigma                       right singular vectors by one-sided (Hestenes) Jacobi in
//                                      MpFloat arithmetic: the reference's MPFR right SVD
//                                      (mpfr_svd.rs, Golub-Kahan + dqds + inverse iteration) is
//                                      replaced by a method whose rotations of disjoint column
//                                      pairs run in parallel (their column sums exact dots);
//                                      singular values are the final column norms, sorted
//                                      descending
//   lambda = sigma, Lambda^-1/2 = 1 / sqrt(sigma)
//   R = L1 V Lambda^-1/2,  Rinv = Lambda^1/2 (L1^-T V)',  G = R R' (upper)
// V is unique up to the signs of its columns (and rotations within clusters of equal singular
// values); R, Rinv change with it as the reference's do, G, lambda and the congruences they define
// do not.  Per-block status: 0, or SDPXG_ST_CHOL_FAIL (s or z not interior), or
// SDPXG_ST_SVD_UNCONVERGED, and then the block's outputs are zeros; SDPXG_ST_EXACT_SPREAD in the shared status word when an exact dot
// exceeds the accumulator.
#include <stdexcept>

#include "device.cuh"
#include "mp.cuh"
#include "mp_ldl.cuh"

namespace sdpxg {
namespace {

using mpd::Val;

// Up to 4 limbs 16 warps (128 registers a thread hold a dot's accumulator, operands and product);
// above, 8 warps.
template <int N>
constexpr int kNtThreads = N <= 4 ? 512 : 256;
constexpr int kNtMaxSweeps = 80;
constexpr int kNtMax = 64;  // block order
constexpr int kPairs = kNtMax / 2;

__device__ __forceinline__ void named_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// Exact-dot Cholesky (lower, in place, column-major ld n) by a group of `nt` threads that
// synchronise on named barrier `bar`: the group's first warp forms each pivot (its dot split over
// the lanes), then eight lanes take a row's dot and one thread a row its difference and quotient.
template <int N>
__device__ void chol_group(unsigned char* L, int n, int t, int nt, int bar, unsigned char* sd, unsigned char* sdot,
                           volatile int* fail, uint32_t* status) {
  constexpr int esz = 8 * N + 8, G = 8;
  auto at = [&](int i, int k) { return L + ((long)i + (long)k * n) * esz; };
  bool ok = true;
  for (int j = 0; j < n; ++j) {
    if (t < 32) {  // the group's first warp forms the pivot's dot, its lane 0 the rest
      const Val<N> dot = mpd::dot<N, 32>(nullptr, at(j, 0), n, at(j, 0), n, j, &ok);
      if (t == 0) {
        const Val<N> d = mpd::addsub<N>(mpd::load<N>(at(j, j)), dot, -1);
        if (d.zero || d.neg) {
          *fail = 1;
        } else {
          const Val<N> r = mpd::root<N>(d);
          mpd::store<N>(at(j, j), r, status);
          mpd::store<N>(sd, r, status);
        }
      }
    } else {
      for (int i = j + 1 + (t - 32) / G; i < n; i += (nt - 32) / G) {  // group-uniform
        const Val<N> dot = mpd::dot<N, G>(nullptr, at(i, 0), n, at(j, 0), n, j, &ok);
        if ((t & (G - 1)) == 0) mpd::stage<N>(sdot + i * esz, dot);
      }
    }
    named_sync(bar, nt);
    if (*fail) break;
    if (t < n - 1 - j) {
      const int i = j + 1 + t;
      const Val<N> d = mpd::addsub<N>(mpd::load<N>(at(i, j)), mpd::unstage<N>(sdot + i * esz), -1);
      mpd::store<N>(at(i, j), mpd::divide<N>(d, mpd::load<N>(sd)), status);
    }
    named_sync(bar, nt);
  }
  if (!ok) atomicOr(status, SDPXG_ST_EXACT_SPREAD);
}

// The rotation of a pair of columns with x'x = aa, y'y = bb, x'y = gg: false when the pair is
// orthogonal to working accuracy (|gamma| <= 2^-(64N-8) sqrt(ab)), else c and sn:
// zeta = (b - a) / (2 g), t = sign(zeta) / (|zeta| + sqrt(1 + zeta^2)), c = 1/sqrt(1+t^2), sn = c t.
template <int N>
__device__ __noinline__ bool rotation(const Val<N>& aa, const Val<N>& bb, const Val<N>& gg, Val<N>& c, Val<N>& sn) {
  if (gg.zero || aa.zero || bb.zero) return false;
  {
    Val<N> ab = mpd::mul<N>(aa, bb);
    ab.s -= 2LL * (64 * N - 8);
    if (mpd::cmp<N>(mpd::mul<N>(gg, gg), ab) <= 0) return false;
  }
  const Val<N> one = mpd::one_val<N>();
  Val<N> g2 = gg;
  g2.s += 1;
  Val<N> zeta = mpd::mul<N>(mpd::addsub<N>(bb, aa, -1), mpd::recip_approx<N>(g2));
  Val<N> t;
  if (zeta.zero) {
    t = one;
  } else if (zeta.s + 64LL * N > 32LL * N + 8) {  // |zeta| > 2^(32N+8): t = 1 / (2 zeta)
    Val<N> z2 = zeta;
    z2.s += 1;
    t = mpd::recip_approx<N>(z2);
  } else {
    Val<N> az = zeta;
    az.neg = false;
    const Val<N> w = mpd::addsub<N>(one, mpd::mul<N>(zeta, zeta), 1);
    const Val<N> sq = mpd::mul<N>(w, mpd::rsqrt_approx<N>(w));
    t = mpd::recip_approx<N>(mpd::addsub<N>(az, sq, 1));
    t.neg = zeta.neg;
  }
  c = mpd::rsqrt_approx<N>(mpd::addsub<N>(one, mpd::mul<N>(t, t), 1));
  sn = mpd::mul<N>(c, t);
  return true;
}

// Columns of a round-robin round r over mm positions: pair k holds positions k and mm - 1 - k
// (position 0 fixed, the others rotating).  False when the pair holds the padding column.
__device__ __forceinline__ bool round_pair(int k, int r, int mm, int n, int* p, int* q) {
  const int pb = mm - 1 - k;
  *p = k == 0 ? 0 : 1 + (k - 1 + r) % (mm - 1);
  *q = 1 + (pb - 1 + r) % (mm - 1);
  return *p < n && *q < n;
}

// One CTA per block (see the file comment).  Work: five n x n matrices per block at element
// 5 * mat (L1, L2, the Jacobi matrix A, V, X), two n-vectors at element 2 * vec (sigma, sqrt sigma).
// Bound by the chain of the Jacobi rounds.  A round is three phases: the 3 n / 2 column sums (exact
// dots, eight lanes each); the rotations, one lane a pair -- the chain of some fifty MpFloat
// operations runs once for all pairs of the round, on one warp -- while the other warps apply the
// previous round's rotations to V, which no dot reads; and the rotations of A, one thread an entry
// pair.  (With a warp a pair and the whole round on it, every lane repeats that chain, and four
// warps a scheduler repeat it against one another.)
template <int N>
__global__ void __launch_bounds__(kNtThreads<N>) k_mp_nt_scale(const MpNtBlock* __restrict__ blocks,
                                                               const unsigned char* __restrict__ s,
                                                               const unsigned char* __restrict__ z,
                                                               const unsigned char* __restrict__ frac,
                                                               unsigned char* __restrict__ work,
                                                               unsigned char* __restrict__ wvec,
                                                               unsigned char* __restrict__ lam,
                                                               unsigned char* __restrict__ lisqrt,
                                                               unsigned char* __restrict__ R,
                                                               unsigned char* __restrict__ Rinv,
                                                               unsigned char* __restrict__ G, int* __restrict__ bstatus,
                                                               uint32_t* __restrict__ status) {
  constexpr int T = kNtThreads<N>, esz = 8 * N + 8, LG = 8;
  __shared__ __align__(8) unsigned char sd[2][esz];
  __shared__ __align__(8) unsigned char ssum[3 * kPairs * esz];        // column sums (Cholesky: dots of both halves)
  __shared__ __align__(8) unsigned char srot[2][2 * kPairs * esz];     // c and sn of this round and the last
  __shared__ int spair[2][2 * kPairs];                                 // their columns; first -1: not rotated
  __shared__ volatile int fail[2];
  __shared__ int rotated;
  __shared__ int perm[kNtMax];
  static_assert(3 * kPairs >= kNtMax, "Cholesky staging");
  const MpNtBlock B = blocks[blockIdx.x];
  const int n = B.n, nn = n * n, tid = threadIdx.x;
  auto el = [&](unsigned char* base, long e) { return base + e * esz; };
  unsigned char* L1 = work + 5 * B.mat * esz;
  unsigned char* L2 = L1 + (long)nn * esz;
  unsigned char* A = L2 + (long)nn * esz;
  unsigned char* V = A + (long)nn * esz;
  unsigned char* X = V + (long)nn * esz;
  unsigned char* sig = wvec + 2 * B.vec * esz;
  unsigned char* root = sig + n * esz;
  if (tid == 0) {
    fail[0] = fail[1] = 0;
    bstatus[blockIdx.x] = 0;
  }
  // S and Z, lower triangles (svec upper column order: (i, j), j <= i, at i (i + 1) / 2 + j)
  const Val<N> fv = mpd::load<N>(frac);
  for (int e = tid; e < nn; e += T) {
    const int i = e % n, j = e / n;
    Val<N> sv = mpd::zero_val<N>(), zv = sv;
    if (i >= j) {
      const long t = (long)i * (i + 1) / 2 + j;
      sv = mpd::load<N>(s + (B.svec + t) * esz);
      zv = mpd::load<N>(z + (B.svec + t) * esz);
      if (i != j) {
        sv = mpd::mul<N>(sv, fv);
        zv = mpd::mul<N>(zv, fv);
      }
    }
    mpd::store<N>(el(L1, e), sv, status);
    mpd::store<N>(el(L2, e), zv, status);
  }
  __syncthreads();
  if (tid < T / 2)
    chol_group<N>(L1, n, tid, T / 2, 1, sd[0], ssum, &fail[0], status);
  else
    chol_group<N>(L2, n, tid - T / 2, T / 2, 2, sd[1], srot[0], &fail[1], status);
  __syncthreads();
  // a failed block's outputs are zeros
  auto zero_outputs = [&]() {
    const Val<N> zv = mpd::zero_val<N>();
    for (int e = tid; e < nn; e += T) {
      mpd::store<N>(el(R, B.mat + e), zv, status);
      mpd::store<N>(el(Rinv, B.mat + e), zv, status);
      mpd::store<N>(el(G, B.mat + e), zv, status);
    }
    for (int r = tid; r < n; r += T) {
      mpd::store<N>(el(lam, B.vec + r), zv, status);
      mpd::store<N>(el(lisqrt, B.vec + r), zv, status);
    }
  };
  if (fail[0] || fail[1]) {
    if (tid == 0) bstatus[blockIdx.x] = SDPXG_ST_CHOL_FAIL;
    zero_outputs();
    return;
  }
  bool ok = true;
  // A = M = L2' L1 (entry (i, j): rows k >= max(i, j)), V = I
  for (int e = tid; e < nn; e += T) {
    const int i = e % n, j = e / n, k0 = i > j ? i : j;
    const Val<N> m = mpd::dot<N, 1>(nullptr, el(L2, k0 + (long)i * n), 1, el(L1, k0 + (long)j * n), 1, n - k0, &ok);
    mpd::store<N>(el(A, e), m, status);
    mpd::store<N>(el(V, e), i == j ? mpd::one_val<N>() : mpd::zero_val<N>(), status);
  }
  // rotate the rows of M2's columns (p, q) of the pairs stored in buffer `buf`, threads t of nt
  const int mm = n + (n & 1), P = mm / 2;
  auto rotate = [&](unsigned char* M2, int buf, int t, int nt) {
    for (int e = t; e < P * n; e += nt) {
      const int k = e / n, i = e % n, p = spair[buf][2 * k], q = spair[buf][2 * k + 1];
      if (p < 0) continue;
      const Val<N> c = mpd::unstage<N>(srot[buf] + 2 * k * esz), sn = mpd::unstage<N>(srot[buf] + (2 * k + 1) * esz);
      unsigned char* xp = el(M2, i + (long)p * n);
      unsigned char* xq = el(M2, i + (long)q * n);
      const Val<N> vp = mpd::load<N>(xp), vq = mpd::load<N>(xq);
      mpd::store<N>(xp, mpd::addsub<N>(mpd::mul<N>(c, vp), mpd::mul<N>(sn, vq), -1), status);
      mpd::store<N>(xq, mpd::addsub<N>(mpd::mul<N>(sn, vp), mpd::mul<N>(c, vq), 1), status);
    }
  };
  // One-sided Jacobi: sweeps of round-robin rounds until one without a rotation.
  int cur = 0;
  if (tid < 2 * kPairs) spair[0][tid] = spair[1][tid] = -1;
  bool converged = n <= 1;
  for (int sweep = 0; sweep < kNtMaxSweeps && !converged; ++sweep) {
    __syncthreads();
    if (tid == 0) rotated = 0;
    for (int r = 0; r < mm - 1; ++r, cur ^= 1) {
      __syncthreads();  // A is rotated
      for (int d = tid / LG; d < 3 * P; d += T / LG) {  // group-uniform
        int p, q;
        if (!round_pair(d / 3, r, mm, n, &p, &q)) continue;
        const int x = d % 3 == 1 ? q : p, y = d % 3 == 0 ? p : q;  // (p, p), (q, q), (p, q)
        const Val<N> v = mpd::dot<N, LG>(nullptr, el(A, (long)x * n), 1, el(A, (long)y * n), 1, n, &ok);
        if ((tid & (LG - 1)) == 0) mpd::stage<N>(ssum + d * esz, v);
      }
      __syncthreads();
      if (tid < 32) {
        if (tid < P) {
          int p, q;
          Val<N> c, sn;
          bool rot = round_pair(tid, r, mm, n, &p, &q);
          if (rot)
            rot = rotation<N>(mpd::unstage<N>(ssum + 3 * tid * esz), mpd::unstage<N>(ssum + (3 * tid + 1) * esz),
                              mpd::unstage<N>(ssum + (3 * tid + 2) * esz), c, sn);
          spair[cur][2 * tid] = rot ? p : -1;
          spair[cur][2 * tid + 1] = q;
          if (rot) {
            mpd::stage<N>(srot[cur] + 2 * tid * esz, c);
            mpd::stage<N>(srot[cur] + (2 * tid + 1) * esz, sn);
            atomicAdd(&rotated, 1);
          }
        }
      } else {
        rotate(V, cur ^ 1, tid - 32, T - 32);  // the last round's rotations
      }
      __syncthreads();
      rotate(A, cur, tid, T);
    }
    __syncthreads();
    converged = rotated == 0;
  }
  rotate(V, cur ^ 1, tid, T);  // the last round of the last sweep (none rotated once converged)
  if (!ok) atomicOr(status, SDPXG_ST_EXACT_SPREAD);
  if (!converged) {
    if (tid == 0) bstatus[blockIdx.x] = SDPXG_ST_SVD_UNCONVERGED;
    zero_outputs();
    return;
  }
  __syncthreads();
  // singular values: column norms (exact sums of squares, correctly rounded roots), descending
  for (int j = tid / LG; j < n; j += T / LG) {
    const Val<N> ss = mpd::dot<N, LG>(nullptr, el(A, (long)j * n), 1, el(A, (long)j * n), 1, n, &ok);
    if ((tid & (LG - 1)) == 0) mpd::store<N>(el(sig, j), mpd::root<N>(ss), status);
  }
  __syncthreads();
  for (int j = tid; j < n; j += T) {
    const Val<N> sj = mpd::load<N>(el(sig, j));
    int rank = 0;
    for (int k = 0; k < n; ++k) {
      if (k == j) continue;
      const int c = mpd::cmp<N>(mpd::load<N>(el(sig, k)), sj);
      rank += (c > 0 || (c == 0 && k < j)) ? 1 : 0;
    }
    perm[rank] = j;
  }
  __syncthreads();
  for (int r = tid; r < n; r += T) {
    const Val<N> sg = mpd::load<N>(el(sig, perm[r]));
    const Val<N> rt = mpd::root<N>(sg);
    mpd::store<N>(el(lam, B.vec + r), sg, status);
    mpd::store<N>(el(root, r), rt, status);
    mpd::store<N>(el(lisqrt, B.vec + r), mpd::recip<N>(rt), status);
  }
  __syncthreads();
  // R = L1 V Lambda^-1/2 (row i of L1 has entries k <= i); X = L1^-T V (back substitution, eight
  // lanes a column)
  for (int e = tid; e < nn; e += T) {
    const int i = e % n, r = e / n;
    const Val<N> d = mpd::dot<N, 1>(nullptr, el(L1, i), n, el(V, (long)perm[r] * n), 1, i + 1, &ok);
    mpd::store<N>(el(R, B.mat + e), mpd::mul<N>(d, mpd::load<N>(el(lisqrt, B.vec + r))), status);
  }
  {
    const unsigned gmask = 0xffu << (tid & 24);
    for (int r = tid / LG; r < n; r += T / LG) {
      for (int i = n - 1; i >= 0; --i) {
        const Val<N> b = mpd::load<N>(el(V, i + (long)perm[r] * n));
        const Val<N> d = mpd::dot<N, LG>(&b, el(L1, i + 1 + (long)i * n), 1, el(X, i + 1 + (long)r * n), 1, n - 1 - i,
                                         &ok);
        if ((tid & (LG - 1)) == 0)
          mpd::store<N>(el(X, i + (long)r * n), mpd::divide<N>(d, mpd::load<N>(el(L1, i + (long)i * n))), status);
        __syncwarp(gmask);  // x_i visible to the group's next dot
      }
    }
  }
  __syncthreads();
  // Rinv(r, j) = sqrt(sigma_r) X(j, r); G = R R' (upper: exact dots of rows of R)
  for (int e = tid; e < nn; e += T) {
    const int r = e % n, j = e / n;
    mpd::store<N>(el(Rinv, B.mat + e),
                  mpd::mul<N>(mpd::load<N>(el(X, j + (long)r * n)), mpd::load<N>(el(root, r))), status);
    Val<N> g = mpd::zero_val<N>();
    if (r <= j) g = mpd::dot<N, 1>(nullptr, el(R, B.mat + r), n, el(R, B.mat + j), n, n, &ok);
    mpd::store<N>(el(G, B.mat + e), g, status);
  }
  if (!ok) atomicOr(status, SDPXG_ST_EXACT_SPREAD);
}

// The working-precision 1/sqrt 2 (FloatConst::FRAC_1_SQRT_2): sqrt(1/2) rounded once.
template <int N>
__global__ void k_mp_frac_sqrt2(unsigned char* out, uint32_t* status) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  Val<N> h = mpd::one_val<N>();
  h.s -= 1;  // 1/2
  mpd::store<N>(out, mpd::root<N>(h), status);
}

}  // namespace

void mp_launch_nt_scale(const MpNtBlock* blocks, int nblk, int N, const unsigned char* s, const unsigned char* z,
                        unsigned char* frac, unsigned char* work, unsigned char* wvec, unsigned char* lam,
                        unsigned char* lisqrt, unsigned char* R, unsigned char* Rinv, unsigned char* G, int* bstatus,
                        uint32_t* status, cudaStream_t st) {
  if (N < 1 || N > mpd::kMaxN) throw std::invalid_argument("MPFR NT scaling: limbs must be in 1..8");
  if (nblk <= 0) return;
  mpd::by_limbs(N, [&](auto l) {
    constexpr int L = l();
    ++g_launches, k_mp_frac_sqrt2<L><<<1, 32, 0, st>>>(frac, status);
    ++g_launches, k_mp_nt_scale<L><<<nblk, kNtThreads<L>, 0, st>>>(blocks, s, z, frac, work, wvec, lam, lisqrt, R,
                                                                   Rinv, G, bstatus, status);
  });
  check(cudaGetLastError(), "k_mp_nt_scale");
}

}  // namespace sdpxg
