// Step-length bound of a PSD block at MPFR width on the GPU: the reference's
// step_length_psd_component for precisions above 64 bits (crates/solver/src/solver/cones/
// psdtrianglecone.rs:1180-1231, with eigval_min_f64 1233-1285, min_eigenvalue_f64 1287-1390,
// admits 1168-1178, lrscale_symmetric 1391-1406).  Per block, from the exact congruence
// Y = W-congruence of the direction (computed beforehand by the exact RNS congruence):
//   wv = svec(Y); Delta = mat(wv) scaled on both sides by Lambda^-1/2 (each product rounded)
//   n > 3: gamma = lambda_min of Delta's binary64 copy (Householder tridiagonalisation and Sturm
//          bisection, the reference's operation order, every FP64 operation rounded separately:
//          no contraction into FMA), accepted when its a priori bound 2 (n+1)^2 eps |Delta|_F is
//          within 1e-10 of max(|gamma|, 1/alpha_max), else certified by an exact-dot Cholesky of
//          I + alpha_c Delta at alpha_c = (1 - 1e-10) min(-1/gamma, alpha_max)
//   otherwise (n <= 3, a non-finite copy, a failed certificate): lambda_min of Delta in MpFloat
//          arithmetic by cyclic two-sided Jacobi (the reference's MPFR eigensolver,
//          algebra/dense/blas/mpfr_eigen.rs, is replaced by it; it agrees to working precision)
//   alpha = min(-1/gamma, alpha_max) when gamma < 0, else alpha_max.
// path[b]: 0 a priori bound, 1 certified, 2 MpFloat eigensolver, 3 the eigensolver did not converge
// (alpha = 0, the reference's zero step for a failed eigensolve).
#include <cfloat>
#include <stdexcept>

#include "device.cuh"
#include "mp.cuh"
#include "mp_ldl.cuh"

namespace sdpxg {
namespace {

using mpd::Val;

constexpr int kStThreads = 256;
constexpr int kStMax = 64;  // block order

// v rounded to binary64, to nearest with ties to even (values beyond the normal range become
// infinities or are rounded once more by ldexp into the subnormals).
template <int N>
__device__ inline double to_double(const Val<N>& v) {
  if (v.zero) return 0.0;
  const unsigned long long top = ((unsigned long long)v.m[2 * N - 1] << 32) | v.m[2 * N - 2];  // top bit set
  unsigned long long mant = top >> 11;  // 53 bits
  const unsigned long long rest = top & 0x7FFull;
  bool sticky = (rest & 0x3FFull) != 0;
#pragma unroll
  for (int q = 0; q < 2 * N - 2; ++q) sticky = sticky || v.m[q] != 0;
  const bool half = (rest >> 10) & 1ull;
  if (half && (sticky || (mant & 1ull))) ++mant;  // may carry to 2^53: still exact in FP64
  // value = mant 2^(s + 64N - 53) (before the carry, mant < 2^53)
  const long long e = v.s + 64LL * N - 53;
  double r;
  if (e > 1100)
    r = HUGE_VAL;
  else if (e < -1200)
    r = 0.0;
  else
    r = ldexp((double)mant, (int)e);
  return v.neg ? -r : r;
}

// The reference's min_eigenvalue_f64 on a (n x n column-major in shared memory, both triangles;
// overwritten), in its operation order with every operation rounded on its own.  d, e: n-entry
// shared scratch, red one shared double.  Returns false for a non-finite Gershgorin interval.  Every
// thread of the CTA calls it.  Bound by the serial sums that the order fixes: each sum runs on one
// thread, and what the order leaves independent in parallel -- the scaled column, the products
// a v (one thread an entry, its terms in order) and the rank-two update (one thread an entry); the
// bisection evaluates the 31 midpoints of its next five levels at once (each midpoint by the
// reference's formula from its own bracket), so a round takes five of its steps.
__device__ bool min_eigenvalue_f64(double* a, int n, double* d, double* e, double* red, double* out) {
  auto at = [&](int i, int j) -> double& { return a[i + j * n]; };
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int i = tid; i < n; i += nt) d[i] = e[i] = 0.0;
  __syncthreads();
  for (int i = n - 1; i >= 1; --i) {
    const int l = i - 1;
    if (l == 0) {
      if (tid == 0) {
        e[i] = at(i, l);
        d[i] = 0.0;
      }
      __syncthreads();
      continue;
    }
    if (tid == 0) {
      double scale = -0.0;
      for (int k = 0; k <= l; ++k) scale = __dadd_rn(scale, fabs(at(i, k)));
      red[0] = scale;
    }
    __syncthreads();
    const double scale = red[0];
    if (scale == 0.0) {
      if (tid == 0) {
        e[i] = at(i, l);
        d[i] = 0.0;
      }
      __syncthreads();
      continue;
    }
    for (int k = tid; k <= l; k += nt) at(i, k) = __ddiv_rn(at(i, k), scale);
    __syncthreads();
    if (tid == 0) {
      double h = 0.0;
      for (int k = 0; k <= l; ++k) h = __dadd_rn(h, __dmul_rn(at(i, k), at(i, k)));
      const double f = at(i, l);
      const double g = f >= 0.0 ? -__dsqrt_rn(h) : __dsqrt_rn(h);
      e[i] = __dmul_rn(scale, g);
      h = __dsub_rn(h, __dmul_rn(f, g));
      at(i, l) = __dsub_rn(f, g);
      d[i] = h;
    }
    __syncthreads();
    const double h = d[i];
    for (int j = tid; j <= l; j += nt) {
      double gg = 0.0;
      for (int k = 0; k <= j; ++k) gg = __dadd_rn(gg, __dmul_rn(at(j, k), at(i, k)));
      for (int k = j + 1; k <= l; ++k) gg = __dadd_rn(gg, __dmul_rn(at(k, j), at(i, k)));
      e[j] = __ddiv_rn(gg, h);
    }
    __syncthreads();
    if (tid == 0) {
      double f = 0.0;
      for (int j = 0; j <= l; ++j) f = __dadd_rn(f, __dmul_rn(e[j], at(i, j)));
      red[0] = __ddiv_rn(f, __dadd_rn(h, h));
    }
    __syncthreads();
    const double hh = red[0];
    for (int j = tid; j <= l; j += nt) e[j] = __dsub_rn(e[j], __dmul_rn(hh, at(i, j)));
    __syncthreads();
    for (int t = tid; t < (l + 1) * (l + 1); t += nt) {
      const int j = t % (l + 1), k = t / (l + 1);
      if (k <= j) at(j, k) = __dsub_rn(at(j, k), __dadd_rn(__dmul_rn(at(i, j), e[k]), __dmul_rn(e[j], at(i, k))));
    }
    __syncthreads();
  }
  if (tid == 0) e[0] = 0.0;
  for (int i = tid; i < n; i += nt) d[i] = at(i, i);
  __syncthreads();
  const double tiny = __ddiv_rn(DBL_MIN, DBL_EPSILON);
  auto below = [&](double x) {
    int count = 0;
    double q = __dsub_rn(d[0], x);
    for (int i = 0; i < n; ++i) {
      if (i > 0) q = __dsub_rn(__dsub_rn(d[i], x), __ddiv_rn(__dmul_rn(e[i], e[i]), q));
      if (q == 0.0) q = -tiny;
      if (q < 0.0) ++count;
    }
    return count;
  };
  double lo = HUGE_VAL, hi = -HUGE_VAL;
  for (int i = 0; i < n; ++i) {
    const double r = __dadd_rn(fabs(e[i]), i + 1 < n ? fabs(e[i + 1]) : 0.0);
    lo = fmin(lo, __dsub_rn(d[i], r));
    hi = fmax(hi, __dadd_rn(d[i], r));
  }
  if (!isfinite(lo) || !isfinite(hi)) return false;
  const double width = fmax(__dsub_rn(hi, lo), __dmul_rn(fmax(fabs(hi), fabs(lo)), DBL_EPSILON));
  lo = __dsub_rn(lo, __dmul_rn(width, DBL_EPSILON));
  hi = __dadd_rn(hi, __dmul_rn(width, DBL_EPSILON));
  if (tid < 32) {
    const int node = tid + 1;  // node of the tree of the next five midpoints: children 2v, 2v + 1
    bool stop = false;
    for (int it = 0; it < 128 && !stop; it += 5) {
      double nl = lo, nh = hi, mid = __dmul_rn(0.5, __dadd_rn(nl, nh));
      const int depth = 31 - __clz(node);
      for (int b = depth - 1; b >= 0; --b) {  // from the root down: a 1 bit takes the upper half
        if ((node >> b) & 1)
          nl = mid;
        else
          nh = mid;
        mid = __dmul_rn(0.5, __dadd_rn(nl, nh));
      }
      const bool end = mid <= nl || mid >= nh;
      const bool low = !end && node < 32 && below(mid) >= 1;
      const unsigned ends = __ballot_sync(0xffffffffu, end), lows = __ballot_sync(0xffffffffu, low);
      int v = 1;
      for (int step = 0; step < 5 && it + step < 128 && !stop; ++step) {  // walk the five steps
        const double m = __shfl_sync(0xffffffffu, mid, v - 1);
        if ((ends >> (v - 1)) & 1u) {
          stop = true;
        } else if ((lows >> (v - 1)) & 1u) {
          hi = m;
          v = 2 * v;
        } else {
          lo = m;
          v = 2 * v + 1;
        }
      }
    }
    if (tid == 0) red[0] = __dmul_rn(0.5, __dadd_rn(lo, hi));
  }
  __syncthreads();
  *out = red[0];
  return true;
}


// lambda_min of the symmetric n x n A (column-major, full; overwritten) by cyclic two-sided Jacobi
// in MpFloat arithmetic, one warp (lanes over rows and columns).  false when 60 sweeps leave an
// off-diagonal entry above 2^-(64N-8) sqrt|a_pp a_qq|.
template <int N>
__device__ bool jacobi_min_eig(unsigned char* A, int n, Val<N>* out, uint32_t* status) {
  constexpr long esz = 8L * N + 8;
  const int lane = threadIdx.x & 31;
  auto el = [&](int i, int j) { return A + ((long)i + (long)j * n) * esz; };
  const Val<N> one = mpd::one_val<N>();
  auto turn = [&](unsigned char* xp, unsigned char* xq, const Val<N>& c, const Val<N>& sn) {
    const Val<N> p = mpd::load<N>(xp), q = mpd::load<N>(xq);
    mpd::store<N>(xp, mpd::addsub<N>(mpd::mul<N>(c, p), mpd::mul<N>(sn, q), -1), status);
    mpd::store<N>(xq, mpd::addsub<N>(mpd::mul<N>(sn, p), mpd::mul<N>(c, q), 1), status);
  };
  bool converged = n <= 1;
  for (int sweep = 0; sweep < 60 && !converged; ++sweep) {
    int rotations = 0;
    for (int p = 0; p < n; ++p)
      for (int q = p + 1; q < n; ++q) {
        const Val<N> apq = mpd::load<N>(el(p, q));
        if (apq.zero) continue;
        const Val<N> app = mpd::load<N>(el(p, p)), aqq = mpd::load<N>(el(q, q));
        Val<N> pp = mpd::mul<N>(app, aqq);
        pp.neg = false;
        pp.s -= 2LL * (64 * N - 8);
        if (!pp.zero && mpd::cmp<N>(mpd::mul<N>(apq, apq), pp) <= 0) continue;
        ++rotations;
        Val<N> a2 = apq;
        a2.s += 1;
        const Val<N> th = mpd::mul<N>(mpd::addsub<N>(aqq, app, -1), mpd::recip_approx<N>(a2));
        Val<N> t;
        if (th.zero) {
          t = one;
        } else if (th.s + 64LL * N > 32LL * N + 8) {
          Val<N> t2 = th;
          t2.s += 1;
          t = mpd::recip_approx<N>(t2);
        } else {
          Val<N> ath = th;
          ath.neg = false;
          const Val<N> w = mpd::addsub<N>(mpd::mul<N>(th, th), one, 1);
          t = mpd::recip_approx<N>(mpd::addsub<N>(ath, mpd::mul<N>(w, mpd::rsqrt_approx<N>(w)), 1));
          t.neg = th.neg;
        }
        const Val<N> c = mpd::rsqrt_approx<N>(mpd::addsub<N>(one, mpd::mul<N>(t, t), 1));
        const Val<N> sn = mpd::mul<N>(c, t);
        __syncwarp();
        for (int k = lane; k < n; k += 32) turn(el(k, p), el(k, q), c, sn);  // columns p, q
        __syncwarp();
        for (int k = lane; k < n; k += 32) turn(el(p, k), el(q, k), c, sn);  // rows p, q
        __syncwarp();
      }
    converged = rotations == 0;
  }
  Val<N> mn = mpd::load<N>(el(0, 0));
  for (int i = 1; i < n; ++i) {
    const Val<N> v = mpd::load<N>(el(i, i));
    if (mpd::cmp<N>(v, mn) < 0) mn = v;
  }
  *out = mn;
  return converged;
}

// One CTA per block: Delta from the congruence Y (n x n at element `mat`), then the bound.
// consts: the working-precision 1/sqrt 2 and alpha_max.
// work: 2 n^2 elements per block at 2 * mat (Delta, then I + alpha_c Delta or the Jacobi copy).
template <int N>
__global__ void __launch_bounds__(kStThreads) k_mp_step_bound(const MpStepBlock* __restrict__ blocks,
                                                              const unsigned char* __restrict__ Y,
                                                              const unsigned char* __restrict__ lisqrt,
                                                              const unsigned char* __restrict__ consts,
                                                              unsigned char* __restrict__ work,
                                                              unsigned char* __restrict__ alpha, int* __restrict__ path,
                                                              uint32_t* __restrict__ status) {
  constexpr int esz = 8 * N + 8, G = 8;
  __shared__ __align__(8) unsigned char s_alc[esz], s_piv[esz];
  __shared__ int s_mode, s_fail, s_bad;  // mode: 0 accepted, 1 to certify, 2 eigensolver, 4 certified
  __shared__ double s_gamma, s_sum, s_red;
  __shared__ double a[kStMax * kStMax], s_d[kStMax], s_e[kStMax];
  const MpStepBlock B = blocks[blockIdx.x];
  const int n = B.n, nn = n * n, tid = threadIdx.x;
  auto el = [&](unsigned char* base, long e) { return base + e * esz; };
  auto cel = [&](const unsigned char* base, long e) { return base + e * esz; };
  unsigned char* D = work + 2 * B.mat * esz;
  unsigned char* C = D + (long)nn * esz;
  const Val<N> frac = mpd::load<N>(cel(consts, 0)), amax = mpd::load<N>(cel(consts, 1));
  if (tid == 0) {
    s_mode = 2;
    s_fail = s_bad = 0;
  }
  // Delta(r, c) = mat(svec(Y))(r, c) * (d_r d_c), the upper entry (r <= c) mirrored: svec's
  // off-diagonal is (Y_rc + Y_cr) / sqrt 2 (Y exactly symmetric: 2 Y_rc exactly), mat's is that
  // times 1/sqrt 2, each product rounded once (matrix_math.rs:156-180, 231-260); a is its
  // binary64 copy
  for (int e = tid; e < nn; e += kStThreads) {
    const int r = e % n, c = e / n;
    if (r > c) continue;
    Val<N> v = mpd::load<N>(cel(Y, B.mat + r + (long)c * n));
    if (r != c) {
      if (!v.zero) v.s += 1;
      v = mpd::mul<N>(mpd::mul<N>(v, frac), frac);
    }
    const Val<N> dd = mpd::mul<N>(mpd::load<N>(cel(lisqrt, B.vec + r)), mpd::load<N>(cel(lisqrt, B.vec + c)));
    v = mpd::mul<N>(v, dd);
    mpd::store<N>(el(D, e), v, status);
    if (r != c) mpd::store<N>(el(D, c + (long)r * n), v, status);
    a[e] = a[c + r * n] = to_double<N>(v);
  }
  __syncthreads();
  if (n > 3) {
    const double amx = to_double<N>(amax);
    for (int e = tid; e < nn; e += kStThreads)
      if (!isfinite(a[e]) || fabs(a[e]) > 1e150) s_bad = 1;
    if (tid == 0) {  // the sum in the reference's order
      double sumsq = 0.0;
      for (int e = 0; e < nn; ++e) sumsq = __dadd_rn(sumsq, __dmul_rn(a[e], a[e]));
      s_sum = sumsq;
    }
    __syncthreads();
    double gamma = 0.0;
    const bool ok = isfinite(amx) && !s_bad && min_eigenvalue_f64(a, n, s_d, s_e, &s_red, &gamma);
    if (ok && tid == 0) {
      const double bound = __dmul_rn(__dmul_rn(__dmul_rn(2.0, (double)(n + 1) * (double)(n + 1)), DBL_EPSILON),
                                     __dsqrt_rn(s_sum));
      const double floor = (amx > 0.0 && isfinite(amx)) ? __ddiv_rn(1.0, amx) : 0.0;
      s_gamma = gamma;
      if (bound <= __dmul_rn(1e-10, fmax(fabs(gamma), floor))) {
        s_mode = 0;
      } else {
        s_mode = 1;
        Val<N> alc = amax;
        if (gamma < 0.0 && __ddiv_rn(-1.0, gamma) < amx)
          alc = mpd::from_double<N>(__ddiv_rn(-__dsub_rn(1.0, 1e-10), gamma), 0);
        mpd::store<N>(s_alc, alc, status);
      }
    }
  }
  __syncthreads();
  if (s_mode == 1) {  // admits: exact-dot Cholesky of alpha_c Delta + I (symmetric: the lower factor)
    const Val<N> alc = mpd::load<N>(s_alc), one = mpd::one_val<N>();
    bool ok = true;
    for (int e = tid; e < nn; e += kStThreads) {
      Val<N> v = mpd::mul<N>(mpd::load<N>(el(D, e)), alc);
      if (e % n == e / n) v = mpd::addsub<N>(v, one, 1);
      mpd::store<N>(el(C, e), v, status);
    }
    __syncthreads();
    for (int j = 0; j < n; ++j) {
      if (tid < 32) {  // warp 0 forms the pivot's dot, its lane 0 the rest
        const Val<N> dot = mpd::dot<N, 32>(nullptr, el(C, j), n, el(C, j), n, j, &ok);
        if (tid == 0) {
          const Val<N> d = mpd::addsub<N>(mpd::load<N>(el(C, j + (long)j * n)), dot, -1);
          if (d.zero || d.neg) {
            s_fail = 1;
          } else {
            const Val<N> r = mpd::root<N>(d);
            mpd::store<N>(el(C, j + (long)j * n), r, status);
            mpd::store<N>(s_piv, r, status);
          }
        }
      }
      __syncthreads();
      if (s_fail) break;
      const Val<N> r = mpd::load<N>(s_piv);
      for (int i = j + 1 + tid / G; i < n; i += kStThreads / G) {  // group-uniform
        const Val<N> dot = mpd::dot<N, G>(nullptr, el(C, i), n, el(C, j), n, j, &ok);
        if ((tid & (G - 1)) == 0) {
          unsigned char* p = el(C, i + (long)j * n);
          mpd::store<N>(p, mpd::divide<N>(mpd::addsub<N>(mpd::load<N>(p), dot, -1), r), status);
        }
      }
      __syncthreads();
    }
    if (!ok) atomicOr(status, SDPXG_ST_EXACT_SPREAD);
    __syncthreads();
    if (tid == 0) s_mode = s_fail ? 2 : 4;
    __syncthreads();
  }
  Val<N> gamma = mpd::zero_val<N>();
  int pth = s_mode == 0 ? 0 : (s_mode == 4 ? 1 : 2);
  bool eig_ok = true;
  if (s_mode == 2) {  // the MpFloat eigensolver on a copy of Delta
    for (int e = tid; e < nn; e += kStThreads) mpd::store<N>(el(C, e), mpd::load<N>(el(D, e)), status);
    __syncthreads();
    if (tid < 32) eig_ok = jacobi_min_eig<N>(C, n, &gamma, status);
  }
  if (tid != 0) return;
  if (s_mode != 2) gamma = mpd::from_double<N>(s_gamma, 0);
  Val<N> al;
  if (!eig_ok) {
    al = mpd::zero_val<N>();
    pth = 3;
  } else if (!gamma.zero && gamma.neg) {
    Val<N> ng = mpd::recip<N>(gamma);
    ng.neg = !ng.neg;
    al = mpd::cmp<N>(ng, amax) < 0 ? ng : amax;
  } else {
    al = amax;
  }
  mpd::store<N>(el(alpha, blockIdx.x), al, status);
  path[blockIdx.x] = pth;
}
// X_b = mat(d_b): full symmetric, off-diagonals times the working-precision 1/sqrt 2 (rounded).
template <int N>
__global__ void k_mp_smat_blocks(const MpStepBlock* __restrict__ blocks, const unsigned char* __restrict__ d,
                                 const unsigned char* __restrict__ consts, unsigned char* __restrict__ X,
                                 uint32_t* __restrict__ status) {
  constexpr int esz = 8 * N + 8;
  const MpStepBlock B = blocks[blockIdx.x];
  const int n = B.n;
  const Val<N> frac = mpd::load<N>(consts);
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int r = e % n, c = e / n, lo = r < c ? r : c, hi = r < c ? c : r;
    Val<N> v = mpd::load<N>(d + (B.svec + (long)hi * (hi + 1) / 2 + lo) * esz);
    if (r != c) v = mpd::mul<N>(v, frac);
    mpd::store<N>(X + (B.mat + e) * esz, v, status);
  }
}

// The working-precision 1/sqrt 2 into consts[0] (sqrt(1/2) rounded once).
template <int N>
__global__ void k_mp_step_consts(unsigned char* consts, uint32_t* status) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  Val<N> h = mpd::one_val<N>();
  h.s -= 1;
  mpd::store<N>(consts, mpd::root<N>(h), status);
}

}  // namespace

void mp_launch_step_smat(const MpStepBlock* blocks, int nblk, int N, const unsigned char* d, unsigned char* consts,
                         unsigned char* X, uint32_t* status, cudaStream_t st) {
  if (N < 1 || N > mpd::kMaxN) throw std::invalid_argument("MPFR step length: limbs must be in 1..8");
  if (nblk <= 0) return;
  mpd::by_limbs(N, [&](auto l) {
    ++g_launches, k_mp_step_consts<l()><<<1, 32, 0, st>>>(consts, status);
    ++g_launches, k_mp_smat_blocks<l()><<<nblk, 256, 0, st>>>(blocks, d, consts, X, status);
  });
  check(cudaGetLastError(), "k_mp_smat_blocks");
}

void mp_launch_step_bound(const MpStepBlock* blocks, int nblk, int N, const unsigned char* Y,
                          const unsigned char* lisqrt, unsigned char* consts, unsigned char* work,
                          unsigned char* alpha, int* path, uint32_t* status, cudaStream_t st) {
  if (N < 1 || N > mpd::kMaxN) throw std::invalid_argument("MPFR step length: limbs must be in 1..8");
  if (nblk <= 0) return;
  mpd::by_limbs(N, [&](auto l) {
    ++g_launches, k_mp_step_bound<l()><<<nblk, kStThreads, 0, st>>>(blocks, Y, lisqrt, consts, work, alpha, path,
                                                                    status);
  });
  check(cudaGetLastError(), "k_mp_step_bound");
}

}  // namespace sdpxg
