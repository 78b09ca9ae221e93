// CTA-level dense eigen / singular-value routines for PSD blocks of order <= SDPXG_NMAX.
//
//  * cta_jacobi_left: one-sided (Hestenes) Jacobi with the parallel odd-even ordering,
//    register-resident.  It orthogonalises the columns of M in place.  Relative accuracy of
//    the small singular values is what the NT scaling
//    needs (the reference takes the SVD of L2'L1 directly instead of an eigensolve of the
//    squared matrix, cones/psdtrianglecone.rs:378-386).
//  * cta_tridiagonalize: Householder reduction of a symmetric matrix to tridiagonal form.
//  * sturm / cta_eig_*: eigenvalues of the tridiagonal by Sturm-sequence multisection
//    (the reference bisects for its binary64 lambda_min bound,
//    cones/psdtrianglecone.rs:1250-1290), every loop bounded.
#pragma once
#include "common.cuh"

#define SDPXG_JACOBI_MAX_SWEEPS 60

namespace jacobi_detail {

// x'y over the R rows a lane holds, in four chains.
template <int R>
__device__ __forceinline__ double dot_rows(const double (&x)[R], const double (&y)[R]) {
  double p[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) p[u] = x[u] * y[u];
#pragma unroll
  for (int k = 4; k < R; ++k) p[k & 3] = fma(x[k], y[k], p[k & 3]);
  return (p[0] + p[1]) + (p[2] + p[3]);
}

// Sum of the four warps' partials b[0], b[32], b[64], b[96] (the same bits in every warp).
__device__ __forceinline__ double sum4(const double* b) { return (b[0] + b[32]) + (b[64] + b[96]); }

// Rotation x' = c x - s y, y' = s x + c y with x'y' = 0 for a pair with ||x||^2 = a, ||y||^2 = b,
// x'y = g, by the half-angle formulas (|theta| <= pi/4):
//   cos 2t = |h| / r, sin 2t = sign(h) 2g / r, r = sqrt(h^2 + 4g^2), h = b - a,
//   c = sqrt((1 + cos 2t) / 2), s = sin 2t / (2c);
// c >= 1/sqrt 2, so nothing cancels, and c^2 + s^2 = 1 to rounding.  tg = (s / c) g, with which
// ||x'||^2 = a - tg and ||y'||^2 = b + tg.  No branch (an in-order warp pays for each): a pair that
// is not `on`, or whose r^2 < 2^-1000 (next to columns of norm 2^200), gets the identity and false.
__device__ __forceinline__ bool rotation(double a, double b, double g, bool on, double& c, double& s, double& tg) {
  const double h = b - a, g2 = g + g, r2 = fma(g2, g2, h * h);
  const bool rot = on && mid_range(r2);
  const double ir = rsqrt_mid(r2), cc = fma(0.5 * fabs(h), ir, 0.5), ic = rsqrt_mid(cc);
  const double t = (h < 0.0 ? -g : g) * ir * ic;
  c = rot ? cc * ic : 1.0;
  s = rot ? t : 0.0;
  tg = rot ? t * ic * g : 0.0;
  return rot;
}

// R rows per warp (n <= 4 R).
template <int R>
__device__ __forceinline__ int sweep_columns(double* M, int n, double* part) {
  constexpr double kTol2 = 1e-30, kBig2 = 1e-20;
  constexpr unsigned kFull = 0xffffffffu;
  const int warp = threadIdx.x >> 5, j = threadIdx.x & 31;
  const int N = n + (n & 1), H = N / 2;
  int iA = j < H ? 2 * j : -1, iB = j < H ? 2 * j + 1 : -1;
  double A[R], B[R], nA = 0.0, nB = 0.0, mx = 0.0;
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int row = 4 * k + warp;
    A[k] = (row < n && iA >= 0 && iA < n) ? SM(M, row, iA) : 0.0;
    B[k] = (row < n && iB >= 0 && iB < n) ? SM(M, row, iB) : 0.0;
    mx = fmax(mx, fmax(fabs(A[k]), fabs(B[k])));
  }
  // largest entry to 2^199 .. 2^200 by a power of two: the room that the norms' squares have
  mx = warp_max(mx);
  if (j == 0) part[warp] = mx;
  asm volatile("bar.sync 1, 128;" ::: "memory");
  mx = fmax(fmax(part[0], part[1]), fmax(part[2], part[3]));
  int ex = 0;
  if (mx > 0.0 && isfinite(mx)) ex = max(-800, min(1000, ilogb(mx) - 199));
  const double down = ldexp(1.0, -ex), up = ldexp(1.0, ex);
#pragma unroll
  for (int k = 0; k < R; ++k) {
    A[k] *= down;
    B[k] *= down;
  }
  int sweeps = (n < 2) ? 0 : -1;
  int phase = 1;  // part[0..3] may still be read
  for (int sweep = 0; n >= 2 && sweep < SDPXG_JACOBI_MAX_SWEEPS; ++sweep) {
    bool rotated = false, big = false;
    for (int r = 0; r < N; r += 2) {
      {  // pairs (2j, 2j+1): both columns in this lane
        double* buf = part + phase * 384;
        phase ^= 1;
        buf[warp * 32 + j] = dot_rows<R>(A, B);
        if (r == 0) {
          buf[128 + warp * 32 + j] = dot_rows<R>(A, A);
          buf[256 + warp * 32 + j] = dot_rows<R>(B, B);
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (r == 0) {
          nA = sum4(buf + 128 + j);
          nB = sum4(buf + 256 + j);
        }
        const double a = nA, b = nB, ab = a * b, g = sum4(buf + j), gg = g * g;
        double c, s, tg;
        rotated |= rotation(a, b, g, j < H && gg > kTol2 * ab, c, s, tg);
        big |= j < H && gg > kBig2 * ab;
#pragma unroll
        for (int k = 0; k < R; ++k) {  // rotate and trade places: A <- y', B <- x'
          const double x = A[k], y = B[k];
          A[k] = fma(s, x, c * y);
          B[k] = fma(c, x, -s * y);
        }
        nA = b + tg;
        nB = a - tg;
        const int t = iA;
        iA = iB;
        iB = t;
      }
      {  // pairs (2j+1, 2j+2): this lane's B and lane j+1's A
        double An[R], Bp[R];
#pragma unroll
        for (int k = 0; k < R; ++k) An[k] = __shfl_down_sync(kFull, A[k], 1);
        const double nAn = __shfl_down_sync(kFull, nA, 1);
        double* buf = part + phase * 384;
        phase ^= 1;
        buf[warp * 32 + j] = dot_rows<R>(B, An);
        asm volatile("bar.sync 1, 128;" ::: "memory");
        const double* bj = buf + j;
        const double q0 = bj[0], q1 = bj[32], q2 = bj[64], q3 = bj[96];
#pragma unroll
        for (int k = 0; k < R; ++k) Bp[k] = __shfl_up_sync(kFull, B[k], 1);
        const int iAn = __shfl_down_sync(kFull, iA, 1), iBp = __shfl_up_sync(kFull, iB, 1);
        const bool exists = j + 1 < H;  // pair (2j+1, 2j+2)
        const double a = nB, b = nAn, ab = a * b, g = (q0 + q1) + (q2 + q3), gg = g * g;
        double c, s, tg;
        rotated |= rotation(a, b, g, exists && gg > kTol2 * ab, c, s, tg);
        big |= exists && gg > kBig2 * ab;
        const double nAl = __shfl_up_sync(kFull, a - tg, 1);
        double cl = __shfl_up_sync(kFull, c, 1), sl = __shfl_up_sync(kFull, s, 1);
        const bool recv = j >= 1 && j < H;  // lane j's A is the right column of pair j-1
        c = exists ? c : 0.0;               // no pair: B stays
        s = exists ? s : 1.0;
        cl = recv ? cl : 0.0;
        sl = recv ? sl : -1.0;
#pragma unroll
        for (int k = 0; k < R; ++k) {
          B[k] = fma(s, B[k], c * An[k]);     // y' of pair j
          A[k] = fma(cl, Bp[k], -sl * A[k]);  // x' of pair j-1
        }
        nB = exists ? b + tg : nB;
        iB = exists ? iAn : iB;
        nA = recv ? nAl : nA;
        iA = recv ? iBp : iA;
      }
    }
    if (!__any_sync(kFull, rotated) || !__any_sync(kFull, big)) {
      sweeps = sweep + 1;
      break;
    }
  }
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int row = 4 * k + warp;
    if (row < n && j < H) {
      if (iA < n) SM(M, row, iA) = A[k] * up;
      if (iB < n) SM(M, row, iB) = B[k] * up;
    }
  }
  return sweeps;
}

}  // namespace jacobi_detail

// One-sided (Hestenes) Jacobi on the columns of M (n x n, n <= 64, column-major shared memory
// with leading dimension SDPXG_LD): on return M holds M V = U diag(sigma), columns in their
// original order; V itself is not formed.  Returns the number of sweeps, or -1 when the sweep
// bound was hit.  Every thread of the CTA calls it (blockDim.x >= 128).
//
// The matrix stays in registers for the whole iteration.  Warps 0..3 take part: warp w holds
// the rows 4k + w, lane j the columns at positions 2j (A) and 2j+1 (B) of a line of
// N = n rounded up to even positions (an odd n gets a zero column that never rotates).  The
// pairs follow the odd-even ordering of Luk and Park: rounds alternate between the pairs
// (2j, 2j+1), which a lane holds itself, and (2j+1, 2j+2), whose second column comes from lane
// j+1 by a warp shuffle; after every rotation the two columns trade places, so in N rounds
// every pair meets once (the moves are those of odd-even transposition sort on a reversed
// line).  Only the across-lane rounds move data (two shuffles per row, one of them under the
// exchange of the partials), and the lane that computes a pair's rotation hands (c, s) to its right
// neighbour.  A pair's inner product is the sum of the four warps' row partials, taken in a fixed tree
// order, so every warp holds the same bits and takes the same decisions without a broadcast; one named
// barrier per round (the partials are double-buffered in `part`, 768 doubles of shared memory).
// Squared column norms are summed exactly at the start of every sweep and carried through its rotations
// (a - tg, b + tg).  A pair rotates while |x'y| > 1e-15 sqrt(||x||^2 ||y||^2); the sweeps stop
// after one without a rotation, or after one in which every cosine was below 1e-10 (the
// rotations of that sweep leave cosines of order 1e-20: one-sided Jacobi converges
// quadratically).
// One warp per SM quarter, not two: a round is bound by its chain (inner product, exchange, two roots,
// rotation), every warp repeats the scalars, and half the warps read half the partials: 1110 cycles a
// pair of rounds at n = 64 against 1600.  Of these the rotations' chains take 360, the FP64 pipe's
// issue of inner products and rotations 400, the shuffles 140.
__device__ inline int cta_jacobi_left(double* M, int n, double* part, int* out) {
  if (threadIdx.x < 128) {
    const int sweeps = n <= 16 ? jacobi_detail::sweep_columns<4>(M, n, part)
                     : n <= 32 ? jacobi_detail::sweep_columns<8>(M, n, part)
                               : jacobi_detail::sweep_columns<16>(M, n, part);
    if (threadIdx.x == 0) *out = sweeps;
  }
  __syncthreads();
  const int res = *out;
  __syncthreads();
  return res;
}

namespace tridiag_detail {

// Shared memory of cta_tridiagonalize (SDPXG_TRIDIAG_WORK doubles): the step's column x and the next
// one, x in column order per warp, the warps' partials of A x, and per warp p in its column order.
constexpr int kX = 0, kY = 64, kXp = 128, kPart = 208, kPw = 464, kRow = 20;
static_assert(kPw + 4 * kRow == SDPXG_TRIDIAG_WORK, "layout");

// Position k of the padded matrix is at hand: warp k & 3 publishes its first column as x (rows above
// k + 1 zero, and d[k]), the warp of column k + 1 that one as y.
template <bool LOW>
__device__ __forceinline__ void publish(int k, int off, double unscale, const double (&a0)[16],
                                        const double (&a1)[16], double* d, double* ws) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, t = k >> 2;
  if (w == (k & 3)) {
    const double x0 = (LOW && lane > k) ? a0[0] : 0.0, x1 = lane + 32 > k ? a1[0] : 0.0;
    ws[kX + lane] = x0;
    ws[kX + lane + 32] = x1;
    double* xp = ws + kXp + (lane & 3) * kRow;  // the columns that are gone leave zeros at the end
    xp[((lane >> 2) - t) & 15] = x0;
    xp[((lane >> 2) + 8 - t) & 15] = x1;
    if (lane == (k & 31)) d[k - off] = ((LOW && k < 32) ? a0[0] : a1[0]) * unscale;
  }
  const int j = (k & 3) == 3;  // column k + 1 is its warp's first or, of warp 0, the second
  if (w == ((k + 1) & 3)) {
    if (LOW) ws[kY + lane] = j ? a0[1] : a0[0];
    ws[kY + lane + 32] = j ? a1[1] : a1[0];
  }
}

// Steps k0 .. k1-1 (positions of the padded matrix) with NJ columns alive per warp; LOW: rows 0 .. 31 too.
template <int NJ, bool LOW>
__device__ __forceinline__ void steps(int k0, int k1, int off, double unscale, double (&a0)[16], double (&a1)[16],
                                      double* d, double* e, double* ws) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int k = k0; k < k1; ++k) {
    asm volatile("bar.sync 1, 128;" ::: "memory");
    const double x0 = LOW ? ws[kX + lane] : 0.0, x1 = ws[kX + lane + 32], xk = ws[kX + k + 1];
    const double y0 = LOW ? ws[kY + lane] : 0.0, y1 = ws[kY + lane + 32];
    double vc[NJ];
#pragma unroll
    for (int j = 0; j < NJ; j += 2) {
      const double2 t = *reinterpret_cast<const double2*>(ws + kXp + w * kRow + j);
      vc[j] = t.x;
      vc[j + 1] = t.y;
    }
    const double nrm2 = warp_sum(LOW ? fma(x0, x0, x1 * x1) : x1 * x1);
    double p0 = 0.0, p1 = 0.0, s0 = 0.0, s1 = 0.0;  // A x: this warp's columns
#pragma unroll
    for (int j = 0; j < NJ; j += 2) {
      if (LOW) p0 = fma(a0[j], vc[j], p0);
      p1 = fma(a1[j], vc[j], p1);
      if (LOW) s0 = fma(a0[j + 1], vc[j + 1], s0);
      s1 = fma(a1[j + 1], vc[j + 1], s1);
    }
    if (LOW) ws[kPart + 64 * w + lane] = p0 + s0;
    ws[kPart + 64 * w + lane + 32] = p1 + s1;
    const bool live = __double2hiint(nrm2) >= 0x01700000;  // 2^-1000 or more
    const double rs = live ? rsqrt_mid(nrm2) : 0.0;
    const double alpha = -copysign(nrm2 * rs, xk), u = xk - alpha;
    const double c = recip_mid(fma(fabs(xk), rs, 1.0));  // 2 / |v rs|^2, in [1/2, 1]
    const double up = live ? fma(xk, rs, copysign(1.0, xk)) : 0.0;
    const double v0 = lane == k + 1 ? up : x0 * rs, v1 = lane + 32 == k + 1 ? up : x1 * rs;
    if (threadIdx.x == 0) e[k - off] = live ? alpha * unscale : 0.0;
    vc[0] = w == (k & 3) + 1 ? u : vc[0];  // column k + 1
    vc[1] = w + 3 == (k & 3) ? u : vc[1];
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (LOW) {
      const double* b = ws + kPart + lane;
      p0 = fma(-alpha, y0, (b[0] + b[64]) + (b[128] + b[192]));
    }
    {
      const double* b = ws + kPart + lane + 32;
      p1 = fma(-alpha, y1, (b[0] + b[64]) + (b[128] + b[192]));
    }
    {
      const int j = (lane >> 2) - (k >> 2);
      if ((lane & 3) == w) {
        if (LOW) ws[kPw + w * kRow + (j & 15)] = j >= 0 ? p0 : 0.0;
        ws[kPw + w * kRow + ((j + 8) & 15)] = j + 8 >= 0 ? p1 : 0.0;
      }
    }
    __syncwarp();
    p0 *= rs;
    p1 *= rs;
    const double S = warp_sum(LOW ? fma(v0, p0, v1 * p1) : v1 * p1);
    const double cr = c * rs, f0 = -cr * v0, f1 = -cr * v1;
#pragma unroll
    for (int j = 0; j < NJ; j += 2) {
      const double2 t = *reinterpret_cast<const double2*>(ws + kPw + w * kRow + j);
      if (LOW) {
        a0[j] = fma(f0, t.x, a0[j]);
        a0[j + 1] = fma(f0, t.y, a0[j + 1]);
      }
      a1[j] = fma(f1, t.x, a1[j]);
      a1[j + 1] = fma(f1, t.y, a1[j + 1]);
    }
    const double cs = c * S, g0 = cr * fma(cs, v0, -p0), g1 = cr * fma(cs, v1, -p1);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      if (LOW) a0[j] = fma(g0, vc[j], a0[j]);
      a1[j] = fma(g1, vc[j], a1[j]);
    }
    if ((k & 3) == 3) {  // the warps' first columns are done with
#pragma unroll
      for (int j = 0; j + 1 < NJ; ++j) {
        if (LOW) a0[j] = a0[j + 1];
        a1[j] = a1[j + 1];
      }
      if (LOW) a0[NJ - 1] = 0.0;
      a1[NJ - 1] = 0.0;
    }
    publish<LOW>(k + 1, off, unscale, a0, a1, d, ws);
  }
}

}  // namespace tridiag_detail

// Householder tridiagonalisation of the symmetric A (n <= 64, shared memory).  d[0..n), e[0..n-1).
// `ws` is SDPXG_TRIDIAG_WORK doubles of shared memory, 16-byte aligned.  Every thread of the CTA calls
// it (blockDim.x >= 128); warps 0..3 take part.
// The matrix stays in registers, as the last n rows and columns of a 64 x 64 one (so that every order
// ends with the same short steps): warp w holds the columns 4j + w, its first register the first column
// that is still alive, lane l the rows l and l + 32.  Step k reflects column k below the diagonal, x =
// A[k+1:, k], by v = x - alpha e1, alpha = -sign(x_1) |x|; with r = 1/|x|, c = 1/(1 + |x_1| r) and p = A v
// = A x - alpha A e1:
//   A <- A - c (vr) (pr)' - c (pr) (vr)' + c^2 ((vr)'(pr)) (vr) (vr)'
// (scaled by r so that no product leaves the range that |x|^2 allows).  A x needs neither |x| nor alpha:
// the warps' partials of it cross shared memory while |x| is summed; the terms with p' are applied while
// (vr)'(pr) is summed.  Rows up to k carry on without being read (they see an orthogonal factor on one
// side); from k = 32 on only the rows 32 .. 63 are kept up.
// Bound by the step's chain -- two barriers, two warp sums (180 cycles each), a root, the published
// column: 1140 cycles a step at n = 64.  One warp for the scalars between four CTA barriers and operands
// in shared memory took 3200; eight warps, each summing all eight partials again, 2290.
__device__ inline void cta_tridiagonalize(const double* A, int n, double* d, double* e, double* ws) {
  using namespace tridiag_detail;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, off = SDPXG_NMAX - n;
  double unscale = 1.0;
  if (w < 4) {
    double a0[16], a1[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int c = 4 * (j + (off >> 2)) + w - off, r = lane - off;
      const bool in = c >= 0 && c < n;
      a0[j] = in && r >= 0 ? SM(A, r, c) : 0.0;
      a1[j] = in && r + 32 >= 0 ? SM(A, r + 32, c) : 0.0;
    }
    // entries below one in magnitude by a power of two: |x|^2 < 2^-1000 is then nothing
    double mx = 0.0;
#pragma unroll
    for (int j = 0; j < 16; ++j) mx = fmax(mx, fmax(fabs(a0[j]), fabs(a1[j])));
    mx = warp_max(mx);
    if (lane == 0) ws[kPart + w] = mx;
    // the steps from row 32 on write half of a warp's row of p and read all of it, gone columns too: those
    // have to be numbers, since a gone column's zero in x does not silence a NaN
    if (lane < kRow) ws[kPw + w * kRow + lane] = 0.0;
    asm volatile("bar.sync 1, 128;" ::: "memory");
    mx = fmax(fmax(ws[kPart], ws[kPart + 1]), fmax(ws[kPart + 2], ws[kPart + 3]));
    int ex = 0;
    if (mx > 0.0 && isfinite(mx)) ex = max(-1000, min(1000, ilogb(mx) + 1));
    const double scale = ldexp(1.0, -ex);
    unscale = ldexp(1.0, ex);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      a0[j] *= scale;
      a1[j] *= scale;
    }
    publish<true>(off, off, unscale, a0, a1, d, ws);
    steps<16, true>(off, 16, off, unscale, a0, a1, d, e, ws);
    steps<12, true>(max(off, 16), 32, off, unscale, a0, a1, d, e, ws);
    steps<8, false>(max(off, 32), 48, off, unscale, a0, a1, d, e, ws);
    steps<4, false>(max(off, 48), SDPXG_NMAX - 2, off, unscale, a0, a1, d, e, ws);
  }
  __syncthreads();
  if (threadIdx.x == 0 && n >= 2) {
    e[n - 2] = ws[kX + SDPXG_NMAX - 1] * unscale;
    d[n - 1] = ws[kY + SDPXG_NMAX - 1] * unscale;
  }
  __syncthreads();
}

// The tridiagonal (d, e) made ready for the Sturm sequences: t[i] = (d_i, e_{i-1}^2) times a power of
// two (its square) that brings the Gershgorin interval to about one, e^2 at least 2^-200 (a perturbation
// of 2^-100 relative to the norm keeps every sequence from stopping at zero; `raised` when there is one),
// padded to a multiple of eight rows with (4, 0), which change no sign.  lo and hi: the interval in the
// scaled units.  `t` is 16-byte aligned shared memory, SDPXG_STURM_WORK doubles.  The same in every thread.
// `finite` is false for a (d, e) with a NaN or an infinity, which minima, maxima and sign tests would pass
// over.
struct SturmRange {
  double lo, hi, scale, unscale;
  bool finite, raised;
};
__device__ inline SturmRange sturm_prepare(const double* d, const double* e, int n, double2* t) {
  const int lane = threadIdx.x & 31;
  double l = 1e300, h = -1e300;
  bool fin = true;
  for (int i = lane; i < n; i += 32) {
    const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < n ? fabs(e[i]) : 0.0);
    fin = fin && isfinite(d[i]) && isfinite(r);
    l = fmin(l, d[i] - r);
    h = fmax(h, d[i] + r);
  }
  l = -warp_max(-l);
  h = warp_max(h);
  const double span = fmax(fabs(l), fabs(h));
  l -= 2.0 * 2.220446049250313e-16 * span;
  h += 2.0 * 2.220446049250313e-16 * span;
  int ex = 0;
  if (span > 0.0 && isfinite(span)) ex = max(-1000, min(1000, ilogb(span) + 1));
  SturmRange r;
  r.scale = ldexp(1.0, -ex);
  r.unscale = ldexp(1.0, ex);
  r.lo = l * r.scale - 0x1p-200;
  r.hi = h * r.scale + 0x1p-200;
  bool small = false;
  for (int i = lane; i + 1 < n; i += 32) small = small || fabs(e[i]) * r.scale < 0x1p-100;
  r.finite = __all_sync(0xffffffffu, fin);
  r.raised = __any_sync(0xffffffffu, small);
  const int np = (n + 7) & ~7;
  for (int i = threadIdx.x; i < np; i += blockDim.x) {
    const double v = (i > 0 && i < n) ? e[i - 1] * r.scale : 0.0;
    t[i] = i < n ? make_double2(d[i] * r.scale, fmax(v * v, 0x1p-200)) : make_double2(4.0, 0.0);
  }
  __syncthreads();
  return r;
}

// An eigenvalue x (scaled units) that the raised e^2 may have moved by more than a rounding: they move it
// by up to 2^-99.  It is found again by quotients, from e^2 as it is, and to kSturmFine.
constexpr double kSturmCoarse = 0x1p-200, kSturmFine = 0x1p-250;  // brackets of an eigenvalue zero end here
__device__ __forceinline__ bool sturm_again(const SturmRange& r, double x) { return r.raised && fabs(x) < 0x1p-46; }

// Eigenvalues of the tridiagonal below x / s by the quotients q_i = d_i - x - e_{i-1}^2 / q_{i-1}, |q_i| at
// least the smallest normal number.
static __device__ __noinline__ int sturm_quotients(const double* d, const double* e, int n, double s, double x) {
  int cnt = 0;
  double q = 1.0;
  for (int i = 0; i < n; ++i) {
    const double v = i > 0 ? e[i - 1] * s : 0.0;
    q = (d[i] * s - x) - v * v / q;
    if (fabs(q) < 0x1p-1022) q = -0x1p-1022;
    cnt += q < 0.0;
  }
  return cnt;
}

// The leading principal minors of T - x for the tridiagonal prepared by sturm_prepare, p_i = (d_i - x)
// p_{i-1} - e_{i-1}^2 p_{i-2}: COUNT ? the number of their sign changes, the eigenvalues below x : the
// sign of any (at least one eigenvalue below x).  Each step perturbs d_i - x and e_{i-1}^2 by a few
// units in the last place, as the quotient form q_i = d_i - x - e_{i-1}^2 / q_{i-1} does, but its chain
// is one multiply-add (8 cycles) instead of a reciprocal (about 110).  Every eighth step rescales the
// pair by a power of two (eight steps change it by at most 2^16 upwards and about 2^-800 downwards).
template <bool COUNT>
__device__ __forceinline__ int sturm(const double2* t, int n, double x) {
  double p0 = 0.0, p1 = 1.0;
  int cnt = 0;
  double2 r[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) r[u] = t[u];
  for (int i = 0; i < n; i += 8) {
    double2 next[8];
    const double2* tn = t + (i + 8 < n ? i + 8 : 0);
#pragma unroll
    for (int u = 0; u < 8; ++u) next[u] = tn[u];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const double p2 = fma(r[u].x - x, p1, -(r[u].y * p0));
      if (COUNT) cnt += (int)((unsigned)(__double2hiint(p2) ^ __double2hiint(p1)) >> 31);
      else cnt |= __double2hiint(p2);
      p0 = p1;
      p1 = p2;
    }
    const int m = max(__double2hiint(p0) & 0x7ff00000, __double2hiint(p1) & 0x7ff00000);
    const double s = __hiloint2double(0x7fe00000 - min(max(m, 0x00100000), 0x7fd00000), 0);
    p0 *= s;
    p1 *= s;
#pragma unroll
    for (int u = 0; u < 8; ++u) r[u] = next[u];
  }
  return COUNT ? cnt : (int)((unsigned)cnt >> 31);
}

// Smallest eigenvalue in scaled units by CTA-wide multisection: each round every thread evaluates one
// Sturm sequence on an even grid over the current bracket and the bracket shrinks to the first grid cell
// holding an eigenvalue.  With 256 threads a round is bound by the sequence's chain and gives 8 bits; with
// 512 it is bound by issue and gives 9.  *ok = false if the round bound is hit.
template <bool QUOTIENTS>
__device__ __forceinline__ double multisect_min(const double* d, const double* e, int n, const double2* t,
                                                const SturmRange& r, int* best, bool* ok) {
  const int T = blockDim.x;
  double lo = r.lo, hi = r.hi;
  for (int round = 0; round < 40; ++round) {
    if (!(hi - lo > 2.0 * 2.220446049250313e-16 * fmax(fabs(lo), fabs(hi)) + (QUOTIENTS ? kSturmFine : kSturmCoarse))) {
      *ok = true;
      return 0.5 * (lo + hi);
    }
    const double step = (hi - lo) / (T + 1);
    if (threadIdx.x == 0) *best = T;
    __syncthreads();
    const double x = lo + step * (threadIdx.x + 1);
    const unsigned bal = __ballot_sync(0xffffffffu, x > lo && x < hi &&
                                       (QUOTIENTS ? sturm_quotients(d, e, n, r.scale, x) : sturm<false>(t, n, x)));
    if (bal && (threadIdx.x & 31) == 0) atomicMin(best, (int)threadIdx.x + __ffs(bal) - 1);
    __syncthreads();
    const int b = *best;
    __syncthreads();
    const double nlo = (b == 0) ? lo : lo + step * b;
    const double nhi = (b == T) ? hi : lo + step * (b + 1);
    lo = nlo;
    hi = nhi;
  }
  *ok = false;
  return 0.5 * (lo + hi);
}
static __device__ __noinline__ double multisect_min_again(const double* d, const double* e, int n, SturmRange r,
                                                          int* best, bool* ok) {
  return multisect_min<true>(d, e, n, nullptr, r, best, ok);
}

// Smallest eigenvalue of the tridiagonal (d, e), resolved relative to itself down to about 2^-200 of the
// norm: at most 26 rounds, and 32 more by quotients.  Uniform result; `best` is one int of shared memory, `t`
// SDPXG_STURM_WORK doubles.  *ok = false if the round bound is hit or (d, e) is not finite.
__device__ inline double cta_eig_min(const double* d, const double* e, int n, double2* t, int* best, bool* ok) {
  if (n == 1) {  // orthant rows come as such blocks, thousands at a time
    *ok = isfinite(d[0]);
    return d[0];
  }
  const SturmRange r = sturm_prepare(d, e, n, t);
  *ok = false;
  if (!r.finite) return 0.0;
  double x = multisect_min<false>(d, e, n, t, r, best, ok);
  if (*ok && sturm_again(r, x)) x = multisect_min_again(d, e, n, r, best, ok);
  return x * r.unscale;
}

// Eigenvalue k in scaled units by the 16 lanes of a group (lane sl, the warp's lanes from `base` on):
// multisection with 15 Sturm counts per round (the bracket shrinks 16-fold per round).
template <bool QUOTIENTS>
__device__ __forceinline__ double multisect_kth(const double* d, const double* e, int n, const double2* t,
                                                const SturmRange& r, int k, bool* ok) {
  constexpr int P = 16;
  const int sl = threadIdx.x % P, base = threadIdx.x & 16;
  const unsigned gmask = 0xFFFFu << base;
  double lo = r.lo, hi = r.hi;
  for (int round = 0; round < 64; ++round) {
    if (!(hi - lo > 2.0 * 2.220446049250313e-16 * fmax(fabs(lo), fabs(hi)) + (QUOTIENTS ? kSturmFine : kSturmCoarse))) {
      *ok = true;
      return 0.5 * (lo + hi);
    }
    const double step = (hi - lo) / P;
    const double x = lo + step * (sl + 1);
    const bool above = (sl < P - 1) && x > lo && x < hi &&
                       (QUOTIENTS ? sturm_quotients(d, e, n, r.scale, x) : sturm<true>(t, n, x)) > k;
    const unsigned bal = (__ballot_sync(gmask, above) >> base) & 0xFFFFu;
    const int c = bal ? __ffs(bal) - 1 : P - 1;  // eigenvalue k lies in cell c
    const double nlo = (c == 0) ? lo : lo + step * c;
    const double nhi = (c == P - 1) ? hi : lo + step * (c + 1);
    lo = nlo;
    hi = nhi;
  }
  *ok = false;
  return 0.5 * (lo + hi);
}
static __device__ __noinline__ double multisect_kth_again(const double* d, const double* e, int n, SturmRange r, int k,
                                                          bool* ok) {
  return multisect_kth<true>(d, e, n, nullptr, r, k, ok);
}

// Every eigenvalue of the tridiagonal (d, e), ascending, into eig[0..n): 16-lane groups, one
// eigenvalue per group, no CTA barrier inside.  `t`: SDPXG_STURM_WORK doubles.
// Sets the status bit SDPXG_ST_EIG_FAIL for an eigenvalue whose round bound was hit and for a (d, e) that
// is not finite.
__device__ inline void cta_eig_all(const double* d, const double* e, int n, double2* t, double* eig,
                                   uint32_t* status) {
  const SturmRange r = sturm_prepare(d, e, n, t);
  if (!r.finite && threadIdx.x == 0) atomicOr(status, SDPXG_ST_EIG_FAIL);
  for (int k = threadIdx.x / 16; k < n; k += blockDim.x / 16) {
    bool ok;
    double x = multisect_kth<false>(d, e, n, t, r, k, &ok);
    if (ok && sturm_again(r, x)) x = multisect_kth_again(d, e, n, r, k, &ok);
    if (threadIdx.x % 16 == 0) {
      eig[k] = x * r.unscale;
      if (!ok) atomicOr(status, SDPXG_ST_EIG_FAIL);
    }
  }
}
