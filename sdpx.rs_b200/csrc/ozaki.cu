// Split-precision FP64 products (Ozaki scheme II) on the INT8 tensor cores; see ozaki.cuh.
#include <cmath>
#include <mutex>
#include <stdexcept>

#include "i8_gemm.cuh"
#include "ozaki.cuh"

namespace sdpxg {
namespace {

// Sixteen pairwise coprime moduli <= 256 (256 = 2^8, 255 = 3*5*17, 253 = 11*23, 247 = 13*19,
// 217 = 7*31, the rest prime): their product P is about 2^126.4.  A constant function of the
// index, so that in the kernels' unrolled loops every reduction is by a literal modulus.
__host__ __device__ constexpr int oz_mod(int t) {
  return t == 0 ? 256 : t == 1 ? 255 : t == 2 ? 253 : t == 3 ? 251 : t == 4 ? 247 : t == 5 ? 241 : t == 6 ? 239
       : t == 7 ? 233 : t == 8 ? 229 : t == 9 ? 227 : t == 10 ? 223 : t == 11 ? 217 : t == 12 ? 211
       : t == 13 ? 199 : t == 14 ? 197 : 193;
}
constexpr int kModuli[kOzMod] = {oz_mod(0),  oz_mod(1),  oz_mod(2),  oz_mod(3),  oz_mod(4),  oz_mod(5),
                                 oz_mod(6),  oz_mod(7),  oz_mod(8),  oz_mod(9),  oz_mod(10), oz_mod(11),
                                 oz_mod(12), oz_mod(13), oz_mod(14), oz_mod(15)};

constexpr int kOzTriples = (kOzMod + 2) / 3;  // moduli 3g, 3g + 1, 3g + 2
// Tables of the residue and reconstruction kernels, in constant memory (every index is a literal after
// unrolling).  With P the product of the moduli and W_t = P / p_t:
struct OzTables {
  uint32_t wlo[kOzMod], whi[kOzMod];  // 256^k mod p for the bytes k of a 64-bit integer
  uint32_t init[kOzMod];              // floor(p / 2) - 2^62 mod p
  uint32_t magic[kOzMod];             // ceil(2^32 / p): floor(x / p) = x magic >> 32 for x < 2^24
  uint32_t inv[kOzMod];               // W_t^-1 mod p
  uint32_t div[kOzMod];               // floor(2^22 / p)
  uint32_t co[kOzMod];                // product of the other moduli of the triple of p
  uint32_t W[kOzTriples][4], P[4];    // P / (a triple's product) and P in 32-bit limbs
};
constexpr OzTables oz_tables() {
  OzTables T{};
  unsigned __int128 P = 1;
  for (int t = 0; t < kOzMod; ++t) P *= (unsigned)oz_mod(t);
  for (int l = 0; l < 4; ++l) T.P[l] = (uint32_t)(P >> (32 * l));
  for (int t = 0; t < kOzMod; ++t) {
    const uint32_t p = (uint32_t)oz_mod(t);
    uint32_t w = 1;
    for (int k = 0; k < 8; ++k) {
      (k < 4 ? T.wlo[t] : T.whi[t]) |= w << (8 * (k & 3));
      w = w * 256u % p;
    }
    T.init[t] = p / 2 + (p - (uint32_t)((1ull << 62) % p)) % p;
    T.magic[t] = (uint32_t)(((1ull << 32) + p - 1) / p);
    T.div[t] = (1u << 22) / p;
    uint32_t triple = p;
    for (int u = t / 3 * 3; u < kOzMod && u < t / 3 * 3 + 3; ++u)
      if (u != t) triple *= (uint32_t)oz_mod(u);
    T.co[t] = triple / p;
    for (int l = 0; l < 4; ++l) T.W[t / 3][l] = (uint32_t)(P / triple >> (32 * l));
    const unsigned __int128 W = P / p;
    const uint32_t wm = (uint32_t)(W % p);
    for (uint32_t x = 1; x < p; ++x)  // the inverse by search (p <= 256)
      if (wm * x % p == 1) T.inv[t] = x;
  }
  return T;
}
__constant__ OzTables kOz = oz_tables();
constexpr double kOzLead = 1.0 / ((double)oz_tables().P[3] + (double)oz_tables().P[2] * 0x1p-32);  // 2^96 / P

double log2_product() {
  double s = 0;
  for (int p : kModuli) s += std::log2((double)p);
  return s;
}

// Per-line maxima of |X| as FP64 bit patterns (non-negative doubles order like their bits), by
// atomicMax into a zeroed array; a non-finite entry sets SDPXG_ST_NONFINITE.
// ALONG_K (sk == 1): one warp per line reading along k.  Otherwise (consecutive lines
// consecutive in memory): CTAs of 32 lines x 8 warps over a 256-wide k range, lanes along lines.
template <bool ALONG_K>
__global__ void k_oz_amax(const double* __restrict__ X, int rows, int K, long sr, long sk,
                          unsigned long long* __restrict__ amax, uint32_t* __restrict__ status) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double m = 0.0;
  bool bad = false;
  int row;
  if (ALONG_K) {
    row = (int)(((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (row >= rows) return;
    for (int k = lane; k < K; k += 32) {
      const double v = X[row * sr + k];
      bad |= !isfinite(v);
      m = fmax(m, fabs(v));
    }
    for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    bad = __any_sync(0xffffffffu, bad);
    if (lane != 0) return;
  } else {
    __shared__ double part[8][32];
    row = blockIdx.x * 32 + lane;
    const int k0 = blockIdx.y * 256, k1 = min(K, k0 + 256);
    if (row < rows)
      for (int k = k0 + warp; k < k1; k += 8) {
        const double v = X[row + (long)k * sk];
        bad |= !isfinite(v);
        m = fmax(m, fabs(v));
      }
    part[warp][lane] = bad ? __longlong_as_double(0x7ff8000000000000LL) : m;
    __syncthreads();
    if (warp != 0 || row >= rows) return;
    m = 0.0;
    for (int w = 0; w < 8; ++w) {
      const double v = part[w][lane];
      bad |= isnan(v);
      m = isnan(v) ? m : fmax(m, v);
    }
  }
  if (bad) {
    atomicOr(status, SDPXG_ST_NONFINITE);
    m = __longlong_as_double(0x7ff0000000000000LL);
  }
  atomicMax(amax + row, (unsigned long long)__double_as_longlong(m));
}

// Shift of a line with maximum `bits`: b - 1 - floor(log2 max) puts the line below 2^b; 0 for a
// zero or non-finite line.
__device__ __forceinline__ int oz_shift(unsigned long long bits, int b) {
  const int e = (int)(bits >> 52);
  if (e == 0) return bits ? b - 1 - ilogb(__longlong_as_double((long long)bits)) : 0;
  return e == 2047 ? 0 : b - 1 - (e - 1023);
}

__device__ __forceinline__ double oz_pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }  // |e| <= 1022

// Residues of the quantised lines as signed-byte planes: out[(l * Rpad + x) * Kld + k] =
// rint(X(x, k) 2^shift[x]) mod p_l (symmetric), zeros in the padding.  One CTA per tile of
// 32 lines x 128 k, staged in shared memory so that both the reads (along whichever index is
// contiguous) and the 16-byte plane writes are coalesced.
// A thread has four consecutive k of a line, so that a modulus costs one 4-byte store for the four.  A
// residue is a dot product of the integer's bytes with 256^k mod p (two dp4a; 2^62 added first makes it
// non-negative) and one reduction by a multiply-high: 24 instructions for four residues, where a byte
// at a time with three reductions each had 60.  4.2e6 entries took 92 us and take 33, with half of the issue
// slots used: the staged planes leave three blocks an SM, whose warps wait for their lines and for the integer
// pipes about equally.
constexpr int kResPitch = 144;  // bytes per staged line (128 + 16: 16-byte aligned rows)
__global__ void __launch_bounds__(256) k_oz_residues(const double* __restrict__ X, int rows, int K, long sr, long sk,
                                                     const unsigned long long* __restrict__ amax, int b,
                                                     int8_t* __restrict__ out, int Rpad, int Kld) {
  extern __shared__ int8_t tile[];  // [kOzMod][32][kResPitch]
  __shared__ double scale[32][2];   // 2^shift of a line as two factors: the exponent may exceed 1023
  const int r0 = blockIdx.y * 32, k0 = blockIdx.x * 128;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < 32) {
    const int sh = r0 + lane < rows ? oz_shift(amax[r0 + lane], b) : 0, h = sh / 2;
    scale[lane][0] = oz_pow2(h);
    scale[lane][1] = oz_pow2(sh - h);
  }
  __syncthreads();
  const bool along_k = (sk == 1);
#pragma unroll 1
  for (int pass = 0; pass < 4; ++pass) {
    // a warp: one line of 128 k, or 8 lines x 16 k where the lines are contiguous
    const int task = pass * 8 + warp;
    const int rr = along_k ? task : 8 * (task & 3) + (lane & 7);
    const int kk = along_k ? 4 * lane : 16 * (task >> 2) + 4 * (lane >> 3);
    const int x = r0 + rr;
    const double s0 = scale[rr][0], s1 = scale[rr][1];
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = x < rows && k0 + kk + u < K ? X[(long)x * sr + (long)(k0 + kk + u) * sk] : 0.0;
    uint32_t lo[4], hi[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long q = isfinite(v[u]) ? __double2ll_rn(v[u] * s0 * s1) : 0;
      const unsigned long long w = (unsigned long long)q + (1ull << 62);
      lo[u] = (uint32_t)w;
      hi[u] = (uint32_t)(w >> 32);
    }
#pragma unroll
    for (int l = 0; l < kOzMod; ++l) {
      uint32_t r[4];  // residue + floor(p / 2), non-negative
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t y = __dp4a(hi[u], kOz.whi[l], __dp4a(lo[u], kOz.wlo[l], kOz.init[l]));
        r[u] = y - __umulhi(y, kOz.magic[l]) * (uint32_t)oz_mod(l);
      }
      const uint32_t w = __byte_perm(__byte_perm(r[0], r[1], 0x0040), __byte_perm(r[2], r[3], 0x0040), 0x5410);
      const uint32_t h = (uint32_t)(oz_mod(l) / 2) * 0x01010101u, top = 0x80808080u;
      *reinterpret_cast<uint32_t*>(tile + (l * 32 + rr) * kResPitch + kk) =
          ((w | top) - (h & ~top)) ^ ((w ^ ~h) & top);  // bytewise w - h
    }
  }
  __syncthreads();
  const int rr = threadIdx.x >> 3, c = threadIdx.x & 7;
#pragma unroll 4
  for (int l = 0; l < kOzMod; ++l) {
    const uint4 v = *reinterpret_cast<const uint4*>(tile + (l * 32 + rr) * kResPitch + 16 * c);
    *reinterpret_cast<uint4*>(out + ((size_t)l * Rpad + r0 + rr) * Kld + k0 + 16 * c) = v;
  }
}

// C(i, j) = alpha * 2^-(sL_i + sR_j) * X_ij + beta * C(i, j), X_ij the integer product rebuilt from its
// residues: X = sum_t y_t W_t - k P with y_t = x_t W_t^-1 mod p_t (in [0, 2 p_t)), three moduli at a time
// (y_0 p_1 p_2 + y_1 p_0 p_2 + y_2 p_0 p_1) P / (p_0 p_1 p_2), exact in 32-bit limbs, and k = round(sum / P)
// from the leading bits (|X| <= P / 4 leaves the quotient a quarter from a tie); rounded to FP64 once.  A
// thread has four consecutive entries of the planes (one 4-byte load a modulus).
// Bound by instruction issue (71 % of the slots, the integer pipes ahead); mixed-radix digits (a triangle of 120 products and three reductions a
// digit) and a double-double Horner evaluation took 167 us for 4.2e6 entries, one modulus at a time in
// limbs 84, this 62.
__global__ void __launch_bounds__(256) k_oz_crt(const int8_t* __restrict__ PC, long plane, int M, int N,
                                                const unsigned long long* __restrict__ aL,
                                                const unsigned long long* __restrict__ aR, int b, double alpha,
                                                double beta, double* __restrict__ C, long ldc, int upper_only) {
  const long total = (long)M * N, idx0 = 4 * ((long)blockIdx.x * blockDim.x + threadIdx.x);
  if (idx0 >= total) return;
  int j = (int)(idx0 / M), i = (int)(idx0 - (long)j * M);
  if (upper_only && i > j && i + 3 < M) return;  // four entries of a column below the diagonal
  uint32_t word[kOzMod];
  const bool whole = idx0 + 4 <= total && (plane & 3) == 0;
#pragma unroll
  for (int t = 0; t < kOzMod; ++t) {
    if (whole) {
      word[t] = __ldg(reinterpret_cast<const uint32_t*>(PC + t * plane + idx0));
    } else {
      word[t] = 0;
      for (int u = 0; u < 4; ++u)
        if (idx0 + u < total) word[t] |= (uint32_t)(uint8_t)PC[t * plane + idx0 + u] << (8 * u);
    }
  }
#pragma unroll 1
  for (int u = 0; u < 4; ++u, ++i) {
    if (i == M) {
      i = 0;
      ++j;
    }
    if (j >= N) return;
    unsigned long long s0 = 0, s1 = 0, s2 = 0, s3 = 0;
#pragma unroll
    for (int g = 0; g < kOzTriples; ++g) {
      uint32_t z = 0;  // below 2^27
#pragma unroll
      for (int t = 3 * g; t < kOzMod && t < 3 * g + 3; ++t) {
        const int p = oz_mod(t), r = (int)(int8_t)(uint8_t)word[t];
        word[t] >>= 8;
        const uint32_t x = (uint32_t)(r + p) * kOz.inv[t];             // r >= -128 > -p; below 2^17
        z += (x - (x * kOz.div[t] >> 22) * (uint32_t)p) * kOz.co[t];  // the quotient is at most one short
      }
      s0 += (unsigned long long)z * kOz.W[g][0];
      s1 += (unsigned long long)z * kOz.W[g][1];
      s2 += (unsigned long long)z * kOz.W[g][2];
      s3 += (unsigned long long)z * kOz.W[g][3];
    }
    if (upper_only && i > j) continue;
    const unsigned long long top = s3 + (s2 >> 32);  // sum / 2^96, below 2^36; its double without a conversion
    const double lead = __hiloint2double(0x43300000 | (int)(top >> 32), (int)top) - 0x1p52;
    const uint32_t k = (uint32_t)__double2loint(fma(lead, kOzLead, 0x1.8p52));  // rounded to the nearest
    // differences of less than 2^62 in each limb; arithmetic carries
    const long long d0 = (long long)(s0 - (unsigned long long)k * kOz.P[0]);
    const long long d1 = (long long)(s1 - (unsigned long long)k * kOz.P[1]) + (d0 >> 32);
    const long long d2 = (long long)(s2 - (unsigned long long)k * kOz.P[2]) + (d1 >> 32);
    const long long d3 = (long long)(s3 - (unsigned long long)k * kOz.P[3]) + (d2 >> 32);
    unsigned long long hi = (unsigned long long)d3 << 32 | (uint32_t)d2, lo = (unsigned long long)(uint32_t)d1 << 32 | (uint32_t)d0;
    const bool neg = d3 < 0;
    if (neg) {
      lo = ~lo + 1;
      hi = ~hi + (lo == 0);
    }
    int e = 0;
    if (hi) {  // the top 64 bits, the rest as a sticky bit: one rounding
      const int z = __clzll((long long)hi);  // at least 1: |X| < 2^127
      e = 64 - z;
      const unsigned long long rest = lo << z;
      lo = hi << z | lo >> (64 - z) | (rest != 0);
    }
    double x = __ull2double_rn(lo);
    if (neg) x = -x;
    e -= oz_shift(aL[i], b) + oz_shift(aR[j], b);
    x = e >= -1022 && e <= 1023 ? x * oz_pow2(e) : ldexp(x, e);
    double* c = C + i + (long)j * ldc;
    *c = beta == 0.0 ? alpha * x : fma(alpha, x, beta * *c);
  }
}

template <typename T>
void grow(DevBuf<T>& b, size_t n) {
  if (b.n < std::max<size_t>(n, 1)) b.alloc(std::max<size_t>(n, 1));
}

void line_maxima(const double* X, int rows, int K, long sr, long sk, unsigned long long* amax, uint32_t* status,
                 cudaStream_t st) {
  check(cudaMemsetAsync(amax, 0, (size_t)rows * sizeof(unsigned long long), st), "memset");
  if (sk == 1) {
    ++g_launches, k_oz_amax<true><<<(unsigned)(((long)rows * 32 + 255) / 256), 256, 0, st>>>(X, rows, K, sr, sk,
                                                                                              amax, status);
  } else {
    if (sr != 1) throw std::invalid_argument("split GEMM: one operand index must be contiguous");
    ++g_launches, k_oz_amax<false><<<dim3((unsigned)((rows + 31) / 32), (unsigned)((K + 255) / 256)), 256, 0, st>>>(
        X, rows, K, sr, sk, amax, status);
  }
}

}  // namespace

int ozaki_bits(int K) {
  int lg = 0;
  while ((1L << lg) < std::max(K, 1)) ++lg;
  const int b = (int)std::floor((log2_product() - 2.0 - lg) / 2.0);
  return std::min(b, 62);
}

void ozaki_gemm(OzakiWorkspace& ws, cudaStream_t st, int M, int N, int K, const double* L, long l_sr, long l_sk,
                const double* R, long r_sr, long r_sk, double alpha, double beta, double* C, long ldc,
                int upper_only) {
  if (M <= 0 || N <= 0) return;
  if (K <= 0 || K > (1 << 16)) throw std::invalid_argument("split GEMM: K must be in 1..65536");
  if (!L || !R || !C) throw std::invalid_argument("split GEMM: null operand");
  if (!ws.init) {
    grow(ws.moduli, kOzMod);
    ws.moduli.upload(kModuli, kOzMod, st);
    grow(ws.status, 1);
    grow(ws.err, 1);
    check(cudaMemsetAsync(ws.status.p, 0, sizeof(uint32_t), st), "memset");
    check(cudaMemsetAsync(ws.err.p, 0, sizeof(int), st), "memset");
    static std::once_flag attr;
    std::call_once(attr, [] {
      check(cudaFuncSetAttribute(k_oz_residues, cudaFuncAttributeMaxDynamicSharedMemorySize, kOzMod * 32 * kResPitch),
            "oz residues smem");
    });
    ws.init = true;
  }
  const int b = ozaki_bits(K);
  const int Mpad = (M + 127) / 128 * 128, Npad = (N + 255) / 256 * 256, Kld = (K + 127) / 128 * 128;
  grow(ws.amaxL, M);
  grow(ws.amaxR, N);
  grow(ws.PL, (size_t)kOzMod * Mpad * Kld);
  grow(ws.PR, (size_t)kOzMod * Npad * Kld);
  grow(ws.PC, (size_t)kOzMod * M * N);
  line_maxima(L, M, K, l_sr, l_sk, ws.amaxL, ws.status, st);
  line_maxima(R, N, K, r_sr, r_sk, ws.amaxR, ws.status, st);
  const size_t rsm = (size_t)kOzMod * 32 * kResPitch;
  ++g_launches, k_oz_residues<<<dim3(Kld / 128, Mpad / 32), 256, rsm, st>>>(L, M, K, l_sr, l_sk, ws.amaxL, b, ws.PL,
                                                                            Mpad, Kld);
  ++g_launches, k_oz_residues<<<dim3(Kld / 128, Npad / 32), 256, rsm, st>>>(R, N, K, r_sr, r_sk, ws.amaxR, b, ws.PR,
                                                                            Npad, Kld);
  I8GemmArgs ga;
  ga.Mpad = Mpad; ga.Npad = Npad; ga.Kld = Kld; ga.k0 = 0; ga.Kpad = Kld;
  ga.m = M; ga.n = N; ga.L = kOzMod; ga.moduli = ws.moduli; ga.upper_only = upper_only;
  ga.out = ws.PC.p; ga.plane = (long)M * N; ga.err = ws.err.p;
  launch_i8_gemm(1, ws.PL, ws.PR, ga, st);
  ++g_launches, k_oz_crt<<<(unsigned)(((long)M * N + 1023) / 1024), 256, 0, st>>>(
      ws.PC, (long)M * N, M, N, ws.amaxL, ws.amaxR, b, alpha, beta, C, ldc, upper_only);
  check(cudaGetLastError(), "split GEMM launch");
}

}  // namespace sdpxg
