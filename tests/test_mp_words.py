"""The multiword arithmetic under the MPFR kernels (csrc/mp.cuh) against exact integers, on the CPU.

The header's arithmetic compiles for the host with plain C++ in place of the PTX carry chains:
the same rounding, alignment, normalisation and remainder steps.  Every operation is correctly
rounded, so equality is bitwise.  Sizes and operands are those at which a branch changes:
1..8 limbs, mantissas at the ends of their range, operands 0, 1, 63..65 bits and one guard word
apart, cancellations, and dot terms up to the widest span of the register accumulator.
"""
import ctypes as C
import random
import shutil
import subprocess
from fractions import Fraction
from pathlib import Path

import pytest

from oracle import exact as X

CSRC = Path(__file__).resolve().parent.parent / "sdpx.rs_b200" / "csrc"
SRC = r"""
#include "mp.cuh"
using namespace mpd;
template <int N> void op(int code, const unsigned char* a, const unsigned char* b, unsigned char* out) {
  const Val<N> x = load<N>(a), y = load<N>(b);
  uint32_t st = 0;
  Val<N> r = zero_val<N>();
  if (code == 0) r = addsub<N>(x, y, 1);
  if (code == 1) r = addsub<N>(x, y, -1);
  if (code == 2) r = mul<N>(x, y);
  if (code == 3) r = recip<N>(x);
  if (code == 4) r = divide<N>(x, y);
  if (code == 5) r = root<N>(x);
  if (code == 6) r = cmp<N>(x, y) < 0 ? x : y;
  store<N>(out, r, &st);
}
template <int N> int dot_host(const unsigned char* a, const unsigned char* x, const unsigned char* y, int n,
                              unsigned char* out) {
  const long esz = 8 * N + 8;
  long long lo = LLONG_MAX, hi = LLONG_MIN;
  for (int c = 0; c < n; ++c) {
    long long sx, sy;
    if (!load_scale<N>(x + c * esz, &sx) || !load_scale<N>(y + c * esz, &sy)) continue;
    if (sx + sy < lo) lo = sx + sy;
    if (sx + sy > hi) hi = sx + sy;
  }
  const Val<N> av = load<N>(a);
  if (!av.zero) {
    if (av.s < lo) lo = av.s;
    if (av.s - 64LL * N > hi) hi = av.s - 64LL * N;
  }
  if (lo == LLONG_MAX || hi - lo > kSpanBits) return 1;
  Acc<N> acc;
  for (int w = 0; w < Acc<N>::W; ++w) acc.w[w] = 0;
  if (!av.zero) acc_add_value<N>(acc, av, av.s - lo);
  for (int c = 0; c < n; ++c) {
    const Val<N> xv = load<N>(x + c * esz), yv = load<N>(y + c * esz);
    if (xv.zero || yv.zero) continue;
    uint32_t P[4 * N], st = 0;
    mul_words<N>(P, xv.m, yv.m);
    acc_add<N>(acc, P, (int)(xv.s + yv.s - lo), xv.neg == yv.neg);
  }
  uint32_t st = 0;
  store<N>(out, acc_round<N>(acc, lo), &st);
  return 0;
}
#define EACH(F) F(1) F(2) F(3) F(4) F(5) F(6) F(7) F(8)
extern "C" void mp_op(int N, int code, const unsigned char* a, const unsigned char* b, unsigned char* o) {
#define CASE(n) if (N == n) op<n>(code, a, b, o);
  EACH(CASE)
#undef CASE
}
extern "C" int mp_dot(int N, const unsigned char* a, const unsigned char* x, const unsigned char* y, int n,
                      unsigned char* o) {
#define CASE(m) if (N == m) return dot_host<m>(a, x, y, n, o);
  EACH(CASE)
#undef CASE
  return 1;
}
"""


@pytest.fixture(scope="module")
def words(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("mpwords")
    (d / "w.cc").write_text(SRC)
    subprocess.run([gxx, "-O1", "-std=c++17", "-w", "-shared", "-fPIC", "-I", str(CSRC), str(d / "w.cc"), "-o",
                    str(d / "w.so")], check=True)
    return C.CDLL(str(d / "w.so"))


def mantissas(n, rng):
    p = 64 * n
    top = 1 << (p - 1)
    yield from (top, top + 1, (1 << p) - 1, (1 << p) - 2, top | (top >> 1), top + (1 << (p // 2)))
    for _ in range(10):
        yield top | rng.getrandbits(p)
        yield top | (rng.getrandbits(20) << rng.randrange(p - 20))


def values(n, rng):
    return [X.Mp(n, rng.random() < 0.5, m, rng.choice([0, 0, 1, -3, 40])) for m in mantissas(n, rng)]


def run_op(words, n, code, a, b):
    out = C.create_string_buffer(8 * n + 8)
    words.mp_op(n, code, a.pack(), b.pack(), out)
    return X.Mp.unpack(n, out.raw)


@pytest.mark.parametrize("n", range(1, 9))
def test_operations_round_once(words, n):
    rng = random.Random(n)
    vals = values(n, rng) + [X.Mp(n)]
    p = 64 * n
    gaps = [0, 1, 2, 31, 32, 33, 63, 64, 65, 66, p - 1, p, p + 1, p + 62, p + 63, p + 64, p + 65, p + 200]
    for a in vals:
        for b in rng.sample(vals, 8):
            for g in [0] + rng.sample(gaps, 4):
                c = X.Mp(n, b.neg, b.mant, b.exp - g)
                fa, fc = a.fraction(), c.fraction()
                for x, y, fx, fy in ((a, c, fa, fc), (c, a, fc, fa)):
                    assert run_op(words, n, 0, x, y) == X.from_fraction(n, fx + fy)
                    assert run_op(words, n, 1, x, y) == X.from_fraction(n, fx - fy)
                    assert run_op(words, n, 6, x, y) == (x if fx < fy else y)
                assert run_op(words, n, 2, a, c) == X.from_fraction(n, fa * fc)
            if not b.is_zero():
                assert run_op(words, n, 4, a, b) == X.from_fraction(n, a.fraction() / b.fraction())
        if not a.is_zero():
            assert run_op(words, n, 3, a, a) == X.from_fraction(n, 1 / a.fraction())
        for e in (a.exp, a.exp + 1):
            v = X.Mp(n, False, a.mant, e)
            assert run_op(words, n, 5, v, v) == X.mp_sqrt(n, v)


@pytest.mark.parametrize("n", range(1, 9))
def test_exact_dot_in_the_register_accumulator(words, n):
    rng = random.Random(100 + n)
    span = 12 * 32 - 72
    for count, wide in ((1, 0), (2, span), (3, span - 1), (17, 40), (33, span), (64, 200)):
        for cancel in (False, True):
            x = [X.Mp(n, rng.random() < 0.5, (1 << (64 * n - 1)) | rng.getrandbits(64 * n - 1), 0) for _ in range(count)]
            y = [X.Mp(n, rng.random() < 0.5, (1 << (64 * n - 1)) | rng.getrandbits(64 * n - 1),
                      rng.randrange(wide + 1) if wide else 0) for _ in range(count)]
            y[0].exp = 0
            y[-1].exp = wide
            if cancel:  # the second half cancels the first: the sum is what is left of the addend
                x = x + x
                y = y + [X.Mp(n, not v.neg, v.mant, v.exp) for v in y]
            total = sum((u.fraction() * v.fraction() for u, v in zip(x, y)), Fraction(0))
            # addends at both ends of their frame: the last bit and, as a product's top, the first
            for a in (X.Mp(n), X.Mp(n, True, (1 << (64 * n)) - 1, -64 * n), X.Mp(n, False, 1 << (64 * n - 1), wide)):
                out = C.create_string_buffer(8 * n + 8)
                rc = words.mp_dot(n, a.pack(), X.pack_array(x), X.pack_array(y), len(x), out)
                assert rc == 0
                assert X.Mp.unpack(n, out.raw) == X.from_fraction(n, a.fraction() - total)
