// Publications of the chain of the dataflow Cholesky (chol_dataflow.cu), numbered in their order: 2k is
// U_kk^-T of step k, 2k + 1 is U(k, k+1).  The eight MMA warps arrive on the barrier slot(t) once their
// stores of publication t are issued; the publishing warp waits for the phase of parity(t), in order.
//
// A parity wait cannot tell a phase from the one two phases on, so a barrier may not complete twice before
// the publishing warp has seen its first phase.  The chain itself runs ahead of the publications: up to
// U_kk^-T of step k+1 it needs none of step k.  With one barrier per kind it could complete the phase of
// step k+1 first and the publishing warp would wait for that of step k+2, which waits for tiles that
// wait for step k.  Two barriers per kind, taken in turn by step, are enough: the next use of the barrier of
// publication t is t + 4, of step k + 2, whose tiles need publication t (U_kk^-T reaches row k of its
// column, U(k, k+1) the sums of row k+1).
#pragma once

#if defined(__CUDACC__)
#define SDPXG_PUB_FN __host__ __device__ constexpr
#else
#define SDPXG_PUB_FN constexpr
#endif

namespace chol_publish {
constexpr int kSlots = 4;
SDPXG_PUB_FN int slot(int t) { return t & 3; }
SDPXG_PUB_FN int parity(int t) { return (t >> 2) & 1; }
}  // namespace chol_publish
