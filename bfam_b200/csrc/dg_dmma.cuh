// The FP64 matrix instruction on planes and faces of at most 8 x 8 nodes, one
// per warp, held in the instruction's accumulator layout ("C layout"):
// lane 4 r + c holds X[r][2 c], X[r][2 c + 1] (see dg_mma.cuh).
#pragma once

#include "dg_common.cuh"

namespace bfam_b200
{

// d += a b, one 8 x 8 x 4 step
__device__ __forceinline__ void dmma(double2 &d, double a, double b)
{
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
               "{%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d.x), "+d"(d.y)
               : "d"(a), "d"(b));
}

// x[k] = Op x[k]^T for n matrices in C layout; op: Op's left fragment
// (Op[r][2c], Op[r][2c+1])
template <int n>
__device__ __forceinline__ void dmma_t(const double2 op, double2 *x)
{
  double2 y[n];
#pragma unroll
  for (int k = 0; k < n; ++k)
  {
    y[k] = make_double2(0.0, 0.0);
    dmma(y[k], op.x, x[k].x);
  }
#pragma unroll
  for (int k = 0; k < n; ++k)
  {
    dmma(y[k], op.y, x[k].y);
    x[k] = y[k];
  }
}

// Two values of a row from p[0] and p[o1] (adjacent and 16-byte aligned if
// VEC), and their store where they exist (v0, v1).
template <bool VEC>
__device__ __forceinline__ double2 get2(const double *p, int o1 = 1)
{
  return VEC ? *reinterpret_cast<const double2 *>(p)
             : make_double2(p[0], p[o1]);
}
template <bool VEC>
__device__ __forceinline__ void put2(double *p, const double2 x, bool v0, bool v1)
{
  if (VEC)
  {
    if (v0)
      *reinterpret_cast<double2 *>(p) = x;
  }
  else
  {
    if (v0)
      p[0] = x.x;
    if (v1)
      p[1] = x.y;
  }
}

// Two arrays of face nodes, g0 and g1 of the face region x (Nfp values each,
// fpos order), through the tensor product of mortar operator `op` (2: the
// interpolation to a piece, 5: the projection from one; ops: Dr |
// interpolation[3] | projection[3], bottom halves, of which the top halves are
// the reflections) for hanging piece hp (1 to 4), by one warp: result in C
// layout, row the second face axis.
template <int N>
__device__ __forceinline__ void mortar_pair(const double *ops, int op, int hp,
                                            const double *x, int g0, int g1,
                                            double2 *y)
{
  constexpr int Nq = N + 1, P = Nq * Nq;
  const int rr = (threadIdx.x & 31) >> 2, c = threadIdx.x & 3;
  // lanes past the matrix read its last row and column; their values are not
  // stored, and zeros where they meet the operator's
  const int r = rr < Nq ? rr : N;
  const int i0 = 2 * c < Nq ? 2 * c : N, i1 = 2 * c + 1 < Nq ? 2 * c + 1 : N;
  auto frag = [&](int top) {
    const double *A = ops + op * P + (top ? Nq * N + N - r : r);
    const int sk = top ? -Nq : Nq;
    return make_double2(2 * c < Nq ? __ldg(A + sk * i0) : 0.0,
                        2 * c + 1 < Nq ? __ldg(A + sk * i1) : 0.0);
  };
  const double2 a = frag((hp - 1) & 1), b = frag((hp - 1) >> 1);
  const double *x0 = x + g0 * P, *x1 = x + g1 * P;
  y[0] = make_double2(x0[fpos<3, N>(g0, i0 + Nq * r)],
                      x0[fpos<3, N>(g0, i1 + Nq * r)]);
  y[1] = make_double2(x1[fpos<3, N>(g1, i0 + Nq * r)],
                      x1[fpos<3, N>(g1, i1 + Nq * r)]);
  if (Nq < 8)
  {
#pragma unroll
    for (int k = 0; k < 2; ++k)
      y[k] = make_double2(rr < Nq && 2 * c < Nq ? y[k].x : 0.0,
                          rr < Nq && 2 * c + 1 < Nq ? y[k].y : 0.0);
  }
  dmma_t<2>(a, y);
  dmma_t<2>(b, y);
}

} // namespace bfam_b200
