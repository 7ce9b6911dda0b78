// Glue between two domains (faces of different orders): the coupling
// kernel run once per LSRK stage before the stage's element launches.
#pragma once

#include "dg_common.cuh"

namespace bfam_b200
{

constexpr int PGLUE_MAXQ = 8;  // highest compiled order 7
constexpr int PGLUE_THREADS = 256; // 128 per side

// One side of a glue: its domain's stage input, element tables and mortar
// buffer, the glued face of every pair and its mortar slot, and its 1-D
// operators to and from the glue grid (column-major; NULL: identity).
struct PGlueSide
{
  const double *__restrict__ q;
  size_t fs;
  int N;
  const ElemData *__restrict__ ed;
  double *mbuf;
  const int32_t *__restrict__ elem;
  const int8_t *__restrict__ face;
  const int32_t *__restrict__ slot;
  const double *__restrict__ I; // (Ng+1) x (N+1)
  const double *__restrict__ P; // (N+1) x (Ng+1)
};

struct PGlueView
{
  PGlueSide s[2];
  int32_t K;
  int Ng, flux;
};

// volume node of face node (a, b) on face f of an order-N element
template <int DIM>
__device__ __forceinline__ int gmask_rt(int N, int f, int a, int b)
{
  const int Nq = N + 1;
  if (DIM == 2)
    return f == 0 ? a * Nq : (f == 1 ? a * Nq + N : (f == 2 ? a : N * Nq + a));
  switch (f)
  {
  case 0: return Nq * a + Nq * Nq * b;
  case 1: return N + Nq * a + Nq * Nq * b;
  case 2: return a + Nq * Nq * b;
  case 3: return a + Nq * N + Nq * Nq * b;
  case 4: return a + Nq * b;
  default: return a + Nq * b + Nq * Nq * N;
  }
}

// out[i + mo b'] = sum A(i, a) v[a + mi b] along the first face axis (A is
// mo x mi column-major, A == NULL: copy), for the n2 lines b of nf fields;
// `stride` separates the fields in both arrays
__device__ __forceinline__ void pglue_axis0(const double *A, int mo, int mi,
                                            int n2, int nf, int stride,
                                            const double *v, double *out,
                                            int t)
{
  for (int w = t; w < nf * mo * n2; w += PGLUE_THREADS / 2)
  {
    const int c = w / (mo * n2), r = w % (mo * n2);
    const int i = r % mo, b = r / mo;
    const double *x = v + c * stride + mi * b;
    double s = 0;
    if (A)
      for (int a = 0; a < mi; ++a)
        s += A[i + mo * a] * x[a];
    else
      s = x[i];
    out[c * stride + i + mo * b] = s;
  }
}

// the same along the second face axis: out[a + m0 i] = sum A(i, b) v[a + m0 b]
__device__ __forceinline__ void pglue_axis1(const double *A, int mo, int mi,
                                            int m0, int nf, int stride,
                                            const double *v, double *out,
                                            int t)
{
  for (int w = t; w < nf * m0 * mo; w += PGLUE_THREADS / 2)
  {
    const int c = w / (m0 * mo), r = w % (m0 * mo);
    const int a = r % m0, i = r / m0;
    const double *x = v + c * stride + a;
    double s = 0;
    if (A)
      for (int b = 0; b < mi; ++b)
        s += A[i + mo * b] * x[m0 * b];
    else
      s = x[m0 * i];
    out[c * stride + a + m0 * i] = s;
  }
}

// One CTA per glued pair (minus side s[0], plus side s[1], opposite faces of
// one axis, face nodes in the same tangential order), half of its threads per
// side:
//  1. each side's trace (velocity and the stress row of the face axis) is
//     gathered and interpolated to the order-Ng glue grid;
//  2. at every glue node the Riemann problem gives each side's jumps
//     (T* - T-, v* - v-) from its own outward normal and impedances;
//  3. each side's jumps are L2-projected back to its order and stored in
//     its mortar slot, [2 dim][Nfp] in that side's face-node order, which
//     the side's stage kernel lifts like a coarse face with one piece.
// The launch stands before a stage's element launches, few CTAs of a chain of
// dependent passes: its latency bounds it, not its traffic.  With 64 threads
// taking the sides one after the other, a stage of two glued halves of 2,048
// elements of orders 3 and 5 (512 pairs) took 46.8 us, so 44.8.
template <int DIM>
__global__ void __launch_bounds__(PGLUE_THREADS) dg_pglue_kernel(const PGlueView v)
{
  constexpr int NTF = 2 * DIM, NJ = 2 * DIM, HALF = PGLUE_THREADS / 2;
  constexpr int MF = DIM == 3 ? PGLUE_MAXQ * PGLUE_MAXQ : PGLUE_MAXQ;
  __shared__ double tr[2][NTF][MF]; // traces, then glue-grid values
  __shared__ double tmp[2][NTF][MF];
  __shared__ double J[2][NJ][MF];
  const int k = blockIdx.x, sd = threadIdx.x / HALF, t = threadIdx.x % HALF;
  const PGlueSide &S = v.s[sd];
  const int Nq = S.N + 1, nf = DIM == 3 ? Nq * Nq : Nq;
  const int Ngq = v.Ng + 1, nfg = DIM == 3 ? Ngq * Ngq : Ngq;
  const int f = S.face[k], ax = f >> 1;
  const ElemData &me = S.ed[S.elem[k]], &other = v.s[sd ^ 1].ed[v.s[sd ^ 1].elem[k]];
  const double fc[4] = {other.Zp, 1.0 / (me.Zp + other.Zp), other.Zs,
                        1.0 / (me.Zs + other.Zs)};
  const double Zp = me.Zp, Zs = me.Zs;
  grid_launch_dependents();
  grid_dependency_wait();

  // 1. traces to the glue grid
  {
    const double *q = S.q + (size_t)S.elem[k] * (DIM == 3 ? Nq * Nq * Nq : Nq * Nq);
    double *x = S.I ? &tmp[sd][0][0] : &tr[sd][0][0];
    for (int w = t; w < NTF * nf; w += HALF)
    {
      const int c = w / nf, pn = w % nf;
      x[c * MF + pn] = q[trace_field<DIM>(ax, c) * S.fs +
                         gmask_rt<DIM>(S.N, f, pn % Nq, pn / Nq)];
    }
  }
  __syncthreads();
  if (v.s[0].I || v.s[1].I)
  {
    // J is free until step 2
    if (S.I && DIM == 3)
      pglue_axis0(S.I, Ngq, Nq, Nq, NTF, MF, &tmp[sd][0][0], &J[sd][0][0], t);
    else if (S.I)
      pglue_axis0(S.I, Ngq, Nq, 1, NTF, MF, &tmp[sd][0][0], &tr[sd][0][0], t);
    __syncthreads();
    if (DIM == 3)
    {
      if (S.I)
        pglue_axis1(S.I, Ngq, Nq, Ngq, NTF, MF, &J[sd][0][0], &tr[sd][0][0], t);
      __syncthreads();
    }
  }

  // 2. this side's jumps at the glue nodes
  {
    const double sg = (f & 1) ? 1.0 : -1.0;
    for (int pg = t; pg < nfg; pg += HALF)
    {
      double dq[NTF], Jm[6];
#pragma unroll
      for (int c = 0; c < NTF; ++c)
      {
        // the difference across the glue is formed once, from the minus side
        const double d = tr[1][c][pg] - tr[0][c][pg];
        dq[c] = sd ? -d : d;
      }
      flux_jumps<DIM, double>(dq, ax, sg, Zp, Zs, fc, v.flux, Jm);
#pragma unroll
      for (int c = 0; c < NJ; ++c)
        J[sd][c][pg] = Jm[jslot<DIM>(c)];
    }
  }
  __syncthreads();

  // 3. projection to this side's order, into its mortar slot
  double *out = S.mbuf + (size_t)S.slot[k] * NJ * nf;
  if (v.s[0].P || v.s[1].P)
  {
    if (S.P)
      pglue_axis0(S.P, Nq, Ngq, DIM == 3 ? Ngq : 1, NJ, MF, &J[sd][0][0],
                  &tmp[sd][0][0], t);
    __syncthreads();
    if (S.P && DIM == 3)
      pglue_axis1(S.P, Nq, Ngq, Nq, NJ, MF, &tmp[sd][0][0], &tr[sd][0][0], t);
    if (DIM == 3)
      __syncthreads();
  }
  const double *y = !S.P ? &J[sd][0][0] : (DIM == 3 ? &tr[sd][0][0] : &tmp[sd][0][0]);
  for (int w = t; w < NJ * nf; w += HALF)
    out[w] = y[(w / nf) * MF + w % nf];
}

} // namespace bfam_b200
