// Stage kernel for elements of few nodes (2D, and 3D orders 1 and 2): the
// element update of dg_stage.cuh, with the same arithmetic, for several
// elements per CTA whose nodes fill its threads.
//
// One element per CTA left these shapes with a warp or two per CTA, half of
// its lanes idle, and at most 16 CTAs per SM (2D N = 3: 28 % of the warps, 890
// warp instructions per 16-node element, DRAM 21 %).  Here a thread is a node
// of one of E elements (128 threads; 256 where 128 would leave a fifth of them
// idle), the state comes by 8-byte copies that coalesce over neighbouring
// elements whatever the parity of Np, dq is loaded into registers ahead of the
// barriers, and later items' rows are prefetched into L2, a line per thread.
// Measured on 30 M DOF bricks, G DOF-updates/s before -> now (plain form,
// conforming and with 30 % of the base cells refined): 2D N = 1 28 -> 86 and
// 22 -> 63, N = 2 48 -> 117 and 36 -> 81, N = 3 82 -> 143 and 56 -> 116, N = 4
// 81 -> 143 and 68 -> 110, N = 5 91 -> 143 and 65 -> 112, N = 6 81 -> 126 and
// 67 -> 97, N = 7 141 -> 150 and 103 -> 118, N = 8 (precision form) 105 -> 135
// and 89 -> 106; 3D N = 1 56 -> 96 and 38 -> 62, N = 2 80 -> 98 and 58 -> 72.  Not
// used where the one-element kernel is faster: 3D N = 3 (156 against 123) and 4,
// the shapes of use_pack, and launches too small for it (pack_from).
// What bounds it now is latency (long scoreboard) beside the LSU pipe (60 %).
#pragma once

#include "dg_common.cuh"
#include "dg_stage.cuh"
#include "dg_volume.cuh"

namespace bfam_b200
{

constexpr int even(int n) { return n + n % 2; }

// E elements of Np nodes on NT threads, a node each.  Shared memory in
// doubles: the state field-major over the CTA's nodes; per element and face
// the neighbour's trace, then the flux jumps; the mortar jumps of at most DIM
// fine faces per element; flux constants, element data and D; the precision
// form's FP32 state; then integers (fine-face list).
template <int DIM, int N, typename CT> struct PackShape
{
  using S = Shape<DIM, N>;
  static constexpr int NT = DIM == 2 && (N == 6 || N == 8) ? 256 : 128;
  static constexpr int E = NT / S::Np, NV = E * S::Np;
  static constexpr int OFF_PT = even(S::NFLD * NV);
  static constexpr int OFF_MJ = OFF_PT + even(E * S::NF * S::NTF * S::Nfp);
  static constexpr int OFF_FC = OFF_MJ + even(E * DIM * S::NJ * S::Nfp);
  static constexpr int OFF_ED = OFF_FC + E * S::NF * 4;
  static constexpr int OFF_D = OFF_ED + E * 8;
  // the mortar passes by value (line_values) read Ib and Pb here
  static constexpr bool VALUES = DIM == 2 && N >= 6;
  static constexpr int OFF_IB = OFF_D + even(S::Nq * S::Nq);
  static constexpr int OFF_QV = OFF_IB + (VALUES ? 2 * even(S::Nq * S::Nq) : 0);
  static constexpr bool NARROW = sizeof(CT) < sizeof(double);
  static constexpr int OFF_I = OFF_QV + (NARROW ? (S::NFLD * NV + 3) / 4 * 2 : 0);
  // face descriptors, mortar slots, elements, fine faces and their number
  static constexpr int INTS = 3 * E * S::NF + E + E * DIM + 1;
  static constexpr size_t BYTES = OFF_I * sizeof(double) + INTS * sizeof(int);
  static constexpr int BY_SMEM = (int)(233472 / (BYTES + 1024));
  static constexpr int WANT = NT == 256 ? 5 : DIM == 2 && N >= 3 ? 10 : 8;
  static constexpr int MINB = BY_SMEM < WANT ? BY_SMEM : WANT;
};

// Shapes and arithmetic the kernel serves.  Not, of 2D's, the precision form at
// N = 7, and the plain form at N = 8, whose one element of 81 nodes per CTA,
// its rows by bulk copies, is as fast on large meshes (74,000 elements 1,259 us
// per step against 1,278 here, refined 1,562 and 1,583) and faster on small ones
// (1,501 refined 60.5 and 70.7) and in batches (73,600 refined 1,699 and 1,798).
template <int DIM, int N, typename CT>
__host__ __device__ constexpr bool use_pack()
{
  return DIM == 2 ? N < 7 || N == (sizeof(CT) == sizeof(double) ? 7 : 8) : N <= 2;
}

// In batches of several domains not the plain form at 3D N = 2: the
// node-per-thread kernel is faster or equal (5,256 conforming elements 91 us per
// step against 112 here, 242,649 3,352 and 3,419; refined 39,335 826 and 847,
// 248,268 4,781 and 4,733).
template <int DIM, int N, typename CT> constexpr bool use_pack_batch()
{
  return use_pack<DIM, N, CT>() &&
         !(DIM == 3 && N == 2 && sizeof(CT) == sizeof(double));
}

// Low orders, whose CTA holds many elements: on a small mesh a CTA takes only
// so many that every SM gets four CTAs.  The passes before the node pass run
// over a CTA's faces, so fewer elements per CTA shorten the chain of latencies
// that bounds a small mesh (us per step, full CTAs -> spread; one element per
// CTA of the node-per-thread kernel in brackets): 2D N = 1, 1,822 refined
// elements 47 -> 36 (38), 6,895 50 -> 38 (58); 2D N = 2, 1,822 46 -> 37 (42);
// 3D N = 1, 398 67 -> 40 (53), 6,425 85 -> 66 (96); 3D N = 2, 398 67 -> 53
// (52).  One CTA per SM instead of four: 36, 45, 38, 40, 79, 62.  At the other
// orders (two to eight elements per CTA) it gave nothing and the variable
// count cost 2-6 % (2D N = 6 397 -> 415), so it is a constant there.
template <int DIM, int N> __host__ __device__ constexpr bool pack_spreads()
{
  return N <= 2;
}

// sp with the elements per CTA for n elements
template <int DIM, int N, int E>
inline StageParams pack_params(int n, StageParams sp)
{
  const int spread = (n + 4 * sp.sms - 1) / (4 * sp.sms);
  sp.per = pack_spreads<DIM, N>() && spread < E ? spread : E;
  return sp;
}

inline int pack_ctas(int n, const StageParams &sp)
{
  return (n + sp.per - 1) / sp.per;
}

// Launches of a served shape that are too small for it: the passes over a CTA's
// fine faces go on among few of its threads, and in batches each of its elements
// reaches its domain through two tables, so on meshes of a few elements per SM
// the node-per-thread kernel's many small CTAs are faster.  The elements per SM
// below which a launch goes there (with hanging faces or without, in a batch of
// several domains or not; in 2D those of the stage's widest launch, whose levels
// then go together) lie where the sides meet; us per step node-per-thread and
// packed:
//   3D N = 2, FP64: 9,969 refined elements 206 and 207, 24,254 468 and 461;
//     conforming 2,197 46 and 57, 42,875 566 and 578, 64,000 827 and 822;
//   FP32: 1,597 refined 64 and 76; conforming 1,331 34 and 35, 2,197 49 and 48;
//     batches 5,077 refined 132 and 138, 125,382 2,374 and 2,427, conforming
//     5,256 91 and 100, 40,661 571 and 573, 82,620 1,132 and 1,121;
//   2D N = 6, batches: FP64 5,198 refined 108 and 116, 7,805 154 and 142,
//     conforming 990 29.5 and 33.5, 1,521 41 and 40; FP32 alike;
//   2D N = 7, FP64, batches: 5,198 refined 105 and 117, 11,557 216 and 220,
//     17,246 321 and 312, conforming 3,384 59 and 65, 47,099 578 and 584;
//   2D N = 8, FP32, batches: 3,401 refined 103 and 110, 5,198 150 and 135,
//     conforming 990 31.4 and 37.5, 1,521 45.8 and 45.0.
template <int DIM, int N, typename CT>
constexpr int pack_from(bool hanging, bool batch)
{
  constexpr bool f64 = sizeof(CT) == sizeof(double);
  constexpr int always = 1 << 20;
  if (DIM == 3 && N == 2)
    return batch ? (hanging ? always : 400)
                 : (hanging ? 48 : f64 ? 400 : 12);
  if (DIM == 3 || N < 6 || !batch)
    return 0;
  return N == 6   ? (hanging ? 32 : 10)
         : N == 7 ? (hanging ? 60 : always)
                  : (hanging ? 22 : 8);
}
template <int DIM, int N, typename CT> constexpr bool pack_has_small(bool batch)
{
  return pack_from<DIM, N, CT>(true, batch) > 0;
}
// n elements in a stage whose largest launch has `widest`
template <int DIM, int N, typename CT>
bool pack_too_small(int n, int widest, int sms, int mode, bool batch)
{
  return (DIM == 2 ? widest : n) <
         (int64_t)pack_from<DIM, N, CT>(mode != MODE_STAGE_CF, batch) * sms;
}

// The 1-D mortar pass of line_apply on `lines` faces of NC fields each (2D
// orders 6 and up), a thread per value instead of per line: a CTA has few
// lines there, and a thread per line left most of it waiting for Nq x Nq
// serial products (refined meshes, G DOF-updates/s by line and by value: N = 8
// 60 and 93, N = 7 73 and 118, N = 6 82 and 95; but N = 5 110 and 107, N = 3
// 113 and 107).  A: the
// bottom-half operator in shared memory (the precision form's interpolation
// is applied to the line minus its first value, as in line_apply); at(l, c,
// top) gives line c of face l and its half.  Ends with the CTA's barrier.
template <int N, typename T, int NC, int NT, int LINES, typename At>
__device__ __forceinline__ void line_values(const T *A, int lines, int t,
                                            const At &at)
{
  constexpr int Nq = N + 1, IT = (LINES * NC * Nq + NT - 1) / NT;
  constexpr bool OFFSET = sizeof(T) < sizeof(double);
  double out[IT];
#pragma unroll
  for (int k = 0; k < IT; ++k)
  {
    const int w = t + k * NT;
    if (w < lines * NC * Nq)
    {
      int top;
      const double *x = at(w / (NC * Nq), w / Nq % NC, top);
      const double ref = OFFSET ? x[0] : 0.0;
      const int m = top ? N - w % Nq : w % Nq;
      T s = 0;
#pragma unroll
      for (int i = 0; i < Nq; ++i)
      {
        const double xi = x[top ? N - i : i];
        s += A[m + Nq * i] * (OFFSET ? T(xi - ref) : T(xi));
      }
      out[k] = OFFSET ? ref + double(s) : double(s);
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < IT; ++k)
  {
    const int w = t + k * NT;
    if (w < lines * NC * Nq)
    {
      int top;
      at(w / (NC * Nq), w / Nq % NC, top)[w % Nq] = out[k];
    }
  }
  __syncthreads();
}

template <int DIM, int N, int MODE, typename CT, typename Item>
__device__ __forceinline__ void pack_elements(const Item &item, int n,
                                              const StageParams &sp,
                                              const DiffOp<N, CT> &dop)
{
  using S = Shape<DIM, N>;
  using K = PackShape<DIM, N, CT>;
  constexpr int Nq = S::Nq, Np = S::Np, Nfp = S::Nfp, NF = S::NF,
                NFLD = S::NFLD, NJ = S::NJ, NPC = S::NPC, ROWS = S::ROWS,
                NTF = S::NTF, NT = K::NT, NV = K::NV, FN = NF * Nfp;
  extern __shared__ __align__(16) double smem[];
  double *qs = smem, *pt = smem + K::OFF_PT, *mj = smem + K::OFF_MJ;
  double *fcf = smem + K::OFF_FC;
  const ElemData *ed = reinterpret_cast<const ElemData *>(smem + K::OFF_ED);
  CT *sD = reinterpret_cast<CT *>(smem + K::OFF_D);
  int2 *desc = reinterpret_cast<int2 *>(smem + K::OFF_I);
  int *fidx = reinterpret_cast<int *>(desc + K::E * NF); // mortar slot or -1
  int *elem = fidx + K::E * NF;
  int *flist = elem + K::E, *fcount = flist + K::E * DIM;
  const int t = threadIdx.x, per = pack_spreads<DIM, N>() ? sp.per : K::E;
  const int first = blockIdx.x * per;
  const int ne = n - first < per ? n - first : per; // elements here
  const bool rd = MODE != MODE_RHS && !sp.first_stage;
  constexpr bool HANGS = MODE != MODE_STAGE_CF; // any hanging face

  CT *sI = reinterpret_cast<CT *>(smem + K::OFF_IB);
  double *sP = smem + K::OFF_IB + even(Nq * Nq);
  for (int w = t; w < Nq * Nq; w += NT)
  {
    sD[w] = dop.D[w];
    if (K::VALUES)
    {
      sI[w] = dop.Ib[w];
      sP[w] = dop.Pb[w];
    }
  }
  if (t == 0)
    *fcount = 0;
  __syncthreads();
  // descriptors, and the fine faces of the CTA's elements (in no particular
  // order)
  for (int w = t; w < ne * NF; w += NT)
  {
    const int es = w / NF, e = item.elem(first + es);
    const int2 ds = item.view(first + es).fdesc[(size_t)e * NF + w % NF];
    int at = -1;
    if (HANGS && (ds.y & 3) == 1 && ((ds.y >> 8) & 7) != 0)
    {
      at = atomicAdd(fcount, 1);
      flist[at] = w;
    }
    fidx[w] = at;
    desc[w] = ds;
    if (w % NF == 0)
      elem[es] = e;
  }
  __syncthreads();
  grid_dependency_wait(); // the stage input is complete

  // ------------------------------------------------------------------ loads
  const int ms = t / Np, mn = t % Np; // my element and node
  const bool mine = t < NV && ms < ne;
  const DomainView &md = item.view(first + (mine ? ms : 0));
  const int me_ = elem[mine ? ms : 0];
  const size_t mat = (size_t)me_ * Np + mn;
  if (mine)
  {
#pragma unroll
    for (int c = 0; c < NFLD; ++c)
      cp_async8(qs + c * NV + t, md.qin + c * md.fs + mat);
  }
  for (int w = t; w < ne * FN; w += NT)
  {
    const int es = w / FN, f = w % FN / Nfp, pn = w % Nfp;
    const DomainView &d = item.view(first + es);
    const size_t ef = (size_t)elem[es] * NF + f;
    const int2 ds = desc[es * NF + f];
    const int k = ds.y & 3;
    if (k == 2)
      continue;
    if (k != 3)
    {
      const double *src =
          d.qin + (size_t)ds.x * Np + gmask<DIM, N>((ds.y >> 2) & 7, pn);
      double *dst = pt + (es * NF + f) * NTF * Nfp + pn;
#pragma unroll
      for (int c = 0; c < NTF; ++c)
        cp_async8(dst + c * Nfp, src + trace_field<DIM>(f >> 1, c) * d.fs);
    }
    if (pn == 0)
    {
      const double *fc = reinterpret_cast<const double *>(d.fcE + ef);
      cp_async16(fcf + 4 * (es * NF + f), fc);
      cp_async16(fcf + 4 * (es * NF + f) + 2, fc + 2);
    }
  }
  for (int w = t; w < ne * 4; w += NT)
    cp_async16(smem + K::OFF_ED + 2 * w,
               reinterpret_cast<const double *>(item.view(first + w / 4).ed +
                                                elem[w / 4]) +
                   2 * (w % 4));
  cp_async_commit();
  // later items' state and dq rows into L2, a line each
  if (sp.ahead > 0)
  {
    constexpr int L = (Np * 8 + 127) / 128 + (Np % 16 ? 1 : 0);
    for (int w = t; w < per * L; w += NT)
    {
      const int ia = first + sp.ahead + w / L;
      if (ia < n)
      {
        const DomainView &d = item.view(ia);
        const int x = 16 * (w % L);
        const size_t at = (size_t)item.elem(ia) * Np + (x < Np ? x : Np - 1);
#pragma unroll
        for (int c = 0; c < NFLD; ++c)
        {
          prefetch_l2(d.qin + c * d.fs + at);
          if (rd)
            prefetch_l2(d.dq + c * d.fs + at);
        }
      }
    }
  }
  double qd[NFLD];
#pragma unroll
  for (int c = 0; c < NFLD; ++c)
    qd[c] = mine && rd ? md.dq[c * md.fs + mat] : 0.0;
  cp_async_wait<0>();
  __syncthreads();
  const int nfine = HANGS ? *fcount : 0;

  // FP32 state minus the element's first node (see dg_stage.cuh)
  const CT *qv;
  if constexpr (K::NARROW)
  {
    CT *o = reinterpret_cast<CT *>(smem + K::OFF_QV);
    if (mine)
    {
#pragma unroll
      for (int c = 0; c < NFLD; ++c)
        o[c * NV + t] = CT(qs[c * NV + t] - qs[c * NV + ms * Np]);
    }
    qv = o;
  }
  else
    qv = qs;

  // ------------------------------------- fine side: coarse trace -> my piece
  if (nfine)
  {
    if constexpr (K::VALUES)
      line_values<N, CT, NTF, NT, K::E * DIM>(sI, nfine, t, [&](int l, int c, int &top) {
        const int fw = flist[l];
        top = (((desc[fw].y >> 8) & 7) - 1) & 1;
        return pt + (fw * NTF + c) * Nfp;
      });
    else
      for (int pass = 0; pass < (DIM == 3 ? 2 : 1); ++pass)
      {
        for (int w = t; w < nfine * NTF * ROWS; w += NT)
        {
          const int fw = flist[w / (NTF * ROWS)], r = w % (NTF * ROWS);
          const int hp = (desc[fw].y >> 8) & 7;
          const int c = r / ROWS, line = r % ROWS;
          double *x = pt + (fw * NTF + c) * Nfp;
          if (pass == 0)
            line_apply<DIM, N, true, false, CT, CT>(dop, (hp - 1) & 1, x, 0, line);
          else
            line_apply<DIM, N, false, false, CT, CT>(dop, (hp - 1) >> 1, x, 0, line);
        }
        __syncthreads();
      }
  }

  // -------------------------------- flux jumps, in place of the traces; the
  // coarse side of hanging faces sums its pieces' projected jumps
  for (int w = t; w < ne * FN; w += NT)
  {
    const int es = w / FN, f = w % FN / Nfp, pn = w % Nfp;
    const DomainView &d = item.view(first + es);
    const int2 ds = desc[es * NF + f];
    const int k = ds.y & 3;
    double *x = pt + (es * NF + f) * NTF * Nfp + pn;
    if (k != 2)
    {
      const double *own = qs + es * Np + gmask<DIM, N>(f, pn);
      CT dq[NTF], J[6];
      const bool free_surface = k == 3 && ((ds.y >> 2) & 3) == 0;
#pragma unroll
      for (int c = 0; c < NTF; ++c)
      {
        const double qm = own[trace_field<DIM>(f >> 1, c) * NV];
        const double qp = k != 3 ? x[c * Nfp]
                                 : (free_surface ? (c < DIM ? qm : -qm) : 0.0);
        dq[c] = CT(qp - qm);
      }
      const CT sg = (f & 1) ? CT(1) : CT(-1);
      flux_jumps<DIM, CT>(dq, f >> 1, sg, CT(ed[es].Zp), CT(ed[es].Zs),
                          fcf + 4 * (es * NF + f), sp.flux, J);
      const int at = HANGS ? fidx[es * NF + f] : -1;
      if (at >= 0)
      {
        double *o = mj + at * NJ * Nfp + pn;
#pragma unroll
        for (int c = 0; c < NJ; ++c)
        {
          const int sl = jslot<DIM>(c);
          const CT v = sl < 3 ? sg * dq[DIM + sl] - J[sl] : J[sl] - dq[sl - 3];
          o[c * Nfp] = double(v);
        }
      }
#pragma unroll
      for (int c = 0; c < NJ; ++c)
        put_jump<CT>(x + c * Nfp, J[jslot<DIM>(c)]);
    }
    else if (MODE != MODE_STAGE_NC && HANGS)
    {
      const double *mb = d.mbuf + (size_t)ds.x * NJ * Nfp + pn;
#pragma unroll
      for (int c = 0; c < NJ; ++c)
      {
        double sum = 0;
#pragma unroll
        for (int p = 0; p < NPC; ++p)
          sum += mb[(p * NJ + c) * Nfp];
        put_jump<CT>(x + c * Nfp, CT(sum));
      }
    }
  }

  // ------------- fine side: L2 projection of the coarse side's jumps (FP64)
  if (nfine)
  {
    __syncthreads();
    if constexpr (K::VALUES)
      line_values<N, double, NJ, NT, K::E * DIM>(sP, nfine, t, [&](int l, int c, int &top) {
        top = (((desc[flist[l]].y >> 8) & 7) - 1) & 1;
        return mj + (l * NJ + c) * Nfp;
      });
    else
      for (int pass = 0; pass < (DIM == 3 ? 2 : 1); ++pass)
      {
        for (int w = t; w < nfine * NJ * ROWS; w += NT)
        {
          const int fw = flist[w / (NJ * ROWS)];
          const int hp = (desc[fw].y >> 8) & 7;
          const int g = w / ROWS, line = w % ROWS;
          if (pass == 0)
            line_apply<DIM, N, true, true, double, CT>(dop, (hp - 1) & 1,
                                                       mj + g * Nfp, 0, line);
          else
            line_apply<DIM, N, false, true, double, CT>(dop, (hp - 1) >> 1,
                                                        mj + g * Nfp, 0, line);
        }
        __syncthreads();
      }
    for (int w = t; w < nfine * NJ * Nfp; w += NT)
    {
      const int fw = flist[w / (NJ * Nfp)];
      const int es = fw / NF;
      const DomainView &d = item.view(first + es);
      d.mbuf[(size_t)d.fslot[(size_t)elem[es] * NF + fw % NF] * NJ * Nfp +
             w % (NJ * Nfp)] = mj[w];
    }
  }
  __syncthreads();
  grid_launch_dependents(); // as in dg_stage.cuh, not earlier
  if (!mine)
    return;

  // ------------------------------ volume, face contributions and the update
  const double a = MODE != MODE_RHS ? sp.A : 0.0;
  const double s = MODE != MODE_RHS ? md.dt : 1.0;
  const ElemData &me = ed[ms];
  const int i = mn % Nq, j = (mn / Nq) % Nq, k = mn / (Nq * Nq);
  CT rv[NFLD];
  volume_node<DIM, N, CT>([&](int c) { return qv + c * NV + ms * Np; }, sD, dop,
                          me, s, i, j, k, rv);
#pragma unroll
  for (int ax = 0; ax < DIM; ++ax)
  {
    const int idx = ax == 0 ? i : (ax == 1 ? j : k);
    if (idx != 0 && idx != N)
      continue;
    const int side = idx == N;
    const int pn = DIM == 3 ? (ax == 0 ? j + Nq * k
                                       : (ax == 1 ? i + Nq * k : i + Nq * j))
                            : (ax == 0 ? j : i);
    const double *x = pt + (ms * NF + 2 * ax + side) * NTF * Nfp + pn;
    CT J[6] = {0, 0, 0, 0, 0, 0}, lc[NFLD];
#pragma unroll
    for (int c = 0; c < NJ; ++c)
      J[jslot<DIM>(c)] = get_jump<CT>(x + c * Nfp);
    const CT lfac =
        CT(s * (ax == 0 ? me.rx : (ax == 1 ? me.ry : me.rz)) * dop.iwend);
    lift_face<DIM, CT>(J, ax, side ? CT(1) : CT(-1), lfac, me, lc);
#pragma unroll
    for (int c = 0; c < NFLD; ++c)
      rv[c] += lc[c];
  }
  double acc[NFLD];
#pragma unroll
  for (int c = 0; c < NFLD; ++c)
    acc[c] = double(rv[c]);
  // point source on the velocity: s f(t_stage) F phi_n(x_s) / (rho w_n J)
  if (me_ == md.src.elem)
  {
    const double ts = md.clock->time + sp.C * md.dt;
    const double g =
        s * ricker(ts, md.src.f0, md.src.t0) * md.src.w[mn] * me.irho;
#pragma unroll
    for (int c = 0; c < DIM; ++c)
      acc[c] += g * md.src.force[c];
  }
  if constexpr (MODE != MODE_RHS)
  {
#pragma unroll
    for (int c = 0; c < NFLD; ++c)
    {
      if (rd)
        acc[c] += a * qd[c];
      // streaming stores, as in dg_stage.cuh
      __stcs(md.dq + c * md.fs + mat, acc[c]);
      __stcs(md.qout + c * md.fs + mat, qs[c * NV + t] + sp.B * acc[c]);
    }
  }
  else
  {
#pragma unroll
    for (int c = 0; c < NFLD; ++c)
      md.rhs[c * md.fs + mat] = acc[c];
  }
}

// one domain: CTA b takes the work items from b sp.per on
template <int DIM, int N, int MODE, typename CT>
__global__ void __launch_bounds__(PackShape<DIM, N, CT>::NT,
                                  PackShape<DIM, N, CT>::MINB)
    dg_pack_kernel(DomainView d, int n, StageParams sp,
                   const __grid_constant__ DiffOp<N, CT> dop)
{
  pack_elements<DIM, N, MODE, CT>(SingleItems{d}, n, sp, dop);
}

// many domains: work[idx] = (domain, element)
template <int DIM, int N, int MODE, typename CT>
__global__ void __launch_bounds__(PackShape<DIM, N, CT>::NT,
                                  PackShape<DIM, N, CT>::MINB)
    dg_pack_batch_kernel(const DomainView *__restrict__ views,
                         const int2 *__restrict__ work, int n, StageParams sp,
                         const __grid_constant__ DiffOp<N, CT> dop)
{
  pack_elements<DIM, N, MODE, CT>(BatchItems{views, work}, n, sp, dop);
}

} // namespace bfam_b200
