// Fused DG stage kernel for the isotropic velocity-stress elastic system on
// affine Cartesian elements (sm_100a).
//
// One element per CTA iteration does:
//   issue   : every global read of the element is issued up front -- its own
//             q (and dq, where the shape stages it) and its faces' flux
//             constants by TMA bulk copies into
//             shared memory, the neighbours' face traces by 8-byte cp.async
//             gathers straight into shared memory, addressed from a
//             per-face descriptor.  This is the
//             on-device replacement of vmapP and of the bfam_communicator
//             ghost exchange (src/bfam.c:6783-6877, 2418-2679).  Only the six
//             trace fields the flux uses are gathered (velocity and the stress
//             row of the face normal);
//   face    : upwind flux on the gathered traces (conforming faces and the
//             fine side of hanging faces): six jumps per face node, stored
//             in place of its trace;
//   mortar  : faces that go through the glue grid (2:1 hanging faces,
//             src/bfam.c:7328-7520).  The fine element interpolates the coarse
//             neighbour's trace to its mortar piece (interpolation[1..2]) and
//             evaluates the flux there; from the same Riemann solution it
//             forms the coarse side's jumps on the piece, L2-projects them to
//             the coarse face (projection[1..2]) and stores them in a mortar
//             buffer slot.  The coarse element, launched after its fine
//             neighbours (elements are launched by level), sums its pieces'
//             projected jumps;
//   volume  : one thread per node, the tensor-product LGL derivative along each
//             axis (the BFAM_KRON_IXIXA / IXAXI / AXIXI contractions of
//             src/bfam.c:3519-3624 at one node), plus the jumps of the faces
//             the node lies on, lifted with the lumped LGL mass;
//   update  : the 2N-storage LSRK stage dq = A dq + dt rhs, q' = q + B dq
//             (bfamo_lsrk_t, src/bfam.h:1840-1846) in FP64, writing the new
//             state to the other state buffer so that every element's
//             neighbours read the stage input unchanged.
//
// Template parameters: NT threads per CTA and MINB CTAs per SM targeted by the
// register allocation (the tile shape chosen per order), MODE (stage update or
// right-hand side only) and CT, the arithmetic of the right-hand side (double
// for the plain form; float for the precision form, where the volume
// derivative, flux, lift and mortar interpolation run in FP32 while the state,
// dq, the mortar L2 projection and the update stay FP64; the face jumps and
// lifts stay FP32 until one widening per field).
//
// State layout in HBM: field-major, element, node (bfam's per-field arrays
// stacked): q[f * K * Np + e * Np + n], n = i + Nq (j + Nq k).
#pragma once

#include "dg_common.cuh"
#include "dg_dmma.cuh"
#include "dg_volume.cuh"

namespace bfam_b200
{

// index of the i-th set bit of m
__device__ __forceinline__ int nth_bit(int m, int i)
{
  for (; i > 0; --i)
    m &= m - 1;
  return __ffs(m) - 1;
}

// Two passes over face arrays of LINES lines each, arrays shared out to the
// warps of a (sub-)element of NT threads (wid: this warp's turn), a thread per
// line: the second pass of an array follows the first in the same warp, without
// the other warps
template <int LINES, int NT, typename First, typename Second>
__device__ __forceinline__ void for_arrays(int wid, int arrays,
                                           const First &first,
                                           const Second &second)
{
  constexpr int PER = 32 / LINES; // arrays per warp
  const int lane = threadIdx.x & 31;
  for (int a0 = wid * PER; a0 < arrays; a0 += NT / 32 * PER)
  {
    const int a = a0 + lane / LINES, line = lane % LINES;
    const bool mine = lane < PER * LINES && a < arrays;
    if (mine)
      first(a, line);
    __syncwarp();
    if (mine)
      second(a, line);
    __syncwarp();
  }
}

// The mode of a launch over a mesh without hanging faces: compiled without the
// mortar passes (N = 3 157 -> 161 and 162 -> 166 G DOF-updates/s in the two
// forms, N = 4 137 -> 140 and 154 -> 158; the packed kernel's 2D N = 5 138 -> 143), but for two
// shapes that ran slower so (the plain form at N = 5 spills: 158 against 162;
// the precision form at 2D N = 7: 171 against 174)
template <int DIM, int N, typename CT>
__host__ __device__ constexpr int conforming_mode()
{
  return (DIM == 3 && N == 5 && sizeof(CT) == sizeof(double)) ||
                 (DIM == 2 && N == 7 && sizeof(CT) < sizeof(double))
             ? MODE_STAGE_NC
             : MODE_STAGE_CF;
}

// Shapes (the precision form in 3D) whose mortar passes stay within a warp: the
// interpolation's two passes over an array by the same warp (for_arrays, one
// barrier instead of two), and the L2 projection (FP64) on the matrix
// instruction, a warp per pair of face fields (mortar_pair), without barriers
// and after the node pass.  A thread per line between CTA barriers took 3,700
// and 3,000 of the 20,800 cycles of an N = 7 element with two fine faces.
// Refined meshes, G DOF-updates/s before -> with the projection -> with both:
// N = 7 112.7 -> 118.4 -> 121.3, N = 6 112 -> 117 -> 118 (121 with the
// differentiation rows of y and z from the parameter space), N = 5 123 -> 130.1
// -> 130.4, N = 4 117 -> 118.5 -> 119.3 (122 with all rows from there), N = 3
// 115.9 -> 117.0 -> 117.9.  The plain form's kernels here have no registers for
// it (N = 3 114 -> 110, N = 4 107 -> 101).
template <int DIM, int N, typename CT>
__host__ __device__ constexpr bool mma_mortars()
{
  return DIM == 3 && N >= 3 && sizeof(CT) < sizeof(double);
}

// Per cent of a wave of resident CTAs from which a stage does not let the next
// launch's CTAs in before its end; 85: never (as in
// the packed kernel).  The short launches of 2D and of 3D orders up to 3 lose more by waiting than they gain (N = 3, 1,338 elements
// with hanging faces 63.5 -> 65.4 us per step, 2D N = 5, 1,600 22.6 -> 25.1), and
// at N = 7 in the precision form two CTAs per SM leave little to gain (204 with
// hanging faces 96.3 -> 98.9).
// The others' lines lie where the sides meet: N = 5 FP64 conforming 360 elements
// (0.49) 39.5 early and 41.4 late, 400 (0.54) 48.2 and 42.0; N = 5 FP32 256 (0.43)
// 33.5 and 29.2, 360 (0.61) 38.7 and 37.3.
template <int DIM, int N, typename CT> constexpr int late_from()
{
  return DIM == 2 || N <= 3 || N == 7 ? 85 : sizeof(CT) < sizeof(double) ? 42 : 50;
}

// Node of thread t in the volume/update pass.  Nodes go in order (i
// fastest), except in 3D when a k-plane holds between 32 and 64 nodes (N = 5,
// 6): then warp w < Nq takes the first 32 nodes of plane w and the remaining
// warps the rest of every plane, so that the lines along y a warp reads lie
// in one plane (two planes per warp put lines of both at the same shared
// memory banks).  Threads past the last node get Np.
template <int DIM, int N, int NT>
__device__ __forceinline__ int node_of_thread(int t)
{
  constexpr int Nq = N + 1, P = Nq * Nq, Np = DIM == 3 ? P * Nq : P;
  if constexpr (DIM == 3 && P > 32 && P < 64 && NT >= Np)
  {
    if (t < 32 * Nq)
      return (t >> 5) * P + (t & 31);
    const int r = t - 32 * Nq;
    constexpr int REST = P - 32;
    return r < REST * Nq ? (r / REST) * P + 32 + r % REST : Np;
  }
  else
    return t < Np ? t : Np;
}

// A face node's flux jump in its trace slot (one double): stored at the
// precision of the right-hand side (a float in the slot's first four bytes
// in the precision form), so that it is never widened and narrowed again.
template <typename CT> __device__ __forceinline__ void put_jump(double *slot, CT v)
{
  *reinterpret_cast<CT *>(slot) = v;
}
template <typename CT> __device__ __forceinline__ CT get_jump(const double *slot)
{
  return *reinterpret_cast<const CT *>(slot);
}

// Shared-memory layout of one CTA (in doubles, every region 16-byte
// aligned): state, dq where it is staged, face traces / flux jumps, face flux
// constants, the mortar scratch, the differentiation matrix, the mbarriers (q
// and dq) and the precision form's FP32 tile.
template <int DIM, int N, typename CT, bool DQS = true> struct Tile
{
  using S = Shape<DIM, N>;
  // DQS: the element's dq rows are staged in shared memory (TMA); otherwise
  // they are read from global memory by the update, in L2 by the lookahead of
  // an earlier CTA (prefetching them once more with the element's own loads
  // cost 1-2 % at N = 5 and 7)
  static constexpr int BUF =
      S::SM_QS + (DQS ? S::SM_DQ : 0) + S::SM_PT + 4 * S::NF;
  static constexpr int OFF_MJ = BUF;
  static constexpr int OFF_OPS = OFF_MJ + S::SM_MJ;
  static constexpr int OFF_BAR = OFF_OPS + S::SM_IP;
  static constexpr int OFF_QV = OFF_BAR + 2;
  static constexpr bool NARROW = sizeof(CT) < sizeof(double);
  static constexpr int TOTAL = OFF_QV + (NARROW ? S::SM_QF : 0);
  static constexpr size_t BYTES = (size_t)TOTAL * sizeof(double);
};

// the shape's register budget in resident CTAs per SM for arithmetic CT
template <int DIM, int N, typename CT> __host__ __device__ constexpr int shape_minb()
{
  return sizeof(CT) < sizeof(double) ? Shape<DIM, N>::MINB_NARROW
                                     : Shape<DIM, N>::MINB;
}

// CTAs per SM that the shape's register budget and shared memory admit
// (228 KB of shared memory per SM, 1 KB reserved per CTA)
template <int DIM, int N, typename CT, bool DQS = true>
__host__ __device__ constexpr int resident_ctas()
{
  constexpr size_t bytes = Tile<DIM, N, CT, DQS>::BYTES;
  constexpr int by_smem = bytes > 227 * 1024 ? 0 : (int)(233472 / (bytes + 1024));
  constexpr int m = shape_minb<DIM, N, CT>();
  return m < by_smem ? m : by_smem;
}

// dq staged in shared memory (TMA) unless the shape reads it from L2 in the
// update (Shape::DQ_L2 / DQ_L2_NARROW: 3D N=7, and the precision form at
// 3D N=5, where staging measured 9 % slower), or unless leaving it out admits
// more resident CTAs (the plain form at 3D N=5: five CTAs instead of four)
template <int DIM, int N, typename CT> __host__ __device__ constexpr bool stage_dqs()
{
  if (Shape<DIM, N>::DQ_L2 ||
      (Shape<DIM, N>::DQ_L2_NARROW && sizeof(CT) < sizeof(double)))
    return false;
  return resident_ctas<DIM, N, CT, true>() >=
         resident_ctas<DIM, N, CT, false>();
}

// Elements per CTA: a CTA of EPC * NT threads holds EPC sub-elements of NT
// threads, each with its own shared-memory tile (Tile::TOTAL doubles, one
// after the other) and its own barrier -- the CTA's barrier when EPC = 1, the
// warp's when NT = 32, else named barrier 1 + sub -- so that sub-elements
// whose branches differ (fine or coarse faces) never wait for each other.
template <int NT, int EPC> struct Sub
{
  static_assert(EPC >= 1 && (EPC == 1 || NT == 32 || EPC <= 15),
                "named barriers 1..15");
  static_assert(NT % 32 == 0, "whole warps per sub-element");
  __device__ __forceinline__ static int t()
  {
    return EPC == 1 ? (int)threadIdx.x : (int)threadIdx.x % NT;
  }
  __device__ __forceinline__ static int id()
  {
    return EPC == 1 ? 0 : (int)threadIdx.x / NT;
  }
  __device__ __forceinline__ static void sync()
  {
    if constexpr (EPC == 1)
      __syncthreads();
    else if constexpr (NT == 32)
      __syncwarp();
    else
      asm volatile("bar.sync %0, %1;" ::"r"(1 + id()), "n"(NT) : "memory");
  }
};

// shared-memory tile of this thread's sub-element
template <typename T, int NT, int EPC>
__device__ __forceinline__ double *sub_smem()
{
  extern __shared__ __align__(16) double smem[];
  return EPC == 1 ? smem : smem + Sub<NT, EPC>::id() * T::TOTAL;
}

// The element's buffer in the tile.
template <int DIM, int N, typename CT, int NT = 32, int EPC = 1>
struct TileBuf
{
  double *qs, *R, *pt, *fcf;
  uint64_t *bq, *bdq;
  __device__ __forceinline__ TileBuf()
  {
    using S = Shape<DIM, N>;
    constexpr bool DQS = stage_dqs<DIM, N, CT>();
    using T = Tile<DIM, N, CT, DQS>;
    double *smem = sub_smem<T, NT, EPC>();
    qs = smem;
    R = qs + S::SM_QS;
    pt = R + (DQS ? S::SM_DQ : 0);
    fcf = pt + S::SM_PT;
    bq = reinterpret_cast<uint64_t *>(smem + T::OFF_BAR);
    bdq = bq + 1;
  }
};

// Issue every global read of element e: q and (after the first stage, where it
// is staged) dq by TMA bulk copies completing on the mbarriers, the
// neighbours' face traces by cp.async, as one commit group.  ds0: descriptor
// of the face of thread t's first face node.
template <int DIM, int N, int NT, int MODE, typename CT, int EPC = 1>
__device__ __forceinline__ void issue_element(const DomainView &d,
                                              const StageParams &sp, int e,
                                              int2 ds0)
{
  using S = Shape<DIM, N>;
  constexpr int Np = S::Np, Nfp = S::Nfp, NF = S::NF, NFLD = S::NFLD,
                NTF = S::NTF, PITCH = S::PITCH;
  const TileBuf<DIM, N, CT, NT, EPC> tb;
  double *qs = tb.qs, *R = tb.R, *pt = tb.pt, *fcf = tb.fcf;
  uint64_t *bar_q = tb.bq, *bar_dq = tb.bdq;
  const int t = Sub<NT, EPC>::t();
  const size_t fs = d.fs;
  const size_t eoff = (size_t)e * Np;
  const bool rd = MODE != MODE_RHS && !sp.first_stage;
  const int2 *desc = d.fdesc + (size_t)e * NF;
  if (t == 0)
  {
    const RowShift<Np> sh(d.K, e);
    // row c of `src` to its slot; the last row of an odd-sized array has no
    // value after it to copy, and its own last one goes by itself
    const bool last = Np % 2 && e == d.K - 1 && (d.K & 1);
    auto rows = [&](double *dst, const double *src, uint64_t *bar, int more) {
      if (last)
        dst[(NFLD - 1) * PITCH + Np - 1] = src[(NFLD - 1) * fs + eoff + Np - 1];
      mbar_expect_tx(bar, (NFLD * PITCH - (last ? 2 : 0) + more) * sizeof(double));
#pragma unroll
      for (int c = 0; c < NFLD; ++c)
        bulk_g2s(dst + c * PITCH, src + c * fs + eoff - sh(c),
                 (PITCH - (last && c == NFLD - 1 ? 2 : 0)) * sizeof(double), bar);
    };
    fence_proxy_async(); // the copies complete on barriers set up just now
    // the face flux constants with the state, so that no thread needs
    // another thread's copies before the face phase
    rows(qs, d.qin, bar_q, 4 * NF);
    bulk_g2s(fcf, d.fcE + (size_t)e * NF, NF * sizeof(double4), bar_q);
    if constexpr (stage_dqs<DIM, N, CT>())
    {
      if (rd)
        rows(R, d.dq, bar_dq, 0);
    }
  }

  // neighbour traces of conforming faces and coarse partners of fine-side
  // glue faces, gathered into pt in this element's face-node order
  for (int w = t; w < NF * Nfp; w += NT)
  {
    const int f = w / Nfp, pn = w % Nfp;
    const int2 ds = NF * Nfp <= NT || w == t ? ds0 : desc[f];
    const int k = ds.y & 3;
    if (k == 2)
      continue;
    if (k != 3) // a boundary face's ghost trace comes from the element itself
    {
      // the neighbour's opposite face, nodes in the same order (aligned
      // trees: the host refuses any other pairing or orientation)
      const int src_n = gmask<DIM, N>((ds.y >> 2) & 7, pn);
      const double *src = d.qin + (size_t)ds.x * Np + src_n;
#pragma unroll
      for (int c = 0; c < NTF; ++c)
      {
        const int g = f * NTF + c;
        cp_async8(pt + g * Nfp + fpos<DIM, N>(g, pn),
                  src + trace_field<DIM>(f >> 1, c) * fs);
      }
    }
  }
  cp_async_commit(); // the face traces

}

// L2 prefetch of everything issue_element will read of element e itself
// (state rows, dq rows after the first stage, face descriptors, element
// data, flux constants); one thread, no completion to wait for.
template <int DIM, int N, int MODE>
__device__ __forceinline__ void prefetch_element(const DomainView &d,
                                                 const StageParams &sp, int e)
{
  using S = Shape<DIM, N>;
  {
    constexpr int Np = S::Np, NF = S::NF, NFLD = S::NFLD;
    const size_t eoff = (size_t)e * Np;
    const RowShift<Np> sh(d.K, e);
    // the 16-byte aligned part of each row, never past its end
    auto rows = [&](const double *src) {
#pragma unroll
      for (int c = 0; c < NFLD; ++c)
        bulk_prefetch_l2(src + c * d.fs + eoff - sh(c),
                         (Np % 2 ? Np - 1 + 2 * sh(c) : Np) * sizeof(double));
    };
    rows(d.qin);
    if (MODE != MODE_RHS && !sp.first_stage)
      rows(d.dq);
    bulk_prefetch_l2(d.fdesc + (size_t)e * NF, NF * sizeof(int2));
    bulk_prefetch_l2(d.ed + e, sizeof(ElemData));
    bulk_prefetch_l2(d.fcE + (size_t)e * NF, NF * sizeof(double4));
    if constexpr (MODE != MODE_STAGE_NC && MODE != MODE_STAGE_CF)
    {
      // the mortar slots of its coarse faces (written by an earlier launch)
      constexpr int NJ = S::NJ, Nfp = S::Nfp, NPC = S::NPC;
#pragma unroll 1
      for (int f = 0; f < NF; ++f)
      {
        const int2 ds = d.fdesc[(size_t)e * NF + f];
        if ((ds.y & 3) == 2)
          bulk_prefetch_l2(d.mbuf + (size_t)ds.x * NJ * Nfp,
                           NPC * NJ * Nfp * sizeof(double));
      }
    }
  }
}

// Compute element e, its loads issued by issue_element.
template <int DIM, int N, int NT, int MODE, typename CT, int EPC = 1>
__device__ __forceinline__ void compute_element(const DomainView &d,
                                                const StageParams &sp,
                                                const DiffOp<N, CT> &dop,
                                                int e)
{
  using S = Shape<DIM, N>;
  using T = Tile<DIM, N, CT, stage_dqs<DIM, N, CT>()>;
  constexpr int Nq = S::Nq, Np = S::Np, Nfp = S::Nfp, NF = S::NF,
                NFLD = S::NFLD, NJ = S::NJ, NPC = S::NPC, ROWS = S::ROWS,
                NTF = S::NTF, PITCH = S::PITCH;
  // this sub-element's tile, derived from the dynamic shared array itself
  // (not a pointer parameter), so that all accesses stay in the shared
  // window with 32-bit addressing
  double *smem = sub_smem<T, NT, EPC>();
  const TileBuf<DIM, N, CT, NT, EPC> tb;
  double *qs = tb.qs, *pt = tb.pt, *fcf = tb.fcf;
  uint64_t *bar_q = tb.bq, *bar_dq = tb.bdq;
  // field rows of the state and of dq
  const RowShift<Np> sh(d.K, e);
  auto row = [&](int c) { return qs + c * PITCH + sh(c); };
  auto dq_row = [&](int c) { return tb.R + c * PITCH + sh(c); };
  double *mj = smem + T::OFF_MJ; // [DIM][NJ][Nfp] coarse-side jumps, by fine rank
  const CT *sD = reinterpret_cast<const CT *>(smem + T::OFF_OPS); // D
  // the volume pass's copy of q: q itself in the plain form; in the
  // precision form FP32 q minus the element's first node per field (the
  // derivative of a constant is zero), so that rounding is relative to the
  // variation inside the element
  constexpr bool NARROW = T::NARROW;
  CT *qv = nullptr;
  if constexpr (NARROW)
    qv = reinterpret_cast<CT *>(smem + T::OFF_QV);

  const int t = Sub<NT, EPC>::t();
  const size_t fs = d.fs;
  const size_t eoff = (size_t)e * Np;
  // the update is dq = a dq + s rhs; the right-hand-side mode uses a = 0, s = 1
  const bool rd = MODE != MODE_RHS && !sp.first_stage;
  const double a = MODE != MODE_RHS ? sp.A : 0.0;
  const double s = MODE != MODE_RHS ? d.dt : 1.0;
  const ElemData me = d.ed[e];
  const int2 *desc = d.fdesc + (size_t)e * NF;

  constexpr bool HANGS = MODE != MODE_STAGE_CF; // any hanging face
  constexpr bool NO_COARSE = MODE == MODE_STAGE_NC || !HANGS;
  int coarse_mask = 0, fine_mask = 0, pieces = 0; // 3 bits a face
#pragma unroll
  for (int f = 0; HANGS && f < NF; ++f)
  {
    const int y = desc[f].y;
    coarse_mask |= ((y & 3) == 2) << f;
    if ((y & 3) == 1 && ((y >> 8) & 7) != 0)
    {
      fine_mask |= 1 << f;
      pieces |= ((y >> 8) & 7) << (3 * f);
    }
  }
  const int ncoarse = HANGS ? __popc(coarse_mask) : 0,
            nfine = HANGS ? __popc(fine_mask) : 0;

  // ------------------------------------------------- phase 1: faces, mortars
  if (!mbar_wait(bar_q, 0))
    atomicExch(d.err, 1);
  cp_async_wait<0>();
  if constexpr (NARROW)
  {
    for (int n = t; n < Np; n += NT)
    {
#pragma unroll
      for (int c = 0; c < NFLD; ++c)
        qv[c * Np + n] = CT(row(c)[n] - row(c)[0]);
    }
  }
  // The state and flux constants come by TMA, and a thread's face pass reads
  // only its own gathered trace slots (its own cp.async group), so only the
  // fine-side interpolation, which reads whole lines, needs the barrier.
  if (HANGS && nfine)
    Sub<NT, EPC>::sync();
  // lift factor of face axis ax: s (2/h_ax) / w_0
  CT lfac[3];
#pragma unroll
  for (int ax = 0; ax < 3; ++ax)
    lfac[ax] =
        CT(s * (ax == 0 ? me.rx : (ax == 1 ? me.ry : me.rz)) * dop.iwend);

  // fine side: coarse partner trace -> my piece, in place (rows, then columns)
  constexpr bool MMA = mma_mortars<DIM, N, CT>();
  constexpr int NW = NT / 32;
  const int wid = t >> 5;
  if (nfine)
  {
    if constexpr (MMA)
    {
      // an array's rows, then its columns, by the same warp
      for_arrays<Nq, NT>(wid, nfine * NTF, [&](int a, int line) {
        const int f = nth_bit(fine_mask, a / NTF), g = f * NTF + a % NTF;
        const int hp = (pieces >> (3 * f)) & 7;
        line_apply<DIM, N, true, false, CT, CT>(dop, (hp - 1) & 1, pt + g * Nfp,
                                                g, line);
      }, [&](int a, int line) {
        const int f = nth_bit(fine_mask, a / NTF), g = f * NTF + a % NTF;
        const int hp = (pieces >> (3 * f)) & 7;
        line_apply<DIM, N, false, false, CT, CT>(dop, (hp - 1) >> 1,
                                                 pt + g * Nfp, g, line);
      });
      Sub<NT, EPC>::sync();
    }
    else
      for (int pass = 0; pass < (DIM == 3 ? 2 : 1); ++pass)
      {
        for (int w = t; w < nfine * NTF * ROWS; w += NT)
        {
          const int f = nth_bit(fine_mask, w / (NTF * ROWS)),
                    r = w % (NTF * ROWS);
          const int hp = (pieces >> (3 * f)) & 7;
          const int c = r / ROWS, line = r % ROWS;
          const int half = pass == 0 ? (hp - 1) & 1 : (hp - 1) >> 1;
          const int g = f * NTF + c;
          if (pass == 0)
            line_apply<DIM, N, true, false, CT, CT>(dop, half, pt + g * Nfp, g, line);
          else
            line_apply<DIM, N, false, false, CT, CT>(dop, half, pt + g * Nfp, g, line);
        }
        Sub<NT, EPC>::sync();
      }
  }

  // flux on conforming and fine-side faces: the face node's jumps (T* - T-,
  // v* - v-), written in place over the node's own trace slots (a thread
  // reads only its own node's slots: partners' face nodes are in the same
  // order on aligned trees) and lifted by the node pass.  On a fine face
  // the coarse side's jumps follow from the same Riemann solution (star
  // state v*, S* n shared by both sides, coarse normal -n):
  //   coarse (T* - T-) = -(fine J_T) + [T],  coarse (v* - v-) = fine J_v - [v]
  // with [.] = coarse - fine as seen from the fine side; they go to mj in the
  // coarse piece's node order.
  for (int w = t; w < NF * Nfp; w += NT)
  {
    {
      const int f = w / Nfp, pn = w % Nfp;
      const int y = desc[f].y;
      const int k = y & 3;
      if (k != 2)
      {
        const int vm = gmask<DIM, N>(f, pn);
        const int pp = pn;
        CT dq[NTF], J[6];
        // boundary faces: ghost state v+ = v-, S+ = -S- (free surface) or
        // q+ = 0 (absorbing)
        const bool free_surface = k == 3 && ((y >> 2) & 3) == 0;
#pragma unroll
        for (int c = 0; c < NTF; ++c)
        {
          const double qm = row(trace_field<DIM>(f >> 1, c))[vm];
          const int g = f * NTF + c;
          const double qp = k != 3 ? pt[g * Nfp + fpos<DIM, N>(g, pp)]
                                   : (free_surface ? (c < DIM ? qm : -qm) : 0.0);
          dq[c] = CT(qp - qm);
        }
        const CT sg = (f & 1) ? CT(1) : CT(-1);
        flux_jumps<DIM, CT>(dq, f >> 1, sg, CT(me.Zp), CT(me.Zs),
                            fcf + 4 * f, sp.flux, J);
        if (HANGS && ((fine_mask >> f) & 1))
        {
          // rank of f among the fine faces (an element has at most DIM)
          const int fr = __popc(fine_mask & ((1 << f) - 1));
#pragma unroll
          for (int c = 0; c < NJ; ++c)
          {
            const int sl = jslot<DIM>(c);
            const CT v = sl < 3 ? sg * dq[DIM + sl] - J[sl] : J[sl] - dq[sl - 3];
            const int g = fr * NJ + c;
            mj[g * Nfp + fpos<DIM, N>(g, pp)] = double(v);
          }
        }
#pragma unroll
        for (int c = 0; c < NJ; ++c)
        {
          const int g = f * NTF + c;
          put_jump<CT>(pt + g * Nfp + fpos<DIM, N>(g, pp), J[jslot<DIM>(c)]);
        }
      }
    }
  }

  // coarse side: the pieces' projected jumps, summed in glue order (stored
  // at the precision of the right-hand side, like the flux jumps)
  for (int w = t; !NO_COARSE && w < ncoarse * Nfp; w += NT)
  {
    const int f = nth_bit(coarse_mask, w / Nfp), pn = w % Nfp;
    const double *mb = d.mbuf + (size_t)desc[f].x * NJ * Nfp + pn;
#pragma unroll
    for (int c = 0; c < NJ; ++c)
    {
      double sum = 0;
#pragma unroll
      for (int p = 0; p < NPC; ++p)
        sum += mb[(p * NJ + c) * Nfp];
      const int g = f * NTF + c;
      put_jump<CT>(pt + g * Nfp + fpos<DIM, N>(g, pn), CT(sum));
    }
  }

  // fine side: L2 projection of the coarse-side jumps to the coarse face
  // (FP64), then out to the mortar buffer for the coarse element (on the
  // matrix instruction: after the node pass)
  if (!MMA && nfine)
  {
    Sub<NT, EPC>::sync();
    for (int w = t; w < nfine * NJ * ROWS; w += NT)
    {
      const int fr = w / (NJ * ROWS), r = w % (NJ * ROWS);
      const int hp = (pieces >> (3 * nth_bit(fine_mask, fr))) & 7;
      const int g = fr * NJ + r / ROWS, line = r % ROWS;
      line_apply<DIM, N, true, true, double, CT>(
          dop, (hp - 1) & 1, mj + g * Nfp, g, line);
    }
    Sub<NT, EPC>::sync();
    if (DIM == 3)
    {
      for (int w = t; w < nfine * NJ * Nq; w += NT)
      {
        const int fr = w / (NJ * Nq), r = w % (NJ * Nq);
        const int hp = (pieces >> (3 * nth_bit(fine_mask, fr))) & 7;
        const int g = fr * NJ + r / Nq, col = r % Nq;
        line_apply<DIM, N, false, true, double, CT>(
            dop, (hp - 1) >> 1, mj + g * Nfp, g, col);
      }
      Sub<NT, EPC>::sync();
    }
    for (int w = t; w < nfine * NJ * Nfp; w += NT)
    {
      const int fr = w / (NJ * Nfp), r = w % (NJ * Nfp);
      const int f = nth_bit(fine_mask, fr), g = fr * NJ + r / Nfp;
      d.mbuf[(size_t)d.fslot[(size_t)e * NF + f] * NJ * Nfp + r] =
          mj[g * Nfp + fpos<DIM, N>(g, r % Nfp)];
    }
  }
  Sub<NT, EPC>::sync();

  // The next launch may start from here (all CTAs past this point): released
  // at the kernel's start instead, its waiting CTAs crowd onto the SMs that
  // drain first (N = 5 on 1,057 elements 133 us per step against 127, 129
  // without the overlap)
  if (late_from<DIM, N, CT>() == 85 || sp.early)
    grid_launch_dependents();
  // ------------------------ phase 2: volume, face contributions and update
  constexpr bool DQS = stage_dqs<DIM, N, CT>();
  if (MODE != MODE_RHS && rd && DQS)
  {
    if (!mbar_wait(bar_dq, 0))
      atomicExch(d.err, 2);
  }
  constexpr int NODE_ITERS = (Np + NT - 1) / NT;
#pragma unroll 1
  for (int it = 0; it < NODE_ITERS; ++it)
  {
    const int n = node_of_thread<DIM, N, NT>(t + it * NT);
    if (n >= Np)
      break;
    const int i = n % Nq, j = (n / Nq) % Nq, k = n / (Nq * Nq);
    // s times the right-hand side in CT: the volume term, then the lifted
    // jumps of the faces this node lies on (at most one per axis, in face
    // order); widened to FP64 once for the update
    CT rv[NFLD];
    if constexpr (NARROW)
      volume_node<DIM, N, CT>([&](int c) { return qv + c * Np; }, sD, dop, me, s,
                              i, j, k, rv);
    else
      volume_node<DIM, N, CT>(row, sD, dop, me, s, i, j, k, rv);
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
      const int g0 = (2 * ax + side) * NTF;
      CT J[6] = {0, 0, 0, 0, 0, 0}, lc[NFLD];
#pragma unroll
      for (int c = 0; c < NJ; ++c)
        J[jslot<DIM>(c)] =
            get_jump<CT>(pt + (g0 + c) * Nfp + fpos<DIM, N>(g0 + c, pn));
      lift_face<DIM, CT>(J, ax, side ? CT(1) : CT(-1), lfac[ax], me, lc);
#pragma unroll
      for (int c = 0; c < NFLD; ++c)
        rv[c] += lc[c];
    }
    double acc[NFLD];
#pragma unroll
    for (int c = 0; c < NFLD; ++c)
      acc[c] = double(rv[c]);

    // point source on the velocity: s f(t_stage) F phi_n(x_s) / (rho w_n J)
    if (e == d.src.elem)
    {
      const double ts = d.clock->time + sp.C * d.dt;
      const double g = s * ricker(ts, d.src.f0, d.src.t0) * d.src.w[n] * me.irho;
#pragma unroll
      for (int c = 0; c < DIM; ++c)
        acc[c] += g * d.src.force[c];
    }

    if constexpr (MODE != MODE_RHS)
    {
      if (rd)
      {
#pragma unroll
        for (int c = 0; c < NFLD; ++c)
          acc[c] += a * (DQS ? dq_row(c)[n] : d.dq[c * fs + eoff + n]);
      }
      // streaming stores: the next stage reads these rows a whole stage
      // later (from DRAM), so they should not push the lines in reuse out
      // of L2 (+0.3-0.8 % at cfg1)
#pragma unroll
      for (int c = 0; c < NFLD; ++c)
      {
        __stcs(d.dq + c * fs + eoff + n, acc[c]);
        __stcs(d.qout + c * fs + eoff + n, row(c)[n] + sp.B * acc[c]);
      }
    }
    else
    {
#pragma unroll
      for (int c = 0; c < NFLD; ++c)
        d.rhs[c * fs + eoff + n] = acc[c];
    }
  }

  // Fine side: L2 projection of the coarse-side jumps to the coarse face
  // (FP64) and their store to the mortar buffer for the coarse element, after
  // the node pass and from the last warp on (at N = 7 the first warps have a
  // second pass of nodes): no other warp waits for it
  if constexpr (HANGS && MMA)
  {
    __syncwarp(); // the matrix instruction takes whole warps
    for (int w = NW - 1 - wid; w < 3 * nfine; w += NW)
    {
      const int fr = w / 3, c = w % 3, f = nth_bit(fine_mask, fr);
      double2 y[2];
      mortar_pair<N>(d.ops, 5, (pieces >> (3 * f)) & 7, mj, fr * NJ + c,
                     fr * NJ + c + 3, y);
      double *out =
          d.mbuf + ((size_t)d.fslot[(size_t)e * NF + f] * NJ + c) * Nfp;
      const int r = (t & 31) >> 2, i0 = 2 * (t & 3);
#pragma unroll
      for (int k = 0; k < 2; ++k)
        put2<Nq % 2 == 0>(out + 3 * k * Nfp + i0 + Nq * r, y[k],
                          r < Nq && i0 < Nq, r < Nq && i0 + 1 < Nq);
    }
  }
}


// The launch's work items: item.view(idx) and item.elem(idx) give item idx's
// domain view and element; a CTA does one item (EPC of them), and the block
// scheduler balances the uneven element costs.
template <int DIM, int N, int NT, int MODE, typename CT, typename Item,
          int EPC = 1>
__device__ __forceinline__ void stage_loop(const Item &item, int n,
                                           const StageParams &sp,
                                           const DiffOp<N, CT> &dop)
{
  using T = Tile<DIM, N, CT, stage_dqs<DIM, N, CT>()>;
  using SB = Sub<NT, EPC>;
  constexpr int Nq = N + 1;
  double *smem = sub_smem<T, NT, EPC>();
  const int lt = SB::t();
  if (lt == 0)
  {
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + T::OFF_BAR);
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
  }
  // the differentiation matrix into shared memory (rows indexed per
  // thread in the volume pass; the mortar operators are read from the
  // parameter bank at unrolled indices)
  {
    CT *sD = reinterpret_cast<CT *>(smem + T::OFF_OPS);
    for (int w = lt; w < Nq * Nq; w += NT)
      sD[w] = dop.D[w];
  }
  SB::sync();
  // one element per sub-element (the grid covers every item)
  const int idx = (int)blockIdx.x * EPC + SB::id();
  if (idx >= n)
    return;
  // the tables are constant: the element and the descriptor of this thread's
  // first face node are read while the launch before still runs (two trips to
  // memory per launch: 3D N = 3 on 211 elements 48.3 -> 44.2 us per step, N = 7
  // 99 -> 94; refined 30 M DOF meshes +1 %)
  constexpr int NF = Shape<DIM, N>::NF, Nfp = Shape<DIM, N>::Nfp;
  const DomainView &d = item.view(idx);
  const int e = item.elem(idx), f0 = lt / Nfp;
  const int2 ds0 = d.fdesc[(size_t)e * NF + (f0 < NF ? f0 : NF - 1)];
  grid_dependency_wait(); // the stage input is complete
  issue_element<DIM, N, NT, MODE, CT, EPC>(d, sp, e, ds0);
  // a thread of another warp than the TMA issuer prefetches a later
  // item's element while this one's loads fly
  const int ia = idx + sp.ahead;
  if (sp.ahead > 0 && ia < n && lt == (NT > 32 ? 32 : 0))
    prefetch_element<DIM, N, MODE>(item.view(ia), sp, item.elem(ia));
  compute_element<DIM, N, NT, MODE, CT, EPC>(d, sp, dop, e);
}

// one domain: item idx is element idx, or the idx-th of an element list
struct SingleItems
{
  const DomainView &d;
  __device__ __forceinline__ const DomainView &view(int) const { return d; }
  __device__ __forceinline__ int elem(int idx) const
  {
    return d.elist ? d.elist[idx] : idx;
  }
  // the item's own entry into L2
  __device__ __forceinline__ void prefetch(int idx) const
  {
    if (d.elist)
      prefetch_l2(d.elist + idx);
  }
};

// many domains: item idx is work[idx] = (domain, element)
struct BatchItems
{
  const DomainView *__restrict__ views;
  const int2 *__restrict__ work;
  __device__ __forceinline__ const DomainView &view(int idx) const
  {
    return views[work[idx].x];
  }
  __device__ __forceinline__ int elem(int idx) const { return work[idx].y; }
  __device__ __forceinline__ void prefetch(int idx) const
  {
    prefetch_l2(work + idx);
  }
};

// One domain: item idx is element idx, or the idx-th of the launch's
// element list (meshes with hanging faces launch their elements by level).
template <int DIM, int N, int NT, int MINB, int MODE, typename CT>
__global__ void __launch_bounds__(NT, MINB)
    dg_stage_kernel(DomainView d, int n, StageParams sp,
                    const __grid_constant__ DiffOp<N, CT> dop)
{
  stage_loop<DIM, N, NT, MODE, CT>(SingleItems{d}, n, sp, dop);
}

// Many domains of the same order: item idx is work[idx] = (domain, element),
// each domain with its own arrays and time step.  EPC elements per CTA of
// EPC * NT threads.
template <int DIM, int N, int NT, int MINB, int MODE, typename CT,
          int EPC = 1>
__global__ void __launch_bounds__(NT *EPC, MINB)
    dg_stage_batch_kernel(const DomainView *__restrict__ views,
                          const int2 *__restrict__ work, int nwork,
                          StageParams sp,
                          const __grid_constant__ DiffOp<N, CT> dop)
{
  stage_loop<DIM, N, NT, MODE, CT, BatchItems, EPC>(
      BatchItems{views, work}, nwork, sp, dop);
}

// dynamic shared memory of one CTA of the stage kernels (EPC sub-elements)
template <int DIM, int N, typename CT, int EPC = 1>
__host__ __device__ constexpr size_t stage_smem_bytes()
{
  return EPC * Tile<DIM, N, CT, stage_dqs<DIM, N, CT>()>::BYTES;
}

// resident CTAs per SM the register budget is sized for: the shape's choice,
// capped by what the shared memory allows (228 KB per SM, 1 KB reserved per
// CTA)
template <int DIM, int N, typename CT>
__host__ __device__ constexpr int stage_min_ctas()
{
  constexpr int by_smem = (int)(233472 / (stage_smem_bytes<DIM, N, CT>() + 1024));
  constexpr int m = shape_minb<DIM, N, CT>() < by_smem ? shape_minb<DIM, N, CT>() : by_smem;
  return m < 1 ? 1 : m;
}

} // namespace bfam_b200
