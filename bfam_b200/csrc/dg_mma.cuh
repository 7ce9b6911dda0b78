// Stage kernel of the plain (FP64) form for 3D orders 5 to 7: the fused
// element update of dg_stage.cuh with its small dense operators on the FP64
// matrix instruction (mma.sync m8n8k4, the only tensor-core form of FP64).
//
// Every operator of the element is a matrix of at most 8 x 8 applied along
// the lines of a plane or a face, so one warp holds one plane (or one face)
// as an 8 x 8 matrix in the instruction's accumulator layout,
//   lane 4 r + c holds X[r][2 c], X[r][2 c + 1]            ("C layout"),
// rows the plane's second axis, columns its first; past N lanes repeat the
// last row or columns, which meet zeros in the operators' fragments or land
// where nothing is stored.  The order of the contracted index is free as long as both
// operands agree on it, so with kstep s taking the indices 2 c + s
//   X D^T     takes the C layout of X as its left operand unchanged, and
//   Op X^T    takes the C layout of X as its right operand unchanged;
// a tensor product Op_b X Op_a^T is Op_b (Op_a X^T)^T: two such products,
// with no data movement in between.
//
// Per element, one CTA of Nq warps:
//   issue : the state by TMA bulk copies into shared memory; warp f loads
//           face f's neighbour trace (or the coarse side's projected jumps)
//           from global memory straight into registers, in C layout;
//   z     : warp j derives its plane j = const along z (rows k) and leaves
//           the six derivatives in shared memory, since z lines cross the
//           planes k = const that the update works on;
//   face  : warp f computes face f: interpolation of a coarse trace to the
//           mortar piece, the upwind flux, the projection of the coarse
//           side's jumps and their store to the mortar buffer, all in its
//           registers; the flux jumps go to shared memory, scaled by the
//           lift so that they add to the derivative along the face's axis;
//   update: warp k derives plane k along x and y, adds the z derivatives and
//           the face corrections and does the LSRK update with 16-byte
//           accesses (8-byte ones where Nq is odd).
// Two CTA barriers per element (after the barrier set-up and before the
// update) instead of up to eight.
//
// What bounded the node-per-thread kernel here was shared memory: at N = 7 it
// read 18 lines of 8 values per node (LSU pipe 61 % busy, DRAM 32 %), and at
// N = 6 one CTA of 11 warps filled an SM's registers.  In C layout a plane's
// x derivative reads each value once and its y and z derivatives twice
// (8,100 warp instructions per N = 7 element instead of 19,300).  Measured
// on 29-32 M DOF bricks, G DOF-updates/s before -> now, conforming and with
// 30 % of the base cells refined: N = 7 131.9 -> 180 and 105.5 -> 155, N = 6
// 75.0 -> 130 and 58.9 -> 114; N = 5 with hanging faces 122 -> 127 (on 197 M
// DOFs 116 -> 125).  Lower orders and conforming N = 5 keep the
// node-per-thread kernel: their planes leave too much of an 8 x 8 matrix
// empty (N = 4, 25 of 64 entries: 89 against 95 conforming).
// What bounds it now is latency: two CTAs of 8 warps per SM at N = 7 (82 KB
// each), each in turn waiting for its loads (4,700 cycles of 14,000), at 84 %
// and 72 % of the HBM bandwidth.
#pragma once

#include "dg_common.cuh"
#include "dg_dmma.cuh"
#include "dg_stage.cuh"

namespace bfam_b200
{

template <int N> struct MmaShape
{
  static constexpr int Nq = N + 1, P = Nq * Nq, Np = P * Nq;
  static constexpr int NW = Nq, NT = 32 * NW; // >= 6 faces
  // an element's field row in shared memory: rows of an odd number of nodes
  // start on an 8-byte boundary in global memory for every other element,
  // so they are copied from the 16-byte boundary below, one value longer
  // At N = 7 planes are 4 values apart instead of adjacent: their 512 bytes
  // would put a line along z on one pair of banks
  static constexpr int PP = N == 7 ? P + 4 : P;
  static constexpr int PITCH = Nq * PP + Np % 2;
  static constexpr int OFF_Z = 9 * PITCH;
  static constexpr int OFF_J = OFF_Z + 6 * Np + (6 * Np) % 2;
  static constexpr int OFF_FC = OFF_J + 36 * P;
  static constexpr int OFF_BAR = OFF_FC + 32;
  static constexpr size_t BYTES = (OFF_BAR + 2) * sizeof(double);
  static constexpr int MINB = N == 5 ? 5 : N == 6 ? 3 : 2;
};

// Orders and arithmetic the kernel serves: always at orders 6 and 7, and at
// order 5 where the domain's mesh has hanging faces (mesh_hangs): with 30 %
// of the base cells refined 127 G DOF-updates/s here against 123.5 in the
// node-per-thread kernel, conforming 155 against 162.
template <int DIM, int N, typename CT>
__host__ __device__ constexpr bool use_mma()
{
  return DIM == 3 && N >= 6 && sizeof(CT) == sizeof(double);
}
template <int DIM, int N, typename CT>
__host__ __device__ constexpr bool use_mma_hanging()
{
  return DIM == 3 && N == 5 && sizeof(CT) == sizeof(double);
}
// as late_from: N = 5, 331 elements with hanging faces (262 of them, 0.35, in the
// first launch) 76.2 us per step early and 72.3 late, 204 69.1 and 71.3; N = 6,
// 204 (160, 0.36) 83.4 and 89.6 in eager steps, 256 conforming (0.58) 59.9 and
// 46.6; N = 7, 204 (0.54) 67.5 and 71.3, 256 conforming 41.9 and 41.5
template <int N> constexpr int mma_late_from()
{
  return N == 5 ? 34 : N == 6 ? 42 : 85;
}

// hops: an order-N domain's operators Dr | interpolation[3] | projection[3] | w;
// a domain without a glue grid, so without hanging faces, has identities for
// interpolations
inline bool mesh_hangs(const double *hops, int N)
{
  const int n = N + 1;
  const double *bottom = hops + 2 * n * n;
  for (int i = 0; i < n * n; ++i)
    if (bottom[i] != (i % (n + 1) == 0 ? 1.0 : 0.0))
      return true;
  return false;
}

// L2 prefetch of what the CTA of a later work item will read of its element
// e, a line of 128 bytes per thread: state and dq rows, element data and flux
// constants.
// (The bulk prefetches of prefetch_element, 21 from one thread at about 200
// cycles each, held that thread's warp and with it the CTA's barriers: 4,300
// of the 18,800 cycles of an N = 7 element's CTA.)
template <int N, int MODE, int NT>
__device__ __forceinline__ void prefetch_lines(const DomainView &d,
                                               const StageParams &sp, int e,
                                               int t)
{
  constexpr int P = (N + 1) * (N + 1), Np = P * (N + 1);
  // lines a row may touch; past its end: its last value's line
  constexpr int L = (Np * 8 + 127) / 128 + (Np % 16 ? 1 : 0);
  const size_t eoff = (size_t)e * Np;
  const bool rd = MODE != MODE_RHS && !sp.first_stage;
#pragma unroll
  for (int w0 = 0; w0 < 9 * L; w0 += NT)
  {
    const int w = w0 + t;
    if (w < 9 * L)
    {
      const int n = 16 * (w % L);
      const size_t at = (w / L) * d.fs + eoff + (n < Np ? n : Np - 1);
      prefetch_l2(d.qin + at);
      if (rd)
        prefetch_l2(d.dq + at);
    }
  }
  if (t < 6)
    prefetch_l2(d.fcE + (size_t)e * 6 + t);
  else if (t == 6)
    prefetch_l2(d.ed + e);
}

// work item blockIdx.x of n
template <int N, int MODE, typename Item>
__device__ __forceinline__ void mma_element(const Item &item, int n,
                                            const StageParams &sp,
                                            double iwend)
{
  const DomainView &d = item.view(blockIdx.x);
  const int e = item.elem(blockIdx.x);
  using M = MmaShape<N>;
  constexpr int Nq = M::Nq, P = M::P, PP = M::PP, Np = M::Np, PITCH = M::PITCH;
  constexpr bool VEC = Nq % 2 == 0; // rows of a plane are 16-byte aligned
  extern __shared__ __align__(16) double smem[];
  double *zb = smem + M::OFF_Z, *pt = smem + M::OFF_J;
  const double *fcf = smem + M::OFF_FC;
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + M::OFF_BAR);
  const int t = threadIdx.x, w = t >> 5, rr = (t & 31) >> 2, c = t & 3;
  // row and columns of this lane; lanes past the matrix read its last row
  // or columns instead (they land in rows and columns that are not stored;
  // as entries past a contracted index they are replaced by zeros)
  const bool v0 = rr < Nq && 2 * c < Nq, v1 = rr < Nq && 2 * c + 1 < Nq;
  const int r = rr < Nq ? rr : N;
  const int i0 = 2 * c < Nq ? 2 * c : (VEC ? N - 1 : N);
  const int o1 = i0 < N ? 1 : 0; // second column
  const size_t fs = d.fs, eoff = (size_t)e * Np;
  const bool rd = MODE != MODE_RHS && !sp.first_stage;
  // where the field rows start in their shared-memory slots (odd Np): even
  // and odd fields
  const int sh0 = Np % 2 ? e & 1 : 0, sh1 = Np % 2 ? (e + d.K) & 1 : 0;
  auto row = [&](int f) { return smem + f * PITCH + (f & 1 ? sh1 : sh0); };

  // ------------------------------------------------------------------ issue
  if (t == 0)
    mbar_init(bar, 1);
  int2 ds = make_int2(0, 2);
  if (w < 6)
    ds = d.fdesc[(size_t)e * 6 + w];
  grid_dependency_wait(); // the stage input is complete
  if (t == 0)
  {
    fence_proxy_async();
    // the last row of an odd-sized state has no value after it to copy
    const bool last = Np % 2 && e == d.K - 1 && (d.K & 1);
    mbar_expect_tx(bar, (9 * (Np + Np % 2) - (last ? 2 : 0) + 32) *
                            sizeof(double));
    if (PP == P)
    {
#pragma unroll
      for (int f = 0; f < 9; ++f)
      {
        const int sh = f & 1 ? sh1 : sh0;
        const uint32_t n = PITCH - (last && f == 8 ? 2 : 0);
        bulk_g2s(smem + f * PITCH, d.qin + f * fs + eoff - sh,
                 n * sizeof(double), bar);
      }
    }
    bulk_g2s(smem + M::OFF_FC, d.fcE + (size_t)e * 6, 24 * sizeof(double), bar);
    bulk_g2s(smem + M::OFF_FC + 24, d.ed + e, sizeof(ElemData), bar);
    if (last)
      smem[8 * PITCH + Np - 1] = d.qin[8 * fs + eoff + Np - 1];
  }
  if (PP != P)
  {
    // plane by plane, warp k plane k
    __syncthreads(); // the mbarrier is initialised
    if ((t & 31) == 0)
    {
#pragma unroll
      for (int f = 0; f < 9; ++f)
        bulk_g2s(smem + f * PITCH + w * PP, d.qin + f * fs + eoff + w * P,
                 P * sizeof(double), bar);
    }
    __syncwarp();
  }

  // warp f: the trace across face f (kinds 0 and 1), one matrix per trace
  // field; the coarse side's jumps (kind 2) go straight to the jump arrays
  const int f = w, ax = w >> 1;
  const int sa = ax == 0 ? Nq : 1, sb = ax == 2 ? Nq : P; // along the face
  const int sn = ax == 0 ? 1 : (ax == 1 ? Nq : P);        // across it
  // the face's lines along y at N = 7 (columns of an x face): columns c and
  // c + 4, two to a 128-byte line, instead of 2 c and 2 c + 1
  int a0 = i0, da = o1;
  if (N == 7 && ax == 0)
  {
    a0 = c;
    da = 4;
  }
  const int fo = a0 * sa + r * sb, pn = i0 + Nq * r;
  double *pj = pt + f * 6 * P + pn;
  double2 nb[6];
  if (w < 6)
  {
    const int kind = ds.y & 3;
    if (kind < 2)
    {
      const double *x =
          d.qin + (size_t)ds.x * Np + (f & 1 ? 0 : N * sn) + fo;
      if (VEC && ax > 0)
      {
#pragma unroll
        for (int q = 0; q < 6; ++q)
          nb[q] = get2<true>(x + trace_field<3>(ax, q) * fs);
      }
      else
      {
#pragma unroll
        for (int q = 0; q < 6; ++q)
          nb[q] = get2<false>(x + trace_field<3>(ax, q) * fs, da * sa);
      }
    }
    else if (kind == 2)
    {
      // the pieces' projected jumps, summed in glue order
      const double *x = d.mbuf + (size_t)ds.x * 6 * P + pn;
      const double iv = f & 1 ? iwend : -iwend;
#pragma unroll
      for (int q = 0; q < 6; ++q)
      {
        double2 y[4];
#pragma unroll
        for (int p = 0; p < 4; ++p)
          y[p] = get2<VEC>(x + (p * 6 + q) * P, o1);
        const double sc = q < 3 ? iwend : iv;
        put2<VEC>(pj + q * P,
                  make_double2(sc * (((y[0].x + y[1].x) + y[2].x) + y[3].x),
                               sc * (((y[0].y + y[1].y) + y[2].y) + y[3].y)),
                  v0, v1);
      }
    }
    else
    {
#pragma unroll
      for (int q = 0; q < 6; ++q)
        nb[q] = make_double2(0.0, 0.0);
    }
  }
  // a later item's element, while this one's loads fly
  const int ia = blockIdx.x + sp.ahead;
  int2 dsa = make_int2(0, 0); // its face w
  if (sp.ahead > 0 && ia < n)
  {
    const int ea = item.elem(ia);
    if (w < 6)
      dsa = item.view(ia).fdesc[(size_t)ea * 6 + w];
    prefetch_lines<N, MODE, M::NT>(item.view(ia), sp, ea, t);
    if (t == 8 && ia + sp.ahead < n) // and the entry read here by that CTA
      item.prefetch(ia + sp.ahead);
  }
  // fragments of D, zero past N: for X D^T and Op X^T (column 2 c + s), and
  // along y and z, whose right operands are read from shared memory, with
  // the contracted index that meets fewer bank conflicts (2 c + s or c + 4 s)
  constexpr bool YS = N == 7, ZS = N == 7 || N == 5;
  auto dfrag = [&](int k) {
    return rr < Nq && k < Nq ? __ldg(d.ops + rr + Nq * k) : 0.0;
  };
  if (PP == P)
    __syncthreads(); // the mbarrier is initialised
  // ---------------------------------------------------------------------- z
  // row of plane k = const, line j in the z-derivative buffer: at N = 7 the
  // lines of odd planes are swapped in pairs, so that a warp storing two
  // rows k of one line j does not meet its own banks
  auto zrow = [&](int q, int k, int j) {
    return zb + q * Np + k * P + Nq * (N == 7 ? j ^ (k & 1) : j);
  };
  {
    const int k0 = ZS ? c : 2 * c, k1 = ZS ? c + 4 : 2 * c + 1;
    const double2 fz = make_double2(dfrag(k0), dfrag(k1));
    const int o0 = (k0 < Nq ? k0 : N) * PP + r, o1z = (k1 < Nq ? k1 : N) * PP + r;
    if (!mbar_wait(bar, 0))
      atomicExch(d.err, 1);
    __syncwarp(); // the matrix instruction takes whole warps
    {
      double2 z[6];
#pragma unroll
      for (int q = 0; q < 6; ++q)
      {
        // sxz, syz, szz, vx, vy, vz
        const int f = q == 0 ? 7 : q == 1 ? 8 : q == 2 ? 5 : q - 3;
        z[q] = make_double2(0.0, 0.0);
        dmma(z[q], fz.x, row(f)[w * Nq + o0]);
      }
#pragma unroll
      for (int q = 0; q < 6; ++q)
      {
        const int f = q == 0 ? 7 : q == 1 ? 8 : q == 2 ? 5 : q - 3;
        dmma(z[q], fz.y, k1 < Nq ? row(f)[w * Nq + o1z] : 0.0);
      }
      double *o = zrow(0, r, w) + i0;
      if (v0)
      {
#pragma unroll
        for (int q = 0; q < 6; ++q)
          put2<VEC>(o + q * Np, z[q], true, v1);
      }
    }
  }

  // ------------------------------------------------------------------- face
  const double *em = smem + M::OFF_FC + 24; // irho lam mu Zp Zs rx ry rz
  const int kind = ds.y & 3; // warps without a face: 2, nothing to do
  if (kind != 2)
  {
    const int hp = kind == 1 ? (ds.y >> 8) & 7 : 0;
    const double sg = f & 1 ? 1.0 : -1.0;
    // left fragment of mortar operator `op` (bottom half; the top half is
    // its reflection)
    auto frag = [&](int op, int top, int k0, int k1) {
      const double *A = d.ops + op * P + (top ? Nq * N + N - r : r);
      const int sk = top ? -Nq : Nq;
      return make_double2(rr < Nq && k0 < Nq ? __ldg(A + sk * k0) : 0.0,
                          rr < Nq && k1 < Nq ? __ldg(A + sk * k1) : 0.0);
    };
    // six matrices, whose columns are a0 and a0 + da, through a pair of
    // operators, three at a time; the result has columns 2 c and 2 c + 1
    auto tensor = [&](int op) {
      const bool y4 = N == 7 && da == 4;
      if (Nq < 8)
      {
#pragma unroll
        for (int q = 0; q < 6; ++q)
          nb[q] = make_double2(v0 ? nb[q].x : 0.0, v1 ? nb[q].y : 0.0);
      }
      const double2 oa = frag(op, (hp - 1) & 1, y4 ? c : 2 * c, y4 ? c + 4 : 2 * c + 1),
                    ob = frag(op, (hp - 1) >> 1, 2 * c, 2 * c + 1);
#pragma unroll
      for (int q = 0; q < 6; q += 3)
      {
        dmma_t<3>(oa, nb + q);
        dmma_t<3>(ob, nb + q);
      }
    };
    if (hp) // coarse trace -> my piece
    {
      tensor(2);
      a0 = i0;
      da = o1;
    }
    const int sbs = ax == 2 ? Nq : PP, sns = ax == 2 ? PP : sn; // own trace
    const int own = (f & 1 ? N * sns : 0) + a0 * sa + r * sbs;
    const int pw = a0 + Nq * r - pn; // from this lane's place in C layout
    const double iv = iwend * sg;
    const bool fsurf = kind == 3 && ((ds.y >> 2) & 3) == 0;
    // component a of the flux depends on v_a and row ax of the stress only:
    // the normal component on the P impedances, the others on S
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
      const int ft = trace_field<3>(ax, 3 + a);
      const double *xv = row(a) + own;
      const double *xt = smem + ft * PITCH + (ft & 1 ? sh1 : sh0) + own;
      double2 ov, ot;
      if (VEC && ax > 0)
      {
        ov = get2<true>(xv);
        ot = get2<true>(xt);
      }
      else
      {
        ov = get2<false>(xv, da * sa);
        ot = get2<false>(xt, da * sa);
      }
      if (fsurf)
      {
        // free surface: v+ = v-, S+ = -S- (absorbing: q+ = 0)
        nb[a] = ov;
        nb[3 + a] = make_double2(-ot.x, -ot.y);
      }
      const double2 dv = make_double2(nb[a].x - ov.x, nb[a].y - ov.y);
      const double2 dT = make_double2(sg * (nb[3 + a].x - ot.x),
                                      sg * (nb[3 + a].y - ot.y));
      double2 JT, Jv;
      if (sp.flux == 1)
      {
        JT = make_double2(0.5 * dT.x, 0.5 * dT.y);
        Jv = make_double2(0.5 * dv.x, 0.5 * dv.y);
      }
      else
      {
        const double Zm = em[a == ax ? 3 : 4];
        const double2 zi = *reinterpret_cast<const double2 *>(
            fcf + 4 * f + (a == ax ? 0 : 2)); // Z+, 1 / (Z- + Z+)
        Jv = make_double2((zi.x * dv.x + dT.x) * zi.y,
                          (zi.x * dv.y + dT.y) * zi.y);
        JT = make_double2(Zm * Jv.x, Zm * Jv.y);
      }
      // the coarse side's jumps from the same Riemann solution
      nb[a] = make_double2(dT.x - JT.x, dT.y - JT.y);
      nb[3 + a] = make_double2(Jv.x - dv.x, Jv.y - dv.y);
      const double2 T2 = make_double2(iwend * JT.x, iwend * JT.y),
                    V2 = make_double2(iv * Jv.x, iv * Jv.y);
      if (N == 7 && da == 4)
      {
        pj[a * P + pw] = T2.x;
        pj[a * P + pw + 4] = T2.y;
        pj[(3 + a) * P + pw] = V2.x;
        pj[(3 + a) * P + pw + 4] = V2.y;
      }
      else
      {
        put2<VEC>(pj + a * P, T2, v0, v1);
        put2<VEC>(pj + (3 + a) * P, V2, v0, v1);
      }
    }
    if (hp) // L2 projection of the coarse side's jumps, to its mortar slot
    {
      tensor(5);
      double *o = d.mbuf + (size_t)d.fslot[(size_t)e * 6 + f] * 6 * P + pn;
#pragma unroll
      for (int q = 0; q < 6; ++q)
        put2<VEC>(o + q * P, nb[q], v0, v1);
    }
  }
  // the later item's mortar slots of a coarse face (its descriptor, a trip to
  // memory, has arrived by now: read ahead of the prefetches face by face,
  // six such trips in a row held the CTA)
  if ((dsa.y & 3) == 2)
  {
    constexpr int L = (24 * P * 8 + 127) / 128;
    for (int l = t & 31; l < L; l += 32)
      prefetch_l2(item.view(ia).mbuf + (size_t)dsa.x * 6 * P + 16 * l);
  }
  const double2 fx = make_double2(dfrag(2 * c), dfrag(2 * c + 1));
  const double2 fy = YS ? make_double2(dfrag(c), dfrag(c + 4)) : fx;
  __syncthreads();
  if (sp.early)
    grid_launch_dependents(); // as in dg_stage.cuh, not earlier
  const double a = MODE != MODE_RHS ? sp.A : 0.0;
  const double s = MODE != MODE_RHS ? d.dt : 1.0;
  const int n0 = w * P + r * Nq + i0, m0 = n0 + w * (PP - P);
  const double *dqp = d.dq + eoff + n0;
  // derivatives along x and y of two fields, with the corrections of the
  // faces across the axis (jump components jx, jy) as the start values
  const bool xl = v0 && c == 0, xr = rr < Nq && c == N / 2;
  const bool yl = rr == 0, yr = rr == N;
  const double *px = pt + rr + Nq * w, *py = pt + 12 * P + i0 + Nq * w;
  const int y0 = YS ? c : 2 * c, y1 = YS ? c + 4 : 2 * c + 1;
  const int oy0 = w * PP + (y0 < Nq ? y0 : N) * Nq + r,
            oy1 = w * PP + (y1 < Nq ? y1 : N) * Nq + r;
  // y0 and y1 are indices of a row, for the lanes whose results are stored
  const bool yk0 = N != 5 || v0, yk1 = N == 7 || v1;
  auto startx = [&](int q) {
    double2 y = make_double2(0.0, 0.0);
    if (xl)
      y.x = px[q * P];
    if (xr)
      (N % 2 ? y.y : y.x) = px[(6 + q) * P];
    return y;
  };
  auto starty = [&](int q) {
    double2 y = make_double2(0.0, 0.0);
    if (yl)
      y = get2<VEC>(py + q * P, o1);
    if (yr)
      y = get2<VEC>(py + (6 + q) * P, o1);
    return y;
  };
  auto dxy = [&](int f, int jx, int g, int jy, double2 &X, double2 &Y) {
    double2 x = make_double2(0.0, 0.0);
    if (VEC && v0)
      x = get2<true>(row(f) + m0);
    if (!VEC && v0)
      x.x = row(f)[m0];
    if (!VEC && v1)
      x.y = row(f)[m0 + 1];
    X = startx(jx);
    Y = starty(jy);
    dmma(X, x.x, fx.x);
    dmma(Y, fy.x, yk0 ? row(g)[oy0] : 0.0);
    dmma(X, x.y, fx.y);
    dmma(Y, fy.y, yk1 ? row(g)[oy1] : 0.0);
  };
  // the derivative along z with its faces' corrections (jump component jq)
  const double *pz = zrow(0, w, r) + i0;
  const double *jz = pt + (w == N ? 30 : 24) * P + i0 + Nq * r;
  auto dz = [&](int q, int jq) {
    double2 y = make_double2(0.0, 0.0);
    if (rr < Nq)
      y = get2<VEC>(pz + q * Np, o1);
    if (w == 0 || w == N)
    {
      const double2 j = get2<VEC>(jz + jq * P, o1);
      y.x += j.x;
      y.y += j.y;
    }
    return y;
  };
  // dq of fields [f0, f0 + 3), and their update dq = a dq + acc,
  // q' = q + B dq (or the right-hand side itself)
  auto load_dq = [&](int f0, double2 *u) {
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
      u[k] = make_double2(0.0, 0.0);
      if (MODE != MODE_RHS && rd && rr < Nq)
        u[k] = get2<VEC>(dqp + (f0 + k) * fs, o1);
    }
  };
  auto put = [&](int f0, const double2 *u) {
    const size_t at = eoff + n0 + f0 * fs;
    if constexpr (MODE == MODE_RHS)
    {
#pragma unroll
      for (int k = 0; k < 3; ++k)
        put2<VEC>(d.rhs + at + k * fs, u[k], v0, v1);
    }
    else
    {
      // streaming stores, as in dg_stage.cuh
      if (v0)
      {
        double2 o[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
        {
          const double2 q = get2<VEC>(row(f0 + k) + m0, o1);
          o[k] = make_double2(q.x + sp.B * u[k].x, q.y + sp.B * u[k].y);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
        {
          double *pd = d.dq + at + k * fs, *pq = d.qout + at + k * fs;
          if (VEC)
          {
            __stcs(reinterpret_cast<double2 *>(pd), u[k]);
            __stcs(reinterpret_cast<double2 *>(pq), o[k]);
          }
          else
          {
            __stcs(pd, u[k].x);
            __stcs(pq, o[k].x);
            if (v1)
            {
              __stcs(pd + 1, u[k].y);
              __stcs(pq + 1, o[k].y);
            }
          }
        }
      }
    }
  };
  double2 u[3], X, Y, Z;
  load_dq(0, u);
  const double rx = s * em[5], ry = s * em[6], rz = s * em[7];
  // velocities: (div S) / rho, and the point source, if any:
  // s f(t_stage) F phi_n(x_s) / (rho w_n J)
  {
    const double ir = em[0], cx = ir * rx, cy = ir * ry, cz = ir * rz;
#pragma unroll
    for (int v = 0; v < 3; ++v)
    {
      dxy(trace_field<3>(0, 3 + v), v, trace_field<3>(1, 3 + v), v, X, Y);
      Z = dz(v, v);
      u[v].x = a * u[v].x + (cx * X.x + cy * Y.x + cz * Z.x);
      u[v].y = a * u[v].y + (cx * X.y + cy * Y.y + cz * Z.y);
    }
    if (e == d.src.elem)
    {
      const double ts = d.clock->time + sp.C * d.dt;
      const double gs = s * ricker(ts, d.src.f0, d.src.t0) * ir;
      const double g0 = gs * d.src.w[n0], g1 = gs * d.src.w[n0 + o1];
#pragma unroll
      for (int v = 0; v < 3; ++v)
      {
        u[v].x += g0 * d.src.force[v];
        u[v].y += g1 * d.src.force[v];
      }
    }
  }
  put(0, u);
  load_dq(3, u);
  // normal stresses: lambda tr(grad v) + 2 mu dv_a/dx_a
  {
    const double lam = em[1], m2 = 2.0 * em[2];
    dxy(0, 3, 1, 4, X, Y);
    Z = dz(5, 5);
    X = make_double2(rx * X.x, rx * X.y);
    Y = make_double2(ry * Y.x, ry * Y.y);
    Z = make_double2(rz * Z.x, rz * Z.y);
    const double2 ll = make_double2(lam * (X.x + Y.x + Z.x),
                                    lam * (X.y + Y.y + Z.y));
    u[0].x = a * u[0].x + (ll.x + m2 * X.x);
    u[0].y = a * u[0].y + (ll.y + m2 * X.y);
    u[1].x = a * u[1].x + (ll.x + m2 * Y.x);
    u[1].y = a * u[1].y + (ll.y + m2 * Y.y);
    u[2].x = a * u[2].x + (ll.x + m2 * Z.x);
    u[2].y = a * u[2].y + (ll.y + m2 * Z.y);
  }
  put(3, u);
  load_dq(6, u);
  // shear stresses: mu (dv_a/dx_b + dv_b/dx_a)
  {
    const double mu = em[2], cx = mu * rx, cy = mu * ry, cz = mu * rz;
    dxy(1, 4, 0, 3, X, Y); // sxy
    u[0].x = a * u[0].x + (cx * X.x + cy * Y.x);
    u[0].y = a * u[0].y + (cx * X.y + cy * Y.y);
    dxy(2, 5, 2, 5, X, Y); // sxz, syz
    Z = dz(3, 3);
    u[1].x = a * u[1].x + (cx * X.x + cz * Z.x);
    u[1].y = a * u[1].y + (cx * X.y + cz * Z.y);
    Z = dz(4, 4);
    u[2].x = a * u[2].x + (cy * Y.x + cz * Z.x);
    u[2].y = a * u[2].y + (cy * Y.y + cz * Z.y);
  }
  put(6, u);
}

// one domain, one element per CTA
template <int N, int MINB, int MODE>
__global__ void __launch_bounds__(MmaShape<N>::NT, MINB)
    dg_mma_kernel(DomainView d, int n, StageParams sp, double iwend)
{
  mma_element<N, MODE>(SingleItems{d}, n, sp, iwend);
}

// many domains: work[idx] = (domain, element)
template <int N, int MINB>
__global__ void __launch_bounds__(MmaShape<N>::NT, MINB)
    dg_mma_batch_kernel(const DomainView *__restrict__ views,
                        const int2 *__restrict__ work, int n, StageParams sp,
                        double iwend)
{
  mma_element<N, MODE_STAGE>(BatchItems{views, work}, n, sp, iwend);
}

} // namespace bfam_b200
