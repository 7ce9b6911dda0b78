// Once-per-step work beside the stage kernels: receiver sampling and the
// per-domain clock that the point source reads.
#pragma once

#include "dg_common.cuh"

namespace bfam_b200
{

// What the post-step kernel needs of one domain.
struct PostView
{
  const double *__restrict__ q; // state after the step
  size_t fs;                    // field stride K*Np
  int Np, nfld;
  int nrecv, max_samples;
  const int *__restrict__ relem; // [nrecv] element holding receiver r
  const double *__restrict__ rw; // [nrecv][Np] Lagrange weights phi_n(x_r)
  double *__restrict__ seis;     // [max_samples][nrecv][nfld]
  DomainClock *clock;
  double dt;
};

// Sample every field at the receivers blockIdx.y, blockIdx.y + gridDim.y, ...
// of one domain: one warp per (receiver, field) pair, lane-strided dot product
// with the element's Lagrange weights, then a butterfly sum (deterministic:
// the order does not depend on the grid).  The last of the domain's CTAs to
// finish, by a ticket in its clock, advances the clock by dt.  Samples beyond
// max_samples are dropped; the clock still advances.
// What bounds it is the latency of one (receiver, field) pair, two dependent
// trips to memory: a single CTA took them 18 deep for 16 receivers of nine
// fields, 10 to 14 us of a step (N = 3 and 5), so a CTA of nine warps takes
// one receiver instead.
__device__ __forceinline__ void post_step(const PostView &p)
{
  grid_launch_dependents();
  grid_dependency_wait();
  const int nr = p.nrecv > 1 ? p.nrecv : 1;
  const int parts = nr < (int)gridDim.y ? nr : (int)gridDim.y;
  if ((int)blockIdx.y >= parts)
    return;
  const int s = *static_cast<volatile int *>(&p.clock->nsamp);
  if (s < p.max_samples)
  {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5,
              nw = blockDim.x >> 5;
    for (int r = blockIdx.y; r < p.nrecv; r += parts)
    {
      const size_t at = (size_t)p.relem[r] * p.Np;
      const double *wt = p.rw + (size_t)r * p.Np;
      for (int c = wid; c < p.nfld; c += nw)
      {
        const double *x = p.q + c * p.fs + at;
        double acc = 0;
#pragma unroll 4
        for (int n = lane; n < p.Np; n += 32)
          acc += wt[n] * x[n];
#pragma unroll
        for (int o = 16; o; o >>= 1)
          acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0)
          p.seis[((size_t)s * p.nrecv + r) * p.nfld + c] = acc;
      }
    }
  }
  __syncthreads(); // every warp has read the clock
  if (threadIdx.x == 0)
  {
    bool last = parts == 1;
    if (!last)
    {
      __threadfence(); // this CTA's reads come before its ticket
      last = atomicAdd(&p.clock->ticket, 1) == parts - 1;
    }
    if (last)
    {
      p.clock->time += p.dt;
      p.clock->nsamp = s + 1;
      p.clock->ticket = 0;
    }
  }
}

constexpr int POST_THREADS = 288; // a warp per field
constexpr int POST_PARTS = 64;    // receiver CTAs per domain, at most

// batches: CTAs (domain, part) over the array's domains
__global__ void __launch_bounds__(POST_THREADS)
    dg_post_step_kernel(const PostView *__restrict__ pv)
{
  post_step(pv[blockIdx.x]);
}

// one domain, its view in the parameter bank (captured by value in graphs)
__global__ void __launch_bounds__(POST_THREADS)
    dg_post_step_one(const __grid_constant__ PostView p)
{
  post_step(p);
}

// what & 1: set the time to t; what & 2: restart the sample count
__global__ void dg_set_clock_kernel(DomainClock *clock, double t, int what)
{
  if (what & 1)
    clock->time = t;
  if (what & 2)
    clock->nsamp = 0;
}

} // namespace bfam_b200
