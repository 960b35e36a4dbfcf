// Fused BD loop of the FP64 Newton-3 path: nsteps Brownian-dynamics steps
// (dynamics0-3.mono.f90 driven by the ENERGY force of energy.mono.f90) in one
// cooperative launch: one block an SM, two where no single-particle term is on
// (FLD; the items of a small system are latency).  Per step, two phases between grid barriers:
//   P  every item of the FP64 pair tile (n64_item), round-robin over the
//      blocks; the step's noise, a warp per tile and component, by the blocks
//      that the items reach last;
//   A  a block per quarter tile (half or whole ones where the quarters
//      outnumber the blocks): the tile's partials summed, the ions moved and
//      their single-particle terms formed at the new positions.
// The terms and their summation order are those of the per-kernel steps, bit
// for bit.  Where the terms of a system are few the launches, their gaps and
// the FP64 chains on a handful of SMs were the step: bulk KCl, 260 ions, took
// 55 us a step as fields, ion-ion and assembly kernels, 17 us here.
// Every barrier wait is bounded (gridsync.cuh).
#include <algorithm>

#include "fields64.cuh"
#include "gridsync.cuh"
#include "launch.h"
#include "move64.cuh"
#include "pairs64.cuh"

namespace bgpu {

template <bool RF, bool PBC, bool FLD>
__global__ void __launch_bounds__(kN64Threads, FLD ? 1 : 2)
    k_bd_loop64(const __grid_constant__ KP p, AssembleFlags fl, uint32_t mask, int ii, int srp,
                int variant, uint64_t seed, uint64_t step0, int nsteps) {
  extern __shared__ __align__(16) unsigned char loop64_dsm[];  // Loop64Smem
  N64Smem &sp = *reinterpret_cast<N64Smem *>(loop64_dsm);
  Asm64Smem &sa = *reinterpret_cast<Asm64Smem *>(loop64_dsm + sizeof(N64Smem));
  __shared__ int flag;
  n64_laws(p, sp);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, G = gridDim.x, cap = p.cap;
  const int ntot = p.st->ntot;  // constant during BD
  const int T = live_tiles(ntot, p.nsites), S = n64_split(T), nitem = n3_pairs(T) * S;
  const int nh = 4 * T <= G ? 4 : (2 * T <= G ? 2 : 1);
  double *noise = p.fii;  // [3][cap]: the partials of the chunked kernel, unused here
  unsigned bar = 0;
  double eo[4], e[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // energies: not formed here
  int err = 0;
  if (FLD) {
    for (int u = 8 * (w * G + (int)blockIdx.x); p.nsites + u < ntot; u += 8 * G * (kN64Threads / 32)) {
      const int i = p.nsites + u + (lane >> 2);
      fields_quad_f64(p, i, i < ntot, mask, 1, eo);
    }
    if (!grid_barrier(&p.st->bar_count, ++bar, p.st, &flag)) goto done;
  }
  for (int s = 0; s < nsteps; ++s) {
    if (w < 3)
      for (int t = G - 1 - (int)blockIdx.x; t < T; t += G) {
        const int i = p.nsites + 32 * t + lane;
        if (i < ntot) noise[(size_t)w * cap + i] = bd_noise_one(seed, step0 + s, (uint32_t)i, w);
      }
    for (int it = blockIdx.x; it < nitem; it += G)
      n64_item<RF, PBC, false>(p, ntot, T, S, it, 1, ii != 0, srp != 0, sp, e, err);
    if (!grid_barrier(&p.st->bar_count, ++bar, p.st, &flag)) goto done;
    for (int it = blockIdx.x; it < nh * T; it += G) {
      const int t = it / nh, h = it % nh, n = 32 / nh;
      assemble64<true, RF>(p, fl, 1, variant, seed, step0 + s, ntot, t, 0, h, nh, noise, sa);
      __syncthreads();  // the new positions; the sums' shared memory free again
      if (FLD && s + 1 < nsteps)
        for (int u = 8 * w; u < n; u += 8 * (kN64Threads / 32)) {
          const int i = p.nsites + 32 * t + n * h + u + (lane >> 2);
          fields_quad_f64(p, i, i < ntot, mask, 1, eo);
        }
    }
    if (s + 1 < nsteps && !grid_barrier(&p.st->bar_count, ++bar, p.st, &flag)) goto done;
  }
done:
  if (err) atomicOr(&p.st->err, err);
  launch_exit(p.st);
}

bool bd_loop64_supported(const KP &p, const AssembleFlags &fl) {
  return !fl.fp32_partials && fl.ntile > 0 && !fl.use_total && p.nsites == 0 && !fl.is;
}

template <bool RF, bool PBC, bool FLD>
static cudaError_t launch_loop64_t(const KP &p, const AssembleFlags &fl, uint32_t mask, int ii,
                                   int srp, int variant, uint64_t seed, uint64_t step0,
                                   int nsteps, cudaStream_t stream) {
  auto kern = k_bd_loop64<RF, PBC, FLD>;
  const size_t dsm = sizeof(N64Smem) + sizeof(Asm64Smem);
  int dev = 0, nsm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)dsm);
  if (e != cudaSuccess) return e;
  const int T = fl.ntile;
  const int grid =
      std::max(1, std::min((FLD ? 1 : 2) * nsm, std::max(n3_pairs(T) * n64_split(T), 4 * T)));
  KP pc = p;  // the barrier counters are zero between launches (launch_exit)
  AssembleFlags fc = fl;
  void *args[] = {(void *)&pc,      (void *)&fc,   (void *)&mask,  (void *)&ii,    (void *)&srp,
                  (void *)&variant, (void *)&seed, (void *)&step0, (void *)&nsteps};
  return cudaLaunchCooperativeKernel((const void *)kern, dim3(grid), dim3(kN64Threads), args,
                                     dsm, stream);
}

cudaError_t launch_bd_loop64(const KP &p, const AssembleFlags &fl, uint32_t mask, bool ii,
                             bool srp, int variant, uint64_t seed, uint64_t step0, int nsteps,
                             cudaStream_t stream) {
  auto run = fl.rf_ab ? launch_loop64_t<true, false, true>  // RFPAR: its gathers are a field term
             : fl.nofield
                 ? (p.periodic ? launch_loop64_t<false, true, false>
                               : launch_loop64_t<false, false, false>)
                 : (p.periodic ? launch_loop64_t<false, true, true>
                               : launch_loop64_t<false, false, true>);
  return run(p, fl, mask, ii, srp, variant, seed, step0, nsteps, stream);
}

}  // namespace bgpu
