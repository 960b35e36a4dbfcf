// Force assembly and the Ermak-McCammon BD update (dynamics0-3.mono.f90,
// dynamics0nuc.f90, fixcoor.f90, countions.f90), fused in one kernel: one
// warp per particle sums its partial forces in a fixed order, writes
// fx,fy,fz and, for a BD step, moves the particle with in-register Philox
// noise.
#include "ff.cuh"
#include "launch.h"
#include "physics.cuh"
#include "move32.cuh"
#include "move64.cuh"

namespace bgpu {

constexpr int kAsmWarps = 8;  // particles per assembly block

// One warp per particle: lane c adds chunk partials c, c+32, ...; a fixed
// shuffle tree sums the lanes, so the order is the same every run.
__global__ void __launch_bounds__(32 * kAsmWarps)
    k_assemble(KP p, AssembleFlags fl, int do_bd, int variant, uint64_t seed,
               uint64_t step) {
  const int i = blockIdx.x * kAsmWarps + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int ntot = p.st->ntot;
  if (i >= ntot) return;  // warp-uniform
  const int cap = p.cap;
  double v[3] = {0.0, 0.0, 0.0};
  if (fl.ii && i >= fl.ii_from)
    for (int c = lane; c < fl.nchunk_ii; c += 32)
#pragma unroll
      for (int k = 0; k < 3; ++k) v[k] += p.fii[((size_t)c * 3 + k) * cap + i];
  if (fl.rf && i >= p.nsites)
    for (int c = lane; c < fl.nchunk_rf; c += 32)
#pragma unroll
      for (int k = 0; k < 3; ++k) v[k] += p.frf[((size_t)c * 3 + k) * cap + i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  if (lane != 0) return;
  double f[3];
  if (fl.use_total) {
    f[0] = p.fx[i];
    f[1] = p.fy[i];
    f[2] = p.fz[i];
  } else {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      double w = (fl.nofield ? 0.0 : p.ffield[k * cap + i]) + v[k];
      if (fl.is) w += p.fis[k * cap + i];
      f[k] = w;
    }
    p.fx[i] = f[0];
    p.fy[i] = f[1];
    p.fz[i] = f[2];
  }
  if (do_bd) {
    double g[3];
    bd_noise3(seed, step, (uint32_t)i, g);
    bd_move(p, variant, i, f, g);
  }
}

// The FP64 Newton-3 partials (assemble64): a block per site tile, then four
// per ion tile (eight particles each), so that the FP64 work of a small
// system's moves spreads over the SMs.
constexpr int kAsm64Parts = 4;

template <bool RF>
__global__ void __launch_bounds__(kN64Threads)
    k_assemble64(const __grid_constant__ KP p, AssembleFlags fl, int do_bd, int variant,
                 uint64_t seed, uint64_t step, int sb) {
  after_prev();
  __shared__ Asm64Smem s;
  assemble64<false, RF>(p, fl, do_bd, variant, seed, step, p.st->ntot, blockIdx.x / kAsm64Parts, sb,
                    blockIdx.x % kAsm64Parts, kAsm64Parts, nullptr, s);
}


__global__ void __launch_bounds__(32 * kAsmWarps)
    k_assemble_f32(const __grid_constant__ KP p, AssembleFlags fl, int do_bd, int variant,
                   uint64_t seed, uint64_t step) {
  const int i = blockIdx.x * kAsmWarps + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int ntot = p.st->ntot;
  if (i >= ntot) return;  // warp-uniform
  const int cap = p.cap;
  float s[3] = {0.f, 0.f, 0.f}, c[3] = {0.f, 0.f, 0.f};  // compensated sums
  if (!fl.use_total) {
    if (fl.ii && i >= fl.ii_from)
      for (int ch = lane; ch < fl.nchunk_ii; ch += 32)
#pragma unroll
        for (int k = 0; k < 3; ++k) acc2(s[k], c[k], p.fii_f[((size_t)ch * 3 + k) * cap + i]);
    if (fl.rf && i >= p.nsites)
      for (int ch = lane; ch < fl.nchunk_rf; ch += 32)
#pragma unroll
        for (int k = 0; k < 3; ++k) acc2(s[k], c[k], p.frf_f[((size_t)ch * 3 + k) * cap + i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float s2 = __shfl_xor_sync(0xffffffffu, s[k], o);
        const float c2 = __shfl_xor_sync(0xffffffffu, c[k], o);
        acc2p(s[k], c[k], s2, c2);
      }
  }
  if (lane != 0) return;
  float F[3];
  if (fl.use_total) {
    F[0] = (float)p.fx[i];
    F[1] = (float)p.fy[i];
    F[2] = (float)p.fz[i];
  } else {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (!fl.nofield) acc2(s[k], c[k], p.ffield_f[k * cap + i]);
      if (fl.is) acc2(s[k], c[k], p.fis_f[k * cap + i]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) F[k] = s[k] + c[k];
    if (!do_bd) {  // forces for the host (energy calls)
      p.fx[i] = F[0];
      p.fy[i] = F[1];
      p.fz[i] = F[2];
    }
  }
  if (do_bd) bd_move_f32(p, variant, seed, step, i, F);
}

// The same with one chunk of partials and no cross term (the cell list): a
// thread per particle (a warp's other lanes had nothing to add; 20,000 ions:
// 20 us -> 6 us).
__global__ void __launch_bounds__(128)
    k_assemble_one(const __grid_constant__ KP p, AssembleFlags fl, int do_bd, int variant,
                   uint64_t seed, uint64_t step) {
  after_prev();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.st->ntot) return;
  const int cap = p.cap;
  float F[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float s = i >= fl.ii_from ? p.fii_f[(size_t)k * cap + i] : 0.f, c = 0.f;
    if (!fl.nofield) acc2(s, c, p.ffield_f[k * cap + i]);
    if (fl.is) acc2(s, c, p.fis_f[k * cap + i]);
    F[k] = s + c;
  }
  if (do_bd) {
    bd_move_f32(p, variant, seed, step, i, F);
  } else {
    p.fx[i] = F[0];
    p.fy[i] = F[1];
    p.fz[i] = F[2];
  }
}

constexpr int kTileWarps = 16;  // as the fused loop's phase A: the same sums

__global__ void __launch_bounds__(32 * kTileWarps, 2)
    k_assemble_tiles(const __grid_constant__ KP p, AssembleFlags fl, int do_bd, int variant,
                     uint64_t seed, uint64_t step, int site_blocks) {
  after_prev();
  __shared__ float part[kTileWarps + 1][10][32];
  const int T = fl.wave ? live_tiles(p.st->ntot, p.nsites) : fl.ntile;
  if ((int)blockIdx.x >= site_blocks + T) return;  // the launch is for the host's bound
  assemble_tile<kTileWarps, 4>(p, ctx_asm_sys(p, T, n3_split_of(T, fl.wave), seed), fl, do_bd,
                               variant, step, blockIdx.x, site_blocks, part);
}

void launch_assemble(const KP &p, int ntot_ub, const AssembleFlags &fl,
                     int do_bd, int variant, uint64_t seed, uint64_t step,
                     cudaStream_t stream) {
  if (ntot_ub <= 0) return;
  if (fl.fp32_partials && fl.ntile > 0 && !fl.use_total) {
    const int sb = (p.nsites + 31) / 32;
    launch_after(k_assemble_tiles, sb + fl.ntile, 32 * kTileWarps, stream, p, fl, do_bd, variant,
                 seed, step, sb);
    return;
  }
  if (!fl.fp32_partials && fl.ntile > 0 && !fl.use_total) {
    const int sb = (p.nsites + 31) / 32;
    launch_after(fl.rf_ab ? k_assemble64<true> : k_assemble64<false>,
                 (sb + fl.ntile) * kAsm64Parts, kN64Threads, stream, p, fl, do_bd, variant, seed,
                 step, sb);
    return;
  }
  if (fl.fp32_partials && fl.ii && fl.nchunk_ii == 1 && !fl.rf && !fl.use_total) {
    launch_after(k_assemble_one, (ntot_ub + 127) / 128, 128, stream, p, fl, do_bd, variant, seed,
                 step);
    return;
  }
  const int nb = (ntot_ub + kAsmWarps - 1) / kAsmWarps;
  if (fl.fp32_partials)
    k_assemble_f32<<<nb, 32 * kAsmWarps, 0, stream>>>(p, fl, do_bd, variant, seed, step);
  else
    k_assemble<<<nb, 32 * kAsmWarps, 0, stream>>>(p, fl, do_bd, variant, seed, step);
}

}  // namespace bgpu
