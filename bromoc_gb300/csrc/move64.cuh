// FP64 BD move (dynamics0-3.mono.f90, dynamics0nuc.f90, fixcoor.f90,
// countions.f90) and the assembly of the FP64 Newton-3 partials, shared by the
// assembly kernels (dyn.cu) and the fused FP64 loop (loop64.cu).
#pragma once
#include "launch.h"
#include "move32.cuh"
#include "pairs64.cuh"
#include "physics.cuh"

namespace bgpu {

__device__ __forceinline__ void clamp_bd(double bdmax, double &d) {
  if (fabs(d) > bdmax) d = fsign(bdmax, d);
}

__device__ __forceinline__ void wrap1(double lo, double L, double &v) {
  if (v < lo)
    v += L;
  else if (v >= lo + L)
    v -= L;
}

// fixcoor.f90:19-68; in the extension mode (periodic box) one wrap into the
// box per axis instead of the clamp (BD moves are far shorter than a box).
__device__ __forceinline__ void fixcoor(const KP &p, double &x, double &y,
                                        double &z) {
  if (p.periodic) {
    wrap1(p.lx2m, p.lx, x);
    wrap1(p.ly2m, p.ly, y);
    wrap1(p.lz2m, p.lz, z);
    return;
  }
  if (p.shape == 1) {  // sphere: reflect through the wall
    const double r2 = (x - p.cx) * (x - p.cx) + (y - p.cy) * (y - p.cy) +
                      (z - p.cz) * (z - p.cz);
    if (r2 > p.rsphe2) {
      const double lzrad = 2.0 * p.rsphe / sqrt(r2) - 1.0;
      x = lzrad * (x - p.cx) + p.cx;
      y = lzrad * (y - p.cy) + p.cy;
      z = lzrad * (z - p.cz) + p.cz;
    }
  } else if (p.shape == 2) {  // elliptic cylinder
    const double ex = (x - p.cx) * p.iecx, ey = (y - p.cy) * p.iecy;
    const double r2 = ex * ex + ey * ey;
    if (r2 > 1.0) {
      const double r = 0.999999999999999 / sqrt(r2);
      x = r * (x - p.cx) + p.cx;
      y = r * (y - p.cy) + p.cy;
    }
    if (z < p.lz2m)
      z = p.lz2m;
    else if (z > p.lz2p)
      z = p.lz2p;
  } else {  // box: clamp
    if (x < p.lx2m)
      x = p.lx2m;
    else if (x > p.lx2p)
      x = p.lx2p;
    if (y < p.ly2m)
      y = p.ly2m;
    else if (y > p.ly2p)
      y = p.ly2p;
    if (z < p.lz2m)
      z = p.lz2m;
    else if (z > p.lz2p)
      z = p.lz2p;
  }
}


// countions.f90:25-31
__device__ __forceinline__ void count_crossings(const KP &p, int itype, double zold,
                                                double z) {
  const int it = itype - p.nold - 1;
  for (int j = 0; j < p.cntpts; ++j) {
    const double zc = p.zcont[j];
    if (zold < zc && z >= zc)
      atomicAdd(&p.nforward[it * p.cntpts + j], 1);
    else if (zold >= zc && z < zc)
      atomicAdd(&p.nbackward[it * p.cntpts + j], 1);
  }
}

// BD move of particle i under the assembled force f with the noise g
// (dynamics*.f90), FP64.
__device__ __forceinline__ void bd_move(const KP &p, int variant, int i, const double f[3],
                                        const double g[3]) {
  const int m0 = p.nsites + p.nfix;
  if (i < m0 && (i >= p.nsites || !p.stfree[i])) return;  // fixed ions, frozen sites
  if (i < p.nsites) {  // dynamics0nuc.f90:31-44
    double dx = f[0] * p.fact0n1, dy = f[1] * p.fact0n1, dz = f[2] * p.fact0n1;
    clamp_bd(p.bdmax, dx);
    clamp_bd(p.bdmax, dy);
    clamp_bd(p.bdmax, dz);
    double x = p.x[i] + dx + p.fact0n2 * g[0];
    double y = p.y[i] + dy + p.fact0n2 * g[1];
    double z = p.z[i] + dz + p.fact0n2 * g[2];
    if (!p.qdnafree) fixcoor(p, x, y, z);
    p.x[i] = x;
    p.y[i] = y;
    p.z[i] = z;
    return;
  }
  const int itype = abs(p.typei[i]);
  const double zold = p.z[i];
  double fact1, fact2, dD[3];
  diff_model(p, variant, i, itype, zold, fact1, fact2, dD);
  double dx = f[0] * fact1, dy = f[1] * fact1, dz = f[2] * fact1;
  clamp_bd(p.bdmax, dx);
  clamp_bd(p.bdmax, dy);
  clamp_bd(p.bdmax, dz);
  double x = p.x[i] + dx + fact2 * g[0] + dD[0];
  double y = p.y[i] + dy + fact2 * g[1] + dD[1];
  double z = zold + dz + fact2 * g[2] + dD[2];
  if (p.qcountion) count_crossings(p, itype, zold, z);
  fixcoor(p, x, y, z);
  p.x[i] = x;
  p.y[i] = y;
  p.z[i] = z;
}

// What the move of particle i along one axis needs besides force and noise;
// loaded while the partials are summed.
struct AxisIn {
  double x, fact1, fact2;
  int itype;
  bool moves;
};
__device__ __forceinline__ AxisIn axis_in(const KP &p, int i, int k) {
  AxisIn a;
  const bool site = i < p.nsites;
  a.moves = site ? p.stfree[i] != 0 : i >= p.nsites + p.nfix;  // frozen sites, fixed ions
  a.x = (k == 0 ? p.x : (k == 1 ? p.y : p.z))[i];
  a.itype = site ? 0 : abs(p.typei[i]);
  a.fact1 = site ? p.fact0n1 : p.fact1a[a.itype];
  a.fact2 = site ? p.fact0n2 : p.fact2a[a.itype];
  return a;
}
// bd_move along axis k of a box (or periodic box) with dynamics0.
__device__ __forceinline__ void bd_move_axis(const KP &p, int i, int k, const AxisIn &a, double f,
                                             double g) {
  if (!a.moves) return;
  const bool site = i < p.nsites;
  const int itype = a.itype;
  double *x = k == 0 ? p.x : (k == 1 ? p.y : p.z);
  double d = f * a.fact1;
  clamp_bd(p.bdmax, d);
  const double old = a.x;
  double v = old + d + a.fact2 * g;
  if (k == 2 && !site && p.qcountion) count_crossings(p, itype, old, v);
  if (!(site && p.qdnafree)) {
    const double lo = k == 0 ? p.lx2m : (k == 1 ? p.ly2m : p.lz2m);
    const double hi = k == 0 ? p.lx2p : (k == 1 ? p.ly2p : p.lz2p);
    if (p.periodic)
      wrap1(lo, k == 0 ? p.lx : (k == 1 ? p.ly : p.lz), v);
    else if (v < lo)
      v = lo;
    else if (v > hi)
      v = hi;
  }
  x[i] = v;
}

// Noise component c of slot i at step `step`: bd_noise3's value of it.
__device__ __forceinline__ double bd_noise_one(uint64_t seed, uint64_t step, uint32_t slot,
                                               int c) {
  uint32_t w[4];
  philox4x32_10(slot, (uint32_t)(c >> 1), (uint32_t)step,
                ((uint32_t)(step >> 32) & 0x00FFFFFFu) | (1u << 24), (uint32_t)seed,
                (uint32_t)(seed >> 32), w);
  return c & 1 ? box_muller(w[2], w[3]) : box_muller(w[0], w[1]);
}

struct Asm64Smem {
  double part[kN64Warps + 1][5][32];
  double tot[5][32];
  double g[3][32];
};

// Force and move of the particles of one tile (every thread of the block):
// site tiles are blk 0 .. sb - 1, then the pair kernel's ion tiles; of a tile
// only part h of nh (32 / nh particles).  Warps 3 .. 9 sum the tile's
// partials, each its share with the loads of several entries in flight; warps
// 0 .. 2 draw the noise meanwhile, a component each (the chain of a normal
// deviate is ~4 us; one lane of a particle drew all three in turn before, a
// particle a warp: 23 us for 260 ions), unless it is given (noise, [3][cap]).
template <bool LOOP, bool RF>
__device__ __forceinline__ void assemble64(const KP &p, const AssembleFlags &fl, int do_bd,
                                           int variant, uint64_t seed, uint64_t step, int ntot,
                                           int blk, int sb, int h, int nh, const double *noise,
                                           Asm64Smem &s) {
  constexpr int kSum0 = 3, kSumW = kN64Warps + 1 - kSum0, NC = RF ? 5 : 3, kFly = RF ? 4 : 8;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, cap = p.cap;
  const bool ionblk = blk >= sb;
  const int t = blk - sb, T = live_tiles(ntot, p.nsites), S = n64_split(T);
  const int i = ionblk ? p.nsites + 32 * t + lane : 32 * blk + lane;
  const bool own = lane / (32 / nh) == h && i < ntot && (ionblk || i < p.nsites);
  // a box and the plain move keep the components apart: a warp each (a warp's
  // FP64 chain is the latency here)
  const bool apart = variant == 0 && p.shape == 0;
  double fo = 0.0, d1 = 0.0, d2 = 0.0;  // warp w < 3: of component w
  AxisIn in{};
  if (w < kSum0) {
    if (own) {
      if (do_bd && apart) in = axis_in(p, i, w);
      if (!fl.nofield) fo = __ldcg(p.ffield + w * cap + i);
      if (fl.is) fo += p.fis[w * cap + i];
      if (RF && ionblk) {
        d1 = __ldcg(p.rf_d1 + 3 * (size_t)i + w);
        d2 = __ldcg(p.rf_d2 + 3 * (size_t)i + w);
      }
    }
    if (do_bd && own)
      s.g[w][lane] = noise ? __ldcg(noise + (size_t)w * cap + i)
                           : bd_noise_one(seed, step, (uint32_t)i, w);
  } else {
    double a[NC] = {};
    if (ionblk && own) {
      // entries by group e % S: the diagonal pair's column side, then the
      // tiles (an order that does not depend on T)
      const int n = (T + 1) * S;
      for (int e0 = w - kSum0; e0 < n; e0 += kFly * kSumW) {
        double v[kFly][NC];
#pragma unroll
        for (int j = 0; j < kFly; ++j) {
          const int e = e0 + j * kSumW, u = e / S - 1;
          const bool on = e < n;
          const int q = u < 0 ? n3_index(T, t, t)
                              : (u < t ? n3_index(T, u, t) : n3_index(T, t, u));
          const int side = u < t;  // u < 0 too
          const double *o = p.tp64 + (((size_t)q * S + e % S) * 2 + side) * NC * 32 + lane;
#pragma unroll
          for (int c = 0; c < NC; ++c) v[j][c] = on ? __ldcg(o + 32 * c) : 0.0;
        }
#pragma unroll
        for (int j = 0; j < kFly; ++j)
          if (e0 + j * kSumW < n)
#pragma unroll
            for (int c = 0; c < NC; ++c) a[c] += v[j][c];
      }
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) s.part[w][c][lane] = a[c];
  }
  __syncthreads();
  if (w < NC) {
    double a = 0.0;
#pragma unroll
    for (int u = kSum0; u < kSum0 + kSumW; ++u) a += s.part[u][w][lane];
    s.tot[w][lane] = a;
  }
  __syncthreads();
  if (w < kSum0 && own) {
    double v = s.tot[w][lane];
    if (RF) v += s.tot[3][lane] * d1 + s.tot[4][lane] * d2;
    v += fo;
    if (!LOOP) (w == 0 ? p.fx : (w == 1 ? p.fy : p.fz))[i] = v;
    if (do_bd && apart)
      bd_move_axis(p, i, w, in, v, s.g[w][lane]);
    else if (do_bd)
      s.part[0][w][lane] = v;
  }
  if (!do_bd || apart) return;  // block-uniform
  __syncthreads();
  if (w == 0 && own) {
    const double f[3] = {s.part[0][0][lane], s.part[0][1][lane], s.part[0][2][lane]};
    const double g[3] = {s.g[0][lane], s.g[1][lane], s.g[2][lane]};
    bd_move(p, variant, i, f, g);
  }
}

}  // namespace bgpu
