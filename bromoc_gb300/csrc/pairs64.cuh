// The FP64 Newton-3 pair tile, shared by the FP64 pair kernel (energy.cu)
// and the fused FP64 BD loop (loop64.cu).
//
// GB300 issues an FP64 instruction for a warp every ~64 clocks and one per
// ~16 clocks on an SM, so the pair work is bound by the count of FP64
// instructions, whatever the memory does.  Hence:
//   - each unordered pair once (ion-ion law and RFPAR cross term together),
//     the reaction on the column ion taken from the same numbers;
//   - one reciprocal square root per term (CUDA's rsqrt) where the law's 1/r^2
//     and sqrt(1/r^2) were a division and a square root: ~50 FP64 instructions a pair with RFPAR and energies,
//     where the two target-centred kernels took ~330 for an unordered pair.
// Ions form tiles of 32.  A block takes an item: tile pair (I <= J) and one
// of S groups of its 32 diagonals; at diagonal k lane l (row ion l) meets
// column ion (l + k) mod 32, so the lanes of a step touch distinct columns.
// Eight warps share the group's diagonals.  S (n64_split) cuts the tile pairs
// of small systems finer, so that every SM has work.  The rare SRPMF pairs,
// whose law is three times the rest, go to two more warps beside the others:
// they screen all pairs of the item by their distance in FP32 (with a margin
// above its rounding), queue those near and evaluate them with full lanes, one
// the exponentials, the other sine and cosine (one warp for both was the
// longest chain of a small system's item, 5.5-7.7 us).
// Partials leave per item and side, summed over the warps in a fixed order.
// 2000-ion pore with RFPAR and energies: 627 us as two target-centred kernels,
// 255 us here (the FP64 pipe 85 % busy).
#pragma once
#include "launch.h"
#include "physics.cuh"

namespace bgpu {

// rows of partial sums: eight warps of diagonals, the SRPMF pairs
constexpr int kN64Warps = 9, kN64Threads = 32 * (kN64Warps + 1);

struct Law64 {
  double fct, e24, sg2;  // zero where the pair lacks the term; e24 = 6 epp4
  int flags, is;        // kEfp, kSrp; packed pair index
};

struct N64Smem {
  Law64 law[kN64Types * kN64Types];
  double pos[2][3][32];          // row, column tile
  double srfe[2][32], reff[2][32], q[2][32];
  float posf[2][3][32];
  int code[2][32];               // ion type | mobile << 16 | in the RFPAR map << 17, -1 absent
  double row[kN64Warps][5][32], col[kN64Warps][5][32];
  int hits[2][64];               // the two SRPMF warps' queues (alike)
  double sn[32], cs[32];
};

// The two SRPMF warps meet.
__device__ __forceinline__ void srp_pair_sync() { asm volatile("bar.sync 1, 64;" ::: "memory"); }

__device__ __forceinline__ void n64_laws(const KP &p, N64Smem &s) {
  const int nt = p.nion_t;
  for (int c = threadIdx.x; c < nt * nt; c += blockDim.x) {
    const int is = p.pidx[(p.ndna + c / nt) * p.nttyp + p.ndna + c % nt];
    Law64 l{};
    l.is = is;
    if (is >= 0) {
      const PairParam &q = p.pp[is];
      l.flags = q.flags;
      if (q.flags & kEfp)
        l.flags = kEfp;
      else {
        l.fct = q.flags & kChr ? q.fct : 0.0;
        l.e24 = q.flags & kLj ? 6.0 * q.epp4 : 0.0;
        l.sg2 = q.flags & kLj ? q.sgp2 : 0.0;
      }
    }
    s.law[c] = l;
  }
}

template <bool PBC>
__device__ __forceinline__ double n64_sep(const KP &p, const N64Smem &s, int l, int m, double &dx,
                                          double &dy, double &dz) {
  dx = s.pos[0][0][l] - s.pos[1][0][m];
  dy = s.pos[0][1][l] - s.pos[1][1][m];
  dz = s.pos[0][2][l] - s.pos[1][2][m];
  if (PBC) {  // extension mode: nearest image
    dx -= p.lx * rint(dx / p.lx);
    dy -= p.ly * rint(dy / p.ly);
    dz -= p.lz * rint(dz / p.lz);
  }
  return dx * dx + dy * dy + dz * dz;
}

// The item's SRPMF pairs (two warps, trig: the one with sine and cosine):
// forces into row[8] and col[8].
template <bool PBC>
__device__ __forceinline__ void n64_srpmf(const KP &p, N64Smem &s, bool trig, bool diag, int k0,
                                          int k1, double &esr) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, nt = p.nion_t;
  double rs[3] = {0.0, 0.0, 0.0}, cs[3] = {0.0, 0.0, 0.0};
  const float rx = s.posf[0][0][lane], ry = s.posf[0][1][lane], rz = s.posf[0][2][lane];
  const int rc = s.code[0][lane];
  float far = fmaxf(fmaxf(fabsf(rx), fabsf(ry)), fabsf(rz));
  far = fmaxf(far, fmaxf(fmaxf(fabsf(s.posf[1][0][lane]), fabsf(s.posf[1][1][lane])),
                         fabsf(s.posf[1][2][lane])));
  for (int o = 16; o > 0; o >>= 1) far = fmaxf(far, __shfl_xor_sync(kAll, far, o));
  // a component's rounding moves r^2 by under 4 r far 2^-24 near the cutoff
  const float rth = (float)p.rth, lim = rth + 1e-3f + 2e-6f * sqrtf(rth) * far;
  const float Lx = (float)p.lx, Ly = (float)p.ly, Lz = (float)p.lz;
  int *hits = s.hits[trig];
  int n = 0;
  auto flush = [&](int nb) {
    const bool act = lane < nb;
    const int ent = act ? hits[lane] : 0, l = ent & 31, m = ent >> 5;
    if (trig) {
      if (act) {
        double dx, dy, dz;
        const double d2 = n64_sep<PBC>(p, s, l, m, dx, dy, dz);
        const PairParam &q =
            p.pp[s.law[(s.code[0][l] & 0xffff) * nt + (s.code[1][m] & 0xffff)].is];
        // the law's angle is c3 pi (c1 - r)
        sincospi(q.c3 * (q.c1 - d2 * rsqrt(d2)), &s.sn[lane], &s.cs[lane]);
      }
      srp_pair_sync();
      srp_pair_sync();  // the values are read
      return;
    }
    double gx = 0.0, gy = 0.0, gz = 0.0, dx = 0.0, dy = 0.0, dz = 0.0, d2 = 0.0, idist = 0.0;
    double e1 = 0.0, e3 = 0.0, ft = 0.0, sn = 0.0, c = 0.0;
    const PairParam *q = p.pp;
    bool in = false, taper = false;
    if (act) {
      d2 = n64_sep<PBC>(p, s, l, m, dx, dy, dz);
      in = d2 <= p.rth && !(PBC && d2 >= p.rc2);
      q += s.law[(s.code[0][l] & 0xffff) * nt + (s.code[1][m] & 0xffff)].is;
      idist = rsqrt(d2);
      const double r = d2 * idist;
      taper = r >= p.srpx;
      e1 = q->c0 * exp((q->c1 - r) * q->c2);
      if (taper) ft = exp(-p.srpk * (r - p.srpx));
      e3 = q->c4 * pow6d(q->c1 * idist);
    }
    srp_pair_sync();
    if (act) {
      sn = s.sn[lane];
      c = s.cs[lane];
    }
    srp_pair_sync();
    if (in) {
      double e0 = fma(e1, c, e3);
      double dc = (-q->c2 * c + q->c3 * kPi * sn) * e1 - 6.0 * e3 * idist;
      if (taper) {
        const double fdf = ft - p.srpy;
        dc = dc * fdf - e0 * p.srpk * ft;
        e0 = e0 * fdf;
      }
      esr += e0;
      const double de = -dc * idist;
      gx = de * dx;
      gy = de * dy;
      gz = de * dz;
    }
    for (int t = 0; t < nb; ++t) {  // queue order
      const int lt = __shfl_sync(kAll, l, t), mt = __shfl_sync(kAll, m, t);
      const double vx = __shfl_sync(kAll, gx, t), vy = __shfl_sync(kAll, gy, t),
                   vz = __shfl_sync(kAll, gz, t);
      if (lane == lt) {
        rs[0] += vx;
        rs[1] += vy;
        rs[2] += vz;
      }
      if (lane == mt) {
        cs[0] -= vx;
        cs[1] -= vy;
        cs[2] -= vz;
      }
    }
    __syncwarp();
  };
  for (int k = k0; k < k1; ++k) {
    const int m = (lane + k) & 31, cc = s.code[1][m];
    bool hit = rc >= 0 && cc >= 0 && !(diag && k == 16 && lane >= 16) && ((rc | cc) >> 16 & 1);
    if (hit) {
      float dx = rx - s.posf[1][0][m], dy = ry - s.posf[1][1][m], dz = rz - s.posf[1][2][m];
      if (PBC) {
        dx -= Lx * rintf(dx / Lx);
        dy -= Ly * rintf(dy / Ly);
        dz -= Lz * rintf(dz / Lz);
      }
      hit = !(dx * dx + dy * dy + dz * dz > lim) &&
            (s.law[(rc & 0xffff) * nt + (cc & 0xffff)].flags & kSrp);
    }
    const unsigned b = __ballot_sync(kAll, hit);
    if (!b) continue;
    if (hit) hits[n + __popc(b & ((1u << lane) - 1u))] = lane | m << 5;
    n += __popc(b);
    __syncwarp();
    if (n >= 32) {
      flush(32);
      n -= 32;
      const int v = lane < n ? hits[32 + lane] : 0;
      __syncwarp();
      if (lane < n) hits[lane] = v;
      __syncwarp();
    }
  }
  if (n) flush(n);
  if (trig) return;
  for (int c = 0; c < 3; ++c) {
    s.row[kN64Warps - 1][c][lane] = (rc >> 16 & 1) && rc >= 0 ? rs[c] : 0.0;
    const int cc = s.code[1][lane];
    s.col[kN64Warps - 1][c][lane] = (cc >> 16 & 1) && cc >= 0 ? cs[c] : 0.0;
  }
}

// Item `item` (every thread of the block): partials of its tile pair and
// diagonal group into p.tp64, [item][side][component][lane]: the force and,
// with RF, the A and B sums of the RFPAR chain.  ii: with the ion-ion laws;
// srp: some of them have SRPMF.  e: the thread's energy sums (ecoul, 6 x elj,
// esrpmf, eefpot, erfpar), with EN.
template <bool RF, bool PBC, bool EN>
__device__ __forceinline__ void n64_item(const KP &p, int ntot, int T, int S, int item,
                                         int qforces, bool ii, bool srp, N64Smem &s,
                                         double e[5], int &err) {
  constexpr int NC = RF ? 5 : 3;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, nt = p.nion_t;
  const int m0 = p.nsites + p.nfix;
  int I, J;
  n3_pair(T, item / S, I, J);
  const bool diag = I == J;
  const int G = 32 / S, g0 = (item % S) * G;
  // the group's diagonals; each pair of a diagonal tile lies on 1 .. 16
  const int kb = diag ? max(g0, 1) : g0, ke = diag ? min(g0 + G, 17) : g0 + G;
  __syncthreads();  // the previous item's sums have left
  if (tid < 64) {
    const int side = w, i = p.nsites + 32 * (side ? J : I) + lane;
    double x = 0.0, y = 0.0, z = 0.0, sr = 0.0, re = 0.0, q = 0.0;
    int code = -1;
    if (i < ntot) {
      x = __ldcg(p.x + i);
      y = __ldcg(p.y + i);
      z = __ldcg(p.z + i);
      const int ti = abs(p.typei[i]);
      code = (p.nwtype[ti] - 1 - p.ndna) | (i >= m0 ? 1 << 16 : 0);
      if (RF) {
        q = p.cg[ti];
        sr = __ldcg(p.rf_srfe + i);
        re = __ldcg(p.rf_reff + i);
        code |= __ldcg(p.rf_in + i) ? 1 << 17 : 0;
      }
    }
    s.pos[side][0][lane] = x;
    s.pos[side][1][lane] = y;
    s.pos[side][2][lane] = z;
    s.posf[side][0][lane] = (float)x;
    s.posf[side][1][lane] = (float)y;
    s.posf[side][2][lane] = (float)z;
    s.code[side][lane] = code;
    if (RF) {
      s.srfe[side][lane] = sr;
      s.reff[side][lane] = re;
      s.q[side][lane] = side ? q : p.celec * q;
    }
  }
  __syncthreads();
  if (w < kN64Warps - 1) {
    const int rc = s.code[0][lane];
    const bool rmob = rc >> 16 & 1;
    double srt = 0.0, rft = 0.0, qt = 0.0;
    if (RF) {
      srt = s.srfe[0][lane];
      rft = s.reff[0][lane];
      qt = s.q[0][lane];
    }
    double f[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int c = 0; c < NC; ++c) s.col[w][c][lane] = 0.0;
    const int per = G / (kN64Warps - 1);
    const int k0 = max(kb, g0 + w * per), k1 = min(ke, g0 + (w + 1) * per);
    __syncwarp();
    for (int k = k0; k < k1; ++k) {
      const int m = (lane + k) & 31, cc = s.code[1][m];
      if (rc >= 0 && cc >= 0 && !(diag && k == 16 && lane >= 16)) {
        double dx, dy, dz;
        const double d2 = n64_sep<PBC>(p, s, lane, m, dx, dy, dz);
        const bool cmob = cc >> 16 & 1;
        // -E'/r of the ion-ion law and of the cross term
        double dii = 0.0, drf = 0.0;
        if (!(PBC && d2 >= p.rc2)) {
          if (ii && (rmob || cmob)) {
            const Law64 &lw = s.law[(rc & 0xffff) * nt + (cc & 0xffff)];
            double de;
            if (lw.flags & kEfp) {
              double dist;
              const double u = efp64(p, p.pp[lw.is], d2, de, dist, err);
              if (EN) e[3] += u;
            } else {
              const double ir = rsqrt(d2), ir2 = ir * ir;
              const double cofo = lw.fct * ir;
              double d6 = lw.sg2 * ir2;
              d6 = d6 * d6 * d6;
              const double t = lw.e24 * d6;
              if (EN) {
                e[0] += cofo;
                e[1] = fma(t, d6 - 1.0, e[1]);  // 6 x elj
              }
              de = fma(t, fma(2.0, d6, -1.0), cofo) * ir2;
            }
            dii = de;
          }
          if (RF && (rc & cc & (1 << 17))) {
            // rfpar.f90:177-223: the later ion of the two mobile, the
            // earlier one's srfe not zero
            const double src = s.srfe[1][m];
            const bool ci = !diag || m > lane;
            if ((ci ? cmob : rmob) && (ci ? srt : src) != 0.0) {
              const double rec = s.reff[1][m];
              const double rij = rec * rft;
              const double rd = rsqrt(fma(rij, rij, d2));
              const double a0 = qt * s.q[1][m];
              const double a1 = a0 * (rij * rd), srij = src * srt;
              if (EN) e[4] = fma(a1, srij, e[4]);
              const double a2 = a0 * srij * (rd * rd * rd);
              const double a3 = a2 * fma(0.5, rij, d2);
              f[3] = fma(-a1, src, f[3]);
              f[4] = fma(-a3, rec, f[4]);
              s.col[w][3][m] = fma(-a1, srt, s.col[w][3][m]);
              s.col[w][4][m] = fma(-a3, rft, s.col[w][4][m]);
              if (rmob && cmob)
                dii = fma(a2, rij, dii);
              else
                drf = a2 * rij;
            }
          }
        }
        // the law acts on mobile ions, the cross term on both
        double dr = dii, dc = dii;
        if (!(rmob && cmob)) {
          dr = (rmob ? dii : 0.0) + drf;
          dc = (cmob ? dii : 0.0) + drf;
        }
        f[0] = fma(dr, dx, f[0]);
        f[1] = fma(dr, dy, f[1]);
        f[2] = fma(dr, dz, f[2]);
        s.col[w][0][m] = fma(-dc, dx, s.col[w][0][m]);
        s.col[w][1][m] = fma(-dc, dy, s.col[w][1][m]);
        s.col[w][2][m] = fma(-dc, dz, s.col[w][2][m]);
      }
      __syncwarp();
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) s.row[w][c][lane] = f[c];
  } else if (srp) {
    double esr = 0.0;
    n64_srpmf<PBC>(p, s, w == kN64Warps, diag, kb, ke, esr);
    if (EN) e[2] += esr;
  }
  __syncthreads();
  double *out = p.tp64 + (size_t)item * 2 * NC * 32;
  for (int o = tid; o < 2 * NC * 32; o += kN64Threads) {
    const int side = o / (NC * 32), c = (o / 32) % NC;
    const double(*v)[5][32] = side ? s.col : s.row;
    double a = 0.0;
#pragma unroll
    for (int u = 0; u < kN64Warps - 1; ++u) a += v[u][c][lane];
    if (srp && c < 3) a += v[kN64Warps - 1][c][lane];
    out[o] = qforces ? a : 0.0;
  }
}

}  // namespace bgpu
