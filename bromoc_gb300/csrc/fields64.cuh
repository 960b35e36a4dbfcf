// FP64 single-particle terms, four lanes a particle: shared by the field
// kernel (fields.cu) and the fused FP64 loop (loop64.cu).
//
// An FP64 instruction takes its pipe 64 clocks whatever the lanes do, so the
// work is spread for full warps rather than short chains: lane = 4 e + g, e the
// warp's particle (of eight), g the map: 0 static field, 1 repulsion, 2 gsrfen
// (srfe), 3 greff (reff).  A lane walks its map's eight nodes; the node sum
// factors by axis (over c, then b, then a), which takes 4 multiply-adds a node
// pair instead of 11 products a node.  The 27-point B-spline repulsion takes a
// second pass: three lanes form the weights of an axis each, and the four
// share the 27 nodes by rows.  About 110 and 120 FP64 instructions for eight
// particles; with a warp a particle and a node a lane they were 190 and 100
// for one.  ENERGY of 2000 ions, B-spline repulsion: 46 -> 19 us.
#pragma once
#include "fields32.cuh"
#include "physics.cuh"

namespace bgpu {

// Trilinear weights of the two nodes of one axis (w = 1 - |x - n dcel| / dcel,
// staticf1.f90:78-88) and their signs, zero where the reference takes no slope
// (a weight within kRsmall of 0 or 1).
__device__ __forceinline__ void axis_pair(double xi, int n0, double dcel, double idcel,
                                          double w[2], double s[2]) {
#pragma unroll
  for (int o = 0; o < 2; ++o) {
    const double d = xi - (n0 + o) * dcel;
    w[o] = 1.0 - fabs(d) * idcel;
    s[o] = w[o] < 1.0 - kRsmall && w[o] > kRsmall ? (d >= 0.0 ? 1.0 : -1.0) : 0.0;
  }
}

__device__ __forceinline__ double quad_from(double v, int g) {
  return __shfl_sync(0xffffffffu, v, (threadIdx.x & 28) | g);
}
__device__ __forceinline__ int quad_from(int v, int g) {
  return __shfl_sync(0xffffffffu, v, (threadIdx.x & 28) | g);
}
__device__ __forceinline__ double quad_sum(double v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
__device__ __forceinline__ double pick3(int k, double a, double b, double c) {
  return k == 0 ? a : (k == 1 ? b : c);
}

// Every single-particle term of the quad's particle i in FP64 (a whole warp;
// on: the particle exists): forces into ffield, the RFPAR gathers into rf_*,
// energies (ememb, egsbpa, evdwgd, erfpar) into eo on lanes g == 0.  Positions
// are read past L1: in the fused loop they were written in the same launch.
__device__ __forceinline__ void fields_quad_f64(const KP &p, int i, bool on, uint32_t mask,
                                                int qforces, double eo[4]) {
  const int g = threadIdx.x & 3;
  const bool site = i < p.nsites;
  const bool fixed = !site && i < p.nsites + p.nfix;
  const bool qf = qforces != 0;
  double x = 0.0, y = 0.0, z = 0.0, charge = 0.0;
  int iontype = 0, itype2 = 0;
  if (on) {
    x = __ldcg(p.x + i);
    y = __ldcg(p.y + i);
    z = __ldcg(p.z + i);
    iontype = site ? 0 : abs(p.typei[i]);
    itype2 = site ? p.typtyp[i] : p.nwtype[iontype];
    charge = site ? p.sitecharge[i] : p.cg[iontype];
  }
  // the lane's map
  const Grid3 &g1 = p.g1, &g2 = p.g2, &g3 = p.g3;
  const int mp = g < 2 ? g : 2;
  const double trx = pick3(mp, g1.tranx, g2.tranx, g3.tranx),
               try_ = pick3(mp, g1.trany, g2.trany, g3.trany),
               trz = pick3(mp, g1.tranz, g2.tranz, g3.tranz),
               xbc = pick3(mp, g1.xbcen, g2.xbcen, g3.xbcen),
               ybc = pick3(mp, g1.ybcen, g2.ybcen, g3.ybcen),
               zbc = pick3(mp, g1.zbcen, g2.zbcen, g3.zbcen);
  const bool spl = !p.qtrln;
  bool act = false;  // the particle is in the lane's map
  if (on) {
    bool want;
    if (g == 0)
      want = (mask & 4u) && p.qphix && !fixed && (!site || charge != 0.0);
    else if (g == 1)
      want = (mask & 8u) && p.qphiv && !fixed;
    else
      want = (mask & 16u) && p.qrfpar && !site;
    const double m = g == 1 && spl ? g2.dcel : 0.0;
    const double zhi = g == 1 ? p.vzmax : zbc + trz, zlo = g == 1 ? p.vzmin : zbc - trz;
    act = want && x <= xbc + trx - m && x >= xbc - trx + m && y <= ybc + try_ - m &&
          y >= ybc - try_ + m && z <= zhi && z >= zlo;
  }
  size_t vifir = 0;
  double esvdw = 0.0;
  int vit2 = 0;
  if (g == 1 && act) phiv_select(p, i, iontype, vifir, esvdw, vit2);

  // ---- trilinear maps ----------------------------------------------------
  double le = 0.0, lf0 = 0.0, lf1 = 0.0, lf2 = 0.0, lsum = 0.0;
  if (act && !(g == 1 && spl)) {
    const double dcel = pick3(mp, g1.dcel, g2.dcel, g3.dcel),
                 idc = pick3(mp, g1.idcel, g2.idcel, g3.idcel);
    const int nx = mp == 0 ? g1.nclx : (mp == 1 ? g2.nclx : g3.nclx),
              ny = mp == 0 ? g1.ncly : (mp == 1 ? g2.ncly : g3.ncly),
              nz = mp == 0 ? g1.nclz : (mp == 1 ? g2.nclz : g3.nclz);
    const double xi = x + trx - xbc, yi = y + try_ - ybc, zi = z + trz - zbc;
    int ix = (int)(xi * idc), iy = (int)(yi * idc), iz = (int)(zi * idc);
    if (ix == nx - 1) ix = nx - 2;
    if (iy == ny - 1) iy = ny - 2;
    if (iz == nz - 1) iz = nz - 2;
    const size_t node = (g == 1 ? vifir : (g >= 2 ? rfpar_ifir(p, iontype) : 0)) +
                        (size_t)ix * ny * nz + (size_t)iy * nz + iz;
    float v[8];
    if (g == 0) {
#pragma unroll
      for (int n = 0; n < 8; ++n)
        v[n] = __ldg(p.phix + node + (size_t)(n >> 2) * ny * nz + (size_t)((n >> 1) & 1) * nz +
                     (n & 1));
    } else if (g == 1) {
#pragma unroll
      for (int n = 0; n < 8; ++n)
        v[n] = __ldg(p.phiv + node + (size_t)(n >> 2) * ny * nz + (size_t)((n >> 1) & 1) * nz +
                     (n & 1));
    } else {
      float gs[8];
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const size_t o =
            node + (size_t)(n >> 2) * ny * nz + (size_t)((n >> 1) & 1) * nz + (n & 1);
        gs[n] = __ldg(p.gsrfen + o);
        v[n] = g == 2 ? gs[n] : __ldg(p.greff + o);
      }
      // the reference leaves the innermost (z) loop at a zero gsrfen node:
      // node (a,b,1) counts only if (a,b,0) and (a,b,1) are nonzero, node
      // (a,b,0) only if it is nonzero (rfpar.f90:121)
#pragma unroll
      for (int n = 0; n < 8; n += 2) {
        if (gs[n] == 0.0f || gs[n + 1] == 0.0f) v[n + 1] = 0.0f;
        if (gs[n] == 0.0f) v[n] = 0.0f;
      }
    }
    double wa[2], sa[2], wb[2], sb[2], wc[2], sc[2];
    axis_pair(xi, ix, dcel, idc, wa, sa);
    axis_pair(yi, iy, dcel, idc, wb, sb);
    axis_pair(zi, iz, dcel, idc, wc, sc);
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      double e = 0.0, fb = 0.0, fc = 0.0;
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const double v0 = v[4 * a + 2 * b], v1 = v[4 * a + 2 * b + 1];
        const double s = wc[0] * v0 + wc[1] * v1, d = sc[0] * v0 + sc[1] * v1;
        e += wb[b] * s;
        fb += sb[b] * s;
        fc += wb[b] * d;
      }
      le += wa[a] * e;
      lf0 += sa[a] * e;
      lf1 += wa[a] * fb;
      lf2 += wa[a] * fc;
    }
    if (g == 1) {  // small whole numbers: exact in single precision
      float t = 0.0f;
#pragma unroll
      for (int n = 0; n < 8; ++n) t += v[n];
      lsum = t;
    }
    const double k =
        g == 0 ? p.celec * charge : (g == 1 ? esvdw : (g == 2 ? 1.0 : (double)p.sqrfac));
    le *= k;
    const double kf = qf ? (g >= 2 ? -k : k) * idc : 0.0;  // rfpar.f90:131-144 accumulates -sign
    lf0 *= kf;
    lf1 *= kf;
    lf2 *= kf;
  }

  // ---- 27-point B-spline repulsion ----------------------------------------
  if ((mask & 8u) && p.qphiv && spl) {  // warp-uniform
    const bool in = quad_from((int)act, 1) != 0;
    const size_t vf = __shfl_sync(0xffffffffu, (unsigned long long)vifir, (threadIdx.x & 28) | 1);
    // lanes 0..2: the weights and slopes of the three nodes of an axis
    const int ax = g < 2 ? g : 2, nc = ax == 0 ? g2.nclx : (ax == 1 ? g2.ncly : g2.nclz);
    const double t = pick3(ax, x + g2.tranx - g2.xbcen, y + g2.trany - g2.ybcen,
                           z + g2.tranz - g2.zbcen);
    int n0 = 1, nzb = 0;
    double wm[3], dm[3];
    if (in) n0 = (int)llround(t * g2.idcel);  // nint: half away from zero
    if (n0 == 0) n0 = 1;
    if (n0 == nc - 1) n0 = nc - 2;
#pragma unroll
    for (int o = 0; o < 3; ++o) {
      const double u = 1.5 - (t - (n0 - 1 + o) * g2.dcel) * g2.idcel;
      wm[o] = m3(u);
      dm[o] = dm3(u);
      // a node is visited when none of its axes is cut off
      // (vdwgd1spln.f90:118,125,132)
      if (wm[o] != 0.0 || dm[o] != 0.0) nzb |= 1 << o;
    }
    double A[3], dA[3], B[3], dB[3], C[3], dC[3];
#pragma unroll
    for (int o = 0; o < 3; ++o) {
      A[o] = quad_from(wm[o], 0);
      dA[o] = quad_from(dm[o], 0);
      B[o] = quad_from(wm[o], 1);
      dB[o] = quad_from(dm[o], 1);
      C[o] = quad_from(wm[o], 2);
      dC[o] = quad_from(dm[o], 2);
    }
    const int ix = quad_from(n0, 0) - 1, iy = quad_from(n0, 1) - 1, iz = quad_from(n0, 2) - 1;
    const int na = quad_from(nzb, 0), nb = quad_from(nzb, 1), nz = quad_from(nzb, 2);
    double e1 = 0.0, f0 = 0.0, f1 = 0.0, f2 = 0.0;
    float s1 = 0.0f;  // whole numbers
#pragma unroll
    for (int q = 0; q < 3; ++q) {  // rows (k, l): g, g + 4, and 8 on lane 0
      const int r = g + 4 * q, k = r / 3, l = r - 3 * k;
      if (!in || r > 8 || !((na >> k) & 1) || !((nb >> l) & 1)) continue;
      const int8_t *row = p.phiv + vf + (size_t)(ix + k) * g2.ncly * g2.nclz +
                          (size_t)(iy + l) * g2.nclz + iz;
      double e = 0.0, d = 0.0;
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        const float ph = (nz >> m) & 1 ? (float)__ldg(row + m) : 0.0f;
        s1 += ph;
        e += C[m] * (double)ph;
        d += dC[m] * (double)ph;
      }
      const double a = pick3(k, A[0], A[1], A[2]), da = pick3(k, dA[0], dA[1], dA[2]),
                   b = pick3(l, B[0], B[1], B[2]), db = pick3(l, dB[0], dB[1], dB[2]);
      e1 += a * b * e;
      f0 += da * b * e;
      f1 += a * db * e;
      f2 += a * b * d;
    }
    e1 = quad_sum(e1);
    f0 = quad_sum(f0);
    f1 = quad_sum(f1);
    f2 = quad_sum(f2);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
    if (g == 1 && act) {
      const double kf = qf ? esvdw * g2.idcel : 0.0;
      le = e1 * esvdw;
      lf0 = f0 * kf;
      lf1 = f1 * kf;
      lf2 = f2 * kf;
      lsum = s1;
    }
  }

  // ---- the quad's sums in its lane 0 --------------------------------------
  const bool do_phix = act, phiv_ok = quad_from((int)act, 1) != 0,
             do_rf = quad_from((int)act, 2) != 0;
  const double e_v = quad_from(le, 1), f0_v = quad_from(lf0, 1), f1_v = quad_from(lf1, 1),
               f2_v = quad_from(lf2, 1), s_v = quad_from(lsum, 1);
  const double srfe = quad_from(le, 2), d10 = quad_from(lf0, 2), d11 = quad_from(lf1, 2),
               d12 = quad_from(lf2, 2);
  const double reff = quad_from(le, 3), d20 = quad_from(lf0, 3), d21 = quad_from(lf1, 3),
               d22 = quad_from(lf2, 3);
  vit2 = quad_from(vit2, 1);
  if (g != 0 || !on) return;
  double f[3] = {0.0, 0.0, 0.0};
  if ((mask & 2u) && p.qmemb) {
    if (membrane_one(p, itype2, charge, x, y, z, !fixed && qf, false, eo[0], f))
      atomicAdd(&p.warn[itype2], 1);
  }
  if (do_phix) {
    eo[1] = le;
    f[0] += lf0;
    f[1] += lf1;
    f[2] += lf2;
  }
  if (phiv_ok) {
    eo[2] = e_v;
    f[0] += f0_v;
    f[1] += f1_v;
    f[2] += f2_v;
    if (s_v >= (spl ? p.thold27 : p.thold8)) atomicAdd(&p.warn[vit2], 1);
  }
  if ((mask & 16u) && p.qrfpar && !site) {
    // zero outside the map, where the lanes kept zeros
    const double d1[3] = {d10, d11, d12}, d2[3] = {d20, d21, d22};
    p.rf_in[i] = do_rf ? 1 : 0;
    p.rf_srfe[i] = srfe;
    p.rf_reff[i] = reff;
    for (int k = 0; k < 3; ++k) {
      p.rf_d1[3 * i + k] = d1[k];
      p.rf_d2[3 * i + k] = d2[k];
    }
    if (do_rf && !fixed) {  // self term, rfpar.f90:161-176
      const double tau = p.celec * charge;
      const double aux = tau * charge * srfe;
      eo[3] = 0.5 * aux * srfe;
      if (qf) {
        f[0] -= aux * d1[0];
        f[1] -= aux * d1[1];
        f[2] -= aux * d1[2];
      }
    }
  }
  if (p.qproxdiff && !site)  // dids is rebuilt by the ion-site pass
    for (int m = 0; m < 5; ++m) p.dids[5 * (size_t)i + m] = 0.0;
  p.ffield[i] = f[0];
  p.ffield[p.cap + i] = f[1];
  p.ffield[2 * p.cap + i] = f[2];
}

}  // namespace bgpu
