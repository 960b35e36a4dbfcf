// Reaction field of the MMIJ basis (gsbpmod), FP64 in both modes.
//
// ENERGY (rect_rf1.f90, sphe_rf1.f90):
//   k_mmij_tab    one thread per particle (RECTBOX: and axis): in-region flag
//                 and the basis tables of its position (RECTBOX: Legendre
//                 values and slopes per axis; SPHERE: r^l, cos/sin(m phi),
//                 P_l^m and dP_l^m/d cos(theta)), into its row of
//                 MmijDev::tab;
//   k_mmij_coef   one thread per basis function and ion chunk: the chunk's
//                 sum of q_i b(r_i) into coefp (no atomics);
//   k_mmij_sum    a warp per basis function: coef, its chunk sums; the SPHERE
//                 forces' 10/sin(theta) of the last ion in the sphere;
//   k_mmij_rows   one warp per row: mq = M coef (x rfscal for RECTBOX), lanes
//                 over the row, a fixed shuffle tree; the last block done
//                 forms egsbpb = celec sum coef mq / 2 into an energy slot;
//   k_mmij_force  eight lanes per ion in the region, every eighth function
//                 each: -q celec sum_k grad b_k mq_k, added to the field
//                 forces (ffield / ffield_f).
// Every kernel here is a chain of FP64 instructions of ~64 clocks each, so its
// time is the longest thread's count of them: chunks of 16 ions (of 256 the
// coefficients of 500 ions and 80 functions took 80 us, on two blocks) and
// eight lanes an ion in the forces (43 us with one).
// INTERACT (rect_rf0.f90, sphe_rf0.f90): the same tables with particle j at
// the trial position (an extra row for an insertion trial), coef2 = coef -
// q_j b(r_j), then per row k the terms of E(coef) - E(coef2) over l >= k
// and their sum, added to INTERACT's result.  Particles outside the region,
// and j that is not a mobile ion, contribute nothing.
#include <algorithm>

#include "launch.h"
#include "physics.cuh"

namespace bgpu {

constexpr int kMmThreads = 128;

template <bool F32>
__device__ __forceinline__ void mm_pos(const KP &p, int i, double r[3]) {
  if (F32) {
    const float4 h = p.pk1[i], l = p.pk2[i];
    r[0] = (double)h.x + (double)l.x;
    r[1] = (double)h.y + (double)l.y;
    r[2] = (double)h.z + (double)l.z;
  } else {
    r[0] = p.x[i];
    r[1] = p.y[i];
    r[2] = p.z[i];
  }
}

// Sphere table layout within a row of tab
struct SpheLayout {
  int lmax, mc, w;  // w: (l, m) row width of P and dP
  __host__ __device__ int ar() const { return 0; }
  __host__ __device__ int ac() const { return lmax + 1; }
  __host__ __device__ int as() const { return lmax + 1 + mc + 1; }
  __host__ __device__ int ap() const { return lmax + 1 + 2 * (mc + 1); }
  __host__ __device__ int adp() const { return ap() + (lmax + 2) * w; }
  __host__ __device__ int ang() const { return adp() + (lmax + 2) * w; }  // st, ct, cp, sp
  __host__ __device__ int width() const { return ang() + 4; }
};

__host__ __device__ inline SpheLayout sphe_layout(int nmpol) {
  SpheLayout L;
  L.lmax = nmpol - 1;
  L.mc = L.lmax > 3 ? L.lmax : 3;
  L.w = L.lmax + 2;
  return L;
}

// The tables of one position into t; false when outside the region.
// istnum is 10 for ENERGY (sphe_rf1.f90:46) and 1 for INTERACT.  RECTBOX: of
// axis `axis` alone (the region test is of all).
__device__ bool mm_tables(const KP &p, const double r[3], double istnum, int axis, double *t,
                          double &ist) {
  const MmijDev &m = p.mm;
  ist = 0.0;
  if (m.rect) {
    if (!(r[0] >= -m.xmax && r[0] <= m.xmax && r[1] >= -m.ymax && r[1] <= m.ymax &&
          r[2] >= -m.zmax && r[2] <= m.zmax))
      return false;
    const double sc[3] = {m.xscal, m.yscal, m.zscal};
    const int np[3] = {m.nx, m.ny, m.nz};
    int off = 0;
    for (int a = 0; a < 3; off += 2 * np[a], ++a) {
      if (a != axis) continue;
      const double xs = sc[a] * r[a];
      double *v = t + off, *d = t + off + np[a];
      // rect_rf1.f90:33-55 and :88-118 (values, then slopes, scaled)
      double v0 = 1.0, v1 = xs, v2 = 0.5 * (3.0 * xs * xs - 1.0);
      double d0 = 0.0, d1 = 1.0, d2 = 3.0 * xs;
      v[0] = v0;
      d[0] = d0 * sc[a];
      if (np[a] > 1) {
        v[1] = v1;
        d[1] = d1 * sc[a];
      }
      if (np[a] > 2) {
        v[2] = v2;
        d[2] = d2 * sc[a];
      }
      double vm2 = v1, vm1 = v2, dm1 = d2;
      for (int n = 3; n <= np[a] - 1; ++n) {
        const double vn = ((2.0 * n - 1) * xs * vm1 - (n - 1.0) * vm2) / n;
        const double dn = xs * dm1 + n * vm1;
        v[n] = vn;
        d[n] = dn * sc[a];
        vm2 = vm1;
        vm1 = vn;
        dm1 = dn;
      }
    }
    return true;
  }
  const double r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
  if (!(r2 <= m.srdist2)) return false;
  const SpheLayout L = sphe_layout(m.nmpol);
  const double rr = sqrt(r2), ir = 1.0 / rr;
  double ct = r[2] * ir;
  double st = sqrt(1.0 - ct * ct);
  ist = istnum / st;
  double cp = r[0] * ir * ist, sp = r[1] * ir * ist;
  if (r2 < 1e-3) {  // rsmall: at the origin
    ct = st = cp = sp = 0.0;
  } else if (r[0] > -1e-3 && r[0] < 1e-3 && r[1] > -1e-3 && r[1] < 1e-3) {  // z axis
    ct = r[2] < 0.0 ? -1.0 : 1.0;
    cp = sp = 0.0;
  } else if (r[2] > -1e-3 && r[2] < 1e-3) {  // xy plane
    ct = 0.0;
    cp = r[0] * ir;
    sp = r[1] * ir;
  }
  double *ar = t + L.ar(), *ac = t + L.ac(), *as = t + L.as();
  double *ap = t + L.ap(), *adp = t + L.adp();
  ar[0] = 1.0;  // rpowerl2
  for (int i = 1; i <= L.lmax; ++i) ar[i] = ar[i - 1] * rr;
  ac[0] = 1.0;  // cosmphi2, sinmphi2
  ac[1] = cp;
  ac[2] = 2.0 * cp * cp - 1.0;
  ac[3] = (2.0 * ac[2] - 1.0) * cp;
  as[0] = 0.0;
  as[1] = sp;
  as[2] = 2.0 * cp * sp;
  as[3] = 2.0 * cp * as[2] - sp;
  for (int i = 4; i <= L.lmax; ++i) {
    ac[i] = 2.0 * cp * ac[i - 1] - ac[i - 2];
    as[i] = 2.0 * cp * as[i - 1] - as[i - 2];
  }
  const int W = L.w, lmax = L.lmax, mmax = L.lmax;
  for (int k = 0; k < (lmax + 2) * W; ++k) ap[k] = 0.0;  // P_l^m = 0 for m > l
  const double xc = ct;
  ap[0] = 1.0;  // alpol2
  const double somx2 = sqrt((1.0 - xc) * (1.0 + xc));
  double fact = 1.0;
  for (int mm = 1; mm <= mmax; ++mm) {
    ap[mm * W + mm] = ap[(mm - 1) * W + mm - 1] * fact * somx2;
    fact = fact + 2.0;
  }
  for (int mm = 0; mm <= mmax; ++mm) ap[(mm + 1) * W + mm] = xc * (2 * mm + 1) * ap[mm * W + mm];
  for (int l = 2; l <= lmax; ++l)
    for (int mm = 0; mm <= l - 2; ++mm)
      ap[l * W + mm] =
          (xc * (2.0 * l - 1) * ap[(l - 1) * W + mm] - (l + mm - 1) * ap[(l - 2) * W + mm]) /
          (l - mm);
  if (xc == 1.0 || xc == -1.0) {  // dalpol2
    for (int l = 0; l <= lmax; ++l) {
      double v = 0.0;
      if (xc == 1.0) v = l * (l + 1.0) * 0.5;
      if (xc == -1.0) v = ((l + 1) % 2 ? -1.0 : 1.0) * l * (l + 1.0) * 0.5;
      adp[l * W] = v;
      for (int mm = 1; mm <= mmax; ++mm) adp[l * W + mm] = 0.0;
    }
  } else {
    for (int l = 0; l <= lmax; ++l)
      for (int mm = 0; mm <= mmax; ++mm) {
        const double f = 1.0 / sqrt(1.0 - xc * xc);
        adp[l * W + mm] = f * (ap[l * W + mm + 1] - f * mm * xc * ap[l * W + mm]);
      }
  }
  double *ang = t + L.ang();
  ang[0] = st;
  ang[1] = ct;
  ang[2] = cp;
  ang[3] = sp;
  return true;
}

// basis function k (without its norm) of a table row
__device__ __forceinline__ double mm_value(const MmijDev &m, int k, const double *t) {
  const int3 o = m.lst[k];
  if (m.rect) return t[o.x] * t[2 * m.nx + o.y] * t[2 * m.nx + 2 * m.ny + o.z];
  const SpheLayout L = sphe_layout(m.nmpol);
  const int l = o.x, mm = o.y;
  if (mm == 0) return t[L.ar() + l] * t[L.ap() + l * L.w];
  if (mm > 0) return t[L.ar() + l] * t[L.ac() + mm] * t[L.ap() + l * L.w + mm];
  return t[L.ar() + l] * t[L.as() - mm] * t[L.ap() + l * L.w - mm];
}

// Row of particle i in tab: the trial's row (index cap) stands in for
// particle j in INTERACT mode.
template <bool F32>
__global__ void __launch_bounds__(kMmThreads) k_mmij_tab(KP p, int mode) {
  after_prev();
  const MmijDev &m = p.mm;
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = m.rect ? u / 3 : u, axis = m.rect ? u % 3 : 0;
  const int ntot = p.st->ntot, i0 = p.nsites + p.nfix;
  double r[3], ist = 0.0;
  int row;
  if (mode == 1 && i == ntot) {  // INTERACT: the trial position
    const Trial tr = *p.trial;
    r[0] = tr.x;
    r[1] = tr.y;
    r[2] = tr.z;
    row = p.cap;
  } else {
    if (i >= ntot || i < i0) return;
    mm_pos<F32>(p, i, r);
    row = i;
  }
  double *t = m.tab + (size_t)row * m.tabw;
  const bool in = mm_tables(p, r, mode == 1 ? 1.0 : 10.0, axis, t, ist);
  if (axis == 0) {
    m.in[row] = in ? 1 : 0;
    m.ist[row] = ist;
  }
}

// Chunk c of the ions: thread k sums q_i b_k(r_i) over the chunk's ions in the
// region, listed first (in ion order), so that the sum's loads need no test
// and several ions' are in flight.
__global__ void __launch_bounds__(kMmThreads) k_mmij_coef(KP p, int mode) {
  after_prev();
  const MmijDev &m = p.mm;
  __shared__ int rows[kMmChunk], n;
  __shared__ double qs[kMmChunk];
  const int k = blockIdx.y * blockDim.x + threadIdx.x;
  const int c = blockIdx.x;  // (a grid holds 65535 blocks in y: a million ions)
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const int ntot = p.st->ntot, i = p.nsites + p.nfix + c * kMmChunk + lane;
    int row = i, iend = ntot, type = 0;
    if (lane < kMmChunk && mode == 1) {  // INTERACT: particle j's row is the trial's
      const Trial tr = *p.trial;
      if (tr.insert) iend = ntot + 1;
      if (i == tr.j - 1) {
        row = p.cap;
        type = tr.itype;
      }
    }
    const bool in = lane < kMmChunk && i < iend && m.in[row];
    const unsigned b = __ballot_sync(0xffffffffu, in);
    if (in) {
      const int u = __popc(b & ((1u << lane) - 1u));
      rows[u] = row;
      qs[u] = p.cg[row == p.cap ? type : abs(p.typei[i])];
    }
    if (lane == 0) n = __popc(b);
  }
  __syncthreads();
  if (k >= m.ntpol) return;
  double v = 0.0;
#pragma unroll 4
  for (int u = 0; u < n; ++u) v = fma(qs[u], mm_value(m, k, m.tab + (size_t)rows[u] * m.tabw), v);
  m.coefp[(size_t)c * m.ntpol + k] = v * m.bnorm[k];
}

// A warp per function: the lanes take every 32nd chunk, then a fixed shuffle
// tree.
__global__ void __launch_bounds__(kMmThreads) k_mmij_sum(KP p, int mode, int nchunk) {
  after_prev();
  const MmijDev &m = p.mm;
  const int k = blockIdx.x * (kMmThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (blockIdx.x == 0 && threadIdx.x == 0) *m.done = 0;  // k_mmij_rows' count
  double v = 0.0;
  if (k < m.ntpol) {
    for (int c = lane; c < nchunk; c += 32) v += m.coefp[(size_t)c * m.ntpol + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  }
  if (k < m.ntpol && lane == 0) {
    m.coef[k] = v;
    if (mode == 1) {  // coef2 = coef - q_j b_k(r_j), j a mobile ion in the region
      const Trial tr = *p.trial;
      const int j = tr.j - 1, i0 = p.nsites + p.nfix;
      const bool jin = j >= i0 && m.in[p.cap];
      m.coef2[k] = jin ? v - p.cg[tr.itype] * m.bnorm[k] *
                                 mm_value(m, k, m.tab + (size_t)p.cap * m.tabw)
                       : v;
    }
  }
  if (mode == 0 && !m.rect && blockIdx.x == 0 && threadIdx.x == 0) {
    // sphe_rf1.f90's forces use the ist of the last ion in the sphere
    const int ntot = p.st->ntot;
    double ist = 0.0;
    for (int i = ntot - 1; i >= p.nsites + p.nfix; --i)
      if (m.in[i]) {
        ist = m.ist[i];
        break;
      }
    m.ist[p.cap + 1] = ist;
  }
}

// mode 0: mq_k = sum_l M_kl coef_l (x rfscal); mode 1: row k of
// E(coef) - E(coef2): (c_k^2 - c2_k^2) M_kk / 2 + sum_{l>k} (c_k c_l - c2_k c2_l) M_kl.
// The last block done totals the rows: mode 0: egsbpb into energy slot `slot`;
// mode 1: INTERACT's term added to *dener.
__global__ void __launch_bounds__(kMmThreads)
    k_mmij_rows(KP p, int mode, int slot, double *dener) {
  after_prev();
  const MmijDev &m = p.mm;
  __shared__ double red[kMmThreads / 32];
  __shared__ double tot[1];
  __shared__ bool last;
  const int k = blockIdx.x * (kMmThreads / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int n = m.ntpol;
  const double *row = m.m + (size_t)k * n;
  double v = 0.0;
  if (k >= n) {
  } else if (mode == 0) {
    for (int l = lane; l < n; l += 32) v += m.rect ? row[l] * m.coef[l] * m.rfscal : row[l] * m.coef[l];
  } else {
    const double ck = m.coef[k], c2k = m.coef2[k];
    for (int l = k + 1 + lane; l < n; l += 32) v += (ck * m.coef[l] - c2k * m.coef2[l]) * row[l];
    if (lane == 0) v += 0.5 * (ck * ck - c2k * c2k) * row[k];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (k < n && lane == 0) (mode == 0 ? m.mq : m.rowe)[k] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(m.done, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  double e[1] = {0.0};
  for (int c = threadIdx.x; c < n; c += blockDim.x)
    e[0] += mode == 0 ? 0.5 * m.coef[c] * __ldcg(m.mq + c) : __ldcg(m.rowe + c);
  block_sum<1>(e, red, tot);
  if (threadIdx.x != 0) return;
  if (mode == 0) {
    double *dst = p.epart + (size_t)slot * kNTerms;
    for (int k = 0; k < kNTerms; ++k) dst[k] = 0.0;
    dst[11] = tot[0] * p.celec;
  } else {
    *dener += m.rect ? tot[0] * p.celec * m.rfscal : tot[0] * p.celec;
  }
}

constexpr int kMmLanes = 8;  // lanes per ion of the forces

template <bool F32>
__global__ void __launch_bounds__(kMmThreads) k_mmij_force(KP p) {
  after_prev();
  const MmijDev &m = p.mm;
  // eight lanes an ion; an ion out of range or region keeps its lanes for the
  // shuffles
  const int i = p.nsites + p.nfix + (blockIdx.x * blockDim.x + threadIdx.x) / kMmLanes;
  const int k0 = threadIdx.x % kMmLanes;
  const bool on = i < p.st->ntot && m.in[i];
  const int nf = on ? m.ntpol : 0;
  const double *t = m.tab + (size_t)(on ? i : 0) * m.tabw;
  double f[3] = {0.0, 0.0, 0.0};
  if (m.rect) {  // rect_rf1.f90:119-135
    const double *lx = t, *dlx = t + m.nx, *ly = t + 2 * m.nx, *dly = ly + m.ny;
    const double *lz = t + 2 * m.nx + 2 * m.ny, *dlz = lz + m.nz;
    for (int k = k0; k < nf; k += kMmLanes) {
      const int3 o = m.lst[k];
      const double w = m.bnorm[k] * m.mq[k];
      const double xl = lx[o.x], yl = ly[o.y], wz = w * lz[o.z];
      f[0] = fma(-dlx[o.x] * yl, wz, f[0]);
      f[1] = fma(-xl * dly[o.y], wz, f[1]);
      f[2] = fma(-xl * yl, w * dlz[o.z], f[2]);
    }
  } else {  // sphe_rf1.f90:120-160
    const SpheLayout L = sphe_layout(m.nmpol);
    const double *ar = t + L.ar(), *ac = t + L.ac(), *as = t + L.as();
    const double *ap = t + L.ap(), *adp = t + L.adp(), *ang = t + L.ang();
    const double st = ang[0], ct = ang[1], cp = ang[2], sp = ang[3];
    const double ist = m.ist[p.cap + 1];
    const int W = L.w;
    for (int k = k0; k < nf; k += kMmLanes) {
      const int l = m.lst[k].x;
      int mm = m.lst[k].y;
      double dr = 0.0, ddt = 0.0, dp = 0.0;
      if (mm == 0) {
        if (l != 0) {
          const double rpl = ar[l - 1];
          dr = l * rpl * ap[l * W];
          ddt = -rpl * adp[l * W] * st;
        }
      } else if (mm > 0) {
        const double rpl = ar[l - 1], cmp = ac[mm], apl = ap[l * W + mm];
        dr = l * rpl * cmp * apl;
        ddt = -rpl * cmp * adp[l * W + mm] * st;
        dp = st == 0.0 ? 0.0 : -rpl * mm * as[mm] * apl * ist;
      } else {
        mm = -mm;
        const double rpl = ar[l - 1], smp = as[mm], apl = ap[l * W + mm];
        dr = l * rpl * smp * apl;
        ddt = -rpl * smp * adp[l * W + mm] * st;
        dp = st == 0.0 ? 0.0 : rpl * mm * ac[mm] * apl * ist;
      }
      const double nrm = m.bnorm[k], mq = m.mq[k];
      f[0] -= nrm * (dr * st * cp + ddt * ct * cp - dp * sp) * mq;
      f[1] -= nrm * (dr * st * sp + ddt * ct * sp + dp * cp) * mq;
      f[2] -= nrm * (dr * ct - ddt * st) * mq;
    }
  }
#pragma unroll
  for (int o = kMmLanes / 2; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < 3; ++c) f[c] += __shfl_xor_sync(0xffffffffu, f[c], o);
  if (!on || k0 != 0) return;
  const double ccc = p.cg[abs(p.typei[i])] * p.celec;
  const int cap = p.cap;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (F32)
      p.ffield_f[c * cap + i] += (float)(f[c] * ccc);
    else
      p.ffield[c * cap + i] += f[c] * ccc;
  }
}

int mmij_chunks(const KP &p, int ntot_ub) {
  return std::max(1, (std::max(0, ntot_ub + 1 - p.nsites - p.nfix) + kMmChunk - 1) / kMmChunk);
}

int launch_mmij_energy(const KP &p, bool fp32, int ntot_ub, int slot, cudaStream_t stream) {
  const MmijDev &m = p.mm;
  const int nt = m.ntpol, nch = mmij_chunks(p, ntot_ub);
  const int tb = ((m.rect ? 3 : 1) * ntot_ub + kMmThreads - 1) / kMmThreads;
  const int wb = (nt + kMmThreads / 32 - 1) / (kMmThreads / 32);  // a warp per function
  if (tb > 0)
    launch_after(fp32 ? k_mmij_tab<true> : k_mmij_tab<false>, tb, kMmThreads, stream, p, 0);
  launch_after(k_mmij_coef, dim3(nch, (nt + kMmThreads - 1) / kMmThreads), kMmThreads, stream, p, 0);
  launch_after(k_mmij_sum, wb, kMmThreads, stream, p, 0, nch);
  launch_after(k_mmij_rows, wb, kMmThreads, stream, p, 0, slot, nullptr);
  return 4;
}

// Adds to the field forces: after the field kernel and the energy's kernels.
int launch_mmij_force(const KP &p, bool fp32, int ntot_ub, cudaStream_t stream) {
  const int nion = std::max(0, ntot_ub - p.nsites - p.nfix);
  if (nion == 0) return 0;
  launch_after(fp32 ? k_mmij_force<true> : k_mmij_force<false>,
               (nion * kMmLanes + kMmThreads - 1) / kMmThreads, kMmThreads, stream, p);
  return 1;
}

void launch_mmij_tables(const KP &p, int ntot_ub, cudaStream_t stream) {
  const MmijDev &m = p.mm;
  const int nt = m.ntpol, nch = mmij_chunks(p, ntot_ub);
  // positions are FP64 in INTERACT (the context keeps them current)
  const int wb = (nt + kMmThreads / 32 - 1) / (kMmThreads / 32);
  launch_after(k_mmij_tab<false>, ((m.rect ? 3 : 1) * (ntot_ub + 1) + kMmThreads - 1) / kMmThreads,
               kMmThreads, stream, p, 1);
  launch_after(k_mmij_coef, dim3(nch, (nt + kMmThreads - 1) / kMmThreads), kMmThreads, stream, p, 1);
  launch_after(k_mmij_sum, wb, kMmThreads, stream, p, 1, nch);
}

void launch_mmij_total(const KP &p, double *dener, cudaStream_t stream) {
  const int wb = (p.mm.ntpol + kMmThreads / 32 - 1) / (kMmThreads / 32);
  launch_after(k_mmij_rows, wb, kMmThreads, stream, p, 1, 0, dener);
}

int mmij_table_width(int rect, int nx, int ny, int nz, int nmpol) {
  return rect ? 2 * (nx + ny + nz) : sphe_layout(nmpol).width();
}

}  // namespace bgpu
