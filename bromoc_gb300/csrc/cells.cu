// Cell list of the periodic extension mode, FP32 path, and the pair kernel
// that walks it.  The reference evaluates every ion pair
// (energy.mono.f90:117-194); the extension mode adds a minimum-image box and
// a plain cutoff rc, and with a cutoff only the pairs within rc count.  The
// box is cut into cells of edge at least rc (1 + 1e-4): a pair within rc then
// always lies in the same or a neighbouring cell, even when rounding puts an
// ion near a cell face on the other side of it.
//
// Built on the device every energy evaluation (the ions move every step):
//   count  : each ion's cell from its float-float position (an ion outside the
//            box counts at its image inside), its arrival number in the cell
//            (the count's atomic);
//   scan   : exclusive prefix sum of the counts (one block);
//   fill   : ions into their cell's stretch at their arrival number;
//   sort   : each cell's stretch in ascending ion order (a warp per cell: an
//            ion's place is the number of smaller ones), so a run always sums a
//            particle's pairs in one order, and the ions' records in that
//            order, so that the pair kernel reads its candidates in line.
// Pair kernel: a block per cell.  The cells of one z row are consecutive, so
// the ions of the 27 neighbour cells are nine runs of records (and, at the
// box's z faces, nine more); the block lays them in shared memory, moved by
// the box lengths that their run wraps, and its warps take the cell's ions in
// turn.  A warp tests 32 candidates at a time against its ion's cutoff (one in
// eight is within it; the high parts of the records settle most), queues those
// inside and evaluates the law with full lanes; SRPMF pairs are queued once
// more, over the warp's ions.  Sums are over lanes in a fixed shuffle tree and,
// for SRPMF, in queue order.
// Each pair is evaluated by both of its ions, weight 1/2 per mobile source,
// the conventions of the chunked kernel k_pairs32 (FP32 partials fii_f,
// chunk 0; block partial energies).  Used when every axis holds at least four
// cells; smaller boxes keep the all-pairs Newton-3 tile.
// 20,000 ions, 1728 cells of 12: pairs 48 -> 37 us (before: four lanes an ion
// walking the cells through an index, the law on every candidate's iteration;
// with the records in line and eight lanes 45), sort 28 -> 5 us; a step 60 us
// in a long run (64 with both parts of the records in the first test), ~52 with
// the launches overlapped.  Bound
// by the candidates' tests (6 M of them for 0.8 M within the cutoff) and the
// blocks' barriers.
#include <algorithm>

#include "launch.h"
#include "pairs_n3.cuh"

namespace bgpu {

constexpr int kCellThreads = 256;
constexpr int kCpWarps = 4;      // warps of a cell's block in the pair kernel
constexpr int kCpMax = 512;      // candidates in shared memory at a time
constexpr int kCpGrid = 2048;    // blocks at most; they take cells in turn
constexpr int kCpQ = 64;         // pair queue and SRPMF queue of a warp
constexpr int kCpIons = 16;      // ions whose SRPMF pairs a warp queues together

// An ion outside the box (only a caller's starting position), moved into it by
// whole box lengths, the rounding in the low part: the cells and the pair kernel
// go by the moved record, so that its neighbours are its image's.
__device__ __forceinline__ void fold_in(const KP &p, float4 &h, float4 &l) {
  float *hh[3] = {&h.x, &h.y, &h.z}, *ll[3] = {&l.x, &l.y, &l.z};
  const BoxF &b = p.f.box;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float v = *hh[a];
    if (!(v < b.bh[2 * a] || v > b.bh[2 * a + 1])) continue;
    const float k = floorf(((v - b.bh[2 * a]) + (*ll[a] - b.bl[2 * a])) * p.f.iL[a]);
    const float u = __fmul_rn(-k, b.Lh[a]), s = v + u, t = s - v;
    // the product's rounding, the box length's low part, the sum's rounding
    const float w = *ll[a] + (fmaf(-k, b.Lh[a], -u) - k * b.Ll[a] + ((v - (s - t)) + (u - t)));
    *hh[a] = s + w;
    *ll[a] = w - (*hh[a] - s);
  }
}

__device__ __forceinline__ int cell_of(const KP &p, const float4 &h, const float4 &l) {
  const float hh[3] = {h.x, h.y, h.z}, ll[3] = {l.x, l.y, l.z};
  int c[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float u = ((hh[a] - p.f.box.bh[2 * a]) + (ll[a] - p.f.box.bl[2 * a])) * p.cinv[a];
    c[a] = min(max((int)floorf(u), 0), p.nc[a] - 1);
  }
  return (c[0] * p.nc[1] + c[1]) * p.nc[2] + c[2];
}

__global__ void __launch_bounds__(kCellThreads) k_cell_count(KP p) {
  after_prev();
  const int i = p.nsites + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.st->ntot) return;
  float4 h = p.pk1[i], l = p.pk2[i];
  fold_in(p, h, l);
  const int c = cell_of(p, h, l);
  p.ion_cell[i] = c;
  p.ion_rank[i] = atomicAdd(p.cell_n + c, 1);
}

// Exclusive prefix sum of the counts into cell_start[0..ncells]; the counts
// are cleared for the next build.  One block of 1024 threads, each over a
// contiguous run of cells.
__global__ void __launch_bounds__(1024) k_cell_scan(KP p) {
  after_prev();
  __shared__ int part[1024];
  const int n = p.ncells, per = (n + 1023) / 1024;
  const int b0 = min(n, (int)threadIdx.x * per), b1 = min(n, b0 + per);
  int s = 0;
  for (int c = b0; c < b1; ++c) s += p.cell_n[c];
  part[threadIdx.x] = s;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {  // inclusive scan of the run totals
    const int v = threadIdx.x >= (unsigned)o ? part[threadIdx.x - o] : 0;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  int run = threadIdx.x ? part[threadIdx.x - 1] : 0;
  for (int c = b0; c < b1; ++c) {
    const int k = p.cell_n[c];
    p.cell_start[c] = run;
    run += k;
    p.cell_n[c] = 0;
  }
  if (threadIdx.x == 1023) p.cell_start[n] = part[1023];
}

__global__ void __launch_bounds__(kCellThreads) k_cell_fill(KP p) {
  after_prev();
  const int i = p.nsites + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.st->ntot) return;
  p.cell_any[p.cell_start[p.ion_cell[i]] + p.ion_rank[i]] = i;
}

__global__ void __launch_bounds__(kCellThreads) k_cell_sort(KP p) {
  after_prev();
  const int c = blockIdx.x * (kCellThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (c >= p.ncells) return;  // warp-uniform
  const int o = p.cell_start[c], n = p.cell_start[c + 1] - o;
  for (int a = 0; a < n; a += 32) {
    const int x = a + lane < n ? p.cell_any[o + a + lane] : -1;
    int place = 0;
    for (int b = 0; b < n; b += 32) {
      const int y = b == a ? x : (b + lane < n ? p.cell_any[o + b + lane] : -1);
      const int nb = min(32, n - b);
      for (int k = 0; k < nb; ++k) place += __shfl_sync(0xffffffffu, y, k) < x;
    }
    if (x >= 0) {
      float4 h = p.pk1[x], l = p.pk2[x];
      fold_in(p, h, l);
      p.cell_ion[o + place] = x;
      p.cell_pk1[o + place] = h;
      p.cell_pk2[o + place] = l;
    }
  }
}

struct CellSmem {
  float4 h[kCpMax], l[kCpMax];  // candidates: moved record (hi, type code), lo
  int off[19], beg[18];         // runs: first place in the list, first slot
  float sh[18][3], sl[18][3];   // box lengths added to their positions (hi, lo)
  int q[kCpWarps][kCpQ], sq[kCpWarps][kCpQ];
  float f[kCpWarps][kCpIons][3];
};

template <bool EFP>
__global__ void __launch_bounds__(32 * kCpWarps)
    k_pairs_cell(const __grid_constant__ KP p, int qforces, int slot0) {
  constexpr unsigned kAll = 0xffffffffu;
  __shared__ CellSmem S;
  __shared__ float4 tab[EFP ? 1 : kIpqMax];
  __shared__ float red[kCpWarps * 4];
  __shared__ float tot[4];
  const int nt = p.nion_t, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (!EFP)
    for (int k = threadIdx.x; k < nt * ipq_stride(nt); k += blockDim.x) tab[k] = __ldg(p.ipq + k);
  after_prev();
  const int m0 = p.nsites + p.nfix;
  const float rc2 = p.f.rc2;
  // the first test takes the high parts alone, against a cutoff wider by more
  // than the low parts and the roundings can move a distance in the box
  float cm = 0.f;
#pragma unroll
  for (int a = 0; a < 6; ++a) cm = fmaxf(cm, fabsf(p.f.box.bh[a]));
#pragma unroll
  for (int a = 0; a < 3; ++a) cm = fmaxf(cm, p.f.box.Lh[a]);
  const float rw = fmaf(cm, 2e-6f, sqrtf(rc2)), rc2w = rw * rw;
  const unsigned below = (1u << lane) - 1u;
  float e[4] = {0.f, 0.f, 0.f, 0.f};  // ecoul, elj (6 x elj with the dense table), esrpmf, eefpot
  int *q = S.q[w], *sq = S.sq[w];
  for (int c = blockIdx.x; c < p.ncells; c += gridDim.x) {
    const int t0 = p.cell_start[c], nt0 = p.cell_start[c + 1] - t0;
    if (nt0 == 0) continue;  // block-uniform
    const int n1 = p.nc[1], n2 = p.nc[2];
    const int cz = c % n2, cy = (c / n2) % n1, cx = c / (n1 * n2);
    __syncthreads();  // the previous cell's list
    if (threadIdx.x < 18) {
      // run r: row (r % 9), its unwrapped z cells (r < 9) or its wrapped one
      const int r = threadIdx.x, row = r % 9, z = r / 9;
      int ax = cx + row / 3 - 1, ay = cy + row % 3 - 1;
      const int wx = ax < 0 ? -1 : (ax >= p.nc[0] ? 1 : 0), wy = ay < 0 ? -1 : (ay >= n1 ? 1 : 0);
      const int wz = z == 0 ? 0 : (cz == 0 ? -1 : 1);
      ax -= wx * p.nc[0];
      ay -= wy * n1;
      const int *cs = p.cell_start + (ax * n1 + ay) * n2;
      int b0, b1;
      if (z == 0) {
        b0 = cs[max(cz - 1, 0)];
        b1 = cs[min(cz + 1, n2 - 1) + 1];
      } else {
        const bool on = cz == 0 || cz == n2 - 1;
        const int zw = cz == 0 ? n2 - 1 : 0;
        b0 = on ? cs[zw] : 0;
        b1 = on ? cs[zw + 1] : 0;
      }
      S.beg[r] = b0;
      S.off[r + 1] = b1 - b0;
      const int wv[3] = {wx, wy, wz};
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        S.sh[r][a] = wv[a] * p.f.box.Lh[a];
        S.sl[r][a] = wv[a] * p.f.box.Ll[a];
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      S.off[0] = 0;
      for (int r = 0; r < 18; ++r) S.off[r + 1] += S.off[r];
    }
    __syncthreads();
    const int ncand = S.off[18];
    // the cell's own ions in the list: row 4's run
    const int own0 = S.off[4] + (t0 - S.beg[4]);
    // the ions in groups of a warp each, kCpIons a warp before the SRPMF flush
    for (int g0 = 0; g0 < nt0; g0 += kCpWarps * kCpIons) {
      const int ng = min(kCpIons, (nt0 - g0 - w + kCpWarps - 1) / kCpWarps);  // may be < 1
      int sn = 0;  // queued SRPMF pairs: ion of the group << 16 | candidate
      for (int k = lane; k < kCpIons * 3; k += 32) (&S.f[w][0][0])[k] = 0.f;
      __syncwarp();  // lane 0 adds to them; a later group has no block barrier in between
      for (int c0 = 0; c0 < ncand; c0 += kCpMax) {  // one window but in crowded cells
        const int nc = min(kCpMax, ncand - c0);
        if (c0 > 0 || ncand > kCpMax || g0 == 0) {
          __syncthreads();
          for (int k = threadIdx.x; k < nc; k += blockDim.x) {
            int r = 0;
            while (S.off[r + 1] <= c0 + k) ++r;
            const int s = S.beg[r] + (c0 + k - S.off[r]);
            const float4 h = p.cell_pk1[s], l = p.cell_pk2[s];
            const float hh[3] = {h.x, h.y, h.z}, ll[3] = {l.x, l.y, l.z};
            float mh[3], ml[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {  // the sum's rounding goes to the low part
              const float v = S.sh[r][a];
              mh[a] = hh[a] + v;
              const float t = mh[a] - hh[a];
              ml[a] = ll[a] + (S.sl[r][a] + ((hh[a] - (mh[a] - t)) + (v - t)));
            }
            S.h[k] = make_float4(mh[0], mh[1], mh[2], h.w);
            S.l[k] = make_float4(ml[0], ml[1], ml[2], 0.f);
          }
          __syncthreads();
        }
        auto sep = [&](const float4 &th, const float4 &tl, int k, float &dx, float &dy,
                       float &dz) {
          const float4 h = S.h[k], l = S.l[k];
          dx = (th.x - h.x) + (tl.x - l.x);
          dy = (th.y - h.y) + (tl.y - l.y);
          dz = (th.z - h.z) + (tl.z - l.z);
          return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        };
        auto srp_flush = [&]() {  // warp-uniform
          for (int b = 0; b < sn; b += 32) {
            const bool act = b + lane < sn;
            const int ent = act ? sq[b + lane] : 0, ion = ent >> 16, k = ent & 0xffff;
            float gx = 0.f, gy = 0.f, gz = 0.f;
            if (act) {
              const int slot = t0 + g0 + ion * kCpWarps + w;
              const float4 th = p.cell_pk1[slot], tl = p.cell_pk2[slot];
              float dx, dy, dz;
              const float r2 = sep(th, tl, k, dx, dy, dz);
              const int code = __float_as_int(S.h[k].w);
              const float ds = srpmf32(
                  p, srp_index(p, __float_as_int(th.w), code), r2, rsqrt_nz(r2),
                  (code >> 16) ? 0.5f : 1.0f, e,
                  srp_branch(p, r2, [&] { return pair_r2_64<true>(p, th, tl, S.h[k], S.l[k]); }));
              gx = ds * dx;
              gy = ds * dy;
              gz = ds * dz;
            }
            const int nb = min(32, sn - b);
            for (int t = 0; t < nb; ++t) {  // queue order
              const int it = __shfl_sync(kAll, ion, t);
              const float vx = __shfl_sync(kAll, gx, t), vy = __shfl_sync(kAll, gy, t),
                          vz = __shfl_sync(kAll, gz, t);
              if (lane == 0) {
                S.f[w][it][0] += vx;
                S.f[w][it][1] += vy;
                S.f[w][it][2] += vz;
              }
            }
            __syncwarp();
          }
          sn = 0;
        };
        for (int ion = 0; ion < ng; ++ion) {
          const int place = g0 + ion * kCpWarps + w, i = p.cell_ion[t0 + place];
          if (i < m0) continue;  // a fixed ion is no target (warp-uniform)
          const float4 th = p.cell_pk1[t0 + place], tl = p.cell_pk2[t0 + place];
          const int tcode = __float_as_int(th.w), self = own0 + place - c0;
          const int row =
              EFP ? (tcode & 0xffff) * p.nttyp : ((tcode & 0xffff) - p.ndna) * ipq_stride(nt);
          float fx = 0.f, fy = 0.f, fz = 0.f;
          int n = 0;  // queued pairs
          auto flush = [&](int nb) {
            bool srp = false;
            const int k = lane < nb ? q[lane] : 0;
            float dx, dy, dz;
            float r2 = rc2;
            if (lane < nb) r2 = sep(th, tl, k, dx, dy, dz);
            if (r2 < rc2) {
              const int code = __float_as_int(S.h[k].w);
              const float wt = (code >> 16) ? 0.5f : 1.0f;
              float de;
              if (EFP) {
                de = law32k(p, __ldg(p.pidx + row + (code & 0xffff)), r2, wt, e,
                            [&] { return pair_r2_64<true>(p, th, tl, S.h[k], S.l[k]); });
              } else {
                const float4 t = tab[row + (code & 0xffff) - p.ndna];
                const float ir = rsqrt_nz(r2), ir2 = ir * ir;
                const float cofo = t.x * ir;
                e[0] = fmaf(wt, cofo, e[0]);
                float d6 = t.z * ir2;
                d6 = d6 * d6 * d6;
                const float d12 = d6 * d6;
                e[1] = fmaf(wt, t.y * (d12 - d6), e[1]);
                de = ir2 * fmaf(t.y, fmaf(2.0f, d12, -d6), cofo);
                srp = r2 <= t.w;
              }
              fx = fmaf(de, dx, fx);
              fy = fmaf(de, dy, fy);
              fz = fmaf(de, dz, fz);
            }
            const unsigned b = __ballot_sync(kAll, srp);
            if (srp) sq[sn + __popc(b & below)] = ion << 16 | k;
            sn += __popc(b);
            __syncwarp();
            if (sn > kCpQ - 32) srp_flush();
          };
          for (int k0 = 0; k0 < nc; k0 += 32) {
            const int k = k0 + lane;
            bool hit = false;
            if (k < nc && k != self) {
              const float4 h = S.h[k];
              const float dx = th.x - h.x, dy = th.y - h.y, dz = th.z - h.z;
              hit = fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < rc2w;
            }
            const unsigned b = __ballot_sync(kAll, hit);
            if (!b) continue;
            if (hit) q[n + __popc(b & below)] = k;
            n += __popc(b);
            __syncwarp();
            if (n >= 32) {
              flush(32);
              n -= 32;
              const int v = lane < n ? q[32 + lane] : 0;
              __syncwarp();
              if (lane < n) q[lane] = v;
              __syncwarp();
            }
          }
          if (n) flush(n);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            fx += __shfl_xor_sync(kAll, fx, o);
            fy += __shfl_xor_sync(kAll, fy, o);
            fz += __shfl_xor_sync(kAll, fz, o);
          }
          if (lane == 0) {
            S.f[w][ion][0] += fx;
            S.f[w][ion][1] += fy;
            S.f[w][ion][2] += fz;
          }
        }
        if (sn) srp_flush();  // the queue names places of this window
      }
      __syncwarp();
      if (lane < ng) {
        const int i = p.cell_ion[t0 + g0 + lane * kCpWarps + w];
#pragma unroll
        for (int a = 0; a < 3; ++a)
          p.fii_f[(size_t)a * p.cap + i] = qforces ? S.f[w][lane][a] : 0.f;  // chunk 0
      }
      __syncwarp();
    }
  }
  block_sum_f<4>(e, red, tot);
  if (threadIdx.x == 0) {
    double *dst = p.epart + (size_t)(slot0 + blockIdx.x) * kNTerms;
    for (int m = 0; m < kNTerms; ++m) dst[m] = 0.0;
    dst[1] = tot[0];
    dst[2] = EFP ? (double)tot[1] : (double)tot[1] / 6.0;
    dst[3] = tot[2];
    dst[4] = tot[3];
  }
}

int cell_pair_blocks(const KP &p, int) { return std::min(p.ncells, kCpGrid); }

int launch_cells(const KP &p, int ntot_ub, int qforces, int slot, cudaStream_t stream) {
  const int nion = std::max(0, ntot_ub - p.nsites);
  if (nion == 0 || p.ncells <= 0) return 0;
  const int nb = (nion + kCellThreads - 1) / kCellThreads;
  launch_after(k_cell_count, nb, kCellThreads, stream, p);
  launch_after(k_cell_scan, 1, 1024, stream, p);
  launch_after(k_cell_fill, nb, kCellThreads, stream, p);
  const int cw = kCellThreads / 32;  // a warp per cell
  launch_after(k_cell_sort, (p.ncells + cw - 1) / cw, kCellThreads, stream, p);
  const int npb = cell_pair_blocks(p, ntot_ub);
  if (p.ipq_ok)
    launch_after(k_pairs_cell<false>, npb, 32 * kCpWarps, stream, p, qforces, slot);
  else
    launch_after(k_pairs_cell<true>, npb, 32 * kCpWarps, stream, p, qforces, slot);
  return 5;
}

}  // namespace bgpu
