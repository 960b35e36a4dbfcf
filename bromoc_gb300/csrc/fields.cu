// Single-particle terms of ENERGY, in FP32 with one warp per particle (FP64:
// four lanes per particle, fields64.cuh): static field
// (staticf1.f90), repulsion map (vdwgd1trln.f90 / vdwgd1spln.f90), RFPAR
// gathers and self term (rfpar.f90:75-176) and the membrane (membrane.f90).
//
// Lane layout for the trilinear maps: lane = 8 g + corner, corner = 4a+2b+c
// selects the grid node (ix+a, iy+b, iz+c); g = 0 static field, 1 repulsion,
// 2 gsrfen (srfe), 3 greff (reff).  Each lane gathers one node and forms its
// weight and derivative terms; eight-lane shuffle trees give the sums.  The
// 27-point B-spline repulsion takes lanes 0..26 in a second pass.  The kernel
// works on float-float positions and single-precision weights throughout.
#include "batch.cuh"
#include "ff.cuh"
#include "launch.h"
#include "physics.cuh"
#include "fields32.cuh"
#include "fields64.cuh"

namespace bgpu {

constexpr int kFieldWarps = 4;

// One warp, eight particles: 250 blocks for 2000 ions leave no SM with two
// chains on one FP64 pipe.
__global__ void __launch_bounds__(32)
    k_fields_quad_f64(const __grid_constant__ KP p, uint32_t mask, int qforces, int slot0) {
  after_prev();
  __shared__ double red[4], tot[4];
  const int i = blockIdx.x * 8 + (threadIdx.x >> 2);
  double eo[4] = {0.0, 0.0, 0.0, 0.0};  // lanes g == 0: ememb, egsbpa, evdwgd, erfpar
  fields_quad_f64(p, i, i < p.st->ntot, mask, qforces, eo);
  block_sum<4>(eo, red, tot);
  if (threadIdx.x == 0) {
    double *dst = p.epart + (size_t)(slot0 + blockIdx.x) * kNTerms;
    for (int k = 0; k < kNTerms; ++k) dst[k] = 0.0;
    dst[9] = tot[0];   // EMEMB
    dst[10] = tot[1];  // EGSBPA
    dst[12] = tot[2];  // EVDWGD
    dst[13] = tot[3];  // ERFPAR (self)
  }
}

__global__ void __launch_bounds__(32 * kFieldWarps)
    k_fields_warp_f32(const __grid_constant__ KP p, uint32_t mask, int qforces, int slot0) {
  __shared__ float red[kFieldWarps * 4];
  __shared__ float tot[4];
  __shared__ AxisF ax[12];
  stage_axes(p, ax);
  after_prev();
  const int i = blockIdx.x * kFieldWarps + (threadIdx.x >> 5);
  const int ntot = p.st->ntot;
  float eo[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // lane 0: ememb, egsbpa, evdwgd, erfpar
  if (i < ntot) {  // warp-uniform
    const bool site = i < p.nsites;
    fields_one_f32(p, i, site, !site && i < p.nsites + p.nfix, mask, qforces, eo, ax);
  }
  block_sum_f<4>(eo, red, tot);
  if (threadIdx.x == 0) {
    double *dst = p.epart + (size_t)(slot0 + blockIdx.x) * kNTerms;
    for (int k = 0; k < kNTerms; ++k) dst[k] = 0.0;
    dst[9] = tot[0];
    dst[10] = tot[1];
    dst[12] = tot[2];
    dst[13] = tot[3];
  }
}

// ---------------------------------------------------------------------------
// FP32 mode: FP64 coordinates -> float-float records (also the pair-law type
// code, mobility and charge), and back.
// ---------------------------------------------------------------------------
__global__ void k_pack(KP p) {
  after_prev();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.st->ntot) return;
  const bool site = i < p.nsites;
  const int iontype = site ? 0 : abs(p.typei[i]);
  const int it2 = site ? p.typtyp[i] : p.nwtype[iontype];
  const double q = site ? p.sitecharge[i] : p.cg[iontype];
  const int mobile = i >= p.nsites + p.nfix;
  const double x = p.x[i], y = p.y[i], z = p.z[i];
  const float xh = (float)x, yh = (float)y, zh = (float)z;
  p.pk1[i] = make_float4(xh, yh, zh, __int_as_float((it2 - 1) | (mobile << 16)));
  p.pk2[i] = make_float4((float)(x - (double)xh), (float)(y - (double)yh),
                         (float)(z - (double)zh), 0.0f);
  p.pk3[i] = make_float4(0.0f, (float)q, __int_as_float(mobile << 1), 0.0f);
}

__global__ void k_unpack(KP p) {
  after_prev();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.st->ntot) return;
  const float4 h = p.pk1[i], l = p.pk2[i];
  p.x[i] = (double)h.x + (double)l.x;
  p.y[i] = (double)h.y + (double)l.y;
  p.z[i] = (double)h.z + (double)l.z;
}

void launch_pack(const KP &p, int ntot_ub, bool to_records, cudaStream_t stream) {
  if (ntot_ub <= 0) return;
  const int nb = (ntot_ub + 127) / 128;
  if (to_records)
    launch_after(k_pack, nb, 128, stream, p);
  else
    launch_after(k_unpack, nb, 128, stream, p);
}

// The staging area is pinned host memory: the kernels read and write it
// directly.  A call moves three to eight short arrays; as copies they cost a
// few us each, pageable ones ~10 us with a wait inside.
__global__ void k_stage_in(KP p, int n, const double *xyz, const int *typei,
                           const int *ibuffer) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    p.st->ntot = n;
    *p.live = n;
  }
  if (i >= n) return;
  p.x[i] = xyz[i];
  p.y[i] = xyz[n + i];
  p.z[i] = xyz[2 * (size_t)n + i];
  p.typei[i] = typei[i];
  p.ibuffer[i] = ibuffer ? ibuffer[i] : 0;
}

void launch_stage_in(const KP &p, int n, const double *xyz, const int *typei,
                     const int *ibuffer, cudaStream_t stream) {
  k_stage_in<<<(n + 127) / 128 + (n == 0), 128, 0, stream>>>(p, n, xyz, typei, ibuffer);
}

__global__ void k_stage_out(KP p, StageOut o) {
  after_prev();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int ntot = p.st->ntot;
  if (i == 0) {
    o.head[0] = ntot;
    o.head[1] = p.st->err;
  }
  if (o.terms && i < kNTerms) o.tout[i] = o.terms[i];
  if (o.warn && i < o.nwarn) o.wout[i] = o.warn[i];
  if (i >= ntot || i >= o.nub) return;
  const size_t s = o.stride;
  if (o.ff) {
    const float4 h = p.pk1[i], l = p.pk2[i];
    const double x = (double)h.x + (double)l.x, y = (double)h.y + (double)l.y,
                 z = (double)h.z + (double)l.z;
    p.x[i] = o.out[i] = x;
    p.y[i] = o.out[s + i] = y;
    p.z[i] = o.out[2 * s + i] = z;
  } else {
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (o.a[k]) o.out[k * s + i] = o.a[k][i];
  }
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (o.ia[k]) o.iout[k * s + i] = o.ia[k][i];
}

void launch_stage_out(const KP &p, const StageOut &o, cudaStream_t stream) {
  const int n = o.nub > kNTerms ? o.nub : kNTerms, m = n > o.nwarn ? n : o.nwarn;
  launch_after(k_stage_out, (m + 127) / 128, 128, stream, p, o);
}

// Replica batches: one thread per slot of the batch arrays (one warp per
// slot with a B-spline repulsion map); slots past their replica's live count
// return at once.
constexpr int kBatchFieldThreads = 128;
__global__ void __launch_bounds__(kBatchFieldThreads)
    k_batch_fields_t(const __grid_constant__ KP p, const int *rep_of, const RepDev *rep,
                     float4 *pe, int nslots, uint32_t mask, int qforces) {
  __shared__ AxisF ax[12];
  stage_axes(p, ax);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nslots) return;
  const RepDev &R = rep[rep_of[i]];
  if (i - R.off >= R.n) return;
  float eo[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  fields_one_thread(p, i, mask, qforces, eo, ax);
  pe[i] = make_float4(eo[0], eo[1], eo[2], eo[3]);
}

__global__ void __launch_bounds__(32 * kFieldWarps)
    k_batch_fields(const __grid_constant__ KP p, const int *rep_of, const RepDev *rep,
                   float4 *pe, int nslots, uint32_t mask, int qforces) {
  __shared__ AxisF ax[12];
  stage_axes(p, ax);
  const int i = blockIdx.x * kFieldWarps + (threadIdx.x >> 5);
  if (i >= nslots) return;  // warp-uniform from here on
  const RepDev &R = rep[rep_of[i]];
  if (i - R.off >= R.n) return;
  float eo[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  fields_one_f32(p, i, false, false, mask, qforces, eo, ax);
  if ((threadIdx.x & 31) == 0) pe[i] = make_float4(eo[0], eo[1], eo[2], eo[3]);
}

void launch_batch_fields(const KP &p, const int *rep_of, const RepDev *rep, float4 *pe,
                         int nslots, uint32_t mask, int qforces, cudaStream_t stream) {
  if (nslots <= 0) return;
  if ((mask & 8u) && p.qphiv && !p.qtrln) {
    const int nb = (nslots + kFieldWarps - 1) / kFieldWarps;
    k_batch_fields<<<nb, 32 * kFieldWarps, 0, stream>>>(p, rep_of, rep, pe, nslots, mask,
                                                         qforces);
  } else {
    const int nb = (nslots + kBatchFieldThreads - 1) / kBatchFieldThreads;
    k_batch_fields_t<<<nb, kBatchFieldThreads, 0, stream>>>(p, rep_of, rep, pe, nslots, mask,
                                                            qforces);
  }
}

int fields_blocks(int ntot_ub, bool fp32) {
  return fp32 ? (ntot_ub + kFieldWarps - 1) / kFieldWarps : (ntot_ub + 7) / 8;
}

void launch_fields(const KP &p, int ntot_ub, uint32_t mask, int qforces, bool fp32,
                   int slot0, cudaStream_t stream) {
  const int nb = fields_blocks(ntot_ub, fp32);
  if (nb == 0) return;
  if (fp32)
    launch_after(k_fields_warp_f32, nb, 32 * kFieldWarps, stream, p, mask, qforces, slot0);
  else
    launch_after(k_fields_quad_f64, nb, 32, stream, p, mask, qforces, slot0);
}

}  // namespace bgpu
