// Host-side launch interface between the C ABI (api.cu) and the kernels.
#pragma once
#include "kparams.cuh"

namespace bgpu {

constexpr int kSMs = 152;  // GB300

// A kernel that begins with after_prev (common.cuh), launched so that its
// blocks may take their places while the kernel before it in the stream drains.
// For the kernels of a step that go one by one: five steps of 20,000 ions in
// the cell list 400 -> 323 us, ten of 5000 ions with DNA 809 -> 663, an ENERGY
// call of 8000 ions 246 -> 226.
template <class... P, class... A>
inline void launch_after(void (*kern)(P...), dim3 grid, dim3 block, cudaStream_t stream,
                         A &&...args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = stream;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

// A pair of CUDA events bracketing one launch (diagnostic timing).
struct KTimer {
  cudaEvent_t a, b;
};

// A stream of the context for work beside its main stream's, with the events
// that fork and join it (no stream: the work goes in line).
struct SideStream {
  cudaStream_t s = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  cudaStream_t fork(cudaStream_t main) const {
    if (!s) return main;
    cudaEventRecord(ev_fork, main);
    cudaStreamWaitEvent(s, ev_fork, 0);
    return s;
  }
  void join(cudaStream_t main) const {
    if (!s) return;
    cudaEventRecord(ev_join, s);
    cudaStreamWaitEvent(main, ev_join, 0);
  }
};

struct EnergyPlan {
  int ntot_ub;        // host upper bound of the device-resident ntot
  int nchunk_ii;      // source chunks of the ion-ion kernel
  int nchunk_rf;      // source chunks of the RFPAR cross kernel
  int ntile;          // ion tiles of the Newton-3 pair kernels (0: chunked)
  bool fp32;
  bool nofield = false;  // no single-particle term is on: no field kernel
  int wave = 0;       // FP32: n3_split_of's (0: items are whole)
  bool srp = false;   // FP64: some ion-ion law has SRPMF
  bool cells = false; // FP32 extension mode: the cell-list pair kernel
  bool reduce_energy; // launch the final energy reduction
  bool nuc = false;   // DNA bonded/Go terms (nucl.cu)
  bool mmij = false;  // MMIJ reaction field (mmij.cu)
  KTimer *t_pairs = nullptr, *t_rf = nullptr, *t_fields = nullptr;
  SideStream side;  // where the sites' and MMIJ's work runs beside the ions'
};

// Tile pairs (I <= J) of the Newton-3 pair kernel, row-major: row I holds
// J = I..T-1 and starts at offset I T - I (I - 1) / 2.
constexpr int kN3MaxTiles = 256;  // up to 8192 ions; beyond, the chunked kernel
constexpr int kN64Types = 8;  // ion types of the FP64 Newton-3 kernel's shared law table
// Sites per tile of the FP32 ion-site pair kernel: a warp's 32 ions meet
// them one after another.
constexpr int kIsSiteTile = 8;
__host__ __device__ inline int n3_pairs(int T) { return T * (T + 1) / 2; }
__host__ __device__ inline int n3_index(int T, int I, int J) {
  return I * T - I * (I - 1) / 2 + (J - I);
}
// Work items of the Newton-3 pair kernels, column tile by column tile:
// column J's off-diagonal row tiles 0..J-1 go in pairs (2s, 2s+1), one item
// of 64 row ions against the column's 32 entries; when J is odd, row tile
// J-1 is an item of its own; the diagonal tile pair (J, J) comes last.
// Items before column J: J + floor(J^2 / 4).
__host__ __device__ inline int n3_items_before(int J) { return J + J * J / 4; }
__host__ __device__ inline int n3_items(int T) { return n3_items_before(T); }
// Tile pair q of the row-major list: (I, J).
__host__ __device__ inline void n3_pair(int T, int q, int &I, int &J) {
  const float b = 2.0f * T + 1.0f;
  int i = (int)((b - sqrtf(b * b - 8.0f * q)) * 0.5f);
  i = i < 0 ? 0 : (i > T - 1 ? T - 1 : i);
  while (i > 0 && n3_index(T, i, i) > q) --i;
  while (i + 1 < T && n3_index(T, i + 1, i + 1) <= q) ++i;
  I = i;
  J = i + (q - n3_index(T, i, i));
}
// Item it of T tiles: column J and row tiles I, I2 (I2 < 0: one row tile).
__host__ __device__ inline void n3_item(int T, int it, int &I, int &I2, int &J) {
  int j = (int)(2.0f * (sqrtf((float)it + 1.0f) - 1.0f));
  j = j < 0 ? 0 : (j > T - 1 ? T - 1 : j);
  while (j > 0 && n3_items_before(j) > it) --j;
  while (j + 1 < T && n3_items_before(j + 1) <= it) ++j;
  const int s = it - n3_items_before(j), nd = j >> 1;
  J = j;
  I2 = -1;
  if (s < nd) {
    I = 2 * s;
    I2 = 2 * s + 1;
  } else {
    I = (j & 1) && s == nd ? j - 1 : j;
  }
}

// Targets of the FP32 pair kernel: ion-ion terms act on mobile ions, the
// RFPAR cross term on every ion in the map, so with RFPAR on the targets
// start at the first ion, else at the first mobile ion.
struct PairCfg32 {
  bool ii, rf;
  int t0, ntg;  // first target, number of target slots below ntot_ub
};
inline PairCfg32 pair_cfg32(const KP &p, int ntot_ub, uint32_t mask) {
  PairCfg32 c{};
  c.ii = (mask & 1u) && ntot_ub > p.nsites + p.nfix;
  c.rf = (mask & 16u) && p.qrfpar && ntot_ub > p.nsites;
  c.t0 = c.rf ? p.nsites : p.nsites + p.nfix;
  c.ntg = (c.ii || c.rf) ? ntot_ub - c.t0 : 0;
  return c;
}

struct AssembleFlags {
  int ii, is, rf;     // which partial-force buffers are valid
  int ii_from;        // first particle with ion-ion (fused FP32: pair) partials
  int nchunk_ii, nchunk_rf;
  int fp32_partials;  // FP32 mode: float partials, float-float positions
  int use_total;      // the force is fx,fy,fz as assembled earlier (dynamics())
  int ntile;          // partials are per tile pair (Newton-3 kernels)
  int wave;           // FP32 Newton-3: n3_split_of's
  int rf_ab;          // Newton-3: add A sd1 + B sd2 of the RFPAR chain
  int nofield;        // no single-particle forces: ffield is not read
};

// mmij.cu: MMIJ reaction field (energy into slot `slot`, forces added to
// ffield / ffield_f); INTERACT's term of p.trial added to *dener
constexpr int kMmChunk = 16;  // ions per partial sum of the coefficients
int mmij_chunks(const KP &p, int ntot_ub);
int mmij_table_width(int rect, int nx, int ny, int nz, int nmpol);
int launch_mmij_energy(const KP &p, bool fp32, int ntot_ub, int slot, cudaStream_t stream);
int launch_mmij_force(const KP &p, bool fp32, int ntot_ub, cudaStream_t stream);
void launch_mmij_tables(const KP &p, int ntot_ub, cudaStream_t stream);  // INTERACT's
void launch_mmij_total(const KP &p, double *dener, cudaStream_t stream);

// gcmc.cu: COUNT (count.f90) on the device; ff: positions from the
// float-float records
int launch_count(const KP &p, bool ff, int ntot_ub, cudaStream_t stream);  // launches

// analysis.cu: per-cycle profiles (counts) and .btr frames
struct ProfArgs {
  int rho, rdna, gr;        // which profiles accumulate
  double zmini, idelz;      // z bins: iz = int((z - zmini) idelz) + 1
  int nzmax;
  int igr, npoints;         // RDF centre (0-based) and shells
  double dr;
  unsigned long long *rho_n, *rdna_n, *gr_n;  // [(ntype-nold)*nzmax], [ndna*nzmax], [(ntype-nold)*npoints]
  int *irmax;
};
void launch_profiles(const KP &p, bool fp32, int ntot_ub, const ProfArgs &a,
                     cudaStream_t stream);
void launch_traj_pack(const KP &p, bool fp32, int n, double runtime, uint32_t *w,
                      cudaStream_t stream);

// nucl.cu: DNA bonded and Go-like terms; forces into fis / fis_f of the
// sites (added when accum, else written), energies into one slot
int launch_nucl(const KP &p, bool fp32, uint32_t mask, int qforces, int accum, int slot,
                cudaStream_t stream);
int nucl_slots(const KP &p);  // energy slots launch_nucl writes
// NOTRAN after a BD step: the sites' centre back to notr along the flagged
// axes (one block); returns the launches (0 when off)
int launch_notrans(const KP &p, bool fp32, cudaStream_t stream);
// INTERACT of site j (0-based): adds its bonded/Go terms to *dener
void launch_nucl_interact(const KP &p, uint32_t mask, int j, double *dener,
                          cudaStream_t stream);

// fields.cu: single-particle terms, one warp per particle
int fields_blocks(int ntot_ub, bool fp32);
void launch_fields(const KP &p, int ntot_ub, uint32_t mask, int qforces, bool fp32,
                   int slot0, cudaStream_t stream);
// FP32 mode: FP64 coordinates -> float-float records (to_records) or back
void launch_pack(const KP &p, int ntot_ub, bool to_records, cudaStream_t stream);

// Host arrays through the context's pinned staging area, by one kernel each
// way (fields.cu).  In: n particles from src ([3][n] coordinates, [n] types,
// [n] buffer tags or null: none) and the live count.  Out: the live count and
// error word to head and, where given, the particles' arrays a (positions; ff:
// from the float-float records, also into p.x, p.y, p.z), types and tags, and
// the energy terms and warnings, for the entries below nub.
void launch_stage_in(const KP &p, int n, const double *xyz, const int *typei,
                     const int *ibuffer, cudaStream_t stream);
struct StageOut {
  int nub, stride;
  int ff;                 // positions from the records
  const double *a[3];     // [ntot] each, or null
  double *out;            // [3][stride]
  const int *ia[2];
  int *iout;              // [2][stride]
  const double *terms;
  double *tout;           // [kNTerms]
  const int *warn;
  int *wout, nwarn;
  int *head;              // ntot, err
};
void launch_stage_out(const KP &p, const StageOut &o, cudaStream_t stream);

// energy.cu
int launch_energy(const KP &p, const EnergyPlan &plan, uint32_t mask,
                  int qforces, cudaStream_t stream);
int energy_slots(const KP &p, const EnergyPlan &plan, uint32_t mask);
// cells.cu: the cell list of the FP32 extension mode and its pair kernel
// (block partial energies from `slot`); returns the kernels launched
int launch_cells(const KP &p, int ntot_ub, int qforces, int slot, cudaStream_t stream);
int cell_pair_blocks(const KP &p, int ntot_ub);
// Parts of a work item of the FP32 Newton-3 kernels for T tiles (the column's
// entries are met in one pass or in two halves by two warps), where `wave` warps
// fill the GPU once (n3_wave; 0: whole items): see energy.cu.  The kernels with
// parts take T, and so whether there are any, from the live count, as the FP64
// ones do: a run's rounding must not hang on when a read-back of the count
// arrived.  Where every count that there may be has whole items the host passes
// 0; the kernels are then those without, laid out for the bound (the order of a
// particle's sum is the same for any T).
__host__ __device__ inline int n3_split_of(int T, int wave) {
  return 2 * n3_items(T) <= wave ? 2 : 1;
}
int n3_wave();
inline int n3_split(int T) { return n3_split_of(T, n3_wave()); }
__host__ __device__ inline int n3_work(int T, int split) { return n3_items(T) * split; }
// Entries (64 lanes each) of the partial buffers for up to T tiles.
inline size_t n3_entries(int T) {
  size_t n = 1;
  for (int t = 1; t <= T; ++t) n = n > (size_t)n3_pairs(t) * n3_split(t) ? n : (size_t)n3_pairs(t) * n3_split(t);
  return n;
}
// Warps' items that a launch for a bound of T tiles holds: those of whatever count
// there may be at or below it.
inline int n3_most_work(int T, int wave) {
  int n = 0;
  for (int t = T; t > 0; --t) {
    const int s = n3_split_of(t, wave);
    n = n > n3_work(t, s) ? n : n3_work(t, s);
    if (s == 2 || wave == 0) break;  // fewer tiles have fewer items
  }
  return n;
}
int n3_blocks(int ntile, int wave);  // blocks (energy slots) of the Newton-3 pair kernel

// dyn.cu: force assembly, optionally fused with the BD update
void launch_assemble(const KP &p, int ntot_ub, const AssembleFlags &fl,
                     int do_bd, int variant, uint64_t seed, uint64_t step,
                     cudaStream_t stream);

// loop.cu: nsteps fused BD steps of the FP32 Newton-3 path in one
// cooperative launch (fields_first: evaluate the single-particle terms first)
bool bd_loop_supported(const KP &p, const AssembleFlags &fl);
cudaError_t launch_bd_loop(const KP &p, const AssembleFlags &fl, int ntot_ub, uint32_t mask,
                           int variant, uint64_t seed, uint64_t step0, int nsteps,
                           int fields_first, cudaStream_t stream);

// FP64 Newton-3 pair kernel.  Diagonal groups of a tile pair of T tiles, at
// most four (a group is eight diagonals, one per warp).  An item alone on its
// SM takes least, two on one share the FP64 pipe, and two blocks an SM go round
// by round, so groups pay while every item has an SM, and again where they turn
// two rounds of whole items into three of half ones.  50 steps of the fused
// loop, us, in 1 / 2 / 4 groups: 6 tile pairs 1098 / 861 / 707, 45: 1076 / 828
// / 890, 136: 1060 / 1127 / 1426, 210: 1490 / 1576 / 1806, 325: 2350 / 2069 /
// 2398, 528: 2400 / 2838 / 3363.
__host__ __device__ inline int n64_split(int T) {
  const int n = n3_pairs(T);
  if (4 * n <= kSMs) return 4;
  return 2 * n <= kSMs || (n > 2 * kSMs && n <= 3 * kSMs) ? 2 : 1;
}
// Blocks that share the items, two an SM at most.
__host__ __device__ inline int n64_blocks(int T) {
  const int n = n3_pairs(T) * n64_split(T);
  return n < 2 * kSMs ? n : 2 * kSMs;
}
// The kernels take T from the live count: the host's bound of it depends on
// when a read-back arrived, and a run's rounding must not.  So the items go over
// n64_blocks of the live tiles, and a launch for a bound of T tiles has the
// blocks of whatever count there may be at or below it: n64_blocks rises and
// falls (8 tiles 144, 9 tiles 90, 12 tiles 78).  Blocks beyond the live count's
// return at once.
inline int n64_grid(int T) {
  int n = 0;
  for (int t = 1; t <= T && n < 2 * kSMs; ++t) n = n > n64_blocks(t) ? n : n64_blocks(t);
  return n;
}
__device__ __forceinline__ int live_tiles(int ntot, int nsites) {
  return ntot > nsites ? (ntot - nsites + 31) / 32 : 0;
}
// loop64.cu: nsteps fused BD steps of the FP64 Newton-3 path
bool bd_loop64_supported(const KP &p, const AssembleFlags &fl);
cudaError_t launch_bd_loop64(const KP &p, const AssembleFlags &fl, uint32_t mask, bool ii,
                             bool srp, int variant, uint64_t seed, uint64_t step0, int nsteps,
                             cudaStream_t stream);

// gcmc.cu
// Metropolis moves (mc.cu): the chain's device record, reset per call.
struct McState {
  int iat, skip, draw, naccept;  // the move's ion (0-based), no position found, next draw
  double xn, yn, zn;             // its proposed position
  double e[2];                   // INTERACT at the old and the new position
  double dener;                  // accepted energy change of the call
};
// move.f90:19-45: a position is drawn again while it lies outside the
// system, at most kMcTries times (then the move is skipped).
constexpr int kMcTries = 1000;
// Moves evaluated together in one round of the Metropolis kernel (gcmc.cu),
// each at its old and its new position.
constexpr int kMcSpec = 8, kMcPos = 2 * kMcSpec;
constexpr int kMcMaxGrid = 512;
struct McRound {
  unsigned singles;          // single-particle terms formed since the launch began
  int na;                    // moves of the round (0: the launch ends)
  // per move and position (2k old, 2k + 1 new): the trial, its
  // single-particle terms and its warnings
  Trial tr[kMcPos];
  int nalert[kMcPos];
  double part[kMcMaxGrid][kMcPos];  // block partial sums of the pair terms
  int perr[kMcMaxGrid][kMcPos];     // and their error flags
};
int launch_metropolis(const KP &p, int ntot, uint32_t mask, int nmcm, double mcmax,
                      uint64_t seed, uint64_t cycle, McState *mc, McRound *rd,
                      cudaStream_t stream);
// gcmc.cu: the moves in one cooperative launch, in rounds of up to kMcSpec
cudaError_t launch_metropolis_rounds(const KP &p, int ntot, uint32_t mask, int nmcm,
                                     double mcmax, uint64_t seed, uint64_t cycle, McState *mc,
                                     McRound *rd, cudaStream_t stream);

void launch_interact(const KP &p, int ntot_ub, uint32_t mask, int qalert,
                     double *dener_dev, cudaStream_t stream, const SideStream &side = {});
// gcmc.cu: GRAND one attempt after another (systems with the MMIJ reaction
// field): proposal, INTERACT into *de_dev, acceptance, per attempt; the
// FP64 arrays move; returns the launches
int launch_grand_seq(const KP &p, int ntot_ub, uint32_t mask, uint64_t seed, uint64_t cycle,
                     int ngcmc, double *de_dev, cudaStream_t stream, const SideStream &side);
// GRAND: ngcmc attempts in one cooperative launch (gcmc.cu)
// ffpos: FP32 mode, positions in the float-float records (pk1, pk2)
cudaError_t launch_grand(const KP &p, int ntot_ub, int ipart_slots, uint32_t mask,
                         uint64_t seed, uint64_t cycle, int ngcmc, int ffpos,
                         cudaStream_t stream);
// partial slots for GRAND's widest grid at capacity cap (a lane per
// particle and attempt); INTERACT's need at cap is smaller
int grand_slots(int cap);
int interact_slots(int ntot_ub);

}  // namespace bgpu

// Read-only view of a context's uploaded pair laws, for entry points that
// live outside api.cu.  Returns false until set_system/types/pairs are done.
struct bromoc_ctx;
bool bromoc_ctx_pair_view(const bromoc_ctx *ctx, const bgpu::KP **kp,
                          cudaStream_t *stream, int *precision);
int bromoc_ctx_fail(bromoc_ctx *ctx, int code, const char *msg);
// FP32 prototype for a replica batch: completes its setup (scratch, FP32
// constants) and returns its parameter block.
int bromoc_ctx_prepare_f32(bromoc_ctx *ctx, const bgpu::KP **kp, cudaStream_t *stream);
// Replica batches and adjoint engines borrow their prototype context's
// stream and tables.  They attach a flag to it; a context destroyed before
// them sets the flag, and they then neither touch its stream nor run.
void bromoc_ctx_attach(bromoc_ctx *ctx, int *orphaned);
void bromoc_ctx_detach(bromoc_ctx *ctx, int *orphaned);
