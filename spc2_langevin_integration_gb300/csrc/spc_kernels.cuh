// Kernels of one right-hand-side evaluation and the fused stepper updates,
// for a batch of independent systems in one launch per phase.
//
// One evaluation (the reference's EvaluateInteractionsWithLinkedList,
// ChimeraSystem.cpp:258-426 / :429-645) runs as:
//   k_stage   stage state s + k_coef*dt*k_prev, copy-wrap, cell key  (ChimeraSystem.cpp:270-309)
//   sort      stable counting sort by global cell key (spc_sort.cuh)  (:335-338)
//   k_gather  particles into cell order + float prefilter coordinates
//   k_tile_*  (spc_tile.cuh) one CTA per cell: the 3x3 stencil in the
//             reference's order, the exact FP64 cutoff, the alignment sums,
//             then a fused epilogue (k_next, or the whole stepper update with
//             noise and the engine's periodic wrap).
// When rho > L/4 the reference switches to all pairs (ChimeraSystem.cpp:90-98)
// on unwrapped stage positions; such a system is one "cell" here and
// k_allpairs_pass handles it.
//
// Indexing.  State (x, y, phi, omega, RK4 rates) lives in a particle pool:
// system s owns pool slots [pool_p0, pool_p0 + n).  Each evaluation works on
// the dense list of the active systems' particles, d in [0, n_active) with
// system s at [dense_p0, dense_p0 + n); after the sort, slot p in
// [0, n_active) is cell order.  Cells are global: system s owns cells
// [c0, c0 + nc^2) (one cell for an all-pairs system).  Per-system constants
// come from the SysDesc table, so a single system and a batch of hundreds run
// the same kernels.
#pragma once

#include <cuda_fp16.h>

#include "spc_device.cuh"
#include "spc_sort.cuh"

namespace spc {

enum { kPrecFP64 = 0, kPrecFP32C = 1, kPrecFP32X = 2 };
// what a pass accumulates over the neighbours of i
enum { kKindSin = 0, kKindCos2 = 1, kKindNb = 2 };
// what the pass does with the sums (runtime, warp-uniform)
enum Epilogue {
  kEpiRkK = 0,         // write k_next into k slot `kq_out` (RK form)
  kEpiRk4Combine = 1,  // k4, then the RK4 combine and the wrap
  kEpiEuler = 2,       // StochasticEulerStepper update + wrap
  kEpiSrk1 = 3,        // SRK pass 1: phase rate and n_i in cell order
  kEpiEulerPtr = 4,    // StochasticEulerStepperPtr update + wrap
  kEpiSrk2 = 5,        // SRK pass 2 and the strong-1.5 update + wrap
  kEpiSrk2Out = 6,     // SRK pass 2, derivative / additional_derivative out
  kEpiCount = 7,       // neighbour counts
  kEpiList = 8,        // neighbour indices in visiting order
  kEpiLocalOrder = 9,  // per-particle local order parameter
};

constexpr int kFxyPad = 4;  // the lane kernel reads candidates four at a time
constexpr int kKSlots = 6;  // RK4 k1..k4 (persistent) + two scratch slots for spc_rhs_rk

// One system of a batch.
struct SysDesc {
  SysConst sc;
  int pool_p0;            // first pool slot
  int dense_p0;           // first dense index in the current layout
  int c0;                 // first global cell in the current layout
  int is_vortex;          // natural frequencies in the phase drift
  uint32_t system_id;     // Philox counter word
  uint64_t seed;          // Philox key
  unsigned long long step;     // steps taken before the current call (Philox counter)
  long long remaining;    // steps the system may still take (serving budget)
  int budget;             // steps of the current call it takes; later steps leave it frozen
};

// A particle's stage state and cell key, one 32-byte sector: the gather reads
// them in cell order.
struct alignas(32) StageRec {
  double x, y, phi;
  uint32_t key;
  int sys;
};

struct KArgs {
  const SysDesc *sys;
  int nsys;
  int n_active;                      // dense particles
  int ncell_total;
  int ncell_tile;                    // cells [0, ncell_tile): cell-tile kernels
  int tile_split;                    // cell-tile kernels: CTAs per cell (0 or 1: one)
  int lane_p0, lane_p1, va_p1;       // cell-order slots [lane_p0, lane_p1): lane kernel; [lane_p1, va_p1): vortex arrays
  const int *sys_of_p;               // dense index -> system
  const int *sys_of_c;               // global cell -> system
  // state pool (structure of arrays)
  double *x, *y, *phi;
  const double *omega;
  double *kx[kKSlots], *ky[kKSlots], *kphi[kKSlots];
  // stage (dense order)
  StageRec *stg;
  uint32_t *keys;                    // global cell key (dense order)
  int *arrival;                      // number of the particle among its cell's arrivals (dense order)
  int *cell_cnt;                     // key k's particles at [k << cnt_shift] (zero between evaluations); null: k_rank_gather
  int cnt_shift;
  int *list;                         // dense indices by cell, in order of arrival
  uint32_t *skeys;                   // key of each cell-order slot
  int *cell_start;
  // Sub-cells (SPC_TUNE_SUBCELLS; null when off): the sort key is 2c + h, h = 1
  // for the upper half of cell c (row_offset at least half a cell), and the
  // upper half starts at cell_mid[c].  cell_near[c] = 1 when a particle of
  // cell c lies within kNearHalf cell sides of the half line (cleared by
  // k_stage, set by k_gather).
  int *cell_mid;
  uint8_t *cell_near;
  // cell order
  double *sx, *sy, *sphi;
  float2 *fxy;                       // prefilter coordinates relative to the cell origin (slots [lane_p0,
                                     // va_p1): x relative to the column block's), kFxyPad entries more
  float2 *cs;                        // FP32C: (cos phi, sin phi)
  double2 *dcs;                      // FP64 passes: (cos phi, sin phi) of the stage phase
  uint16_t *rest;                    // and their rests (sincos_phase_rest)
  longlong2 *ics;                    // FP32X: (cos phi, sin phi) in fixed point (2^kXQ)
  // float forms, cell-tile slots: the values of the two passes as digits in
  // halves, 16 bytes (FP32X: 32) a slot (float_digits, fixed_digits); FP32C SRK:
  // pass-1 sum_j cos(phi_j - phi_i - alpha)
  uint4 *dig, *wdig;
  float *scos_f;
  longlong2 *iws;                    // FP32X SRK: phase rate times (cos phi, sin phi), fixed point (2^xq2)
  double *scos;                      // FP32X SRK: pass-1 sum_j cos(phi_j - phi_i - alpha), cell order
  double2 *xsum;                     // FP32X: a pass's exact neighbour sums (c, s), cell order
  int *xcnt;                         // FP32X: a pass's neighbour count, cell order
  int *pidx;                         // pool slot of cell-order slot p
  double *dphi_s;                    // SRK pass 1 phase rate, cell order
  float *dphi_f;                     // same, float (FP32C)
  int *cnt_s;                        // n_i, cell order
  int *va_cnt2;                      // vortex arrays: cohesion partners, cell order
  uint32_t *nbmask;                  // pass-1 neighbour bitmasks for the SRK second pass (mask_at), or null
  // Cell units of the float cell-tile passes (SPC_TUNE_CELL_UNITS; units
  // null when off): the units k_list_units lists for the units kernel
  // (cell, unit), their count (zeroed by k_gather), per staging
  // round r and cell-order slot p at [r * n_active + p] a unit's sums (fixed-point
  // pair) and counts, and a completion counter
  // per 32-particle chunk, indexed by its first slot (zero between launches).
  int2 *units;
  int *unit_count;
  uint8_t *cell_unit;  // per cell-tile cell: 1 if it runs as units (written with the list)
  longlong2 *part_x;
  int *part_n;
  int *unit_done;
  const int *ap_cells;               // global cells of the all-pairs systems
  int n_ap;
  // parity / diagnostics outputs, indexed by pool slot
  double *out_d, *out_a, *out_r;
  int *out_cnt;
  const long long *list_off;
  int *list_idx;
  // stepping
  double dt;
  double sdt;                        // sqrt(dt), rounded once on the host
  int kq_out;                        // k slot written by kEpiRkK / kEpiRk4Combine (k4)
  const double *noise;               // injected normals of this step (pool-indexed), or null
  int noise_m;                       // normals per particle
  int step_off;                      // this step = sys.step + step_off
  unsigned long long *clamped;
  // Verlet rows (null / 0 on the cell-list path)
  const int *gate;                   // binning kernels return at once when *gate == 0
  int *vsys, *vcell;                 // build: system and cell of each cell-order slot
  uint16_t *vrows;                   // row entry k of slot v at vrows[((k / 8) * n_active + v) * 8 + k % 8]
  int *vrowlen;                      // entries of each row, -1: overflow (scan the stencil)
  int vcap;                          // row limit of the current build
  double *vxb, *vyb;                 // stage positions at the build
  int *vflags;                       // [0] rebuild needed this evaluation, [1] forced
  unsigned long long *vrebuilds;
};

// Global cell of cell-order slot p (its sort key, halved with sub-cells).
__device__ __forceinline__ int cell_of_slot(const KArgs &a, int p) {
  const int k = (int)a.skeys[p];
  return a.cell_mid ? k >> 1 : k;
}

// Sub-cells: a stage y's offset above the lower edge of its cell row cy.  It
// decides the half (upper when >= cell / 2) in k_stage and the near flag in
// k_gather, the same expression in both.
__device__ __forceinline__ double row_offset(const SysConst &sc, double y, int cy) {
  return dsub(y, dmul((double)cy, sc.cell));
}

// A half's stencil leaves out the far half of the row beyond it.  The pairs
// left out are more than a cell side (>= rho) apart unless both particles
// lie within rounding of the half line, so each cell records whether any of
// its particles lies within kNearHalf cell sides of the line, and a far cell
// stays whole when both it and the half's own cell do.  2^-20 of a cell is
// far above the rounding of the row offsets and of the reference's distance
// (a few ulps of L, L < 2^30 cells), and holds ~2e-6 of the particles.
constexpr double kNearHalf = 0x1p-20;

// ---------------------------------------------------------------------------
// k_stage: rk = s + (k_coef*dt) * k_prev (ChimeraSystem.cpp:274-276), the copy
// wrap and cell key (:295-308).  kq < 0 means k_prev is all zeros (the Euler
// stepper's zero-filled buffer, StochasticEulerStepper.hpp:34); rk_form = 0 is
// the SRK form, whose stage state is the state itself (:456-458).  With
// sub-cells the key also carries the half of the cell (the upper half when
// the stage y is at least half a cell above the cell's lower edge).
// It also counts the key's particles and numbers its arrivals (spc_sort.cuh).
constexpr int kStageThreads = 256;
constexpr int kRankBits = 12;  // k_rank_gather: a particle's entry of `keys` is key << kRankBits | index

__global__ void __launch_bounds__(kStageThreads) k_stage(KArgs a, int rk_form, int kq, double kcdt) {
  if (a.gate && *a.gate == 0) return;
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (a.cell_mid)  // this evaluation's near flags (set by k_gather)
    for (int c = d; c < a.ncell_total; c += gridDim.x * blockDim.x) a.cell_near[c] = 0;
  if (d >= a.n_active) return;
  const int s = a.sys_of_p[d];
  const SysDesc &sd = a.sys[s];
  const SysConst &sc = sd.sc;
  const int i = d - sd.dense_p0, q = sd.pool_p0 + i;
  double x = a.x[q], y = a.y[q], ph = a.phi[q];
  if (rk_form) {
    const double kx = kq >= 0 ? a.kx[kq][q] : 0.0;
    const double ky = kq >= 0 ? a.ky[kq][q] : 0.0;
    const double kp = kq >= 0 ? a.kphi[kq][q] : 0.0;
    x = dadd(x, dmul(kcdt, kx));
    y = dadd(y, dmul(kcdt, ky));
    ph = dadd(ph, dmul(kcdt, kp));
  }
  uint32_t key;
  int arrival = i;
  if (sc.allpairs) {
    // all pairs use the unwrapped stage positions (ChimeraSystem.cpp:135-153),
    // in index order
    key = a.cell_mid ? 2u * (uint32_t)sd.c0 : (uint32_t)sd.c0;
    if (i == 0 && a.cell_cnt) a.cell_cnt[(size_t)key << a.cnt_shift] = sc.n;
  } else {
    wrap_if_outside(sc, x, y);
    int clamped = 0;
    const int cx = cell_coord(sc, x, clamped);
    const int cy = cell_coord(sc, y, clamped);
    if (clamped) atomicAdd(a.clamped, 1ull);
    key = (uint32_t)(sd.c0 + cy * sc.nc + cx);
    if (a.cell_mid) key = 2u * key + (row_offset(sc, y, cy) >= 0.5 * sc.cell ? 1u : 0u);
    if (a.cell_cnt) arrival = atomicAdd(&a.cell_cnt[(size_t)key << a.cnt_shift], 1);
  }
  StageRec r;
  r.x = x;
  r.y = y;
  r.phi = ph;
  r.key = key;
  r.sys = s;
  a.stg[d] = r;
  if (a.cell_cnt) {
    a.keys[d] = key;
    a.arrival[d] = arrival;
  } else {
    a.keys[d] = key << kRankBits | (uint32_t)d;
    if (d == a.n_active - 1)
      for (int k = d + 1; k & 3; ++k) a.keys[k] = 0xffffffffu;
  }
}

// Phase reduced to about [-pi, pi] in double, then float (FP32C trig input).
__device__ __forceinline__ float reduced_phase_f(double ph) {
  const double two_pi = 6.283185307179586;
  const double inv_two_pi = 0.15915494309189535;
  return (float)(ph - two_pi * rint(ph * inv_two_pi));
}

// Column blocks of a row of nc cells (particle-per-lane passes): blocks of 16,
// the last one up to 31; the first column of cx's block.
__device__ __forceinline__ int block_first(int cx, int nc) {
  return min(cx >> 4, max((nc >> 4) - 1, 0)) << 4;
}

// A candidate's record for the float cell-tile passes (spc_ftile.cuh): signed
// digits, each exact in a half, whose sums the tensor cores keep exact.
// FP32C: three digits in base 4096 each of x and y (|x|, |y| <= 1 up to float
// rounding; units of 2^-35), 1, and 1 if either is not finite.  (A value below
// 2^-11 keeps fewer bits than its float, but the phase's own rounding is 2^-24:
// mean errors of the rates against FP64, n = 16,384, alpha = 0, phases spread by
// 1e-2 to 1e-5 about 1: 2.6e-8, with float sums 2.9e-8; about 0: 3.3e-10 to
// 5.4e-13, with float sums 4.1e-10 to 3.5e-13.)
__device__ __forceinline__ uint32_t halves(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ uint4 float_digits(float x, float y) {
  const bool bad = !(fabsf(x) < 1.5f && fabsf(y) < 1.5f);
  if (bad) x = y = 0.0f;
  const float x2 = rintf(x * 2048.0f), rx = fmaf(x, 2048.0f, -x2) * 4096.0f, x1 = rintf(rx);
  const float y2 = rintf(y * 2048.0f), ry = fmaf(y, 2048.0f, -y2) * 4096.0f, y1 = rintf(ry);
  return make_uint4(halves(x2, x1), halves(rintf((rx - x1) * 4096.0f), y2),
                    halves(y1, rintf((ry - y1) * 4096.0f)), halves(1.0f, bad ? 1.0f : 0.0f));
}
// FP32X: five digits in base 2048 each of x and y (|x|, |y| < 2^54), lowest
// first, 1, and 1 if they are kNotFixed, zeros.
__device__ __forceinline__ void fixed_digits(longlong2 v, uint4 *to) {
  float d[10];
  const bool bad = v.x == kNotFixed;
  if (bad) v = make_longlong2(0, 0);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    long long r = h ? v.y : v.x;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int low = (int)((uint32_t)r << 21) >> 21;
      d[5 * h + k] = (float)low;
      r = (r - low) >> 11;
    }
    d[5 * h + 4] = (float)(int)r;
  }
  to[0] = make_uint4(halves(d[0], d[1]), halves(d[2], d[3]), halves(d[4], d[5]), halves(d[6], d[7]));
  to[1] = make_uint4(halves(d[8], d[9]), halves(1.0f, bad ? 1.0f : 0.0f), 0u, 0u);
}

// What the FP64 passes need of a phase, for slot p.
// REST: false when no system has rests (rest_on).
template <bool REST>
__device__ __forceinline__ void gather_cs64(const KArgs &a, const SysConst &sc, double ph, int p) {
  double s, c;
  if (REST && sc.rest_on)
    a.rest[p] = sincos_phase_rest(ph, s, c);
  else
    sincos_phase(ph, s, c);
  a.dcs[p] = make_double2(c, s);
}

// Dense particle d into cell-order slot p.
template <int PREC, bool REST>
__device__ __forceinline__ void gather_to(const KArgs &a, int d, const StageRec &r, int p) {
  const SysDesc &sd = a.sys[r.sys];
  const SysConst &sc = sd.sc;
  const double x = r.x, y = r.y, ph = r.phi;
  a.skeys[p] = r.key;
  a.sx[p] = x;
  a.sy[p] = y;
  a.sphi[p] = ph;
  a.pidx[p] = sd.pool_p0 + (d - sd.dense_p0);
  const int cell = (int)(a.cell_mid ? r.key >> 1 : r.key);
  if (a.vsys) {  // Verlet build: remember each slot's system and cell until the next build
    a.vsys[p] = r.sys;
    a.vcell[p] = cell;
  }
  if (!sc.allpairs) {
    const int key = cell - sd.c0;
    const int cx = key % sc.nc, cy = key / sc.nc;
    const int ox = p >= a.lane_p0 && p < a.va_p1 ? block_first(cx, sc.nc) : cx;
    a.fxy[p] = make_float2((float)__fma_rn(-(double)ox, sc.cell, x), (float)__fma_rn(-(double)cy, sc.cell, y));
    if (a.cell_mid && fabs(row_offset(sc, y, cy) - 0.5 * sc.cell) < kNearHalf * sc.cell)
      a.cell_near[sd.c0 + key] = 1;
  }
  if constexpr (PREC == kPrecFP32C) {
    float s, c;
    sincosf(reduced_phase_f(ph), &s, &c);
    a.cs[p] = make_float2(c, s);
    if (p < a.lane_p0) a.dig[p] = float_digits(c, s);
  }
  if constexpr (PREC == kPrecFP32X) {
    double s, c;
    sincos_phase(ph, s, c);
    const longlong2 v = to_fixed2(c, s, kXQ);
    a.ics[p] = v;
    if (p < a.lane_p0) fixed_digits(v, a.dig + 2 * (size_t)p);
    if (sc.allpairs) gather_cs64<REST>(a, sc, ph, p);  // its passes are the FP64 ones
  }
  if constexpr (PREC == kPrecFP64) gather_cs64<REST>(a, sc, ph, p);
}

template <int PREC, bool REST>
__global__ void k_gather(KArgs a) {
  if (a.gate && *a.gate == 0) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n_active) return;
  if (t == 0 && a.unit_count) *a.unit_count = 0;  // this evaluation's cell units (k_list_units)
  const int d = a.list[t];
  const StageRec r = a.stg[d];
  int p = t;  // cell-order slot: the cell's indices below d come before it
  if (!a.sys[r.sys].sc.allpairs) {
    const int c0 = key_start(r.key, a.cell_start, a.cell_mid), c1 = key_end(r.key, a.cell_start, a.cell_mid);
    p = c0;
    int k = c0;
    for (; k < c1 && (k & 3); ++k) p += a.list[k] < d ? 1 : 0;
#pragma unroll 4
    for (; k + 3 < c1; k += 4) {
      const int4 v = *reinterpret_cast<const int4 *>(a.list + k);
      p += (v.x < d ? 1 : 0) + (v.y < d ? 1 : 0) + (v.z < d ? 1 : 0) + (v.w < d ? 1 : 0);
    }
    for (; k < c1; ++k) p += a.list[k] < d ? 1 : 0;
  }
  gather_to<PREC, REST>(a, d, r, p);
}

// Few particles: no counting and no list.  Sixteen lanes count the particles
// before a given one in (key, index) order, which is its slot, and likewise
// those before each key's first, which is its start; then the particle is
// gathered.  n^2 compares, but two launches less than the counting sort and no
// chain of dependent loads.  An Euler step with it and with the counting sort,
// FP64, us:
// N = 300 23.2 and 27.7, 1,024 24.9 and 28.6, 2,048 27.0 and 29.2, 3,000 30.1 and
// 29.9, 4,096 31.9 and 31.0; eight lanes 27.7 and thirty-two 27.0 at 1,500 (26.8).
constexpr int kRankMax = 2048;
constexpr int kRankLanes = 16, kRankThreads = 32;
static_assert(kRankMax <= 1 << kRankBits && (uint64_t)kScanOneCta << kRankBits < 0xffffffffu, "ranks fit 32 bits");

template <int PREC, bool REST>
__global__ void __launch_bounds__(kRankThreads) k_rank_gather(KArgs a, int nkeys) {
  if (a.gate && *a.gate == 0) return;
  const int n = a.n_active;
  const int q = (blockIdx.x * kRankThreads + threadIdx.x) / kRankLanes, sub = threadIdx.x % kRankLanes;
  if (q == 0 && sub == 0) {
    a.cell_start[a.ncell_total] = n;
    if (a.unit_count) *a.unit_count = 0;  // this evaluation's cell units (k_list_units)
  }
  // queries [0, n): the particles, [n, n + nkeys): the keys
  const uint32_t key = (uint32_t)min(q - n, nkeys - 1), own = q < n ? a.keys[q] : key << kRankBits;
  int p = 0;
#pragma unroll 4
  for (int j = 4 * sub; j < n; j += 4 * kRankLanes) {
    const uint4 k = *reinterpret_cast<const uint4 *>(a.keys + j);  // padded to fours
    p += (k.x < own ? 1 : 0) + (k.y < own ? 1 : 0) + (k.z < own ? 1 : 0) + (k.w < own ? 1 : 0);
  }
#pragma unroll
  for (int off = 1; off < kRankLanes; off <<= 1) p += __shfl_xor_sync(0xffffffffu, p, off);
  if (sub != 0) return;
  if (q < n)
    gather_to<PREC, REST>(a, q, a.stg[q], p);
  else if (q < n + nkeys)
    (a.cell_mid && (key & 1u) ? a.cell_mid : a.cell_start)[a.cell_mid ? key >> 1 : key] = p;
}

// ---------------------------------------------------------------------------
// Per-i accumulators of one pass.
template <int PREC>
struct Acc;

template <>
struct Acc<kPrecFP64> {
  double s0, s1;  // sin sum | cos/n sum, (dphi) cos/n sum | cos, sin sums
  int n;
  long long rest; // sin sum: the terms' rests, in units of 2^-68 (sine_rest; up to 2^17 each)
  __device__ void init() { s0 = 0.0; s1 = 0.0; n = 0; rest = 0; }
};

template <>
struct Acc<kPrecFP32C> {
  float s0, c0, s1, c1;  // Kahan sums and compensations
  int n;
  __device__ void init() { s0 = c0 = s1 = c1 = 0.0f; n = 0; }
};

// Word w (< 32) of the pass-1 neighbour bitmask of cell-order slot p among n
// active particles.  Four consecutive words of a particle share one 16-byte
// group, and all kernels of a pass that index a buffer this way never share a
// word.  (The Verlet kernels keep a word-major layout of their own: a Verlet
// engine holds one system and runs no other neighbour kernel in the pass.)
__device__ __forceinline__ size_t mask_at(int w, int p, int n) {
  return ((size_t)(w >> 2) * n + p) * 4 + (w & 3);
}

// Float prefilter offset of a candidate at (dx, dy) from a value near rho^2, in
// two fused multiply-adds.  Float error is ~1e-7 rho^2 (1.6e-5 at most over the
// column blocks of the particle-per-lane passes), inside the band of 3e-5 rho^2.
__device__ __forceinline__ float cutoff_offset(float dx, float dy, float nmid) {
  return fmaf(dx, dx, fmaf(dy, dy, nmid));
}

// Every neighbour kernel decides a candidate from one offset: the float cell-tile
// and Verlet kernels from d^2 - mid, inside when off < -band, undecided (the
// reference's FP64 test decides) when |off| <= band; the others (k_tile_fp64,
// k_lane, k_allpairs_pass) from d^2 - lo2, inside when it is negative, undecided
// up to hi2 - lo2; outside otherwise.  The inside and undecided sets are then
// disjoint and leave no gap below hi2.  Deciding instead from d^2 < lo2
// and |d^2 - mid| <= band separately leaves one: mid = (lo2 + hi2) / 2 is
// rounded, and for about one rho in five |lo2 - mid| exceeds band by a
// fraction of an ulp, so a float d^2 equal to lo2 is in neither set and a pair
// just inside the cutoff (d^2 ~ rho^2 (1 - 3e-5)) is dropped.
__device__ __forceinline__ bool float_inside(float off, float band) { return off < -band; }
__device__ __forceinline__ bool float_undecided(float off, float band) { return fabsf(off) <= band; }

__device__ __forceinline__ void kahan_add(float &sum, float &comp, float v) {
  const float y = v - comp;
  const float t = sum + y;
  comp = (t - sum) - y;
  sum = t;
}

// Everything an i lane needs inside the candidate loop.
struct ILane {
  int p;        // cell-order slot
  bool valid;
  float fx, fy; // prefilter coordinates
  double x, y;  // wrapped stage position
  double phi;   // stage phase
  int cnt;      // pass 2: n_i from pass 1
  double dphi;  // pass 2: own phase rate
  float ca, sa; // FP32C: cos(phi + alpha), sin(phi + alpha)
  double dca, dsa;  // FP64: the same in double
  bool rest;        // FP64 pass 1: sine_rest, with the sectors that are near and
  int rest_from, rest_own;  // the own rest (units of 2^-68, with the offset)
  uint32_t dsa_lo, dsa_hi;  // dsa's significand and exponent, for rest_of_product
  int dsa_e;
  float dphif;
};

// FP64 pair terms.  The reference evaluates sin (SRK second pass: cos) of
// phi_j - phi_i - alpha per pair (ChimeraSystem.cpp:412, :634-637).  Here both
// come from the angle-difference identities with each particle's cos phi and
// sin phi, evaluated once by the gather, and with theta_i = phi_i + alpha by
// angle addition: two operations of the FP64 pipe per term instead of the ~25
// of a sine (GB300 runs FP64 at 1/64 of the FP32 rate, and the pair terms
// filled that pipe: 75% busy).  A term's absolute error is below 3.5e-16, as
// that of the sine of the twice rounded difference; a term below 2^-11, whose
// relative error would pass 7e-13 (1e-12 is the right-hand sides' contract),
// is evaluated as the reference writes it: 1 term in 1,600 of unrelated
// phases.  The terms are added in the reference's order as before; the mean of
// 200 terms is 2.4e-17 (uniform phases, before 2.9e-17) to 3.5e-16 (aligned,
// alpha = 1.45: the same as before) from the exact one.  Vortex SRK step,
// N = 65,536: 2.96 -> 0.45 ms on the cell list (0.47 with the rests below).
//
// Between aligned phases (alpha small) 3.5e-16 is far more than the rounding of
// the small sine that the reference gets.  Three things make up that error: the
// rounding of the particles' cosines and sines, which turns either by up to
// 2^-53.4; that of (dca, dsa); and that of one product.  The first two are kept
// as an angle per particle (rest), the third is found by an integer product, and
// where the phases are within two sectors of 22.5 degrees (the cosine of the
// difference is near 1) their sum goes to an integer, so that it depends on no
// order.  Mean of 200 terms, error against 64 bits over that of the sines of the
// differences, phases spread by sd about one phase, alpha = 0: sd 3e-4 54 -> 1.1,
// 1e-3 47 -> 1.0, 1e-2 6.7 -> 1.1, 0.1 1.2 -> 1.0 (20 terms: 170, 139, 18, 2.2 ->
// at most 1.3); alpha = 0.1, sd 1e-2: 1.3 -> 1.0.  From |alpha| = 0.5 on the
// reference's own rounding of the difference is as large, and nothing is kept.
// Some 25 integer instructions a pair, beside the 48 cycles that the FP64 pipe
// takes for a warp's pair, and 28 FP64 operations a particle in the gather: vortex
// SRK, N = 65,536, pass 1 171 -> 189 us and gather 6 -> 9 (with the product's rest
// by a fused multiply-add, pass 1 was 220).
constexpr double kRestAlpha = 0.5;
constexpr uint32_t kRestNear = 5u << 12;
// (c dsa - p) 2^68, p = RN(c dsa), |p| <= 1, by integers: the product of the
// significands from its last place of p on, modulo 2^64, is what rounding left of
// it, a signed number of 52 or 53 bits.
__device__ __forceinline__ int rest_of_product(const ILane &il, double c, double p) {
  const int hi = __double2hiint(c), ep = (__double2hiint(p) >> 20) & 0x7ff;
  const uint32_t lo = (uint32_t)__double2loint(c), mh = ((uint32_t)hi & 0xfffffu) | 0x100000u;
  const uint64_t low = (uint64_t)lo * il.dsa_lo;
  const uint32_t up = (uint32_t)(low >> 32) + lo * il.dsa_hi + mh * il.dsa_lo;
  const int carry = ep - ((hi >> 20) & 0x7ff) - il.dsa_e;  // 1: 53 bits
  const int x = (int)__funnelshift_l((uint32_t)low, up, 12 - carry);
  const int v = x >> min((unsigned)(1039 - ep), 31u);
  return __double2hiint(p) < 0 ? -v : v;
}
// What the term fma(cj.y, dca, -p), p = RN(cj.x dsa), lacks; w: j's rest.
__device__ __forceinline__ int sine_rest(const ILane &il, uint32_t w, double cjx, double p) {
  const int v = (int)((w & 0xfffu) << 4) - il.rest_own - rest_of_product(il, cjx, p);
  return ((w - (uint32_t)il.rest_from) & 0xffffu) < kRestNear ? v : 0;
}
__device__ __noinline__ double sin_of_difference(double pj, double pi, double alpha) {
  return sin(dsub(dsub(pj, pi), alpha));
}
__device__ __noinline__ double cos_of_difference(double pj, double pi, double alpha) {
  return cos(dsub(dsub(pj, pi), alpha));
}
// |t| < 2^-11
__device__ __forceinline__ bool small_term(double t) {
  return (unsigned)(__double2hiint(t) & 0x7fffffff) < 0x3f400000u;
}
// One accepted pair: pass 1 adds the sine, pass 2 the cosine and the cosine
// weighted by the difference of the phase rates.  phase() gives phi_j, rest() its
// rest.  The second pass's quotients by n_i are taken once of each sum
// (finish_pairs).
template <int KIND, class Phase, class Rest>
__device__ __forceinline__ void add_pair(Acc<kPrecFP64> &acc, const SysConst &sc, const ILane &il, double2 cj,
                                         double dj, Phase phase, Rest rest) {
  if constexpr (KIND == kKindSin) {
    const double p = dmul(cj.x, il.dsa);
    double t = __fma_rn(cj.y, il.dca, -p);
    if (small_term(t))
      t = sin_of_difference(phase(), il.phi, sc.alpha);
    else if (il.rest)
      acc.rest += sine_rest(il, rest(), cj.x, p);
    acc.s0 = dadd(acc.s0, t);
  } else {
    double t = __fma_rn(cj.x, il.dca, dmul(cj.y, il.dsa));
    if (small_term(t)) t = cos_of_difference(phase(), il.phi, sc.alpha);
    acc.s0 = dadd(acc.s0, t);
    acc.s1 = __fma_rn(dsub(dj, il.dphi), t, acc.s1);
  }
}
// A particle's neighbours as words of bits (bit 31 of a word is its entry
// `base`): next(bits, base) gives the next word that is not zero, cs(k), rate(k),
// phase(k) and rest(k) what entry k's pair needs.  U neighbours of a word are taken at
// a time: their terms are independent, so only the additions wait for one
// another (a dependent FP64 operation takes over 100 cycles, and the small
// systems have one warp per SM).
template <int KIND, int U, bool REST, class Next, class Cs, class Rate, class Phase, class Rest>
__device__ __forceinline__ void walk_pairs(Acc<kPrecFP64> &acc, const SysConst &sc, const ILane &il, Next next,
                                           Cs cs, Rate rate, Phase phase, Rest rest) {
  uint32_t bits = 0u;
  int base = 0;
  while (bits != 0u || next(bits, base)) {
    int k[U];
    bool has[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      has[u] = bits != 0u;
      const int t = __clz(bits);
      k[u] = has[u] ? base + t : k[0];
      bits &= ~(0x80000000u >> (t & 31));
    }
    double t[U], d[U];
    int r[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const double2 cj = cs(k[u]);
      r[u] = 0;
      if constexpr (KIND == kKindSin) {
        const double p = dmul(cj.x, il.dsa);
        t[u] = __fma_rn(cj.y, il.dca, -p);
        if (REST && il.rest) r[u] = sine_rest(il, rest(k[u]), cj.x, p);
      } else {
        t[u] = __fma_rn(cj.x, il.dca, dmul(cj.y, il.dsa));
      }
      d[u] = KIND == kKindCos2 ? dsub(rate(k[u]), il.dphi) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (small_term(t[u])) {
        t[u] = KIND == kKindSin ? sin_of_difference(phase(k[u]), il.phi, sc.alpha)
                                : cos_of_difference(phase(k[u]), il.phi, sc.alpha);
        r[u] = 0;
      }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!has[u]) continue;
      if constexpr (KIND == kKindSin) acc.rest += r[u];
      acc.s0 = dadd(acc.s0, t[u]);
      if constexpr (KIND == kKindCos2) acc.s1 = __fma_rn(d[u], t[u], acc.s1);
    }
  }
}
template <int KIND>
__device__ __forceinline__ void finish_pairs(Acc<kPrecFP64> &acc, const ILane &il) {
  if constexpr (KIND == kKindSin) {
    if (acc.rest != 0) acc.s0 = __fma_rn((double)acc.rest, 0x1p-68, acc.s0);
  } else if constexpr (KIND == kKindCos2) {
    if (il.cnt > 0) {
      const Count n = count_of(il.cnt);
      acc.s0 = ddiv_by(acc.s0, n.n, n.r);
      acc.s1 = ddiv_by(acc.s1, n.n, n.r);
    }
  }
}

// The float test of 32 staged candidates against one particle (FP64 passes):
// bit 31 - t of the result is the sign of candidate t's d^2 - lo2, set when
// it is inside for certain.  An undecided one (left to the reference's FP64
// test) has an offset in [0, hi2 - lo2]; *um gets the smallest bit pattern of
// the offsets as an unsigned number, in which negative floats come last.  Two
// fused multiply-adds, one funnel shift and one minimum per candidate.
__device__ __forceinline__ uint32_t test32(const float2 *__restrict__ xy, float fx, float fy, float nlo,
                                           uint32_t &um) {
  uint32_t bits = 0u;
#pragma unroll
  for (int t = 0; t < kWarp; t += 2) {
    const float4 c = *reinterpret_cast<const float4 *>(xy + t);
    const float dx0 = c.x - fx, dy0 = c.y - fy, dx1 = c.z - fx, dy1 = c.w - fy;
    const uint32_t o0 = __float_as_uint(cutoff_offset(dx0, dy0, nlo));
    const uint32_t o1 = __float_as_uint(cutoff_offset(dx1, dy1, nlo));
    bits = __funnelshift_l(o0, bits, 1);
    bits = __funnelshift_l(o1, bits, 1);
    um = min(um, min(o0, o1));
  }
  return bits;
}
// bits of the first cnt candidates of a block (0 <= cnt <= 32)
__device__ __forceinline__ uint32_t first_bits(int cnt) {
  return cnt >= kWarp ? 0xffffffffu : ~(0xffffffffu >> cnt);
}
// upper end of the undecided band above lo2, rounded outwards
__device__ __forceinline__ float undecided_width(float lo2, float hi2) { return (hi2 - lo2) * 1.001f; }

template <int PREC, int KIND>
__device__ __forceinline__ void accept_pair(const KArgs &a, const SysDesc &sd, const ILane &il,
                                            Acc<PREC> &acc, int pj, float cjc, float cjs,
                                            float dphij_f, long long &wpos) {
  static_assert(PREC == kPrecFP32C || KIND == kKindNb, "FP64 sums: walk_pairs");
  if constexpr (KIND == kKindSin) {
    // sin(phi_j - (phi_i + alpha)) by the angle-difference identity
    kahan_add(acc.s0, acc.c0, cjs * il.ca - cjc * il.sa);
    acc.n++;
  } else if constexpr (KIND == kKindCos2) {
    const float c = cjc * il.ca + cjs * il.sa;
    kahan_add(acc.s0, acc.c0, c);
    kahan_add(acc.s1, acc.c1, (dphij_f - il.dphif) * c);
    acc.n++;
  } else {
    if (a.list_idx) a.list_idx[wpos++] = a.pidx[pj] - sd.pool_p0;
    if constexpr (PREC == kPrecFP64) {
      if (a.out_r) {
        const double2 cj = a.dcs[pj];
        acc.s0 += cj.x;
        acc.s1 += cj.y;
      }
    }
    acc.n++;
  }
}

__device__ __forceinline__ double noise_at(const KArgs &a, int q, int k, double z0, double z1) {
  if (a.noise) return a.noise[(size_t)q * a.noise_m + k];
  return k == 0 ? z0 : z1;
}

// v + sdt * 0.0 (StochasticEulerStepper.hpp:43: the position's noise is zero),
// by the bit pattern: it turns -0.0 into 0.0, or v into NaN with sdt.
__device__ __forceinline__ double plus_zero(double v, double sdt) {
  if ((__double2hiint(sdt) & 0x7ff00000) == 0x7ff00000) return dadd(v, dmul(sdt, 0.0));
  return __double_as_longlong(v) == (long long)0x8000000000000000ull ? 0.0 : v;
}

// Fused epilogue for the particle in pool slot q (system sd) at cell-order slot p.
template <int PREC, int KIND>
__device__ void epilogue(const KArgs &a, int epi, const SysDesc &sd, const ILane &il,
                         Acc<PREC> &acc, int q, const double2 *cs_known = nullptr) {
  const SysConst &sc = sd.sc;
  const int p = il.p;
  if constexpr (KIND == kKindNb) {
    if (epi == kEpiCount) a.out_cnt[q] = acc.n;
    if (epi == kEpiLocalOrder) {
      const double2 ci = a.dcs[p];
      const double re = acc.s0 + ci.x, im = acc.s1 + ci.y;
      a.out_r[q] = sqrt(re * re + im * im) / (double)(acc.n + 1);
    }
    return;
  }
  // past its step budget a system is frozen: no persistent state changes
  const bool live = a.step_off < sd.budget;
  const int i = q - sd.pool_p0;  // index within the system (Philox counter)
  const unsigned long long step = sd.step + (unsigned long long)a.step_off;
  double z0 = 0.0, z1 = 0.0;
  const bool draws = (epi == kEpiEuler || epi == kEpiEulerPtr || epi == kEpiSrk2) && !a.noise && live;
  const double dt = a.dt;
  if constexpr (PREC == kPrecFP64) {
    if (draws) philox_normal2(sd.seed, sd.system_id, step, (uint32_t)i, z0, z1);
    // cos / sin of the stage phase from the gather: the doubles, or (FP32X)
    // its fixed-point values, exact to 2^-53
    const double2 csp = cs_known ? *cs_known : a.dcs[p];
    const double cph = csp.x, sph = csp.y;
    const double d0 = dmul(sc.v0, cph), d1 = dmul(sc.v0, sph);  // v_0_ * cos(phi_i) (:419-420)
    if constexpr (KIND == kKindSin) {
      // sigma_ * alignment_force_[i] / neighborhood_cardinality_[i] (:421-424)
      const bool has = acc.n != 0;
      const Count cn = count_of(acc.n);
      const double rate = has ? ddiv_by(dmul(sc.sigma, acc.s0), cn.n, cn.r) : 0.0;
      if (epi == kEpiRkK || epi == kEpiRk4Combine) {
        if (!live) return;
        const int k = a.kq_out;
        a.kx[k][q] = d0;
        a.ky[k][q] = d1;
        if (has) a.kphi[k][q] = rate;  // otherwise k_next keeps its value (H5)
        if (epi == kEpiRk4Combine) {
          // RungeKutta4Stepper.cpp:52-54
          const double k4p = a.kphi[k][q];
          double xs = a.x[q], ys = a.y[q], ps = a.phi[q];
          const double sx_ = dadd(dadd(dadd(a.kx[0][q], dmul(2.0, a.kx[1][q])), dmul(2.0, a.kx[2][q])), d0);
          const double sy_ = dadd(dadd(dadd(a.ky[0][q], dmul(2.0, a.ky[1][q])), dmul(2.0, a.ky[2][q])), d1);
          const double sp_ = dadd(dadd(dadd(a.kphi[0][q], dmul(2.0, a.kphi[1][q])), dmul(2.0, a.kphi[2][q])), k4p);
          xs = dadd(xs, ddiv(dmul(sx_, dt), 6.0));
          ys = dadd(ys, ddiv(dmul(sy_, dt), 6.0));
          ps = dadd(ps, dmul(ddiv(sp_, 6.0), dt));
          a.x[q] = wrap_1d(xs, sc.rL, sc.L);  // SimulationEngine.cpp:154
          a.y[q] = wrap_1d(ys, sc.rL, sc.L);
          a.phi[q] = ps;
        }
      } else if (epi == kEpiEuler) {
        if (!live) return;
        // StochasticEulerStepper.hpp:43-45 with AddNoise (ChimeraSystem.cpp:927-930);
        // a vortex system adds its frequency to the phase drift as the
        // SRK-Ptr stepper does (StochasticRungeKuttaStepperPtr.hpp:65)
        const double sdt = a.sdt;
        const double sto = dmul(sc.s2D, noise_at(a, q, 0, z0, z1));
        const double xs = dadd(a.x[q], plus_zero(dmul(dt, d0), sdt));
        const double ys = dadd(a.y[q], plus_zero(dmul(dt, d1), sdt));
        const double drift = sd.is_vortex ? dadd(a.omega[q], rate) : rate;
        a.phi[q] = dadd(a.phi[q], dadd(dmul(dt, drift), dmul(sdt, sto)));
        a.x[q] = wrap_1d(xs, sc.rL, sc.L);
        a.y[q] = wrap_1d(ys, sc.rL, sc.L);
      } else if (epi == kEpiEulerPtr) {
        if (!live) return;
        // StochasticEulerStepperPtr.hpp:44-51
        const double dW = dmul(a.sdt, noise_at(a, q, 0, z0, z1));
        const double xs = dadd(a.x[q], dmul(d0, dt));
        const double ys = dadd(a.y[q], dmul(d1, dt));
        a.phi[q] = dadd(a.phi[q], dadd(dmul(rate, dt), dmul(sc.s2D, dW)));
        a.x[q] = wrap_1d(xs, sc.rL, sc.L);
        a.y[q] = wrap_1d(ys, sc.rL, sc.L);
      } else if (epi == kEpiSrk1) {
        a.dphi_s[p] = rate;  // derivative is zero-filled each step: 0 when isolated
        a.cnt_s[p] = acc.n;
      }
    } else {  // kKindCos2: SRK pass 2 (ChimeraSystem.cpp:642-643)
      const double A0 = dmul(acc.s0, -sc.s2D);
      const double A1 = dadd(acc.s1, dmul(dmul(-2.0, sc.D), il.dphi));
      const double d2 = il.dphi;
      if (epi == kEpiSrk2Out) {
        a.out_d[3 * (size_t)q] = d0;
        a.out_d[3 * (size_t)q + 1] = d1;
        a.out_d[3 * (size_t)q + 2] = d2;
        a.out_a[2 * (size_t)q] = A0;
        a.out_a[2 * (size_t)q + 1] = A1;
      } else {
        if (!live) return;
        // StochasticRungeKuttaStepper.hpp:44-55 (+ omega: StochasticRungeKuttaStepperPtr.hpp:65)
        const double U1 = noise_at(a, q, 0, z0, z1), U2 = noise_at(a, q, 1, z0, z1);
        const double sdt = a.sdt;
        const double dW = dmul(U1, sdt);
        const double dZ = dmul(dmul(dmul(0.5, dt), sdt), dadd(U1, ddiv_by(U2, kSqrt3, kRcpSqrt3)));
        const double D = sc.D;
        const double s2D = sc.s2D;
        const double dtdt_x = dmul(dmul(dmul(0.5, dadd(dmul(d2, d1), dmul(D, d0))), dt), dt);
        const double xs = dadd(a.x[q], dsub(dsub(dmul(d0, dt), dmul(dmul(s2D, d1), dZ)), dtdt_x));
        const double dtdt_y = dmul(dmul(dmul(0.5, dsub(dmul(d2, d0), dmul(D, d1))), dt), dt);
        const double ys = dadd(a.y[q], dadd(dadd(dmul(d1, dt), dmul(dmul(s2D, d0), dZ)), dtdt_y));
        const double drift = sd.is_vortex ? dmul(dadd(a.omega[q], d2), dt) : dmul(d2, dt);
        const double ps = dadd(a.phi[q], dadd(dadd(dadd(drift, dmul(s2D, dW)), dmul(A0, dZ)),
                                              dmul(dmul(dmul(0.5, A1), dt), dt)));
        a.x[q] = wrap_1d(xs, sc.rL, sc.L);
        a.y[q] = wrap_1d(ys, sc.rL, sc.L);
        a.phi[q] = ps;
      }
    }
  } else {
    // FP32C: right-hand sides and increments in float, accumulated into the
    // double positions and phase.
    float f0 = 0.0f, f1 = 0.0f;
    if (draws) philox_normal2_f(sd.seed, sd.system_id, step, (uint32_t)i, f0, f1);
    auto noise_f = [&](int k) -> float {
      if (a.noise) return (float)a.noise[(size_t)q * a.noise_m + k];
      return k == 0 ? f0 : f1;
    };
    // cos / sin of the stage phase, as the gather computed them for this slot
    const float2 csp = a.cs[p];
    const float cph = csp.x, sph = csp.y;
    const float v0 = (float)sc.v0, D = (float)sc.D, dtf = (float)dt;
    const float d0 = v0 * cph, d1 = v0 * sph;
    if constexpr (KIND == kKindSin) {
      const bool has = acc.n != 0;
      const float rate = has ? (float)sc.sigma * acc.s0 / (float)acc.n : 0.0f;
      if (epi == kEpiRkK || epi == kEpiRk4Combine) {
        if (!live) return;
        const int k = a.kq_out;
        a.kx[k][q] = (double)d0;
        a.ky[k][q] = (double)d1;
        if (has) a.kphi[k][q] = (double)rate;
        if (epi == kEpiRk4Combine) {
          const float k4p = (float)a.kphi[k][q];
          const float sx_ = (float)a.kx[0][q] + 2.0f * (float)a.kx[1][q] + 2.0f * (float)a.kx[2][q] + d0;
          const float sy_ = (float)a.ky[0][q] + 2.0f * (float)a.ky[1][q] + 2.0f * (float)a.ky[2][q] + d1;
          const float sp_ = (float)a.kphi[0][q] + 2.0f * (float)a.kphi[1][q] + 2.0f * (float)a.kphi[2][q] + k4p;
          const float sixth = dtf / 6.0f;
          a.x[q] = wrap_1d(a.x[q] + (double)(sx_ * sixth), sc.rL, sc.L);
          a.y[q] = wrap_1d(a.y[q] + (double)(sy_ * sixth), sc.rL, sc.L);
          a.phi[q] = a.phi[q] + (double)(sp_ * sixth);
        }
      } else if (epi == kEpiEuler || epi == kEpiEulerPtr) {
        if (!live) return;
        const float xi = noise_f(0);
        const float sdt = sqrtf(dtf);
        const float s2D = sqrtf(2.0f * D);
        const float drift = (epi == kEpiEuler && sd.is_vortex) ? (float)a.omega[q] + rate : rate;
        a.x[q] = wrap_1d(a.x[q] + (double)(dtf * d0), sc.rL, sc.L);
        a.y[q] = wrap_1d(a.y[q] + (double)(dtf * d1), sc.rL, sc.L);
        a.phi[q] = a.phi[q] + (double)(dtf * drift + sdt * s2D * xi);
      } else if (epi == kEpiSrk1) {
        a.dphi_s[p] = (double)rate;
        a.dphi_f[p] = rate;
        a.cnt_s[p] = acc.n;
      }
    } else {
      const float inv_n = acc.n ? 1.0f / (float)acc.n : 0.0f;
      const float s2D = sqrtf(2.0f * D);
      const float A0 = (acc.s0 * inv_n) * (-s2D);
      const float A1 = acc.s1 * inv_n + (-2.0f * D) * il.dphif;
      const float d2 = il.dphif;
      if (epi == kEpiSrk2Out) {
        a.out_d[3 * (size_t)q] = (double)d0;
        a.out_d[3 * (size_t)q + 1] = (double)d1;
        a.out_d[3 * (size_t)q + 2] = (double)d2;
        a.out_a[2 * (size_t)q] = (double)A0;
        a.out_a[2 * (size_t)q + 1] = (double)A1;
      } else {
        if (!live) return;
        const float U1 = noise_f(0), U2 = noise_f(1);
        const float sdt = sqrtf(dtf);
        const float dW = U1 * sdt;
        const float dZ = 0.5f * dtf * sdt * (U1 + U2 * 0.57735026918962576f);
        const float dx = d0 * dtf - s2D * d1 * dZ - 0.5f * (d2 * d1 + D * d0) * dtf * dtf;
        const float dy = d1 * dtf + s2D * d0 * dZ + 0.5f * (d2 * d0 - D * d1) * dtf * dtf;
        const float drift = (sd.is_vortex ? (float)a.omega[q] + d2 : d2) * dtf;
        const float dp = drift + s2D * dW + A0 * dZ + 0.5f * A1 * dtf * dtf;
        a.x[q] = wrap_1d(a.x[q] + (double)dx, sc.rL, sc.L);
        a.y[q] = wrap_1d(a.y[q] + (double)dy, sc.rL, sc.L);
        a.phi[q] = a.phi[q] + (double)dp;
      }
    }
  }
}

// REST: false when no system of the launch has rests (rest_on).
template <int PREC, int KIND, bool REST = true>
__device__ __forceinline__ void load_i(const KArgs &a, const SysConst &sc, ILane &il, int p, bool valid) {
  il.p = p;
  il.valid = valid;
  il.rest = REST && PREC == kPrecFP64 && KIND == kKindSin && valid && sc.rest_on;
  if (!valid) return;
  il.x = a.sx[p];
  il.y = a.sy[p];
  il.phi = a.sphi[p];
  if (!sc.allpairs) {
    const float2 f = a.fxy[p];
    il.fx = f.x;
    il.fy = f.y;
  }
  if constexpr (PREC == kPrecFP32C) {
    // cos / sin of (phi + alpha) from the stage phase's cos / sin (made by the
    // gather) by the angle-addition identity
    const float2 t = a.cs[p];
    il.ca = t.x * sc.cos_a - t.y * sc.sin_a;
    il.sa = t.y * sc.cos_a + t.x * sc.sin_a;
  }
  if constexpr (PREC == kPrecFP64 && KIND != kKindNb) {
    const double2 t = a.dcs[p];
    const double u = dmul(t.y, sc.sin_ad), v = dmul(t.x, sc.sin_ad);
    il.dca = __fma_rn(t.x, sc.cos_ad, -u);
    il.dsa = __fma_rn(t.y, sc.cos_ad, v);
    if (REST && KIND == kKindSin && il.rest) {
      const uint32_t w = a.rest[p];
      il.rest_from = (int)(w & 0xf000u) + ((sc.rest_sector - 2) << 12);
      il.rest_own = (int)((w & 0xfffu) << 4);
      const int hi = __double2hiint(il.dsa), e = (hi >> 20) & 0x7ff;
      il.dsa_lo = (uint32_t)__double2loint(il.dsa);
      il.dsa_hi = e ? ((uint32_t)hi & 0xfffffu) | 0x100000u : 0u;
      il.dsa_e = e - 1023;
      if (sc.alpha != 0.0) {  // and that of (dca, dsa), from what its roundings left
        const double cl = dsub(dsub(__fma_rn(t.x, sc.cos_ad, -il.dca), u), __fma_rn(t.y, sc.sin_ad, -u));
        const double sl = dadd(dadd(__fma_rn(t.y, sc.cos_ad, -il.dsa), v), __fma_rn(t.x, sc.sin_ad, -v));
        il.rest_own += small_to_int(dadd(__fma_rn(il.dca, sl, -dmul(il.dsa, cl)), sc.rest_alpha), 68);
      }
    }
  }
  if constexpr (KIND == kKindCos2) {
    il.cnt = a.cnt_s[p];
    il.dphi = a.dphi_s[p];
    if constexpr (PREC == kPrecFP32C) il.dphif = a.dphi_f[p];
  } else {
    il.dphi = 0.0;
    il.dphif = 0.0f;
  }
}

// FP32X: one particle's exact neighbour sums.  Pass 1 (kKindSin): c, s =
// sum_j cos phi_j, sum_j sin phi_j; pass 2 (kKindCos2): the same weighted by
// the neighbours' pass-1 phase rates d_j.  The integer sums over all staging
// rounds are converted to double once (from_fixed128).
struct XSums {
  double c, s;
  int n;
};

// FP32X epilogue: the sums become the plain form's accumulators by the
// angle-addition identities (theta_i = phi_i + alpha):
//   sum_j sin(phi_j - theta_i) = cos(theta_i) sum sin phi_j - sin(theta_i) sum cos phi_j
//   sum_j cos(phi_j - theta_i) = cos(theta_i) sum cos phi_j + sin(theta_i) sum sin phi_j
// and the FP64 epilogue finishes the step with the plain form's formulas and
// normals.  The SRK second pass's per-term divisions by n_i
// (ChimeraSystem.cpp:634-637) become one division of each sum.
// TILE: a slot of the cell-tile passes, which take the second pass's values as
// digits.
template <int KIND, bool TILE = false>
__device__ void epilogue_fp32x(const KArgs &a, int epi, const SysDesc &sd, const ILane &il, const XSums &x,
                               int q) {
  const SysConst &sc = sd.sc;
  const int p = il.p;
  const double2 cs = from_fixed2(a.ics[p], kXQ);
  const double ct = __fma_rn(cs.x, sc.cos_ad, -dmul(cs.y, sc.sin_ad));  // cos(phi_i + alpha)
  const double st = __fma_rn(cs.y, sc.cos_ad, dmul(cs.x, sc.sin_ad));   // sin(phi_i + alpha)
  const Count cn = count_of(x.n);
  Acc<kPrecFP64> acc;
  acc.n = x.n;
  acc.s1 = 0.0;
  if constexpr (KIND == kKindSin) {
    acc.s0 = x.n ? __fma_rn(x.s, ct, -dmul(x.c, st)) : 0.0;
    if (epi == kEpiSrk1) {
      // what the second pass needs: this particle's sum of cosines and its
      // rate (the FP64 epilogue's value) times cos phi_i, sin phi_i
      const double rate = x.n ? ddiv_by(dmul(sc.sigma, acc.s0), cn.n, cn.r) : 0.0;
      a.scos[p] = x.n ? __fma_rn(x.c, ct, dmul(x.s, st)) : 0.0;
      const longlong2 w = to_fixed2(dmul(rate, cs.x), dmul(rate, cs.y), sc.xq2);
      if constexpr (TILE)
        fixed_digits(w, a.wdig + 2 * (size_t)p);
      else
        a.iws[p] = w;
    }
  } else {
    const double scs = a.scos[p];
    if (x.n) {
      acc.s0 = ddiv_by(scs, cn.n, cn.r);
      // sum_j (d_j - d_i) cos(phi_j - theta_i) / n_i
      acc.s1 = ddiv_by(dsub(__fma_rn(x.c, ct, dmul(x.s, st)), dmul(il.dphi, scs)), cn.n, cn.r);
    } else {
      acc.s0 = 0.0;
    }
  }
  epilogue<kPrecFP64, KIND>(a, epi, sd, il, acc, q, &cs);
}

// FP32X epilogues as their own dense launch: one thread per cell-order slot,
// so the FP64 per-particle work (rates, noise, the stepper update) runs on
// full warps, while the cell-tile kernels only write each particle's sums
// (xsum, xcnt).  Slots [0, n): the cell-tile systems; the particle-per-lane
// and all-pairs kernels finish their own.
template <int KIND>
__global__ void __launch_bounds__(256) k_epilogue_fp32x(KArgs a, int epi, int n) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const SysDesc &sd = a.sys[a.sys_of_c[cell_of_slot(a, p)]];
  const SysConst &sc = sd.sc;
  ILane il;
  load_i<kPrecFP32X, KIND>(a, sc, il, p, true);
  const double2 v = a.xsum[p];
  const XSums x{v.x, v.y, a.xcnt[p]};
  epilogue_fp32x<KIND, true>(a, epi, sd, il, x, a.pidx[p]);
}

// All pairs (rho > L/4): ChimeraSystem.cpp:117-255.  An all-pairs system's
// particles form one cell, in index order.  A work item is one block of T
// particles of one such system, so a large system spreads over many CTAs;
// one thread per i walks j ascending (the reference's order).  T is the CTA width: 128, or 32
// (one warp per CTA, four times the CTAs) when the all-pairs systems hold too
// few particles to give every SM work at 128 (each thread's sums are the
// same either way).
constexpr int kAllPairsThreads = 128;
constexpr int kAllPairsThreadsSmall = 32;

// The candidates are tested in float first, as in the cell kernels: for two
// positions inside the box |dx| <= L, and the reference's minimum image is
// min(|dx|, L - |dx|).  A position outside the box (an RK4 stage; the all-pairs
// form does not wrap its copies) is staged as NaN, which is never in the band,
// and flagged, so that its pairs are decided by the reference's FP64 test
// alone.  A round of candidates is tested first, which leaves each thread its
// neighbours as bits in shared memory; then each thread walks its bits, so
// the FP64 terms run on nearly full warps.
// Measured, Chimera Euler step of N = 2,000, L = 1, rho = 0.3: the FP64 test
// of every candidate took 2.74 ms; this form 0.20 ms.
constexpr int kAllPairsCap = 704;  // candidates staged per round

template <int PREC, int KIND, int T = kAllPairsThreads>
__global__ void __launch_bounds__(T) k_allpairs_pass(KArgs a, int epi) {
  constexpr bool kPair64 = PREC == kPrecFP64 && KIND != kKindNb;
  constexpr int kWords = kAllPairsCap / kWarp;
  constexpr int kAP64 = T == kAllPairsThreads ? 2 : 4;  // neighbours at a time: more where warps are few
  __shared__ __align__(16) float2 t_xy[kAllPairsCap];
  __shared__ double2 t_cs[kPair64 ? kAllPairsCap : 1];
  __shared__ double t_d[kPair64 && KIND == kKindCos2 ? kAllPairsCap : 1];
  __shared__ uint16_t t_r[kPair64 && KIND == kKindSin ? kAllPairsCap : 1];
  __shared__ float2 t_csf[PREC == kPrecFP32C ? kAllPairsCap : 1];
  __shared__ float t_df[PREC == kPrecFP32C && KIND == kKindCos2 ? kAllPairsCap : 1];
  __shared__ uint32_t t_out[kWords];   // candidates outside the box (first_bits order)
  __shared__ uint32_t t_w[kWords][T];  // each thread's neighbours of the round
  for (int item = blockIdx.x;; item += gridDim.x) {
    // the item's system (w) and particle block (rest), uniform over the CTA
    int w = 0, rest = item, cb = 0, ce = 0;
    for (; w < a.n_ap; ++w) {
      const int cw = a.ap_cells[w];
      cb = a.cell_start[cw];
      ce = a.cell_start[cw + 1];
      const int nb = (ce - cb + T - 1) / T;
      if (rest < nb) break;
      rest -= nb;
    }
    if (w >= a.n_ap) break;
    const int c = a.ap_cells[w];
    const SysDesc &sd = a.sys[a.sys_of_c[c]];
    const SysConst &sc = sd.sc;
    const bool exact_all = sc.exact_all != 0;
    const float Lf = (float)sc.L, nlo = -sc.lo2, wid = undecided_width(sc.lo2, sc.hi2);
    const int i = cb + rest * T + threadIdx.x;
    ILane il;
    Acc<PREC> acc;
    load_i<PREC, KIND>(a, sc, il, i, i < ce);
    acc.init();
    long long wpos = (a.list_idx && il.valid) ? a.list_off[a.pidx[i]] : 0;
    // the box's upper edge counts as outside: at |dx| = L the reference's
    // minimum image is L and not 0 (PeriodicBoundaryConditions.cpp:22-35)
    const double edge = sc.L * (1.0 - 1e-12);
    auto outside = [&](double x, double y) { return !(x >= 0.0 && x < edge && y >= 0.0 && y < edge); };
    const bool i_out = il.valid && outside(il.x, il.y);
    const float fx = il.valid ? (float)il.x : 0.0f, fy = il.valid ? (float)il.y : 0.0f;
    for (int jt = cb; jt < ce; jt += kAllPairsCap) {
      const int cnt = min(kAllPairsCap, ce - jt), nw = (cnt + kWarp - 1) / kWarp;
      __syncthreads();
      for (int k = threadIdx.x; k < nw * kWarp; k += T) {
        const int j = jt + k;
        bool out = false;
        float2 f = make_float2(__int_as_float(0x7fc00000), 0.0f);
        if (k < cnt) {
          const double x = a.sx[j], y = a.sy[j];
          out = outside(x, y);
          if (!out) f = make_float2((float)x, (float)y);
          if constexpr (kPair64) {
            t_cs[k] = a.dcs[j];
            if constexpr (KIND == kKindCos2) t_d[k] = a.dphi_s[j];
            if constexpr (KIND == kKindSin)
              if (sc.rest_on) t_r[k] = a.rest[j];
          }
          if constexpr (PREC == kPrecFP32C) {
            t_csf[k] = a.cs[j];
            if constexpr (KIND == kKindCos2) t_df[k] = a.dphi_f[j];
          }
        }
        t_xy[k] = f;
        const uint32_t o = __brev(__ballot_sync(0xffffffffu, out));  // k is a multiple of 32 apart per warp
        if (threadIdx.x % kWarp == 0) t_out[k / kWarp] = o;
      }
      __syncthreads();
      if (!il.valid) continue;
      for (int wd = 0; wd < nw; ++wd) {
        const int j0 = wd * kWarp;
        uint32_t bits = 0u, um = 0xffffffffu;
#pragma unroll
        for (int t = 0; t < kWarp; t += 2) {
          const float4 cj = *reinterpret_cast<const float4 *>(t_xy + j0 + t);
          const float ax0 = fabsf(cj.x - fx), ay0 = fabsf(cj.y - fy), ax1 = fabsf(cj.z - fx), ay1 = fabsf(cj.w - fy);
          const float dx0 = fminf(ax0, Lf - ax0), dy0 = fminf(ay0, Lf - ay0);
          const float dx1 = fminf(ax1, Lf - ax1), dy1 = fminf(ay1, Lf - ay1);
          const uint32_t o0 = __float_as_uint(cutoff_offset(dx0, dy0, nlo));
          const uint32_t o1 = __float_as_uint(cutoff_offset(dx1, dy1, nlo));
          bits = __funnelshift_l(o0, bits, 1);
          bits = __funnelshift_l(o1, bits, 1);
          um = min(um, min(o0, o1));
        }
        const uint32_t known = first_bits(cnt - j0) & ~((unsigned)(i - jt - j0) < (unsigned)kWarp
                                                            ? 0x80000000u >> (i - jt - j0)
                                                            : 0u);
        const bool all = exact_all || i_out;
        if (all || um <= __float_as_uint(wid) || t_out[wd] != 0u) {  // the reference's FP64 test
          for (int t = 0; t < kWarp; ++t) {
            const uint32_t b = 0x80000000u >> t;
            if (!(known & b)) continue;
            bool ask = all || (t_out[wd] & b) != 0u;
            if (!ask) {
              const float2 cj = t_xy[j0 + t];
              const float ax = fabsf(cj.x - fx), ay = fabsf(cj.y - fy);
              const float off = cutoff_offset(fminf(ax, Lf - ax), fminf(ay, Lf - ay), nlo);
              ask = off >= 0.0f && off <= wid;
            }
            if (!ask) continue;
            const int j = jt + j0 + t;
            bits = exact_within(sc, il.x, il.y, a.sx[j], a.sy[j]) ? bits | b : bits & ~b;
          }
        }
        t_w[wd][threadIdx.x] = bits & known;
      }
      int wd = -1;
      auto next = [&](uint32_t &bits, int &base) {
        while (bits == 0u && ++wd < nw) bits = t_w[wd][threadIdx.x];
        base = wd * kWarp;
        if constexpr (kPair64) acc.n += __popc(bits);
        return bits != 0u;
      };
      if constexpr (kPair64) {
        walk_pairs<KIND, kAP64, true>(
            acc, sc, il, next, [&](int k) { return t_cs[k]; }, [&](int k) { return t_d[KIND == kKindCos2 ? k : 0]; },
            [&](int k) { return a.sphi[jt + k]; },
            [&](int k) { return (uint32_t)t_r[KIND == kKindSin ? k : 0]; });
      } else {
        uint32_t bits = 0u;
        int base = 0;
        while (bits != 0u || next(bits, base)) {
          const int t = __clz(bits), k = base + t;
          bits ^= 0x80000000u >> t;
          float cc = 0.0f, ss = 0.0f, dj = 0.0f;
          if constexpr (PREC == kPrecFP32C) {
            cc = t_csf[k].x;
            ss = t_csf[k].y;
            if constexpr (KIND == kKindCos2) dj = t_df[k];
          }
          accept_pair<PREC, KIND>(a, sd, il, acc, jt + k, cc, ss, dj, wpos);
        }
      }
    }
    if (il.valid) {
      if constexpr (kPair64) finish_pairs<KIND>(acc, il);
      epilogue<PREC, KIND>(a, epi, sd, il, acc, a.pidx[i]);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Per-call step bookkeeping of every system: the call takes
// budget = min(nsteps, remaining) steps, after which the system is frozen.
__global__ void k_begin_call(SysDesc *sys, int nsys, int nsteps) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsys) return;
  const long long r = sys[s].remaining;
  sys[s].budget = (int)(r < (long long)nsteps ? (r > 0 ? r : 0) : nsteps);
}

__global__ void k_end_call(SysDesc *sys, int nsys) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsys) return;
  sys[s].step += (unsigned long long)sys[s].budget;
  sys[s].remaining -= sys[s].budget;
  sys[s].budget = 0;
}

// dense index -> system, and global cell -> system, from the layout tables
__global__ void k_layout_maps(const SysDesc *sys, int nsys, int n_active, int ncell_total,
                              int *sys_of_p, int *sys_of_c) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g < n_active) {
    int lo = 0, hi = nsys - 1;  // last system with dense_p0 <= g
    while (lo < hi) {
      const int mid = (lo + hi + 1) / 2;
      if (sys[mid].dense_p0 <= g) lo = mid; else hi = mid - 1;
    }
    sys_of_p[g] = lo;
  }
  if (g < ncell_total) {
    int lo = 0, hi = nsys - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) / 2;
      if (sys[mid].c0 <= g) lo = mid; else hi = mid - 1;
    }
    sys_of_c[g] = lo;
  }
}

__global__ void k_aos_to_soa(const double *__restrict__ aos, int n, double *x, double *y,
                             double *phi) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  x[i] = aos[3 * (size_t)i];
  y[i] = aos[3 * (size_t)i + 1];
  phi[i] = aos[3 * (size_t)i + 2];
}

__global__ void k_soa_to_aos(const double *x, const double *y, const double *phi, int n,
                             double *__restrict__ aos) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  aos[3 * (size_t)i] = x[i];
  aos[3 * (size_t)i + 1] = y[i];
  aos[3 * (size_t)i + 2] = phi[i];
}

// Philox normals of steps [first, first + nsteps) in the injection layout.
__global__ void k_export_noise(uint64_t seed, uint32_t system_id, uint64_t first, int nsteps,
                               int n, int m, double *out) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (long long)nsteps * n) return;
  const int s = (int)(g / n), i = (int)(g % n);
  double z0, z1;
  philox_normal2(seed, system_id, first + (uint64_t)s, (uint32_t)i, z0, z1);
  double *o = out + ((size_t)s * n + i) * m;
  o[0] = z0;
  if (m > 1) o[1] = z1;
}

// a[i] / b[i] as ddiv and as ddiv_by with the reciprocal; counts the pairs
// whose results differ in any bit (spc_check_division).
__global__ void k_check_division(long long n, const double *__restrict__ a, const double *__restrict__ b,
                                 unsigned long long *bad) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double x = a[i], d = b[i];
    const double q0 = ddiv(x, d), q1 = ddiv_by(x, d, drcp(d));
    if (__double_as_longlong(q0) != __double_as_longlong(q1)) atomicAdd(bad, 1ull);
  }
}

// sin and cos of x[i] from separate launches (nothing to merge) and from one
// sincos, for spc_check_sincos.
__global__ void k_sin_only(long long n, const double *__restrict__ x, double *__restrict__ s) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    s[i] = sin(x[i]);
}
__global__ void k_cos_only(long long n, const double *__restrict__ x, double *__restrict__ c) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    c[i] = cos(x[i]);
}
__global__ void k_sincos_cmp(long long n, const double *__restrict__ x, const double *__restrict__ s,
                             const double *__restrict__ c, unsigned long long *bad) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    double sn, cn;
    sincos(x[i], &sn, &cn);
    if (__double_as_longlong(sn) != __double_as_longlong(s[i]) ||
        __double_as_longlong(cn) != __double_as_longlong(c[i]))
      atomicAdd(bad, 1ull);
  }
}

__global__ void k_philox_kat(U4 c, uint32_t k0, uint32_t k1, uint32_t *out) {
  const U4 o = philox4x32_10(c, k0, k1);
  out[0] = o.x;
  out[1] = o.y;
  out[2] = o.z;
  out[3] = o.w;
}

// Global order parameter partial sums (FP64) of phi[0..n): sum cos, sum sin.
__global__ void k_order_sum(const double *phi, int n, double *out2) {
  __shared__ double sc_[256], ss_[256];
  double c = 0.0, s = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    c += cos(phi[i]);
    s += sin(phi[i]);
  }
  sc_[threadIdx.x] = c;
  ss_[threadIdx.x] = s;
  __syncthreads();
  for (int off = blockDim.x / 2; off > 0; off >>= 1) {
    if (threadIdx.x < off) {
      sc_[threadIdx.x] += sc_[threadIdx.x + off];
      ss_[threadIdx.x] += ss_[threadIdx.x + off];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out2[2 * blockIdx.x] = sc_[0];
    out2[2 * blockIdx.x + 1] = ss_[0];
  }
}

}  // namespace spc
