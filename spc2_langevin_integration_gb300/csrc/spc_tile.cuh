// Cell-tile neighbour passes: one CTA per cell.
//
// The CTA stages the candidates of the cell's 3x3 stencil (in the reference's
// visiting order, ChimeraSystem.cpp:39-44; ascending index inside a cell) into
// shared memory once, with each stencil cell's periodic shift already added to
// the float prefilter coordinates, and then every thread of the CTA works on
// one particle of the cell against that list: no global load in the inner
// loop, and every candidate read is a shared-memory broadcast.
//
// FP32C and FP32X: spc_ftile.cuh, on the tensor cores.
//
// FP64 (k_tile_fp64): one thread per particle walks the whole list in order,
// so each particle's sum keeps the reference's order term for term.  The
// threads first find their neighbours of a staging round as bits and then walk
// the bits, so that the FP64 terms (1/64-rate pipe on GB300) run on nearly
// full warps instead of on the few lanes that accept a given candidate.
//
// Both decide every pair exactly as the reference: float prefilter on
// cell-relative coordinates, the reference's FP64 test for pairs within a
// relative 3e-5 of rho^2 (warp-uniform branch, rare).
#pragma once

#include "spc_kernels.cuh"

namespace spc {

constexpr int kTileCap = 1024;      // FP32C: candidates staged per round
constexpr int kTileCapX = 768;      // FP32X: candidates staged per round (24 mask words)
constexpr int kTileCap64 = 704;     // FP64: candidates staged per round (7 CTAs/SM fit)
constexpr int kTileThreads32 = 128; // float CTA: 4 warps
constexpr int kTileThreads64 = 64;  // FP64 CTA: 2 warps

struct Stencil {
  int start[9];    // cell-order start of each stencil cell
  int prefix[10];  // offsets of each stencil cell in the staged list
};

// half < 0: the 3x3 stencil of cell c.  half 0 / 1 (sub-cells): the stencil
// of the lower / upper half of cell c.  A particle of the lower half is more
// than a cell side (>= rho) below the upper half of the row above, so that
// row's entries keep only their lower half [start, mid); the upper half's
// stencil keeps the upper half [mid, end) of the row below.  The own cell
// (entry 4) stays whole, and so does a far cell when both it and cell c hold
// a particle near the half line (cell_near, kNearHalf).
__device__ __forceinline__ void stencil_cell(const KArgs &a, const SysDesc &sd, int c, int q, int half, int &ja,
                                             int &jb) {
  const SysConst &sc = sd.sc;
  const int nc = sc.nc, cl = c - sd.c0, cx = cl % nc, cy = cl / nc;
  const int ox = (q % 3) - 1, oy = (q / 3) - 1;
  const int cj = sd.c0 + adjust_cell(cy + oy, nc) * nc + adjust_cell(cx + ox, nc);
  ja = a.cell_start[cj];
  jb = a.cell_start[cj + 1];
  if (half >= 0 && oy == (half == 0 ? 1 : -1) && !(a.cell_near[c] && a.cell_near[cj])) {
    if (half == 0)
      jb = a.cell_mid[cj];
    else
      ja = a.cell_mid[cj];
  }
}
__device__ __forceinline__ void stencil_of(const KArgs &a, const SysDesc &sd, int c, Stencil &s,
                                           int half = -1) {
  s.prefix[0] = 0;
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    int ja, jb;
    stencil_cell(a, sd, c, q, half, ja, jb);
    s.start[q] = ja;
    s.prefix[q + 1] = s.prefix[q] + (jb - ja);
  }
}

// Cell-order slot of staged candidate g (0 <= g < prefix[9]) and its stencil
// entry q.  A select chain with constant indices keeps the stencil in
// registers (a dynamic index would put it in local memory).
__device__ __forceinline__ int slot_of(const Stencil &s, int g, int &q_out) {
  int q = 0, base = s.start[0];
#pragma unroll
  for (int k = 1; k < 9; ++k) {
    const bool ge = g >= s.prefix[k];
    q = ge ? k : q;
    base = ge ? s.start[k] - s.prefix[k] : base;
  }
  q_out = q;
  return base + g;
}

// periodic shift of stencil entry q in the float prefilter frame
__device__ __forceinline__ float shift_x(int q, float cell_f) { return (float)(q % 3 - 1) * cell_f; }
__device__ __forceinline__ float shift_y(int q, float cell_f) { return (float)(q / 3 - 1) * cell_f; }

// ---------------------------------------------------------------------------
// The SRK first pass (KIND == kKindSin) records, for cells whose candidate list
// fits one staging round, each particle's neighbour set as bits over that list,
// and the second pass (kKindCos2) tests nothing again there.  The words are
// laid out by mask_at, so the second pass fetches the words of four candidate
// blocks with one 16-byte load.
constexpr int kMaskWords = kTileCap / 32;
static_assert(kMaskWords % 4 == 0, "mask words come in groups of four");

// Work item `item` of the cell-tile kernels: cell c = item / K and part
// item % K of its particles, K = a.tile_split CTAs per cell.  A part is a
// whole number of the kernel's particle groups (GROUP = the CTA's threads,
// the particles it processes at a time), so a cell of at most GROUP
// particles stays one item and is staged once, while the few cells of a
// clustered state that hold several groups are spread over up to K CTAs
// instead of running their groups one after another on one CTA (the tail of
// a single-wave pass).  Items past a cell's last group are empty.  c0 is the
// cell's first particle (the own cell's stencil entry starts there).
struct TileItem {
  int c, c0, cb, ce;
};

__device__ __forceinline__ int tile_items(const KArgs &a) { return a.ncell_tile * max(a.tile_split, 1); }

template <int GROUP>
__device__ __forceinline__ bool tile_item(const KArgs &a, int item, TileItem &t) {
  const int K = max(a.tile_split, 1);
  t.c = item / K;
  const int h = item - t.c * K;
  t.c0 = a.cell_start[t.c];
  const int c1 = a.cell_start[t.c + 1];
  const int groups = (c1 - t.c0 + GROUP - 1) / GROUP;
  const int per = ((groups + K - 1) / K) * GROUP;
  t.cb = t.c0 + h * per;
  t.ce = min(c1, t.cb + per);
  return t.cb < t.ce;
}

// Cell units (tuning SPC_TUNE_CELL_UNITS).  Every cell whose candidate list
// takes at most kSplitRounds staging rounds is cut into units of 32 particles
// x one staging round, and the units kernel runs each unit on its own CTA,
// beside the cell-tile kernel, which keeps only the cells of longer lists.
// On a clustered state the cell-tile kernel's one CTA per 128-particle group
// is badly balanced: a cell of a cluster holds up to ~380 particles with
// ~6,000 candidates, several times a typical cell's work, and its groups set
// the end of the single-wave pass while most SMs idle.  Units of ~32 x 1,024
// pair tests spread that work over every SM.  A unit's four warps take a
// quarter of its round each; the unit stores its per-particle sums of the
// round, and the last unit of a 32-particle chunk to finish (a counter per
// chunk, reset by that unit) adds the rounds in order and finishes the
// particles.  k_list_units lists the units once per evaluation (both passes
// see the same cells).  Which cells are units, and the order of every sum,
// depend on the cell alone, so the results do not depend on the CTAs per cell.
// With sub-cells (SPC_TUNE_SUBCELLS, cell_mid set) each half of a unit cell
// is cut the same way over its own half stencil (stencil_of with half 0 / 1)
// and listed as (2c + half, u); the cell stays a unit cell on its whole
// stencil's round count, which bounds both halves'.
constexpr int kSplitRounds = 8;

__device__ __forceinline__ bool unit_cell(const KArgs &a, int n_c, int total, int cap) {
  return a.units != nullptr && n_c > 0 && total <= kSplitRounds * cap;
}

// List the units of every unit cell of the cell-tile systems (one thread per
// cell), once per evaluation after the gather, for both passes' units kernels,
// and mark those cells for the cell-tile kernels to skip.
// CAP: the form's staging round.
template <int CAP>
__global__ void k_list_units(KArgs a) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.ncell_tile) return;
  const int c0 = a.cell_start[c], n_c = a.cell_start[c + 1] - c0;
  a.cell_unit[c] = 0;
  if (n_c == 0) return;
  const SysDesc &sd = a.sys[a.sys_of_c[c]];
  if (sd.sc.allpairs) return;
  Stencil st;
  stencil_of(a, sd, c, st);
  const int total = st.prefix[9];
  if (!unit_cell(a, n_c, total, CAP)) return;
  a.cell_unit[c] = 1;
  if (a.cell_mid) {
    // sub-cells: each half's units over its own stencil, listed as (2c + half, u)
    const int mid = a.cell_mid[c];
    for (int h = 0; h < 2; ++h) {
      const int n_h = h ? c0 + n_c - mid : mid - c0;
      if (n_h == 0) continue;
      Stencil sh;
      stencil_of(a, sd, c, sh, h);
      const int rounds = (sh.prefix[9] + CAP - 1) / CAP;
      const int units = (n_h + kWarp - 1) / kWarp * rounds;
      const int base = atomicAdd(a.unit_count, units);
      for (int u = 0; u < units; ++u) a.units[base + u] = make_int2(2 * c + h, u);
    }
    return;
  }
  const int rounds = (total + CAP - 1) / CAP;
  const int units = (n_c + kWarp - 1) / kWarp * rounds;
  const int base = atomicAdd(a.unit_count, units);
  for (int u = 0; u < units; ++u) a.units[base + u] = make_int2(c, u);
}

// ---------------------------------------------------------------------------
// FP64 passes.  A staging round is tested first: each thread's neighbours of
// the round become bits, one word per 32 candidates, in its own column of
// shared memory.  Then each thread walks its bits in order (the reference's
// visiting order), taking the next word when one is used up, so the lanes of a
// warp run out of neighbours together (a lane has ~200 +- 14 of them) and the
// FP64 terms run on ~90% full warps.  The SRK first pass keeps the words of
// one-round cells in nbmask and the second pass tests nothing again.
// Bound by the FP64 pipe (3 operations per pair in pass 1, 5 in pass 2).
// Vortex SRK, N = 65,536: pass 1 2.04 ms -> 171 us (189 with the terms' rests,
// for alpha below 0.5), pass 2 0.92 ms -> 250 us (against sines per pair and a queue of accepted candidates).  704
// candidates per round leave room for 7 CTAs per SM in pass 2.
// The neighbour diagnostics (kKindNb: counts, lists in visiting order, local
// order parameters) are the same walk.  Order parameters of N = 65,536 at 64 a
// cell, with upload and readback: 550 -> 278 us against a warp per cell that
// added on the lanes that accept a candidate (even, 2% slower, at 3 a cell).
constexpr int kTileWords64 = kTileCap64 / kWarp;
static_assert(kTileCap64 % kWarp == 0 && (kTileWords64 + 3) / 4 * 4 <= kMaskWords, "FP64 staging round");

template <int KIND>
__global__ void __launch_bounds__(kTileThreads64) k_tile_fp64(KArgs a, int epi) {
  __shared__ __align__(16) float2 s_xy[kTileCap64];  // x+shift, y+shift (prefilter; padded to 32)
  __shared__ double2 s_cs[kTileCap64];               // cos, sin of the stage phase
  __shared__ double s_d[KIND == kKindCos2 ? kTileCap64 : 1];  // pass 2: phase rate
  __shared__ uint16_t s_r[KIND == kKindSin ? kTileCap64 : 1];  // pass 1: rest of the phase
  __shared__ uint32_t s_w[(kTileWords64 + 3) / 4 * 4][kTileThreads64];
  const int tid = threadIdx.x;
  const int n_all = a.n_active;
  const int nitems = tile_items(a);
  for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
    TileItem ti;
    if (!tile_item<kTileThreads64>(a, item, ti)) continue;
    const int c = ti.c, c0 = ti.c0, cb = ti.cb, ce = ti.ce;
    const SysDesc &sd = a.sys[a.sys_of_c[c]];
    const SysConst &sc = sd.sc;
    if (sc.allpairs) continue;
    const float nlo = -sc.lo2, wid = undecided_width(sc.lo2, sc.hi2);
    const bool exact_all = sc.exact_all != 0;
    Stencil st;
    stencil_of(a, sd, c, st);
    const int total = st.prefix[9];
    const int rounds = (total + kTileCap64 - 1) / kTileCap64;
    const bool masked = rounds == 1 && a.nbmask != nullptr && !exact_all;
    for (int ig = cb; ig < ce; ig += kTileThreads64) {
      const int gi = min(kTileThreads64, ce - ig);
      const bool valid = tid < gi;
      const int p = ig + tid;
      ILane il;
      load_i<kPrecFP64, KIND>(a, sc, il, p, valid);
      if (!valid) {
        il.fx = il.fy = 3.0e17f;
        il.x = il.y = 0.0;
      }
      Acc<kPrecFP64> acc;
      acc.init();
      long long wpos = KIND == kKindNb && a.list_idx && valid ? a.list_off[a.pidx[p]] : 0;
      for (int r = 0; r < rounds; ++r) {
        const int rlo = r * kTileCap64, rcnt = min(kTileCap64, total - rlo);
        const int nw = (rcnt + kWarp - 1) / kWarp;
        if (rounds > 1 || ig == cb) {
          __syncthreads();
          for (int k = tid; k < nw * kWarp; k += blockDim.x) {
            if (k < rcnt) {
              int q;
              const int pj = slot_of(st, rlo + k, q);
              s_cs[k] = a.dcs[pj];
              if constexpr (KIND == kKindCos2) s_d[k] = a.dphi_s[pj];
              if constexpr (KIND == kKindSin)
                if (sc.rest_on) s_r[k] = a.rest[pj];
              if (KIND == kKindCos2 && masked) continue;
              const float2 f = a.fxy[pj];
              s_xy[k] = make_float2(f.x + shift_x(q, sc.cell_f), f.y + shift_y(q, sc.cell_f));
            } else {  // padding: never a neighbour, never near the cutoff
              s_xy[k] = make_float2(3.0e18f, 3.0e18f);
            }
          }
          __syncthreads();
        }
        if (!valid) continue;
        uint4 *m4 = reinterpret_cast<uint4 *>(a.nbmask);
        if (KIND == kKindCos2 && masked) {
          for (int g = 0; g * 4 < nw; ++g) {
            const uint4 m = m4[(size_t)g * n_all + p];
            s_w[4 * g][tid] = m.x;
            s_w[4 * g + 1][tid] = m.y;
            s_w[4 * g + 2][tid] = m.z;
            s_w[4 * g + 3][tid] = m.w;
          }
        } else {
          const int self = st.prefix[4] + (p - c0) - rlo;
          for (int w = 0; w < nw; ++w) {
            const int j0 = w * kWarp;
            uint32_t um = 0xffffffffu;
            uint32_t bits = test32(s_xy + j0, il.fx, il.fy, nlo, um);
            uint32_t known = first_bits(rcnt - j0);
            if ((unsigned)(self - j0) < (unsigned)kWarp) known &= ~(0x80000000u >> (self - j0));
            // pairs the float test cannot decide: the reference's FP64 test
            if (exact_all || um <= __float_as_uint(wid)) {
              for (int t = 0; t < kWarp; ++t) {
                const uint32_t b = 0x80000000u >> t;
                if (!(known & b)) continue;
                const float2 cj = s_xy[j0 + t];
                const float off = cutoff_offset(cj.x - il.fx, cj.y - il.fy, nlo);
                if (!(exact_all || (off >= 0.0f && off <= wid))) continue;
                int q;
                const int pj = slot_of(st, rlo + j0 + t, q);
                bits = exact_within(sc, il.x, il.y, a.sx[pj], a.sy[pj]) ? bits | b : bits & ~b;
              }
            }
            bits &= known;
            acc.n += __popc(bits);
            s_w[w][tid] = bits;
          }
          if (KIND == kKindSin && masked)
            for (int g = 0; g * 4 < nw; ++g)  // words past the last one are not read
              m4[(size_t)g * n_all + p] =
                  make_uint4(s_w[4 * g][tid], s_w[4 * g + 1][tid], s_w[4 * g + 2][tid], s_w[4 * g + 3][tid]);
        }
        int w = -1;
        auto next = [&](uint32_t &bits, int &base) {
          while (bits == 0u && ++w < nw) bits = s_w[w][tid];
          base = w * kWarp;
          return bits != 0u;
        };
        if constexpr (KIND == kKindNb) {  // diagnostics
          uint32_t bits = 0u;
          int base = 0;
          if (a.list_idx) {
            while (bits != 0u || next(bits, base)) {
              const int t = __clz(bits);
              bits &= ~(0x80000000u >> t);
              int q;
              a.list_idx[wpos++] = a.pidx[slot_of(st, rlo + base + t, q)] - sd.pool_p0;
            }
          } else if (a.out_r) {
            while (bits != 0u || next(bits, base)) {
              const int t = __clz(bits);
              bits &= ~(0x80000000u >> t);
              const double2 cj = s_cs[base + t];
              acc.s0 = dadd(acc.s0, cj.x);
              acc.s1 = dadd(acc.s1, cj.y);
            }
          }
        } else {
          walk_pairs<KIND, 2, true>(
              acc, sc, il, next, [&](int j) { return s_cs[j]; },
              [&](int j) { return s_d[KIND == kKindCos2 ? j : 0]; },
              [&](int j) {
                int q;
                return a.sphi[slot_of(st, rlo + j, q)];
              },
              [&](int j) { return (uint32_t)s_r[KIND == kKindSin ? j : 0]; });
        }
      }
      if (valid) {
        finish_pairs<KIND>(acc, il);
        epilogue<kPrecFP64, KIND>(a, epi, sd, il, acc, a.pidx[p]);
      }
      __syncthreads();
    }
  }
}

}  // namespace spc
