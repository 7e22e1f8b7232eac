// Particle-per-lane neighbour passes for sparse cells.
//
// At the densities of ensembles of small systems a cell of side ~rho holds
// ~10 particles.  One lane takes one particle: its candidates are three runs of
// cell-order slots, one per row of its 3x3 stencil (three neighbouring cells of
// a row are contiguous in cell order), read straight from the gathered arrays,
// where the lanes of a warp share a few cells and hit L1.  There is no staging,
// no barrier and no work per cell; every lane of a warp has a particle, and the
// fused epilogue runs on full warps.
//
// A lane first tests a row's candidates, four at a time, which gives one bit
// per candidate (d^2 < lo2: inside for certain; the reference's FP64 test
// decides in the band, as everywhere).  Words with neighbours go to the lane's
// list in shared memory with the slot of their first bit; then the lane walks
// its list in order (rows top to bottom, ascending slots: the reference's
// visiting order, ChimeraSystem.cpp:39-44) and adds its terms.  The SRK first
// pass keeps the list for the second.
//
// The prefilter's x is relative to the first column of a block of 16 to 31
// columns and its y to the cell row's edge, so a run of three cells needs no
// shift per candidate unless it leaves the block (or the box): such a row is
// two runs, the second starting on a multiple of four.  The float error of
// d^2 is below 1e-5 rho^2 (31 columns of at most 1.25 rho, 2^-24 relative),
// inside the band of 3e-5 rho^2.
//
// Bound by issue.  96-system Euler ensemble (681,278 particles, ~6 per cell),
// FP32X: the pass and its epilogue take 216 us where one warp per cell took
// 230 and a separate epilogue 170 (168 instructions per 32 tests, most of them
// per cell); N = 1,024 in 100 cells, FP64: 29 us against 64.
#pragma once

#include "spc_tile.cuh"

namespace spc {

constexpr int kLaneThreads = 128;
constexpr int kLaneWords = 16;  // words a lane collects before it walks them
// Saved lists: (bits, slot) pair w of particle p, in the particle's 16-byte
// groups of nbmask (as mask_at, so that the passes of one batch share the
// buffer).  A list of up to kLaneWords - 1 words ends with (0, 0); (0, 1) in
// front says that it was longer.
static_assert(kLaneWords * 2 == kMaskWords, "the saved lists fill the particles' mask words");
__device__ __forceinline__ size_t saved_at(int w, int p, int n) {
  return ((size_t)(w >> 1) * n + p) * 2 + (w & 1);
}
// Cell-list systems with fewer particles per cell than this (on average) run
// the particle-per-lane passes by default.
constexpr double kSparseBelowDefault = 24.0;

// The runs of a row of cx's stencil: cells [a0, a1) and [b0, b1) of the row,
// and the columns to add to a candidate's block-relative x of either run.
struct LaneRuns {
  int a0, a1, b0, b1;
  int sa, sb;
};
__device__ __forceinline__ LaneRuns lane_runs(int cx, int nc) {
  const int f = block_first(cx, nc);
  const int l = (f >> 4) == max((nc >> 4) - 1, 0) ? nc - 1 : f + 15;  // the block's last column
  LaneRuns r{cx - 1, cx + 2, 0, 0, 0, 0};
  if (cx == f) {
    const int left = cx == 0 ? nc - 1 : cx - 1;
    r = LaneRuns{left, left + 1, cx, cx + 2, block_first(left, nc) - (cx == 0 ? nc : 0) - f, 0};
  } else if (cx == l) {
    const int right = cx == nc - 1 ? 0 : cx + 1;
    r = LaneRuns{cx - 1, cx + 1, right, right + 1, 0, block_first(right, nc) + (cx == nc - 1 ? nc : 0) - f};
  }
  return r;
}

// One lane's sums.
template <int PREC, int KIND>
struct LaneSums;

template <int KIND>
struct LaneSums<kPrecFP64, KIND> {
  Acc<kPrecFP64> acc;
  __device__ void init() { acc.init(); }
  __device__ void term(const KArgs &a, const SysConst &sc, const ILane &il, int j) {
    add_pair<KIND>(acc, sc, il, a.dcs[j], KIND == kKindCos2 ? a.dphi_s[j] : 0.0, [&]() { return a.sphi[j]; });
  }
  __device__ void word_end(const ILane &) {}
  __device__ void list_end() {}
  __device__ void finish(const KArgs &a, int epi, const SysDesc &sd, const ILane &il, int n, int q) {
    acc.n = n;
    finish_pairs<KIND>(acc, il);
    epilogue<kPrecFP64, KIND>(a, epi, sd, il, acc, q);
  }
};

// FP32X: exact fixed-point sums, 64 bits over a list (at most 16 x 32
// candidates) and 128 over the lists, so the result is bitwise that of the
// cell-tile kernel.
template <int KIND>
struct LaneSums<kPrecFP32X, KIND> {
  long long c, s;
  __int128 tc, ts;
  __device__ void init() {
    c = s = 0;
    tc = ts = 0;
  }
  __device__ void term(const KArgs &a, const SysConst &, const ILane &, int j) {
    const longlong2 v = KIND == kKindSin ? a.ics[j] : a.iws[j];
    c += v.x;
    s += v.y;
  }
  __device__ void word_end(const ILane &) {}
  __device__ void list_end() {
    tc += c;
    ts += s;
    c = s = 0;
  }
  __device__ void finish(const KArgs &a, int epi, const SysDesc &sd, const ILane &il, int n, int q) {
    const int qv = KIND == kKindSin ? kXQ : sd.sc.xq2;
    epilogue_fp32x<KIND>(a, epi, sd, il, XSums{from_fixed128(tc, qv), from_fixed128(ts, qv), n}, q);
  }
};

// FP32C: a word's neighbours are summed in float, turned into the alignment
// terms by angle addition and added with Kahan compensation.
template <int KIND>
struct LaneSums<kPrecFP32C, KIND> {
  float bc, bs, bdc, bds;
  Acc<kPrecFP32C> acc;
  __device__ void init() {
    bc = bs = bdc = bds = 0.0f;
    acc.init();
  }
  __device__ void term(const KArgs &a, const SysConst &, const ILane &, int j) {
    const float2 t = a.cs[j];
    bc += t.x;
    bs += t.y;
    if constexpr (KIND == kKindCos2) {
      const float d = a.dphi_f[j];
      bdc = fmaf(d, t.x, bdc);
      bds = fmaf(d, t.y, bds);
    }
  }
  __device__ void word_end(const ILane &il) {
    if constexpr (KIND == kKindSin) {
      kahan_add(acc.s0, acc.c0, fmaf(bs, il.ca, -bc * il.sa));
    } else {
      const float b0 = fmaf(bc, il.ca, bs * il.sa);
      kahan_add(acc.s0, acc.c0, b0);
      kahan_add(acc.s1, acc.c1, fmaf(bdc, il.ca, fmaf(bds, il.sa, -il.dphif * b0)));
    }
    bc = bs = bdc = bds = 0.0f;
  }
  __device__ void list_end() {}
  __device__ void finish(const KArgs &a, int epi, const SysDesc &sd, const ILane &il, int n, int q) {
    acc.n = n;
    acc.s0 -= acc.c0;
    acc.s1 -= acc.c1;
    epilogue<kPrecFP32C, KIND>(a, epi, sd, il, acc, q);
  }
};

template <int PREC, int KIND>
__global__ void __launch_bounds__(kLaneThreads) k_lane(KArgs a, int epi) {
  __shared__ uint32_t s_bits[kLaneWords][kLaneThreads];
  __shared__ int s_slot[kLaneWords][kLaneThreads];
  const int tid = threadIdx.x;
  const int p = a.lane_p0 + blockIdx.x * blockDim.x + tid;
  if (p >= a.lane_p1) return;  // no barrier below
  const int n_all = a.n_active;
  const int c = cell_of_slot(a, p);
  const SysDesc &sd = a.sys[a.sys_of_c[c]];
  const SysConst &sc = sd.sc;
  ILane il;
  load_i<PREC, KIND>(a, sc, il, p, true);
  LaneSums<PREC, KIND> sums;
  sums.init();
  int n = 0, nw = 0;
  uint2 *saved = reinterpret_cast<uint2 *>(a.nbmask);

  auto walk = [&]() {  // the listed words (none of them zero), in order
    uint32_t bits = 0u;
    int slot = 0;
    for (int w = 0;;) {
      if (bits == 0u) {
        if (w > 0) sums.word_end(il);
        if (w == nw) break;
        bits = s_bits[w][tid];
        slot = s_slot[w][tid];
        ++w;
      }
      const int t = __clz(bits);
      bits ^= 0x80000000u >> t;
      sums.term(a, sc, il, slot + t);
    }
    sums.list_end();
    nw = 0;
  };

  bool listed = false;  // pass 2: the first pass left its list
  if constexpr (KIND == kKindCos2) {
    if (saved) {
      uint2 e = saved[saved_at(0, p, n_all)];
      listed = e.x != 0u || e.y == 0u;  // (0, 1): the list was too long
      if (listed)
        while (e.x != 0u) {
          s_bits[nw][tid] = e.x;
          s_slot[nw][tid] = (int)e.y;
          n += __popc(e.x);
          ++nw;
          e = saved[saved_at(nw, p, n_all)];
        }
    }
  }
  if (!listed) {
    int nsaved = 0;
    auto put = [&](uint32_t bits, int slot) {
      if (bits == 0u) return;
      s_bits[nw][tid] = bits;
      s_slot[nw][tid] = slot;
      if (KIND == kKindSin && saved && nsaved < kLaneWords - 1)
        saved[saved_at(nsaved, p, n_all)] = make_uint2(bits, (uint32_t)slot);
      ++nsaved;
      ++nw;
    };
    const float nlo = -sc.lo2, wid = undecided_width(sc.lo2, sc.hi2);
    const bool exact_all = sc.exact_all != 0;
    const int nc = sc.nc, cl = c - sd.c0, cy = cl / nc, cx = cl - cy * nc;
    const LaneRuns r = lane_runs(cx, nc);
    const float xa = il.fx - (float)r.sa * sc.cell_f, xb = il.fx - (float)r.sb * sc.cell_f;
    const int *row = a.cell_start + sd.c0 + adjust_cell(cy - 1, nc) * nc;
    int a0 = row[r.a0], a1 = row[r.a1], b0 = row[r.b0], b1 = row[r.b1];
#pragma unroll 1
    for (int k = 0; k < 3; ++k) {
      // the next row's bounds, on their way while this row is tested
      const int *next = a.cell_start + sd.c0 + adjust_cell(cy + k, nc) * nc;
      const int na0 = next[r.a0], na1 = next[r.a1], nb0 = next[r.b0], nb1 = next[r.b1];
      const float y = il.fy - (float)(k - 1) * sc.cell_f;
      // run a takes positions [0, la), run b [la4, la4 + lb)
      const int la = a1 - a0, la4 = (la + 3) & ~3, total = la4 + (b1 - b0);
      for (int base = 0; base < total; base += kWarp) {
        const int cnt = min(kWarp, total - base);
        uint32_t bits = 0u, um = 0xffffffffu;
        int done = 0;
        for (; done < cnt; done += 4) {
          const bool in_a = base + done < la4;
          const float x = in_a ? xa : xb;
          // up to three slots past the run's end are read (the array is padded) and masked
          const float2 *f = a.fxy + ((in_a ? a0 : b0 - la4) + base + done);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float2 fj = f[u];
            const uint32_t o = __float_as_uint(cutoff_offset(fj.x - x, fj.y - y, nlo));
            bits = __funnelshift_l(o, bits, 1);
            um = min(um, o);
          }
        }
        bits <<= kWarp - done;
        const uint32_t part_a = first_bits(min(max(la4 - base, 0), kWarp));
        uint32_t known = first_bits(min(max(la - base, 0), kWarp)) | (first_bits(cnt) & ~part_a);
        if (k == 1) {
          const int self = (p < a1 && p >= a0 ? p - a0 : la4 + p - b0) - base;
          if ((unsigned)self < (unsigned)kWarp) known &= ~(0x80000000u >> self);
        }
        // pairs the float test cannot decide: the reference's FP64 test
        if (exact_all || um <= __float_as_uint(wid)) {
          for (uint32_t ask = known; ask != 0u;) {
            const int t = __clz(ask);
            const uint32_t b = 0x80000000u >> t;
            ask ^= b;
            const bool in_a = base + t < la4;
            const int j = (in_a ? a0 : b0 - la4) + base + t;
            const float2 fj = a.fxy[j];
            const float off = cutoff_offset(fj.x - (in_a ? xa : xb), fj.y - y, nlo);
            if (exact_all || (off >= 0.0f && off <= wid))
              bits = exact_within(sc, il.x, il.y, a.sx[j], a.sy[j]) ? bits | b : bits & ~b;
          }
        }
        bits &= known;
        n += __popc(bits);
        put(bits & part_a, a0 + base);
        put(bits & ~part_a, b0 - la4 + base);
        if (nw > kLaneWords - 2) walk();
      }
      a0 = na0, a1 = na1, b0 = nb0, b1 = nb1;
    }
    if (KIND == kKindSin && saved) {
      if (nsaved < kLaneWords)
        saved[saved_at(nsaved, p, n_all)] = make_uint2(0u, 0u);
      else
        saved[saved_at(0, p, n_all)] = make_uint2(0u, 1u);
    }
  }
  walk();
  sums.finish(a, epi, sd, il, n, a.pidx[p]);
}

}  // namespace spc
