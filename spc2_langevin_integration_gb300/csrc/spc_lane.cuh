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
// A lane tests a row's candidates, four at a time, which gives one bit per
// candidate (d^2 < lo2: inside for certain; the reference's FP64 test decides
// in the band, as everywhere), and walks the bits of each word of 32 (rows top
// to bottom, ascending slots: the reference's visiting order,
// ChimeraSystem.cpp:39-44).  The SRK first pass keeps the words with neighbours
// for the second.
//
// The prefilter's x is relative to the first column of a block of 16 to 31
// columns and its y to the cell row's edge, so a run of three cells needs no
// shift per candidate unless it leaves the block (or the box): such a row is
// two runs, the second starting on a multiple of four.  The float error of
// d^2 is below 1e-5 rho^2 (31 columns of at most 1.25 rho, 2^-24 relative),
// inside the band of 3e-5 rho^2.
//
// Bound by the latency of the loads from L1 (its hit rate is 79%) and by issue
// (43%).  96-system Euler ensemble (681,278 particles, ~6 per cell), FP32X: the
// pass with its update takes 162 us, where one warp per cell took 230 and a
// separate epilogue 170 (168 instructions per 32 tests, most of them per
// cell).  Taking two neighbours of a word at a time gave 176 -> 171, ten CTAs
// per SM (48 registers) 171 -> 162; FP32C (24 systems, 1.0 M particles) 168 ->
// 160 and no gain from fewer registers.  CTAs of 256 and 512 threads and
// prefetching the next row gave nothing.  FP64, N = 1,024 in 100 cells: 29 us
// against 64; there the words are listed first (39 us when each word is walked
// on its own).
#pragma once

#include "spc_tile.cuh"

namespace spc {

constexpr int kLaneThreads = 128;
constexpr int kLaneWords = 16;  // words a lane collects (FP64) before it walks them
constexpr int kLanePairs = 2;   // FP64: neighbours taken at a time
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

// One lane's sums (float forms): value() loads what a neighbour adds, add()
// adds it if p.
template <int PREC, int KIND>
struct LaneSums;

// FP64: the words are listed first and walked together, the lanes of a warp
// running out of neighbours at about the same time.
template <int KIND>
struct LaneSums<kPrecFP64, KIND> {
  Acc<kPrecFP64> acc;
  __device__ void init() { acc.init(); }
  __device__ void finish(const KArgs &a, int epi, const SysDesc &sd, const ILane &il, int n, int q) {
    acc.n = n;
    finish_pairs<KIND>(acc, il);
    epilogue<kPrecFP64, KIND>(a, epi, sd, il, acc, q);
  }
};

// FP32X: exact fixed-point sums, so the result is bitwise that of the
// cell-tile kernel.  A word's neighbours add less than 2^57; after each word the
// multiples of 2^57 move to a 32-bit count (2^57 each).
template <int KIND>
struct LaneSums<kPrecFP32X, KIND> {
  long long c, s;
  int ch, sh;
  __device__ void init() {
    c = s = 0;
    ch = sh = 0;
  }
  typedef longlong2 Value;
  __device__ static Value value(const KArgs &a, int j) { return KIND == kKindSin ? a.ics[j] : a.iws[j]; }
  __device__ void add(const Value &v, bool p) { add2_if(c, s, v, p); }
  __device__ void word_end(const ILane &) {
    constexpr long long low = (1ll << 57) - 1;
    ch += (int)(c >> 57);
    sh += (int)(s >> 57);
    c &= low;
    s &= low;
  }
  __device__ void finish(const KArgs &a, int epi, const SysDesc &sd, const ILane &il, int n, int q) {
    const int qv = KIND == kKindSin ? kXQ : sd.sc.xq2;
    const __int128 tc = ((__int128)ch << 57) + c, ts = ((__int128)sh << 57) + s;
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
  struct Value {
    float2 cs;
    float d;
  };
  __device__ static Value value(const KArgs &a, int j) { return {a.cs[j], KIND == kKindCos2 ? a.dphi_f[j] : 0.0f}; }
  __device__ void add(const Value &v, bool p) {
    addf2_if(bc, bs, v.cs.x, v.cs.y, p);
    if constexpr (KIND == kKindCos2) fmaf2_if(bdc, bds, v.d, v.cs.x, v.cs.y, p);
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
  __device__ void finish(const KArgs &a, int epi, const SysDesc &sd, const ILane &il, int n, int q) {
    acc.n = n;
    acc.s0 -= acc.c0;
    acc.s1 -= acc.c1;
    epilogue<kPrecFP32C, KIND>(a, epi, sd, il, acc, q);
  }
};

template <int PREC, int KIND>
__global__ void __launch_bounds__(kLaneThreads, PREC == kPrecFP32X ? 10 : 1) k_lane(KArgs a, int epi) {
  constexpr bool kList = PREC == kPrecFP64;
  __shared__ uint32_t s_bits[kList ? kLaneWords : 1][kLaneThreads];
  __shared__ int s_slot[kList ? kLaneWords : 1][kLaneThreads];
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
  int n = 0;
  uint2 *saved = reinterpret_cast<uint2 *>(a.nbmask);

  int nw = 0;  // FP64: words listed
  auto walk_list = [&]() {
    if constexpr (kList) {
      int w = -1;
      walk_pairs<KIND, kLanePairs>(
          sums.acc, sc, il,
          [&](uint32_t &bits, int &base) {
            if (++w >= nw) return false;
            bits = s_bits[w][tid];
            base = s_slot[w][tid];
            return true;
          },
          [&](int j) { return a.dcs[j]; }, [&](int j) { return a.dphi_s[j]; }, [&](int j) { return a.sphi[j]; });
      nw = 0;
    }
  };
  // a word with neighbours; bit 31 is slot `slot`
  auto take = [&](uint32_t bits, int slot) {
    n += __popc(bits);
    if constexpr (kList) {
      s_bits[nw][tid] = bits;
      s_slot[nw][tid] = slot;
      ++nw;
    } else {
      while (bits != 0u) {  // two at a time: both loads are on their way together
        const int t0 = __clz(bits);
        bits ^= 0x80000000u >> t0;
        const bool two = bits != 0u;
        const int t1 = two ? __clz(bits) : t0;
        bits &= ~(0x80000000u >> t1);
        const auto v0 = sums.value(a, slot + t0), v1 = sums.value(a, slot + t1);
        sums.add(v0, true);
        sums.add(v1, two);
      }
      sums.word_end(il);
    }
  };

  bool listed = false;  // pass 2: the first pass left its list
  if constexpr (KIND == kKindCos2) {
    if (saved) {
      uint2 e = saved[saved_at(0, p, n_all)];
      listed = e.x != 0u || e.y == 0u;  // (0, 1): the list was too long
      if (listed)
        for (int w = 1; e.x != 0u; ++w) {
          const uint2 next = saved[saved_at(w, p, n_all)];
          take(e.x, (int)e.y);
          e = next;
        }
    }
  }
  if (!listed) {
    int nsaved = 0;
    auto found = [&](uint32_t bits, int slot) {
      if (bits == 0u) return;
      if (KIND == kKindSin && saved) {
        if (nsaved < kLaneWords - 1) saved[saved_at(nsaved, p, n_all)] = make_uint2(bits, (uint32_t)slot);
        ++nsaved;
      }
      take(bits, slot);
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
          uint32_t o[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float2 d = add2(f[u], make_float2(-x, -y));
            o[u] = __float_as_uint(cutoff_offset(d.x, d.y, nlo));
            bits = __funnelshift_l(o[u], bits, 1);
          }
          um = __vimin3_u32(um, o[0], o[1]);
          um = __vimin3_u32(um, o[2], o[3]);
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
        found(bits & part_a, a0 + base);
        if (base + cnt > la4) found(bits & ~part_a, b0 - la4 + base);
        if (kList && nw > kLaneWords - 2) walk_list();
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
  walk_list();
  sums.finish(a, epi, sd, il, n, a.pidx[p]);
}

}  // namespace spc
