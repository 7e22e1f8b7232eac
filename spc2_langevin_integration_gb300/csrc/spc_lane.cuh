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
// two runs, the second starting on a multiple of four.  The float error of d^2
// is below 1.6e-5 rho^2, inside the band of 3e-5 rho^2: coordinates and shifts
// are at most 33 rho (31 columns of rho (nc + 1) / nc), so the roundings of the
// candidate's coordinate, of cell_f, of the shift's product and of its sum with
// the own coordinate are 2e-6 rho each, 8e-6 rho in dx.  (1.2e-5 rho^2 is the
// largest found over the block edges at nc = 29 to 63.)
//
// Bound by the latency of the loads from L1 (its hit rate is 79%) and by issue
// (43%).  96-system Euler ensemble (681,278 particles, ~6 per cell), FP32X: the
// pass with its update takes 165 us, where one warp per cell took 230 and a
// separate epilogue 170 (168 instructions per 32 tests, most of them per
// cell); FP32C (24 systems, 1.0 M particles): 166 us against 290.  Ten CTAs per
// SM (48 registers), rows unrolled and two neighbours of a word at a time each
// gave 3 to 15%; CTAs of 256 and 512 threads and prefetching the next row
// nothing.  FP64, N = 1,024 in 100 cells: 20 us against 64; there the words are
// listed first (10 us more when each word is walked on its own).
#pragma once

#include "spc_tile.cuh"

namespace spc {

constexpr int kLaneThreads = 128;
constexpr int kLaneWords = 16;  // words a lane collects (FP64) before it walks them
constexpr int kLanePairs = 2;   // FP64: neighbours taken at a time
// Few particles: a group of four lanes takes one.  Three of them test a row
// each, and the FP64 terms of four neighbours are formed side by side (their
// additions keep the order).  The sums are the same bit for bit: FP32X's are
// exact, FP32C adds row by row either way.
constexpr int kLaneGroup = 4;
// Up to this many particles, where the GPU's schedulers would hold a few warps
// each (4 lanes and 1 lane per particle, Euler step in us at density 1,000, rho
// = 0.1): FP64 1,024: 27.1 / 34.2, 12,288: 34.3 / 40.0, 16,384: 46.0 / 42.3;
// FP32C 1,024: 20.8 / 29.8, 65,536: 45.3 / 47.1, 81,920: 53.1 / 49.7; FP32X
// 1,024: 24.1 / 33.8, 32,768: 41.8 / 44.3, 49,152: 53.5 / 49.0.
template <int PREC>
constexpr int kLaneGroupMax = PREC == kPrecFP64 ? 14336 : PREC == kPrecFP32C ? 73728 : 38912;

// Saved words: row k of particle p has entries [5 k, 5 k + 5) of (bits, slot)
// pairs, in the particle's 16-byte groups of nbmask (as mask_at, so that the
// passes of one batch share the buffer).  (0, 0) ends a row; (0, 1) in front
// says that it had more words, and the second pass tests it again.
constexpr int kRowWords = 5;
static_assert((3 * kRowWords + 1) * 2 <= kMaskWords, "three rows fit a particle's mask words");
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
// multiples of 2^57 move to a 32-bit count (2^57 each).  A value that is not
// finite (kNotFixed) is found by the smallest high word of the neighbours'.
template <int KIND>
struct LaneSums<kPrecFP32X, KIND> {
  long long c, s;
  int ch, sh, low;
  __device__ void init() {
    c = s = 0;
    ch = sh = low = 0;
  }
  typedef longlong2 Value;
  __device__ static Value value(const KArgs &a, int j) { return KIND == kKindSin ? a.ics[j] : a.iws[j]; }
  __device__ void add(const Value &v, bool p) {
    add2_if(c, s, v, p);
    low = min(low, (int)(v.x >> 32));  // a v that is not added has been
  }
  __device__ void word_end(const ILane &) {
    constexpr long long rest = (1ll << 57) - 1;
    ch += (int)(c >> 57);
    sh += (int)(s >> 57);
    c &= rest;
    s &= rest;
  }
  __device__ void row_end() {}
  __device__ void join_group(unsigned mask, int) {
#pragma unroll
    for (int o = 1; o < kLaneGroup; o <<= 1) {  // four times 2^57 at most
      c += __shfl_xor_sync(mask, c, o);
      s += __shfl_xor_sync(mask, s, o);
      ch += __shfl_xor_sync(mask, ch, o);
      sh += __shfl_xor_sync(mask, sh, o);
      low = min(low, __shfl_xor_sync(mask, low, o));
    }
  }
  __device__ void finish(const KArgs &a, int epi, const SysDesc &sd, const ILane &il, int n, int q) {
    const int qv = KIND == kKindSin ? kXQ : sd.sc.xq2;
    const __int128 tc = ((__int128)ch << 57) + c, ts = ((__int128)sh << 57) + s;
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    const bool bad = low == (int)(kNotFixed >> 32);
    epilogue_fp32x<KIND>(a, epi, sd, il,
                         XSums{bad ? nan : from_fixed128(tc, qv), bad ? nan : from_fixed128(ts, qv), n}, q);
  }
};

// FP32C: a word's neighbours are summed in float, turned into the alignment
// terms by angle addition and added with Kahan compensation, and so are the
// rows' sums.
template <int KIND>
struct LaneSums<kPrecFP32C, KIND> {
  float bc, bs, bdc, bds;
  Acc<kPrecFP32C> tot;
  Acc<kPrecFP32C> acc;
  __device__ void init() {
    bc = bs = bdc = bds = 0.0f;
    acc.init();
    tot.init();
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
  // the row's compensated sums join the total
  __device__ void row_end() {
    join(acc);
    acc.init();
  }
  __device__ void join(const Acc<kPrecFP32C> &row) {
    kahan_add(tot.s0, tot.c0, row.s0);
    kahan_add(tot.s0, tot.c0, -row.c0);
    if constexpr (KIND == kKindCos2) {
      kahan_add(tot.s1, tot.c1, row.s1);
      kahan_add(tot.s1, tot.c1, -row.c1);
    }
  }
  __device__ void join_group(unsigned mask, int lead) {
    const Acc<kPrecFP32C> mine = acc;
    for (int k = 0; k < 3; ++k) {
      Acc<kPrecFP32C> row;
      row.s0 = __shfl_sync(mask, mine.s0, lead + k);
      row.c0 = __shfl_sync(mask, mine.c0, lead + k);
      row.s1 = __shfl_sync(mask, mine.s1, lead + k);
      row.c1 = __shfl_sync(mask, mine.c1, lead + k);
      join(row);
    }
  }
  __device__ void finish(const KArgs &a, int epi, const SysDesc &sd, const ILane &il, int n, int q) {
    acc.n = n;
    acc.s0 = tot.s0 - tot.c0;
    acc.s1 = tot.s1 - tot.c1;
    epilogue<kPrecFP32C, KIND>(a, epi, sd, il, acc, q);
  }
};

// The words that a group's first three lanes listed (lane k: row k), one after
// the other, for walks in which the whole warp stays together: a group whose
// words are used up idles until the last one's are.  skip: an empty list.
struct GroupWords {
  int w0, w1, w2, i;
  __device__ GroupWords(int nw, int lead, bool skip) {
    w0 = __shfl_sync(0xffffffffu, nw, lead);
    w1 = w0 + __shfl_sync(0xffffffffu, nw, lead + 1);
    w2 = w1 + __shfl_sync(0xffffffffu, nw, lead + 2);
    if (skip) w0 = w1 = w2 = 0;
    i = 0;
  }
  // the next word when `bits` is used up; col: the first lane's column
  __device__ void next(const uint32_t (*s_bits)[kLaneThreads], const int (*s_slot)[kLaneThreads], int col,
                       uint32_t &bits, int &slot) {
    if (bits != 0u || i >= w2) return;
    const int row = i < w0 ? 0 : (i < w1 ? 1 : 2);
    const int w = i - (row == 0 ? 0 : (row == 1 ? w0 : w1));
    bits = s_bits[w][col + row];
    slot = s_slot[w][col + row];
    ++i;
  }
};

// Lane g's neighbour of the word's next four (slot of bit 31: `slot`; `none`
// when there are fewer); they leave the word.
__device__ __forceinline__ int group_pick(uint32_t &bits, int slot, int g, int m, int none) {
  int j = none;
#pragma unroll
  for (int u = 0; u < kLaneGroup; ++u) {
    const int t = __clz(bits);
    if (u == g && u < m) j = slot + t;
    bits &= ~(0x80000000u >> (t & 31));
  }
  return j;
}

// G lanes per particle: 1 or kLaneGroup.  REST (FP64 pass 1): some system has
// rests.  (The gather and this kernel compiled without them: an Euler step of N =
// 1,024 at alpha = 1.45 takes 25.2 us, 26.7 with a test at run time.)
template <int PREC, int KIND, int G, bool REST = false>
__global__ void __launch_bounds__(kLaneThreads, PREC != kPrecFP64 && G == 1 ? 10 : 1) k_lane(KArgs a, int epi) {
  constexpr bool kList = PREC == kPrecFP64;
  __shared__ uint32_t s_bits[kList ? kLaneWords : 1][kLaneThreads];
  __shared__ int s_slot[kList ? kLaneWords : 1][kLaneThreads];
  const int tid = threadIdx.x, g = tid % G, lead = tid % kWarp - g;
  const int p_own = a.lane_p0 + (blockIdx.x * blockDim.x + tid) / G;
  if (G == 1 && p_own >= a.lane_p1) return;  // no barrier below
  // groups: the warps stay whole, lanes past the end repeat the last particle
  const int p = min(p_own, a.lane_p1 - 1);
  const int n_all = a.n_active;
  const int c = cell_of_slot(a, p);
  const SysDesc &sd = a.sys[a.sys_of_c[c]];
  const SysConst &sc = sd.sc;
  ILane il;
  load_i<PREC, KIND, REST>(a, sc, il, p, true);
  LaneSums<PREC, KIND> sums;
  sums.init();
  int n = 0;
  uint2 *saved = reinterpret_cast<uint2 *>(a.nbmask);

  int nw = 0;  // FP64: words listed
  bool full = false;  // FP64, G > 1: the row has more words than the list
  auto walk_list = [&]() {
    if constexpr (kList) {
      int w = -1;
      walk_pairs<KIND, kLanePairs, REST>(
          sums.acc, sc, il,
          [&](uint32_t &bits, int &base) {
            if (++w >= nw) return false;
            bits = s_bits[w][tid];
            base = s_slot[w][tid];
            return true;
          },
          [&](int j) { return a.dcs[j]; }, [&](int j) { return a.dphi_s[j]; }, [&](int j) { return a.sphi[j]; },
          [&](int j) { return (uint32_t)a.rest[j]; });
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

  const float nlo = -sc.lo2, wid = undecided_width(sc.lo2, sc.hi2);
  const bool exact_all = sc.exact_all != 0;
  const int nc = sc.nc, cl = c - sd.c0, cy = cl / nc, cx = cl - cy * nc;
  const LaneRuns r = lane_runs(cx, nc);
  const float xa = il.fx - (float)r.sa * sc.cell_f, xb = il.fx - (float)r.sb * sc.cell_f;
  // rows [k0, k1) of the stencil; flush: walk the FP64 list when it is full
  auto rows = [&](int k0, int k1, bool flush) {
    const int *row = a.cell_start + sd.c0 + adjust_cell(cy + k0 - 1, nc) * nc;
    int a0 = row[r.a0], a1 = row[r.a1], b0 = row[r.b0], b1 = row[r.b1];
#pragma unroll(!kList && G == 1 ? 3 : 1)
    for (int k = k0; k < k1; ++k) {
      // the next row's bounds, on their way while this row is tested
      const int *next = a.cell_start + sd.c0 + adjust_cell(cy + min(k, 1), nc) * nc;
      const int na0 = next[r.a0], na1 = next[r.a1], nb0 = next[r.b0], nb1 = next[r.b1];
      // room for a row's saved words (with flush off the list starts empty)
      if (kList && flush && nw > kLaneWords - kRowWords) walk_list();
      bool listed = false;  // pass 2: the first pass left this row's words
      if constexpr (KIND == kKindCos2) {
        if (saved) {
          uint2 e = saved[saved_at(k * kRowWords, p, n_all)];
          listed = e.x != 0u || e.y == 0u;
          if (listed)
            for (int w = 1; e.x != 0u; ++w) {
              const uint2 after = w < kRowWords ? saved[saved_at(k * kRowWords + w, p, n_all)] : make_uint2(0u, 0u);
              take(e.x, (int)e.y);
              e = after;
            }
        }
      }
      if (!listed) {
        int nsaved = 0;
        auto found = [&](uint32_t bits, int slot) {
          if (bits == 0u) return;
          if (KIND == kKindSin && saved) {
            if (nsaved < kRowWords) saved[saved_at(k * kRowWords + nsaved, p, n_all)] = make_uint2(bits, (uint32_t)slot);
            ++nsaved;
          }
          take(bits, slot);
        };
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
          if (kList && nw > kLaneWords - 2) {
            if (flush) {
              walk_list();
            } else {
              full = true;
              return;
            }
          }
        }
        if (KIND == kKindSin && saved) {
          if (nsaved < kRowWords)
            saved[saved_at(k * kRowWords + nsaved, p, n_all)] = make_uint2(0u, 0u);
          else if (nsaved > kRowWords)
            saved[saved_at(k * kRowWords, p, n_all)] = make_uint2(0u, 1u);
        }
      }
      if constexpr (!kList && G == 1) sums.row_end();
      a0 = na0, a1 = na1, b0 = nb0, b1 = nb1;
    }
  };

  if constexpr (G == 1) {
    rows(0, 3, true);
    walk_list();
  } else {
    constexpr unsigned kAll = 0xffffffffu;
    if (g < 3) rows(g, g + 1, false);
    bool alone = false;
    if constexpr (kList) {
      __syncwarp();
      alone = ((__ballot_sync(kAll, full) >> lead) & ((1u << G) - 1u)) != 0u;  // a very long row
      GroupWords words(nw, lead, alone);
      uint32_t bits = 0u;
      int slot = 0;
      while (true) {
        words.next(s_bits, s_slot, tid - g, bits, slot);
        const int m = __popc(bits);
        if (!__any_sync(kAll, m > 0)) break;
        const int j = group_pick(bits, slot, g, m, p);
        const double2 cj = a.dcs[j];
        const double pr = KIND == kKindSin ? -dmul(cj.x, il.dsa) : dmul(cj.y, il.dsa);
        double t = __fma_rn(KIND == kKindSin ? cj.y : cj.x, il.dca, pr);
        const double d = KIND == kKindCos2 ? dsub(a.dphi_s[j], il.dphi) : 0.0;
        if (g < m) {
          if (small_term(t))
            t = KIND == kKindSin ? sin_of_difference(a.sphi[j], il.phi, sc.alpha)
                                 : cos_of_difference(a.sphi[j], il.phi, sc.alpha);
          else if (REST && il.rest)
            sums.acc.rest += sine_rest(il, a.rest[j], cj.x, -pr);
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < G; ++u) {
          const double tu = __shfl_sync(kAll, t, lead + u);
          const double du = KIND == kKindCos2 ? __shfl_sync(kAll, d, lead + u) : 0.0;
          if (u < m) {
            sums.acc.s0 = dadd(sums.acc.s0, tu);
            if constexpr (KIND == kKindCos2) sums.acc.s1 = __fma_rn(du, tu, sums.acc.s1);
          }
        }
      }
    } else {
      __syncwarp();
      sums.join_group(kAll, lead);
    }
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
      n += __shfl_xor_sync(kAll, n, o);
      if constexpr (REST) sums.acc.rest += __shfl_xor_sync(kAll, sums.acc.rest, o);
    }
    if (g != 0 || p_own >= a.lane_p1) return;
    if (alone) {  // the first lane walks as it tests
      n = nw = 0;
      rows(0, 3, true);
      walk_list();
    }
  }
  sums.finish(a, epi, sd, il, n, a.pidx[p]);
}

}  // namespace spc
