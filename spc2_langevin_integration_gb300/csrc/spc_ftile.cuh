// Cell-tile passes of the float forms (FP32C, FP32X) on the tensor cores.
//
// A pass is, for each particle i of a cell, a sum over the candidates j of the
// cell's 3x3 stencil of (cos phi_j, sin phi_j), pass 2: of the phase rate times
// those, where the pair is inside the cutoff: the product of a 0/1 matrix that
// the distance tests make and a matrix of a few columns.  The values are cut
// into signed digits that a half holds exactly, so every product and every
// sum in the 32-bit accumulators is an exact integer (a round's sums are at most
// 2^21): the result depends neither on the order of the list nor on how it is
// cut among warps, rounds and CTAs.  The columns of a candidate are
//   FP32C (8):  three digits each of cos and sin, base 4096 (units of 2^-35:
//               a float's own rounding is 2^-25), 1 (the count), and 1 for a
//               value that is not finite, whose digits are 0
//   FP32X (16): five digits each, base 2048, of the 64-bit fixed-point values,
//               1 (the count), 1 for a value that is not finite, zeros
// A warp takes 32 particles (rows) and 32 candidates at a time; its
// lanes hold the tests in the layout of mma.sync's A operand (lane 4 g + t:
// rows g + 8 k, candidates 8 m + 2 t and the next), so a test becomes an A
// element without leaving its lane.  Eight candidates' 16-byte records are one
// 8x8 matrix of ldmatrix, and are staged as they stand in memory.
//
// A block of 32 x 32 tests takes 64 packed operations for the offsets, 48 for
// signs, A elements and the undecided check, and 4 (FP32X: 8) matrix
// instructions, some 5 instructions a test, where predicated sums took 18
// (FP32C) and 20 (FP32X).  Bound by issue (69% busy over 8,100 cells of 65
// particles, where a CTA's stencil, staging and epilogue are a third of its
// instructions) and, for one wave of CTAs, by the latency of those.
// Against predicated sums, in us: N = 2^22 at 64 a cell, FP32C pass 1 1,480 ->
// 948; vortex SRK N = 65,536, passes 1 and 2: FP32C 41 + 33 -> 31 + 29, FP32X
// clustered with cell units 72 + 76 -> 56 + 68 (with its FP64 epilogues).
//
// tcgen05 would want the 0/1 matrix in tensor memory or shared memory: another
// store per test, and a block of 128 rows where a cell has 64.
#pragma once

#include "spc_tile.cuh"

namespace spc {

constexpr int kPartWarps = kTileThreads32 / kWarp;  // a round's list is cut among a CTA's warps

template <int PREC>
struct FloatTile;
template <>
struct FloatTile<kPrecFP32C> {
  static constexpr int kCap = kTileCap, kNT = 1, kCols = 8;  // kCols: columns summed (padded to 16 bytes)
};
template <>
struct FloatTile<kPrecFP32X> {
  static constexpr int kCap = kTileCapX, kNT = 2, kCols = 12;
};
// The stencil of the CTA's cell, filled by its first warp.
struct TileStencil {
  int start[9];    // cell-order start of each stencil cell
  int prefix[10];  // offsets of each stencil cell in the staged list
  __device__ int slot(int g) const {
    int q = 0;
    while (q < 8 && g >= prefix[q + 1]) ++q;
    return start[q] + g - prefix[q];
  }
};
template <int PREC>
struct TileMem {
  TileStencil st;
  float4 xy[FloatTile<PREC>::kCap / 2];  // x, x', y, y' of candidates 2 k and 2 k + 1, shifted
  uint4 b[FloatTile<PREC>::kNT][FloatTile<PREC>::kCap];
  int sum[kTileThreads32][FloatTile<PREC>::kCols];  // column sums of each particle of the group
};

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
// min(m, |a|, |b|); NaNs are passed over
__device__ __forceinline__ float min_abs(float m, float a, float b) {
  asm("min.abs.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(a), "f"(b));
  return m;
}
// bit 0 (16) set where a (b) is negative
__device__ __forceinline__ uint32_t negative2(float a, float b) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, 0xffbb;" : "=r"(r) : "r"(__float_as_uint(a)), "r"(__float_as_uint(b)));
  return r & 0x00010001u;
}
// The 8x8 half matrices of the 32 records from p on, transposed: r[m] holds
// column `lane / 4` of records 8 m + 2 (lane % 4) and the next.
__device__ __forceinline__ void load_records(const uint4 *p, uint32_t (&r)[4]) {
  const uint32_t at = (uint32_t)__cvta_generic_to_shared(p + threadIdx.x % kWarp);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(at)
               : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void copy16_async(uint4 *to, const uint4 *from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from)
               : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A elements are the half with bit 0 set, 2^-24, so that a test's bit and its
// A element are the same bit; a column's sum comes back as an integer (at most
// kCap digits of at most 2048 each: 2^21).
__device__ __forceinline__ int column_sum(float acc) {
  return __float_as_int(fmaf(acc, 16777216.0f, 12582912.0f)) - 0x4b400000;
}

// Bits of a block: A element (k, m) of a lane is bit 4 k + m (candidate
// 8 m + 2 t) and bit 16 + 4 k + m (the next candidate) of its word.  The four
// lanes of a quad exchange nibbles, so that lane 4 g + t gets row g + 8 t's
// whole word (kept in nbmask between the SRK passes), and back.
__device__ __forceinline__ uint32_t quad_transpose(uint32_t w, int t) {
  uint32_t u = __shfl_xor_sync(0xffffffffu, w, 1);
  w = (t & 1) ? (w & 0xf0f0f0f0u) | ((u >> 4) & 0x0f0f0f0fu) : (w & 0x0f0f0f0fu) | ((u & 0x0f0f0f0fu) << 4);
  u = __shfl_xor_sync(0xffffffffu, w, 2);
  return __byte_perm(w, u, (t & 2) ? 0x3715 : 0x6240);
}

// Fills s.st for cell c (half: as stencil_of) and returns the list's length.
// Called by the whole CTA; ends with all threads past the previous cell.
template <int PREC>
__device__ __forceinline__ int share_stencil(const KArgs &a, const SysDesc &sd, int c, TileMem<PREC> &s,
                                             int half = -1) {
  __syncthreads();
  if (threadIdx.x < kWarp) {
    const int q = threadIdx.x;
    int ja = 0, n = 0;
    if (q < 9) {
      int jb;
      stencil_cell(a, sd, c, q, half, ja, jb);
      n = jb - ja;
    }
    int upto = n;
#pragma unroll
    for (int off = 1; off < 16; off <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, off);
      if (q >= off) upto += v;
    }
    if (q < 9) {
      s.st.start[q] = ja;
      s.st.prefix[q + 1] = upto;
      if (q == 0) s.st.prefix[0] = 0;
    }
  }
  __syncthreads();
  return s.st.prefix[9];
}

// Stage candidates [rlo, rlo + rcnt) of the stencil list, padded to rpad: a
// warp takes stencil cell after stencil cell, 64 members at a time.
constexpr int kStageCopies = 2;
template <int PREC, int KIND>
__device__ __forceinline__ void stage_tile(const KArgs &a, const SysConst &sc, TileMem<PREC> &s, int rlo, int rcnt,
                                           int rpad, bool masked) {
  constexpr int NT = FloatTile<PREC>::kNT;
  const uint4 *dig = KIND == kKindSin ? a.dig : a.wdig;
  const bool coords = !(KIND == kKindCos2 && masked);
  float *xy = reinterpret_cast<float *>(s.xy);
  const int lane = threadIdx.x % kWarp;
  for (int q = threadIdx.x / kWarp; q < 9; q += kPartWarps) {
    const int at = s.st.prefix[q] - rlo, from = s.st.start[q];
    const int i1 = min(s.st.prefix[q + 1] - s.st.prefix[q], rcnt - at);
    const float sx = shift_x(q, sc.cell_f), sy = shift_y(q, sc.cell_f);
    for (int i = max(0, -at) + lane; i < i1; i += kStageCopies * kWarp) {
      float2 f[kStageCopies];
#pragma unroll
      for (int u = 0; u < kStageCopies; ++u) {
        if (i + u * kWarp >= i1) break;
        const int pj = from + i + u * kWarp, k = at + i + u * kWarp;
#pragma unroll
        for (int h = 0; h < NT; ++h) copy16_async(&s.b[h][k], dig + (size_t)pj * NT + h);
        if (coords) f[u] = a.fxy[pj];
      }
      if (coords) {
#pragma unroll
        for (int u = 0; u < kStageCopies; ++u) {
          const int k = at + i + u * kWarp;
          if (i + u * kWarp >= i1) break;
          xy[(k >> 1) * 4 + (k & 1)] = f[u].x + sx;
          xy[(k >> 1) * 4 + 2 + (k & 1)] = f[u].y + sy;
        }
      }
    }
  }
  // padding: never a neighbour, never near the cutoff
  const int k = rcnt + (int)threadIdx.x - (kTileThreads32 - kWarp);
  if (threadIdx.x >= kTileThreads32 - kWarp && k < rpad) {
    xy[(k >> 1) * 4 + (k & 1)] = 3.0e18f;
    xy[(k >> 1) * 4 + 2 + (k & 1)] = 3.0e18f;
#pragma unroll
    for (int h = 0; h < NT; ++h) s.b[h][k] = make_uint4(0u, 0u, 0u, 0u);
  }
  copies_done();
}

// One warp: rows [row0, row0 + rows) (rows <= 32) of the group that starts
// at slot ig, against [jlo, jhi) of the staged round [rlo, rlo + rcnt); the
// column sums are added to s.sum.  Called by all lanes.
template <int PREC, int KIND>
__device__ __forceinline__ void tile_rows(const KArgs &a, const SysConst &sc, TileMem<PREC> &s,
                                          int c0, int ig, int row0, int rows, int rlo, int rcnt, int jlo, int jhi,
                                          bool masked) {
  constexpr int NT = FloatTile<PREC>::kNT, MT = 2, K = 2 * MT;  // two 16-row tiles
  const int n_all = a.n_active;
  const int lane = threadIdx.x % kWarp, g = lane >> 2, t = lane & 3;
  const int p0 = ig + row0;
  const bool exact_all = sc.exact_all != 0;
  const float band = 0.5f * (sc.hi2 - sc.lo2), nmid = -0.5f * (sc.hi2 + sc.lo2);
  const bool words = KIND == kKindCos2 && masked;  // pass 1 left the neighbours' bits
  float nx[K], ny[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    nx[k] = ny[k] = -3.0e17f;
    if (!words && g + 8 * k < rows) {
      const float2 f = a.fxy[p0 + g + 8 * k];
      nx[k] = -f.x;
      ny[k] = -f.y;
    }
  }
  float acc[MT][NT][4] = {};
  // the row whose saved words this lane keeps
  const int wrow = g + 8 * t, wp = p0 + wrow;
  const bool keeps = wrow < rows;
  const int self0 = s.st.prefix[4] + (p0 - c0) - rlo;  // staged index of row 0 itself
  const uint4 *m4 = reinterpret_cast<const uint4 *>(a.nbmask);
  const uint4 none = make_uint4(0u, 0u, 0u, 0u);
  int grp = jlo / kWarp >> 2;
  uint4 cur = none, nxt = none;
  if (KIND == kKindCos2 && words && keeps) {
    if (jlo < jhi) cur = m4[(size_t)grp * n_all + wp];
    if ((grp + 1) * 4 * kWarp < jhi) nxt = m4[(size_t)(grp + 1) * n_all + wp];
  }
  for (int j0 = jlo; j0 < jhi; j0 += kWarp) {
    uint32_t A[K][4];
    uint32_t w = 0u;
    bool expand;
    if (KIND == kKindCos2 && words) {
      const int wd = j0 / kWarp;
      if ((wd >> 2) != grp) {
        ++grp;
        cur = nxt;
        nxt = keeps && (grp + 1) * 4 * kWarp < jhi ? m4[(size_t)(grp + 1) * n_all + wp] : none;
      }
      const int sub = wd & 3;
      w = quad_transpose(sub == 0 ? cur.x : sub == 1 ? cur.y : sub == 2 ? cur.z : cur.w, t);
      expand = true;
    } else {
      float mn = 3.0e38f;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const float4 c = s.xy[(j0 >> 1) + 4 * m + t];
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const float2 dx = add2(make_float2(c.x, c.y), make_float2(nx[k], nx[k]));
          const float2 dy = add2(make_float2(c.z, c.w), make_float2(ny[k], ny[k]));
          const float2 o = fma2(dx, dx, fma2(dy, dy, make_float2(nmid, nmid)));
          mn = min_abs(mn, o.x, o.y);
          A[k][m] = negative2(o.x, o.y);
        }
      }
      const bool selves = j0 < self0 + kWarp && self0 < j0 + kWarp;  // the block holds some rows themselves
      const bool amb = exact_all || mn <= band;
      expand = __any_sync(0xffffffffu, amb) || selves;
      if (expand || (KIND == kKindSin && masked)) {
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
          for (int m = 0; m < 4; ++m) w += A[k][m] << (4 * k + m);
      }
      if (expand) {
        if (amb) {  // pairs the float test cannot decide: the reference's FP64 test
          uint32_t open = 0u;  // the same bits as w
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            const float4 c = s.xy[(j0 >> 1) + 4 * m + t];
#pragma unroll
            for (int k = 0; k < K; ++k) {
              const float o0 = cutoff_offset(c.x + nx[k], c.z + ny[k], nmid);
              const float o1 = cutoff_offset(c.y + nx[k], c.w + ny[k], nmid);
              open |= (exact_all || fabsf(o0) <= band ? 1u : 0u) << (4 * k + m);
              open |= (exact_all || fabsf(o1) <= band ? 1u : 0u) << (16 + 4 * k + m);
            }
          }
          while (open) {
            const int b = __ffs(open) - 1;
            open &= open - 1u;
            const int r = g + 8 * ((b >> 2) & 3), j = j0 + 8 * (b & 3) + 2 * t + (b >> 4);
            if (r >= rows || j >= rcnt) continue;
            const int pj = s.st.slot(rlo + j);
            const bool in = exact_within(sc, a.sx[p0 + r], a.sy[p0 + r], a.sx[pj], a.sy[pj]);
            w = in ? w | (1u << b) : w & ~(1u << b);
          }
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {  // the rows themselves
          const int d = self0 + g + 8 * k - j0;
          if ((unsigned)d < (unsigned)kWarp && ((d >> 1) & 3) == t) w &= ~(1u << (16 * (d & 1) + 4 * k + (d >> 3)));
        }
      }
      if (KIND == kKindSin && masked) {
        const uint32_t row_word = quad_transpose(w, t);
        if (keeps) a.nbmask[mask_at(j0 / kWarp, wp, n_all)] = row_word;
      }
    }
    if (expand) {
#pragma unroll
      for (int k = 0; k < K; ++k)
#pragma unroll
        for (int m = 0; m < 4; ++m) A[k][m] = (w >> (4 * k + m)) & 0x00010001u;
    }
#pragma unroll
    for (int h = 0; h < NT; ++h) {
      uint32_t b[4];
      load_records(&s.b[h][j0], b);
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        mma16816(acc[i][h], A[2 * i][0], A[2 * i + 1][0], A[2 * i][1], A[2 * i + 1][1], b[0], b[1]);
        mma16816(acc[i][h], A[2 * i][2], A[2 * i + 1][2], A[2 * i][3], A[2 * i + 1][3], b[2], b[3]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int h = 0; h < NT; ++h)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int col = 8 * h + 2 * t + (e & 1), row = row0 + 16 * i + g + 8 * (e >> 1);
        if (col < FloatTile<PREC>::kCols) atomicAdd(&s.sum[row][col], column_sum(acc[i][h][e]));
      }
}

// One warp's part of a staged round for a group of gi rows: a quarter of the
// list's blocks.  (Equal shares of all row tiles' blocks, tiles of 16 rows for
// a last tile of at most 16, and 96 members at a time in the staging were each
// within 2%.)
template <int PREC, int KIND>
__device__ __forceinline__ void tile_round(const KArgs &a, const SysConst &sc, TileMem<PREC> &s, int c0, int ig,
                                           int gi, int rlo, int rcnt, int rpad, bool masked) {
  const int w = threadIdx.x / kWarp, nb = rpad / kWarp;
  const int jlo = nb * w / kPartWarps * kWarp, jhi = nb * (w + 1) / kPartWarps * kWarp;
  for (int row0 = 0; row0 < gi; row0 += kWarp)
    tile_rows<PREC, KIND>(a, sc, s, c0, ig, row0, min(kWarp, gi - row0), rlo, rcnt, jlo, jhi, masked);
}

template <int PREC>
__device__ __forceinline__ void clear_sums(TileMem<PREC> &s) {
  int4 *r = reinterpret_cast<int4 *>(s.sum[threadIdx.x]);
#pragma unroll
  for (int k = 0; k < FloatTile<PREC>::kCols / 4; ++k) r[k] = make_int4(0, 0, 0, 0);
}

// A particle's sums over its rounds, as integers.
template <int PREC>
struct RowSums;

template <>
struct RowSums<kPrecFP32C> {
  long long c = 0, s = 0;
  int n = 0, bad = 0;
  __device__ void add(const int (&v)[8]) {
    c += ((long long)v[0] << 24) + (((long long)v[1] << 12) + v[2]);
    s += ((long long)v[3] << 24) + (((long long)v[4] << 12) + v[5]);
    n += v[6];
    bad += v[7];
  }
  __device__ longlong2 pair() const { return make_longlong2(c, s); }
  // a round's count, complemented when a neighbour's value was not finite
  __device__ int count() const { return bad ? ~n : n; }
  __device__ void add(longlong2 v, int m) {
    c += v.x;
    s += v.y;
    if (m < 0) {
      bad = 1;
      m = ~m;
    }
    n += m;
  }
};
template <>
struct RowSums<kPrecFP32X> {
  __int128 c = 0, s = 0;
  int n = 0, bad = 0;
  __device__ void add(const int (&v)[12]) {
    long long p = v[4], q = v[9];
#pragma unroll
    for (int k = 3; k >= 0; --k) {
      p = p * 2048 + v[k];
      q = q * 2048 + v[k + 5];
    }
    c += p;
    s += q;
    n += v[10];
    bad += v[11];
  }
  __device__ longlong2 pair() const { return make_longlong2((long long)c, (long long)s); }  // one round
  __device__ int count() const { return bad ? ~n : n; }
  __device__ void add(longlong2 v, int m) {
    c += v.x;
    s += v.y;
    if (m < 0) {
      bad = 1;
      m = ~m;
    }
    n += m;
  }
};

template <int PREC>
__device__ __forceinline__ void take_row(const TileMem<PREC> &s, RowSums<PREC> &sum) {
  int v[FloatTile<PREC>::kCols];
#pragma unroll
  for (int k = 0; k < FloatTile<PREC>::kCols; k += 4)
    *reinterpret_cast<int4 *>(v + k) = *reinterpret_cast<const int4 *>(s.sum[threadIdx.x] + k);
  sum.add(v);
}

// v 2^-35 as an unevaluated sum of two floats (the whole within 2^-48 of v): below
// 2,048 from two parts that are exact, else v rounded to float and the rest.
__device__ __forceinline__ float2 two_floats(long long v) {
  const long long up = v >> 22;
  if ((unsigned long long)(up + (1ll << 24)) < 1ull << 25) {
    const float a = (float)(int)up * 0x1p-13f, b = (float)(int)(v & 0x3fffff) * 0x1p-35f;
    const float h = a + b, bb = h - a;
    return make_float2(h, (a - (h - bb)) + (b - bb));
  }
  const float h = __ll2float_rn(v);
  return make_float2(h * 0x1p-35f, __ll2float_rn(v - __float2ll_rn(h)) * 0x1p-35f);
}
// x u + y v for such sums x and y
__device__ __forceinline__ float dot2(float2 x, float u, float2 y, float v) {
  const float p = x.x * u, q = y.x * v;
  const float ep = fmaf(x.x, u, -p), eq = fmaf(y.x, v, -q);
  const float r = p + q, bb = r - p;
  const float er = (p - (r - bb)) + (q - bb);
  return r + (er + (ep + eq) + fmaf(x.y, u, y.y * v));
}

// Particle p's sums become the plain form's accumulators by the
// angle-addition identities (theta_i = phi_i + alpha; see epilogue_fp32x) and
// its step is finished; FP32X leaves that to k_epilogue_fp32x.
template <int KIND>
__device__ __forceinline__ void finish_row(const KArgs &a, int epi, const SysDesc &sd, int p,
                                           const RowSums<kPrecFP32C> &sum) {
  const SysConst &sc = sd.sc;
  ILane il;
  load_i<kPrecFP32C, KIND>(a, sc, il, p, true);
  Acc<kPrecFP32C> acc;
  acc.init();
  acc.n = sum.n;
  float2 C = two_floats(sum.c), S = two_floats(sum.s);
  if (sum.bad) C.x = S.x = __int_as_float(0x7fffffff);
  if constexpr (KIND == kKindSin) {
    acc.s0 = dot2(S, il.ca, C, -il.sa);
    if (epi == kEpiSrk1) {
      // for the second pass: the sum of cosines, and the mean of the sines
      // (|rate / sigma|) times cos phi_i and sin phi_i
      a.scos_f[p] = dot2(C, il.ca, S, il.sa);
      const float mean = sum.n ? acc.s0 / (float)sum.n : 0.0f;
      const float2 cs = a.cs[p];
      a.wdig[p] = float_digits(mean * cs.x, mean * cs.y);
    }
  } else {
    acc.s0 = a.scos_f[p];
    // sum_j (d_j - d_i) cos(phi_j - theta_i)
    acc.s1 = fmaf((float)sc.sigma, dot2(C, il.ca, S, il.sa), -il.dphif * acc.s0);
  }
  epilogue<kPrecFP32C, KIND>(a, epi, sd, il, acc, a.pidx[p]);
}
template <int KIND>
__device__ __forceinline__ void finish_row(const KArgs &a, int epi, const SysDesc &sd, int p,
                                           const RowSums<kPrecFP32X> &sum) {
  const int qv = KIND == kKindSin ? kXQ : sd.sc.xq2;
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  a.xsum[p] = sum.bad ? make_double2(nan, nan) : make_double2(from_fixed128(sum.c, qv), from_fixed128(sum.s, qv));
  a.xcnt[p] = sum.n;
}

// UNITS: unit cells are left to the units kernel.
template <int PREC, int KIND, bool UNITS>
__global__ void __launch_bounds__(kTileThreads32, PREC == kPrecFP32C ? 7 : 6) k_tile_float(KArgs a, int epi) {
  constexpr int CAP = FloatTile<PREC>::kCap;
  __shared__ __align__(128) TileMem<PREC> s;
  const int tid = threadIdx.x;
  const int nitems = tile_items(a);
  for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
    TileItem ti;
    if (!tile_item<kTileThreads32>(a, item, ti)) continue;
    if constexpr (UNITS) {
      if (a.cell_unit[ti.c]) continue;  // run by the units kernel
    }
    const SysDesc &sd = a.sys[a.sys_of_c[ti.c]];
    const SysConst &sc = sd.sc;
    if (sc.allpairs) continue;
    const int total = share_stencil(a, sd, ti.c, s);
    const int rounds = (total + CAP - 1) / CAP;
    const bool masked = rounds == 1 && a.nbmask != nullptr && !sc.exact_all && (KIND == kKindCos2 || epi == kEpiSrk1);
    for (int ig = ti.cb; ig < ti.ce; ig += kTileThreads32) {
      const int gi = min(kTileThreads32, ti.ce - ig);
      RowSums<PREC> sum;  // of particle ig + tid
      for (int r = 0; r < rounds; ++r) {
        const int rlo = r * CAP, rcnt = min(CAP, total - rlo);
        const int rpad = (rcnt + kWarp - 1) & ~(kWarp - 1);
        clear_sums(s);
        if (rounds > 1 || ig == ti.cb) {
          if (r > 0 || ig != ti.cb) __syncthreads();
          stage_tile<PREC, KIND>(a, sc, s, rlo, rcnt, rpad, masked);
        }
        __syncthreads();
        tile_round<PREC, KIND>(a, sc, s, ti.c0, ig, gi, rlo, rcnt, rpad, masked);
        __syncthreads();
        if (tid < gi) take_row(s, sum);
      }
      if (tid < gi) finish_row<KIND>(a, epi, sd, ig + tid, sum);
    }
  }
}

// The units of a pass (listed by k_list_units after the gather): unit u of
// cell c is chunk u / rounds (32 particles) x staging round u % rounds.  A
// unit stores its particles' sums of the round and the last unit of a chunk
// to finish adds the rounds.
template <int PREC, int KIND>
__global__ void __launch_bounds__(kTileThreads32, PREC == kPrecFP32C ? 7 : 6) k_units_float(KArgs a, int epi) {
  constexpr int CAP = FloatTile<PREC>::kCap;
  __shared__ __align__(128) TileMem<PREC> s;
  __shared__ int s_last;
  const int n_all = a.n_active;
  const int tid = threadIdx.x;
  const int count = *a.unit_count;
  for (int i = blockIdx.x; i < count; i += gridDim.x) {
    const int2 e = a.units[i];
    // the unit's cell and, with sub-cells, its half: particles [g0, g1)
    const int c = a.cell_mid ? e.x >> 1 : e.x, half = a.cell_mid ? e.x & 1 : -1;
    const int c0 = a.cell_start[c];
    const int g0 = half == 1 ? a.cell_mid[c] : c0;
    const int g1 = half == 0 ? a.cell_mid[c] : a.cell_start[c + 1];
    const SysDesc &sd = a.sys[a.sys_of_c[c]];
    const SysConst &sc = sd.sc;
    const int total = share_stencil(a, sd, c, s, half);
    const int rounds = (total + CAP - 1) / CAP;
    const bool masked = rounds == 1 && a.nbmask != nullptr && !sc.exact_all && (KIND == kKindCos2 || epi == kEpiSrk1);
    const int k = e.y / rounds, r = e.y - k * rounds;
    const int ig = g0 + k * kWarp, gi = min(kWarp, g1 - ig);
    const int rlo = r * CAP, rcnt = min(CAP, total - rlo);
    const int rpad = (rcnt + kWarp - 1) & ~(kWarp - 1);
    clear_sums(s);
    stage_tile<PREC, KIND>(a, sc, s, rlo, rcnt, rpad, masked);
    __syncthreads();
    tile_round<PREC, KIND>(a, sc, s, c0, ig, gi, rlo, rcnt, rpad, masked);
    __syncthreads();
    RowSums<PREC> sum;
    const int p = ig + tid;
    if (tid < gi) take_row(s, sum);
    if (rounds == 1) {
      if (tid < gi) finish_row<KIND>(a, epi, sd, p, sum);
      continue;
    }
    if (tid < gi) {
      a.part_x[(size_t)r * n_all + p] = sum.pair();
      a.part_n[(size_t)r * n_all + p] = sum.count();
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(&a.unit_done[ig], 1) == rounds - 1;
    __syncthreads();
    if (s_last) {
      __threadfence();
      if (tid < gi) {
        RowSums<PREC> all;
        for (int q = 0; q < rounds; ++q)
          all.add(__ldcg(&a.part_x[(size_t)q * n_all + p]), __ldcg(&a.part_n[(size_t)q * n_all + p]));
        finish_row<KIND>(a, epi, sd, p, all);
      }
      if (tid == 0) a.unit_done[ig] = 0;  // for the next pass
    }
  }
}

}  // namespace spc
