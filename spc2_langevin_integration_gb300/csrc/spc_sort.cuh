// Stable counting sort of the particles by cell, and the cell start table.
// Every kernel takes an optional device gate: when it points to 0 the kernel
// returns at once (the Verlet path keeps its rebuild in a captured step and
// runs it only on the evaluations that need one).
//
// This replaces the reference's serial linked-list rebuild
// (`linked_list_[pre_linked_list_[i]].push_back(i)` for i = 0..N-1,
// ChimeraSystem.cpp:335-338), whose cells hold their members in ascending
// index order:
//  1. k_stage counts each key's particles (an atomic per particle, which also
//     numbers the cell's arrivals);
//  2. the counts are scanned into the start table (one CTA up to
//     kScanOneCta keys, else per-chunk sums and a second launch) and cleared
//     for the next evaluation;
//  3. k_place writes each particle's index to its cell's arrival slot;
//  4. k_gather ranks an index among its cell's (they arrive in any order) and
//     gathers the particle to that slot.
// The rank costs one compare per cell member, where the neighbour passes test
// nine cells' members with some ten instructions each (16,384 particles in one
// cell, Euler: the gather takes 385 us, FP32C's pass 29,300).  All-pairs systems are
// one cell with the members already in index order, and are neither counted
// nor ranked.
// Bound by latency (few keys) or by scattered 32-byte sectors.  Against a radix
// sort of (key, index) pairs by 8- to 11-bit digits, in us for stage + sort +
// gather: 96-system ensemble (681,278 particles, 110,312 cells) 145 -> 94, N =
// 2^22 in 65,536 cells 541 -> 335, N = 65,536 in 1,024 cells 37 -> 31.
// Up to kRankMax particles k_rank_gather takes the place of 2 to 4.
#pragma once

#include "spc_device.cuh"

namespace spc {

constexpr int kScanThreads = 1024;
constexpr int kScanChunk = 4 * kScanThreads;  // keys a CTA scans at a time
// With few keys the counters stand 16 bytes apart: the arrivals' atomics then
// spread over more of L2 (N = 65,536 in 1,024 cells: stage 12.9 -> 10.7 us; 8
// and 32 bytes the same within 0.2 us a step).
constexpr int kSpreadShift = 2;
constexpr int kSpreadKeys = kScanChunk;
inline int count_shift(int nkeys) { return nkeys <= kSpreadKeys ? kSpreadShift : 0; }
constexpr int kScanOneCta = 3 * kScanChunk;   // up to here one CTA scans chunk after chunk

// Block-wide exclusive scan of one value per thread (kScanThreads threads);
// *total gets the sum.
__device__ __forceinline__ int block_exclusive_scan(int mine, int *wsum, int *total) {
  const int t = threadIdx.x, lane = t % kWarp, w = t / kWarp;
  int incl = mine;
#pragma unroll
  for (int off = 1; off < kWarp; off <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += y;
  }
  __syncthreads();  // the previous scan's sums are no longer read
  if (lane == kWarp - 1) wsum[w] = incl;
  __syncthreads();
  if (w == 0) {
    const int s = wsum[lane];
    int si = s;
#pragma unroll
    for (int off = 1; off < kWarp; off <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, si, off);
      if (lane >= off) si += y;
    }
    wsum[lane] = si - s;
    if (lane == kWarp - 1) wsum[kWarp] = si;
  }
  __syncthreads();
  *total = wsum[kWarp];
  return wsum[w] + (incl - mine);
}

// Starts of keys [k0, k0 + kScanChunk) from their counts, `before` particles
// having smaller keys; the counts are left zero.  Returns the chunk's
// particles.  With sub-cells (mid) key 2c is cell c's start and 2c + 1 the
// start of its upper half.  (The count table is padded to whole chunks.)
__device__ __forceinline__ int scan_chunk(int *__restrict__ cnt, int shift, int nkeys, int k0, int before,
                                          int *__restrict__ start, int *__restrict__ mid, int *wsum) {
  const int k = k0 + 4 * threadIdx.x;
  int4 c = make_int4(0, 0, 0, 0);
  if (k >= nkeys) {
    // nothing to read
  } else if (shift == 0) {
    int4 *c4 = reinterpret_cast<int4 *>(cnt + k);
    c = *c4;
    *c4 = make_int4(0, 0, 0, 0);
  } else {
    int *c1 = cnt + ((size_t)k << shift);
    const int st = 1 << shift;
    c = make_int4(c1[0], c1[st], c1[2 * st], c1[3 * st]);
    c1[0] = c1[st] = c1[2 * st] = c1[3 * st] = 0;
  }
  int total;
  const int s0 = before + block_exclusive_scan(c.x + c.y + c.z + c.w, wsum, &total);
  const int s[4] = {s0, s0 + c.x, s0 + c.x + c.y, s0 + c.x + c.y + c.z};
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    if (k + u >= nkeys) continue;
    if (mid)
      ((k + u) & 1 ? mid : start)[(k + u) >> 1] = s[u];
    else
      start[k + u] = s[u];
  }
  return total;
}

// Many keys: each chunk's particles, then each chunk's starts.
__global__ void __launch_bounds__(kScanThreads) k_chunk_sums(const int *__restrict__ cnt, int *__restrict__ part,
                                                             const int *gate) {
  if (gate && *gate == 0) return;
  __shared__ int wsum[kWarp + 1];
  const int4 c = reinterpret_cast<const int4 *>(cnt)[(size_t)blockIdx.x * kScanThreads + threadIdx.x];
  int total;
  block_exclusive_scan(c.x + c.y + c.z + c.w, wsum, &total);
  if (threadIdx.x == 0) part[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads)
    k_scan_chunks(int *cnt, const int *__restrict__ part, int nkeys, int ncell, int n, int *start, int *mid,
                  const int *gate) {
  if (gate && *gate == 0) return;
  __shared__ int wsum[kWarp + 1];
  int mine = 0, before;
  for (int b = threadIdx.x; b < blockIdx.x; b += kScanThreads) mine += part[b];
  block_exclusive_scan(mine, wsum, &before);
  scan_chunk(cnt, 0, nkeys, blockIdx.x * kScanChunk, before, start, mid, wsum);
  if (blockIdx.x == 0 && threadIdx.x == 0) start[ncell] = n;
}

// First slot of key k's particles.
__device__ __forceinline__ int key_start(uint32_t k, const int *__restrict__ start, const int *__restrict__ mid) {
  return mid ? ((k & 1u) ? mid : start)[k >> 1] : start[k];
}
// One past the last slot of key k's particles.
__device__ __forceinline__ int key_end(uint32_t k, const int *__restrict__ start, const int *__restrict__ mid) {
  return mid && !(k & 1u) ? mid[k >> 1] : start[(mid ? k >> 1 : k) + 1];
}

__global__ void k_place(const uint32_t *__restrict__ keys, const int *__restrict__ arrival, int n, const int *start,
                        const int *mid, int *__restrict__ list, const int *gate) {
  if (gate && *gate == 0) return;
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d < n) list[key_start(keys[d], start, mid) + arrival[d]] = d;
}

// One CTA scans all keys.
__global__ void __launch_bounds__(kScanThreads)
    k_scan_cells(int *cnt, int shift, int nkeys, int ncell, int n, int *start, int *mid, const int *gate) {
  if (gate && *gate == 0) return;
  __shared__ int wsum[kWarp + 1];
  int before = 0;
  for (int k0 = 0; k0 < nkeys; k0 += kScanChunk)
    before += scan_chunk(cnt, shift, nkeys, k0, before, start, mid, wsum);
  if (threadIdx.x == 0) start[ncell] = n;
}

}  // namespace spc
