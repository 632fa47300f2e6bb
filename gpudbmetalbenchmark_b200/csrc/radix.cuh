// Stable hash-radix partitioning of (key, payload) rows.
// Reference: sf100_radix_histogram / sf100_radix_prefix_sum / sf100_radix_scatter
// (kernels/microbenchmarks.metal:15-99): one 1024-way pass, threadgroup histograms,
// a single-threadgroup Blelloch scan, and an atomic-cursor scatter (unstable, one 4-byte
// write per row anywhere in memory).
//
// B200 design. Partition p = key_hash32(key) & (2^bits - 1) (the reference's hash), in LSD
// passes of at most kRxPassBits bits (one pass up to 1024 partitions). The input is cut into
// G super-tiles, as many as the scatter kernel's blocks that fit on the GPU at once, sized
// on the device from the row count; per pass:
//   rx_hist_kernel    counts each super-tile's rows per digit (shared-memory atomics, one block
//                     per super-tile) into hist[digit][G], and in the first of two passes also
//                     the rows per final partition;
//   rx_offsets_kernel turns hist into where each (digit, super-tile) run starts inside its
//                     digit, one warp per digit, and its last block the digits' starts;
//   rx_scatter_kernel one block per super-tile walks its sub-tiles in order: ranks the rows of
//                     a sub-tile by digit, stages them digit-sorted in shared memory and writes
//                     them out run by run from per-digit cursors that carry across the
//                     super-tile's sub-tiles.
// Stable: the order inside a partition is the input order, so later passes and the final
// result are deterministic.
#pragma once
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "engine.h"
#include "join_common.cuh"
#include "scan.cuh"

namespace gpudb {

constexpr int kRxThreads = 512;                         // histogram blocks
constexpr int kRxPassBits = 10;                         // fan-out of one pass <= 1024
constexpr uint32_t kRxMaxF = 1u << kRxPassBits;
constexpr int kRxFullSmemBits = 13;                     // final-partition counts in shared memory up to 8192

// Plain columns: keys, and a payload column or (null) the row number. Rows [0, n) with
// n = *n_dev when given (a count left on the device by an earlier kernel), capped at n_max.
template <class P>
struct ColumnSource {
  const int32_t* keys;
  const P* pay;
  uint64_t n_max;
  const uint32_t* n_dev;
  __device__ __forceinline__ uint64_t rows() const {
    return n_dev ? min((uint64_t)*n_dev, n_max) : n_max;
  }
  // both columns start on 16 bytes, so every whole sub-tile does (sub-tiles start at
  // multiples of their row count, a multiple of 4)
  __device__ __forceinline__ bool aligned16() const { return (((uintptr_t)keys | (uintptr_t)pay) & 15u) == 0; }
};

__device__ __forceinline__ void rx_load4(const int32_t* p, int32_t* o) {
  const int4 v = __ldcs(reinterpret_cast<const int4*>(p));
  o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
}
__device__ __forceinline__ void rx_load4(const int64_t* p, int64_t* o) {
  const longlong2 a = __ldcs(reinterpret_cast<const longlong2*>(p)), b = __ldcs(reinterpret_cast<const longlong2*>(p) + 1);
  o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
}

// Rows per super-tile for n rows over G super-tiles: whole sub-tiles of `tile` rows, at least
// one. Both kernels of a pass derive it from the same device row count, so a count that an
// earlier kernel left on the device (a filtered input) still spreads over all G blocks.
__host__ __device__ __forceinline__ uint64_t rx_super_rows_for(uint64_t n, uint32_t G, uint32_t tile) {
  const uint64_t per = (n + G - 1) / (G ? G : 1);
  const uint64_t s = (per + tile - 1) / tile * tile;
  return s < (uint64_t)tile ? (uint64_t)tile : s;
}

__device__ __forceinline__ uint32_t rx_digit(int32_t key, int shift, uint32_t mask) {
  return (key_hash32(key) >> shift) & mask;
}

// Inclusive scan of one value per thread across a block of NT threads.
template <int NT>
__device__ __forceinline__ uint32_t rx_block_scan(uint32_t v, uint32_t* warp_tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t o = __shfl_up_sync(FULL_MASK, v, d);
    if (lane >= d) v += o;
  }
  if (lane == 31) warp_tot[warp] = v;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < NT / 32 ? warp_tot[lane] : 0u;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t o = __shfl_up_sync(FULL_MASK, w, d);
      if (lane >= d) w += o;
    }
    if (lane < NT / 32) warp_tot[lane] = w;
  }
  __syncthreads();
  if (warp > 0) v += warp_tot[warp - 1];
  __syncthreads();
  return v;
}

// Digit counts of super-tile blockIdx.x into hist[digit * G + super-tile], and with `full` the
// rows per final partition (fbits bits; zeroed). A thread takes quads of consecutive rows (from
// the first 16-byte boundary on: a row per load and per atomic took 20M rows that start off it
// 282 us a call at 4 bits, against 172) and
// adds each run of equal digits inside a quad once: fact keys are clustered (the rows of one
// order are adjacent), and a warp's atomics on one address serialise.
template <class P>
__global__ void __launch_bounds__(kRxThreads) rx_hist_kernel(ColumnSource<P> src, uint32_t G, uint32_t tile, int shift,
                                                             int dbits, int fbits, uint32_t* __restrict__ hist,
                                                             uint32_t* __restrict__ full) {
  __shared__ uint32_t cnt[kRxMaxF];
  __shared__ uint32_t fcnt[1u << kRxFullSmemBits];
  const uint32_t F = 1u << dbits, dmask = F - 1, fmask = (1u << fbits) - 1;
  const bool fs = full && fbits <= kRxFullSmemBits;
  for (uint32_t i = threadIdx.x; i < F; i += kRxThreads) cnt[i] = 0;
  if (fs)
    for (uint32_t i = threadIdx.x; i <= fmask; i += kRxThreads) fcnt[i] = 0;
  __syncthreads();
  const uint64_t n = src.rows();
  const uint64_t super_rows = rx_super_rows_for(n, G, tile);
  const uint64_t r0 = (uint64_t)blockIdx.x * super_rows;
  const uint32_t rows = r0 < n ? (uint32_t)min(super_rows, n - r0) : 0u;
  if (F == 1) {   // one digit: the rows need no reading
    if (threadIdx.x == 0) hist[blockIdx.x] = rows;
    return;
  }
  const int32_t* keys = src.keys + r0;
  auto add = [&](int32_t k, uint32_t run) {
    const uint32_t h = key_hash32(k);
    atomicAdd(&cnt[(h >> shift) & dmask], run);
    if (fs) atomicAdd(&fcnt[h & fmask], run);
    else if (full) atomicAdd(&full[h & fmask], run);
  };
  auto quad = [&](const int4& k) {
    uint32_t run = 1;
    if (k.x == k.y) run++;
    else { add(k.x, run); run = 1; }
    if (k.y == k.z) run++;
    else { add(k.y, run); run = 1; }
    if (k.z == k.w) run++;
    else { add(k.z, run); run = 1; }
    add(k.w, run);
  };
  constexpr uint32_t U = 4;   // quads in flight per thread
  // the rows before the first 16-byte boundary, then quads, then the rest
  const uint32_t lead = min(rows, (uint32_t)(0u - ((uintptr_t)keys >> 2)) & 3u), quads = (rows - lead) / 4;
  const int4* keys4 = reinterpret_cast<const int4*>(keys + lead);
  if (threadIdx.x < lead) add(__ldg(keys + threadIdx.x), 1u);
  uint32_t q = threadIdx.x;
  for (; q + (U - 1) * kRxThreads < quads; q += U * kRxThreads) {
    int4 k[U];
#pragma unroll
    for (uint32_t u = 0; u < U; u++) k[u] = __ldg(keys4 + q + u * kRxThreads);   // cached: the scatter reads them again
#pragma unroll
    for (uint32_t u = 0; u < U; u++) quad(k[u]);
  }
  for (; q < quads; q += kRxThreads) quad(__ldg(keys4 + q));
  const uint32_t rest = lead + quads * 4 + threadIdx.x;
  if (rest < rows) add(__ldg(keys + rest), 1u);
  __syncthreads();
  for (uint32_t b = threadIdx.x; b < F; b += kRxThreads) hist[(size_t)b * G + blockIdx.x] = cnt[b];
  if (fs)
    for (uint32_t i = threadIdx.x; i <= fmask; i += kRxThreads)
      if (fcnt[i]) atomicAdd(&full[i], fcnt[i]);
}

// hist[digit][G] -> exclusive prefix over the super-tiles of each digit, in place (one warp per
// digit); the last block then scans the digits' totals: base[d] = first output row of digit d,
// offsets (null, or F + 1 words) the same with the total last. `ticket` is left at zero.
constexpr int kRxOffThreads = 256;
static __global__ void __launch_bounds__(kRxOffThreads) rx_offsets_kernel(uint32_t* __restrict__ hist, uint32_t F,
                                                                          uint32_t G, uint32_t* __restrict__ base,
                                                                          uint32_t* __restrict__ offsets,
                                                                          unsigned* ticket) {
  __shared__ uint32_t wt[kRxOffThreads / 32];
  const int lane = threadIdx.x & 31;
  const uint32_t d = blockIdx.x * (kRxOffThreads / 32) + (threadIdx.x >> 5);
  if (d < F) {
    uint32_t carry = 0;
    for (uint32_t g0 = 0; g0 < G; g0 += 32 * 4) {   // four loads in flight
      uint32_t c[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const uint32_t g = g0 + u * 32 + lane;
        c[u] = g < G ? hist[(size_t)d * G + g] : 0u;
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        uint32_t x = c[u];
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
          const uint32_t o = __shfl_up_sync(FULL_MASK, x, s);
          if (lane >= s) x += o;
        }
        const uint32_t g = g0 + u * 32 + lane;
        if (g < G) hist[(size_t)d * G + g] = carry + x - c[u];
        carry += __shfl_sync(FULL_MASK, x, 31);
      }
    }
    if (lane == 0) base[d] = carry;
  }
  if (!grid_last_block(ticket)) return;
  constexpr uint32_t kPer = kRxMaxF / kRxOffThreads;
  uint32_t c[kPer], sum = 0;
#pragma unroll
  for (uint32_t j = 0; j < kPer; j++) {
    const uint32_t b = threadIdx.x * kPer + j;
    c[j] = b < F ? __ldcg(base + b) : 0u;
    sum += c[j];
  }
  const uint32_t inc = rx_block_scan<kRxOffThreads>(sum, wt);
  uint32_t run = inc - sum;
#pragma unroll
  for (uint32_t j = 0; j < kPer; j++) {
    const uint32_t b = threadIdx.x * kPer + j;
    if (b < F) {
      base[b] = run;
      if (offsets) offsets[b] = run;
    }
    run += c[j];
  }
  if (offsets && threadIdx.x == kRxOffThreads - 1) offsets[F] = inc;
}

// Lanes of `live` whose digit (NB bits) equals this lane's: one vote per bit. (20M rows with a
// payload into 256 partitions, whole call: 197 us; 257 us with __match_any_sync, whose time
// grows with the distinct values in a warp; 197 us too with an atomicOr of lane masks into
// shared memory, which needs four times the counters.)
template <int NB>
__device__ __forceinline__ uint32_t rx_match(uint32_t d, uint32_t live) {
  uint32_t m = live;
#pragma unroll
  for (int b = 0; b < NB; b++) {
    const int32_t x = (int32_t)(d << (31 - b)) >> 31;   // all ones where the bit is set
    m &= ~(__ballot_sync(FULL_MASK, x < 0) ^ (uint32_t)x);
  }
  return m;
}

// Shared memory of one scatter block: the digit-sorted staging of one sub-tile, the digit
// counters (stable: per warp, u16; unstable: per block, u32) and per digit its output position
// less its place in the staging.
template <class P, bool PAY, int T, int I, bool STABLE>
__host__ __device__ constexpr size_t rx_scatter_smem(uint32_t F) {
  return (sizeof(int32_t) + (PAY ? sizeof(P) : 0)) * T * I +
         (STABLE ? sizeof(uint16_t) * (T / 32) * (F < 2 ? 2 : F) : sizeof(uint32_t) * F) + 2 * sizeof(uint32_t) * F;
}

// One block of T threads per super-tile (see the file comment), sub-tiles of T * I rows.
// offs, base: rx_offsets_kernel's. The next sub-tile's rows are loaded while this one is
// written out.
// Bound: instructions (48 a row of 32 keys) and the shared-memory pipe of the ranking and the
// staging, not DRAM. 20M rows with a payload, 8 bits: 268 us with input staged through a
// bulk-copy ring, match_any ranking and (key, output row) pairs in the staging, 136 us now; 60M
// clustered keys, 9 bits, unstable: 231 us before, 205 us now.
// STABLE ranks each warp's rows in row order, 32 at a time: the lanes of a digit found by
// votes, the warp's counter for it read by all of them and advanced by the last; a block scan
// over warps x digits turns the counts into staged positions. Otherwise a thread takes quads
// of consecutive rows and a row's rank inside its sub-tile is the arrival order of one
// shared-memory atomic per run of equal digits in a quad (clustered keys put four rows of one
// order side by side); super-tiles and sub-tiles still go out in input order, the rows of one
// sub-tile and digit in any order.
template <class P, bool PAY, int T, int I, bool STABLE, int NB>
__global__ void __launch_bounds__(T, T == 512 ? (PAY && I == 16 ? 1 : 2) : (I == 16 ? 3 : 4)) rx_scatter_kernel(
    ColumnSource<P> src, uint32_t G, int shift, int dbits, const uint32_t* __restrict__ offs,
    const uint32_t* __restrict__ base, int32_t* __restrict__ kout, P* __restrict__ pout) {
  constexpr int W = T / 32, TILE = T * I, WROWS = TILE / W;
  constexpr uint32_t kPer = (kRxMaxF + T - 1) / T;   // digits a thread scans, at most
  extern __shared__ __align__(16) unsigned char rx_smem[];
  __shared__ uint32_t wt[W];
  const uint32_t F = 1u << dbits, dmask = F - 1;
  P* spay = reinterpret_cast<P*>(rx_smem);
  int32_t* skey = reinterpret_cast<int32_t*>(spay + (PAY ? TILE : 0));
  uint32_t* delta = reinterpret_cast<uint32_t*>(skey + TILE);   // [digit] output row - staged position
  uint32_t* start = delta + F;                                  // [digit] its place in the staging
  uint32_t* cnt = start + F;                                    // unstable: [digit]
  uint16_t* wcnt = reinterpret_cast<uint16_t*>(start + F);      // stable: [warp][digit]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t n = src.rows();
  const uint64_t super_rows = rx_super_rows_for(n, G, TILE);
  const uint64_t g0 = (uint64_t)blockIdx.x * super_rows;
  if (g0 >= n) return;   // uniform across the block
  const uint64_t g1 = min(g0 + super_rows, n);
  const bool vec = src.aligned16();
  uint16_t* mine = wcnt + warp * F;
  // digits b0 .. b0 + dpt - 1 are this thread's in the scans; their next output rows
  const uint32_t dpt = (F + T - 1) / T, b0 = threadIdx.x * dpt;
  uint32_t cur[kPer];
#pragma unroll
  for (uint32_t u = 0; u < kPer; u++)
    cur[u] = u < dpt && b0 + u < F ? base[b0 + u] + offs[(size_t)(b0 + u) * G + blockIdx.x] : 0u;
  if (STABLE) {
    for (uint32_t i = lane; i < F; i += 32) mine[i] = 0;
    __syncwarp();
  } else {
    for (uint32_t i = threadIdx.x; i < F; i += T) cnt[i] = 0;
    __syncthreads();
  }
  int32_t key[I];
  P pay[I];
  // this thread's row j of the sub-tile
  auto row_of = [&](int j) {
    return STABLE ? (uint32_t)(warp * WROWS + j * 32 + lane) : (uint32_t)((j >> 2) * 4 * T + 4 * threadIdx.x + (j & 3));
  };
  auto load = [&](uint64_t t0) {
    const int32_t* kp = src.keys + t0;
    const P* pp = src.pay ? src.pay + t0 : nullptr;
    if (t0 + TILE > g1) {
      const uint32_t m = (uint32_t)(g1 - t0);
#pragma unroll
      for (int j = 0; j < I; j++)
        if (row_of(j) < m) {
          key[j] = __ldcs(kp + row_of(j));
          if (PAY) pay[j] = pp ? __ldcs(pp + row_of(j)) : (P)(t0 + row_of(j));
        }
    } else if (STABLE || !vec) {
#pragma unroll
      for (int j = 0; j < I; j++) key[j] = __ldcs(kp + row_of(j));
      if (PAY)
#pragma unroll
        for (int j = 0; j < I; j++) pay[j] = pp ? __ldcs(pp + row_of(j)) : (P)(t0 + row_of(j));
    } else {
#pragma unroll
      for (int j = 0; j < I; j += 4) {
        rx_load4(kp + row_of(j), key + j);
        if (PAY) {
          if (pp) rx_load4(pp + row_of(j), pay + j);
          else for (int u = 0; u < 4; u++) pay[j + u] = (P)(t0 + row_of(j + u));
        }
      }
    }
  };
  load(g0);
  // one sub-tile of m rows; FULL: m == TILE
  auto sub_tile = [&](auto full, uint64_t t0, uint32_t m) {
    constexpr bool FULL = decltype(full)::value;
    uint32_t dr[I];   // digit << 16 | rank (stable: among the warp's rows of that digit)
    if (STABLE) {
#pragma unroll
      for (int j = 0; j < I; j++) {
        const bool v = FULL || row_of(j) < m;
        const uint32_t d = rx_digit(key[j], shift, dmask);
        const uint32_t peers = rx_match<NB>(d, FULL ? FULL_MASK : __ballot_sync(FULL_MASK, v));
        const uint32_t first = v ? (uint32_t)mine[d] : 0u;
        dr[j] = (d << 16) | (first + __popc(peers & lanemask_lt()));
        __syncwarp();
        if (v && (peers & lanemask_gt()) == 0u) mine[d] = (uint16_t)(first + __popc(peers));
        __syncwarp();
      }
    } else {
#pragma unroll
      for (int q = 0; q < I; q += 4) {
        uint32_t d[4], len[4];
#pragma unroll
        for (int u = 0; u < 4; u++) d[u] = FULL || row_of(q + u) < m ? rx_digit(key[q + u], shift, dmask) : ~0u;
        len[3] = 1;
#pragma unroll
        for (int u = 2; u >= 0; u--) len[u] = d[u] == d[u + 1] ? len[u + 1] + 1 : 1u;
        uint32_t at = 0;
#pragma unroll
        for (int u = 0; u < 4; u++) {
          if (u > 0 && d[u] == d[u - 1]) at++;
          else if (FULL || d[u] != ~0u) at = atomicAdd(&cnt[d[u]], len[u]);
          dr[q + u] = (d[u] << 16) | at;
        }
      }
    }
    __syncthreads();
    // digit counts (stable: per warp) -> staged positions, digit-major, and the digits' deltas
    uint32_t c[kPer], sum = 0;
#pragma unroll
    for (uint32_t u = 0; u < kPer; u++) {
      c[u] = 0;
      if (u < dpt && b0 + u < F) {
        if (STABLE) {
#pragma unroll
          for (int w = 0; w < W; w++) {   // counts of earlier warps, in place
            const uint32_t x = wcnt[w * F + b0 + u];
            wcnt[w * F + b0 + u] = (uint16_t)c[u];
            c[u] += x;
          }
        } else {
          c[u] = cnt[b0 + u];
        }
      }
      sum += c[u];
    }
    uint32_t run = rx_block_scan<T>(sum, wt) - sum;
#pragma unroll
    for (uint32_t u = 0; u < kPer; u++)
      if (u < dpt && b0 + u < F) {
        delta[b0 + u] = cur[u] - run;
        start[b0 + u] = run;
        if (!STABLE) cnt[b0 + u] = 0;
        cur[u] += c[u];
        run += c[u];
      }
    __syncthreads();
    // stage digit-sorted
#pragma unroll
    for (int j = 0; j < I; j++)
      if (FULL || row_of(j) < m) {
        const uint32_t d = dr[j] >> 16;
        const uint32_t pos = start[d] + (dr[j] & 0xFFFFu) + (STABLE ? (uint32_t)mine[d] : 0u);
        skey[pos] = key[j];
        if (PAY) spay[pos] = pay[j];
      }
    if (STABLE) {   // the warp's counters are its own: cleared for the next sub-tile
      __syncwarp();
      for (uint32_t i = lane; i < F / 2; i += 32) reinterpret_cast<uint32_t*>(mine)[i] = 0;
      if (F == 1 && lane == 0) mine[0] = 0;
      __syncwarp();
    }
    if (t0 + TILE < g1) load(t0 + TILE);
    __syncthreads();
    // write out: consecutive threads take consecutive staged rows, i.e. consecutive output
    // rows inside each digit's run
#pragma unroll
    for (int j = 0; j < I; j++) {
      const uint32_t i = threadIdx.x + (uint32_t)j * T;
      if (FULL || i < m) {
        const int32_t k = skey[i];
        const uint32_t o = delta[rx_digit(k, shift, dmask)] + i;
        kout[o] = k;
        if (PAY) pout[o] = spay[i];
      }
    }
  };
  uint64_t t0 = g0;
  for (; t0 + TILE <= g1; t0 += TILE) sub_tile(std::true_type{}, t0, (uint32_t)TILE);
  if (t0 < g1) sub_tile(std::false_type{}, t0, (uint32_t)(g1 - t0));
}

// Partitions the rows of `src` (at most n_max) into 2^bits partitions: keys (and payloads
// when PAY) to kout/pout, partition starts to offsets[0 .. 2^bits] (the total last). Two
// passes when bits > kRxPassBits, through ktmp/ptmp (n_max rows each). The scatter kernel
// runs with T threads and I rows per thread; there are as many super-tiles as its blocks fit
// on the GPU at once (fewer for a small input).
template <class P, bool PAY, int T, int I, bool STABLE>
int rx_partition_shaped(Call& call, const ColumnSource<P>& src, uint64_t n_max, int bits, int32_t* kout, P* pout,
                        uint32_t* offsets, int32_t* ktmp, P* ptmp) {
  constexpr uint32_t TILE = T * I;
  gpudb_ctx* ctx = call.ctx();
  cudaStream_t s = call.stream();
  const int passes = bits <= kRxPassBits ? 1 : 2;
  const int d0 = passes == 1 ? bits : (bits + 1) / 2, d1 = bits - d0;
  auto kernel_for = [](int dbits, bool stable) {
    return !stable    ? rx_scatter_kernel<P, PAY, T, I, false, 0>
           : dbits <= 6 ? rx_scatter_kernel<P, PAY, T, I, true, 6>
           : dbits <= 8 ? rx_scatter_kernel<P, PAY, T, I, true, 8>
                        : rx_scatter_kernel<P, PAY, T, I, true, kRxPassBits>;
  };
  // the second pass is always stable: it must keep the first pass's order inside each of its
  // digits, or the rows of one final partition would not be contiguous
  auto k0 = kernel_for(d0, STABLE), k1 = kernel_for(d1, true);
  const size_t smem0 = rx_scatter_smem<P, PAY, T, I, STABLE>(1u << d0);
  const size_t smem1 = rx_scatter_smem<P, PAY, T, I, true>(1u << d1);
  GPUDB_CUDA(ctx, kernel_smem(ctx, (const void*)k0, smem0));
  if (passes > 1) GPUDB_CUDA(ctx, kernel_smem(ctx, (const void*)k1, smem1));
  const int per_sm = kernel_occupancy(ctx, (const void*)k0, T, smem0);
  const uint64_t sub = (std::max<uint64_t>(n_max, 1) + TILE - 1) / TILE;
  const uint32_t G = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(sub, (uint64_t)ctx->sm_count * std::max(per_sm, 1)));
  const size_t hn = (size_t)G << std::max(d0, d1), parts = (size_t)1 << bits;
  // ticket (left at zero), digit starts, hist[digit][G], the final partitions' counts, scan scratch
  constexpr size_t kHead = 64;
  void* sc = nullptr;
  int rc = scratch(ctx, "radix.meta", (kHead + kRxMaxF + hn + parts + scan_tiles_count(parts) + 8) * sizeof(uint32_t), &sc);
  if (rc) return rc;
  unsigned* ticket = static_cast<unsigned*>(sc);
  uint32_t* base = static_cast<uint32_t*>(sc) + kHead;
  uint32_t* hist = base + kRxMaxF;
  uint32_t* full = passes > 1 ? hist + hn : nullptr;
  if (full) GPUDB_CUDA(ctx, cudaMemsetAsync(full, 0, parts * sizeof(uint32_t), s));
  for (int pass = 0; pass < passes; pass++) {
    const int shift = pass == 0 ? 0 : d0, dbits = pass == 0 ? d0 : d1;
    const uint32_t F = 1u << dbits;
    const bool last = pass == passes - 1;
    const ColumnSource<P> in = pass == 0 ? src : ColumnSource<P>{ktmp, PAY ? ptmp : nullptr, src.n_max, src.n_dev};
    GPUDB_LAUNCH(call, (rx_hist_kernel<P>), G, kRxThreads, 0, in, G, TILE, shift, dbits, bits, hist,
                 pass == 0 ? full : (uint32_t*)nullptr);
    GPUDB_LAUNCH(call, rx_offsets_kernel, (F + kRxOffThreads / 32 - 1) / (kRxOffThreads / 32), kRxOffThreads, 0, hist, F,
                 G, base, passes == 1 ? offsets : (uint32_t*)nullptr, ticket);
    GPUDB_LAUNCH(call, (pass == 0 ? k0 : k1), G, T, (pass == 0 ? smem0 : smem1), in, G, shift, dbits,
                 (const uint32_t*)hist, (const uint32_t*)base, last ? kout : ktmp, last ? pout : ptmp);
  }
  if (passes == 1) return GPUDB_OK;
  return exclusive_scan<uint32_t, uint32_t>(call, full, parts, offsets, full + parts, offsets + parts);
}

// The scatter block shape (GPUDB_OPT_RADIX_SHAPE): 0 (default), 1, 5 and 6 512 threads x 16
// rows, 3 512 x 8, 7 256 x 16, 2 and 4 256 x 8. The default is the fastest at many partitions,
// where larger sub-tiles have longer runs per digit (60M keys of the join count: 600 us against
// 638, 670 and 740), and within 15% of the best elsewhere; a caller whose partitionings are of one
// kind may choose. 20M random keys with a payload, us a call for 512 x 16, 512 x 8, 256 x 16,
// 256 x 8: 4 bits 171, 158, 149, 159; 8 bits 194, 187, 217, 272; 10 bits 281, 373, 505, 666; 13
// bits 353, 337, 337, 355; 100K keys, 10 bits 45, 37, 37, 34. STABLE: rows keep their input order
// inside a partition.
template <class P, bool PAY, bool STABLE>
int rx_partition(Call& call, const ColumnSource<P>& src, uint64_t n_max, int bits, int32_t* kout, P* pout,
                 uint32_t* offsets, int32_t* ktmp, P* ptmp) {
  switch (call.ctx()->radix_shape) {
    case 3:
      return rx_partition_shaped<P, PAY, 512, 8, STABLE>(call, src, n_max, bits, kout, pout, offsets, ktmp, ptmp);
    case 7:
      return rx_partition_shaped<P, PAY, 256, 16, STABLE>(call, src, n_max, bits, kout, pout, offsets, ktmp, ptmp);
    case 2: case 4:
      return rx_partition_shaped<P, PAY, 256, 8, STABLE>(call, src, n_max, bits, kout, pout, offsets, ktmp, ptmp);
    default:
      return rx_partition_shaped<P, PAY, 512, 16, STABLE>(call, src, n_max, bits, kout, pout, offsets, ktmp, ptmp);
  }
}

// Plain columns (payload = row id when pay is null); the row count may be on the device.
// STABLE (the C ABI's partitioning) keeps the input order inside each partition; the joins,
// whose results do not depend on it, take the unstable form (for the first pass; a second
// pass is always stable).
template <class P, bool STABLE>
int radix_partition_run(Call& call, const int32_t* keys, const P* pay, uint64_t n_max, const uint32_t* n_dev, int bits,
                        int32_t* keys_out, P* pay_out, uint32_t* offsets, int32_t* keys_tmp, P* pay_tmp) {
  const ColumnSource<P> src{keys, pay, n_max, n_dev};
  return rx_partition<P, true, STABLE>(call, src, n_max, bits, keys_out, pay_out, offsets, keys_tmp, pay_tmp);
}

// Keys only (no payload column is read or written), unstable.
inline int radix_partition_keys(Call& call, const int32_t* keys, uint64_t n, int bits, int32_t* keys_out,
                                uint32_t* offsets, int32_t* keys_tmp) {
  const ColumnSource<int32_t> src{keys, nullptr, n, nullptr};
  return rx_partition<int32_t, false, false>(call, src, n, bits, keys_out, nullptr, offsets, keys_tmp, nullptr);
}

// Partition bits so that the average partition holds about `per_part` rows.
inline int radix_bits_for(uint64_t n, uint64_t per_part) {
  int b = 0;
  while (b < kRadixMaxBits && (n >> b) > per_part) b++;
  return b;
}

}  // namespace gpudb
