// Radix-partitioned joins: the C ABI of the partitioner, all-pairs equi-join and the
// semi-join count. Reference: sf100_radix_* and sf100_partition_join
// (kernels/microbenchmarks.metal:15-156), which the reference never launches.
//
// After both sides are partitioned with the same hash bits (radix.cuh), partition p of the
// build side can only match partition p of the probe side. One block per partition builds
// a shared-memory hash table from the build rows (chunks of at most kChunk rows, so any
// skew is handled by re-probing per chunk) and probes the partition's probe rows against
// it. Output positions come from warp-aggregated atomics on one global counter.
#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "engine.h"
#include "join_common.cuh"
#include "micro.h"
#include "radix.cuh"

namespace gpudb {
namespace {

constexpr int kPJThreads = 256;
constexpr uint32_t kPJCap = 4096;          // shared hash-table slots (32 KB)
constexpr uint32_t kChunk = kPJCap / 2;    // build rows per chunk: <= 50% load
constexpr uint64_t kRowsPerPartition = 2048;   // average build rows per partition: one chunk

__device__ __forceinline__ uint32_t pj_slot(int32_t key) { return key_slot(key, kPJCap - 1); }

__device__ __forceinline__ void pj_build(const int32_t* __restrict__ bk, const int32_t* __restrict__ brow, uint32_t c0,
                                         uint32_t c1, int32_t* hkey, int32_t* hrow) {
  for (uint32_t i = threadIdx.x; i < kPJCap; i += kPJThreads) hkey[i] = kEmptyKey;
  __syncthreads();
  for (uint32_t i = c0 + threadIdx.x; i < c1; i += kPJThreads) {
    const int32_t k = bk[i];
    uint32_t s = pj_slot(k);
    // duplicates take their own slots (multi-map); a chunk never fills the table
    for (uint32_t t = 0; t < kPJCap; t++, s = (s + 1) & (kPJCap - 1))
      if (atomicCAS(&hkey[s], kEmptyKey, k) == kEmptyKey) { if (hrow) hrow[s] = brow[i]; break; }
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kPJThreads) partition_pairs_kernel(
    const int32_t* __restrict__ bk, const int32_t* __restrict__ brow, const uint32_t* __restrict__ boff,
    const int32_t* __restrict__ pk, const int32_t* __restrict__ prow, const uint32_t* __restrict__ poff,
    int32_t* out_b, int32_t* out_p, uint64_t cap, unsigned long long* count) {
  __shared__ int32_t hkey[kPJCap], hrow[kPJCap];
  const uint32_t part = blockIdx.x;
  const uint32_t b0 = boff[part], b1 = boff[part + 1], p0 = poff[part], p1 = poff[part + 1];
  const int lane = threadIdx.x & 31;
  for (uint32_t c0 = b0; c0 < b1; c0 += kChunk) {
    pj_build(bk, brow, c0, min(c0 + kChunk, b1), hkey, hrow);
    // whole warps walk the probe rows so the warp-aggregated append is uniform
    for (uint32_t base = p0 + (threadIdx.x & ~31u); base < p1; base += kPJThreads) {
      const uint32_t i = base + lane;
      const bool valid = i < p1;
      const int32_t k = valid ? pk[i] : kEmptyKey;
      uint32_t m = 0;
      if (valid && k != kEmptyKey)
        for (uint32_t s = pj_slot(k), t = 0; t < kPJCap && hkey[s] != kEmptyKey; t++, s = (s + 1) & (kPJCap - 1))
          m += hkey[s] == k;
      uint32_t inc = m;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        uint32_t o = __shfl_up_sync(FULL_MASK, inc, d);
        if (lane >= d) inc += o;
      }
      const uint32_t total = __shfl_sync(FULL_MASK, inc, 31);
      unsigned long long start = 0;
      if (lane == 31 && total) start = atomicAdd(count, (unsigned long long)total);
      start = __shfl_sync(FULL_MASK, start, 31);
      unsigned long long pos = start + inc - m;
      if (m) {
        const int32_t r = prow[i];
        for (uint32_t s = pj_slot(k), t = 0; t < kPJCap && hkey[s] != kEmptyKey; t++, s = (s + 1) & (kPJCap - 1))
          if (hkey[s] == k) {
            if (pos < cap) { out_b[pos] = hrow[s]; out_p[pos] = r; }
            pos++;
          }
      }
    }
    __syncthreads();
  }
}

// Semi-join count: probe rows with at least one match. One block per partition, a shared table
// of the partition's build keys. key_hash32 is a bijection, so a key of the partition is named
// by the hash bits above the `pbits` partition bits: kPCLog of them pick one of the
// buckets and the rest (at most 15) are its tag, never 0 as stored. A bucket is four 16-bit
// tags in one 64-bit word: a probe is one 8-byte shared load and a compare of four tags,
// without a chain to walk (a linear-probing table of the keys ran a warp as long as the
// longest chain of its 32 probes: 237 us for 7.5M build and 60M probe keys against 167 us; two
// 512-thread blocks per SM with 2^13 buckets each need twice the partitions, which costs the
// scatter 100 us more). A key whose bucket
// is full (0.3% at one key a bucket) goes to the stash, a linear-probing set of full keys,
// which only probes of full buckets look at.
// A partition with more build rows than a chunk of kPCBuckets is joined chunk by chunk, its
// matches marked in `flags` (one byte per partitioned probe row) and counted after the last
// chunk; so is one whose keys overfill the stash (keys made to share buckets), in chunks that
// the stash alone can hold.
constexpr int kPCThreads = 1024;
constexpr int kPCLog = 14;
constexpr uint32_t kPCBuckets = 1u << kPCLog;
constexpr uint32_t kPCStash = 4096;
constexpr uint32_t kPCStashMax = kPCStash / 2;
constexpr int kPCMinBits = 32 - 15 - kPCLog;         // partition bits that leave a tag of at most 15
constexpr uint64_t kCountRowsPerPartition = 15360;   // average build keys per partition (<= kPCBuckets with margin)
constexpr int kPCRows = 16;                          // keys in flight per thread
constexpr size_t kPCSmem = kPCBuckets * 8 + kPCStash * 4;

// A zero 16-bit half in x.
__device__ __forceinline__ bool pc_zero_half(uint32_t x, uint32_t y) {
  return ((((x - 0x10001u) & ~x) | ((y - 0x10001u) & ~y)) & 0x80008000u) != 0u;
}

// f(key) for the keys [i0, i1) of a column, kPCRows of them loaded together per thread.
template <class F>
__device__ __forceinline__ void pc_each(const int32_t* __restrict__ col, uint32_t i0, uint32_t i1, F&& f) {
  uint32_t i = i0 + threadIdx.x;
  for (; i + (kPCRows - 1) * kPCThreads < i1; i += kPCRows * kPCThreads) {
    int32_t k[kPCRows];
#pragma unroll
    for (int u = 0; u < kPCRows; u++) k[u] = __ldcs(col + i + u * kPCThreads);
#pragma unroll
    for (int u = 0; u < kPCRows; u++) f(k[u], i + u * kPCThreads);
  }
  // the last strip, its loads together too
  int32_t k[kPCRows];
#pragma unroll
  for (int u = 0; u < kPCRows; u++) k[u] = i + u * kPCThreads < i1 ? __ldcs(col + i + u * kPCThreads) : kEmptyKey;
#pragma unroll
  for (int u = 0; u < kPCRows; u++)
    if (i + u * kPCThreads < i1) f(k[u], i + u * kPCThreads);
}

__global__ void __launch_bounds__(kPCThreads, 1) partition_count_kernel(
    const int32_t* __restrict__ bk, const uint32_t* __restrict__ boff, const int32_t* __restrict__ pk,
    const uint32_t* __restrict__ poff, int pbits, uint8_t* flags, unsigned long long* count) {
  extern __shared__ __align__(16) unsigned char pc_smem[];
  unsigned long long* bucket = reinterpret_cast<unsigned long long*>(pc_smem);
  int32_t* stash = reinterpret_cast<int32_t*>(bucket + kPCBuckets);
  __shared__ uint32_t stashed;
  const uint32_t part = blockIdx.x;
  const uint32_t b0 = boff[part], b1 = boff[part + 1], p0 = poff[part], p1 = poff[part + 1];
  uint32_t chunk = kPCBuckets;
  bool multi = (b1 - b0) > chunk;   // uniform, as every value a branch around a barrier tests
  uint32_t c = 0;
  if (p0 == p1) return;
  if (multi)
    for (uint32_t i = p0 + threadIdx.x; i < p1; i += kPCThreads) flags[i] = 0;
  for (uint32_t c0 = b0; c0 < b1;) {
    const uint32_t c1 = min(c0 + chunk, b1);
    __syncthreads();   // the previous chunk's probes are done
    for (uint32_t i = threadIdx.x; i < kPCBuckets / 2; i += kPCThreads)
      reinterpret_cast<ulonglong2*>(bucket)[i] = make_ulonglong2(0ull, 0ull);
    for (uint32_t i = threadIdx.x; i < kPCStash / 4; i += kPCThreads)
      reinterpret_cast<int4*>(stash)[i] = make_int4(kEmptyKey, kEmptyKey, kEmptyKey, kEmptyKey);
    if (threadIdx.x == 0) stashed = 0;
    __syncthreads();
    pc_each(bk, c0, c1, [&](int32_t k, uint32_t) {
      if (k == kEmptyKey) return;   // (an INT32_MIN key never matches)
      const uint32_t r = key_hash32(k) >> pbits;
      const uint32_t tag = (r >> kPCLog) + 1u, tt = tag * 0x10001u;
      unsigned long long* b = bucket + (r & (kPCBuckets - 1));
      unsigned long long w = *b;
      while (!pc_zero_half((uint32_t)w ^ tt, (uint32_t)(w >> 32) ^ tt)) {   // not there yet
        const int s = (79 - __clzll((long long)w)) & ~15;                   // places fill from the low end
        if (s < 64) {
          const unsigned long long prev = atomicCAS(b, w, w | ((unsigned long long)tag << s));
          if (prev == w) return;
          w = prev;
          continue;
        }
        bool counted = false;
        for (uint32_t x = key_slot(k, kPCStash - 1);; x = (x + 1) & (kPCStash - 1)) {
          int32_t e = stash[x];
          if (e == kEmptyKey) {
            if (!counted && atomicAdd(&stashed, 1u) >= kPCStashMax) return;   // (the chunk is redone below)
            counted = true;
            e = atomicCAS(&stash[x], kEmptyKey, k);
          }
          if (e == kEmptyKey || e == k) return;
        }
      }
    });
    __syncthreads();
    const uint32_t ns = stashed;
    if (ns > kPCStashMax) {   // the stash overflowed: smaller chunks from this one on
      if (!multi)
        for (uint32_t i = p0 + threadIdx.x; i < p1; i += kPCThreads) flags[i] = 0;
      multi = true;
      chunk = kPCStashMax;
      continue;
    }
    auto found = [&](int32_t k) {
      const uint32_t r = key_hash32(k) >> pbits;
      const uint32_t tt = ((r >> kPCLog) + 1u) * 0x10001u;
      const uint2 w = reinterpret_cast<const uint2*>(bucket)[r & (kPCBuckets - 1)];
      bool hit = pc_zero_half(w.x ^ tt, w.y ^ tt);   // (INT32_MIN is in no table, so it has no hit)
      if (!hit && w.y >= 0x10000u && ns) {   // a full bucket, and keys in the stash
        for (uint32_t z = key_slot(k, kPCStash - 1);; z = (z + 1) & (kPCStash - 1)) {
          const int32_t e = stash[z];
          if (e == kEmptyKey) break;
          if (e == k) { hit = true; break; }
        }
      }
      return hit;
    };
    if (multi) pc_each(pk, p0, p1, [&](int32_t k, uint32_t i) { if (found(k)) flags[i] = 1; });
    else pc_each(pk, p0, p1, [&](int32_t k, uint32_t) { c += found(k); });
    c0 = c1;
  }
  if (multi) {
    __syncthreads();
    for (uint32_t i = p0 + threadIdx.x; i < p1; i += kPCThreads) c += flags[i];
  }
  c = __reduce_add_sync(FULL_MASK, c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, (unsigned long long)c);
}

struct Sides {
  int32_t *bk, *brow, *pk, *prow;   // rows: null when only keys are partitioned
  uint32_t *boff, *poff;
};

// Partitions both sides with `bits` bits into scratch buffers: keys only, or keys with
// their row ids as payload.
int partition_both(Call& call, const int32_t* build, uint64_t nb, const int32_t* probe, uint64_t np, int bits,
                   bool rows, Sides* s) {
  gpudb_ctx* ctx = call.ctx();
  const uint64_t parts = 1ull << bits;
  const size_t nmax = std::max<uint64_t>(std::max(nb, np), 1);
  const int k = rows ? 2 : 1;
  void *keys, *offs;
  int rc = scratch(ctx, "rjoin.keys", (size_t)k * (nb + np + nmax + 3 * 48) * sizeof(int32_t), &keys);
  if (!rc) rc = scratch(ctx, "rjoin.offs", (2 * (parts + 1) + 64) * sizeof(uint32_t), &offs);
  if (rc) return rc;
  int32_t* p = static_cast<int32_t*>(keys);
  auto take = [&p](uint64_t n) { int32_t* q = p; p += (n + 16 + 31) / 32 * 32; return q; };   // 128-byte aligned
  s->bk = take(nb);
  s->pk = take(np);
  int32_t* ktmp = take(nmax);
  s->brow = rows ? take(nb) : nullptr;
  s->prow = rows ? take(np) : nullptr;
  int32_t* ptmp = rows ? take(nmax) : nullptr;
  s->boff = static_cast<uint32_t*>(offs);
  s->poff = s->boff + parts + 16;
  if (rows) {
    rc = radix_partition_run<int32_t, false>(call, build, nullptr, nb, nullptr, bits, s->bk, s->brow, s->boff, ktmp, ptmp);
    if (!rc) rc = radix_partition_run<int32_t, false>(call, probe, nullptr, np, nullptr, bits, s->pk, s->prow, s->poff, ktmp, ptmp);
  } else {
    rc = radix_partition_keys(call, build, nb, bits, s->bk, s->boff, ktmp);
    if (!rc) rc = radix_partition_keys(call, probe, np, bits, s->pk, s->poff, ktmp);
  }
  return rc;
}

}  // namespace

int radix_join_count(Call& call, const int32_t* build_keys, uint64_t n_build, const int32_t* probe_keys, uint64_t n_probe,
                     unsigned long long* count) {
  if (n_build == 0 || n_probe == 0) return GPUDB_OK;
  const int bits = std::max(kPCMinBits, radix_bits_for(n_build, kCountRowsPerPartition));
  Sides s;
  int rc = partition_both(call, build_keys, n_build, probe_keys, n_probe, bits, false, &s);
  if (rc) return rc;
  void* flags = nullptr;
  rc = scratch(call.ctx(), "rjoin.flags", n_probe + 16, &flags);
  if (rc) return rc;
  GPUDB_CUDA(call.ctx(), kernel_smem(call.ctx(), (const void*)partition_count_kernel, kPCSmem));
  GPUDB_LAUNCH(call, partition_count_kernel, 1u << bits, kPCThreads, kPCSmem, (const int32_t*)s.bk, (const uint32_t*)s.boff,
               (const int32_t*)s.pk, (const uint32_t*)s.poff, bits, (uint8_t*)flags, count);
  return GPUDB_OK;
}

}  // namespace gpudb

using namespace gpudb;

extern "C" int gpudb_radix_partition(gpudb_ctx* ctx, const int32_t* keys, const int32_t* payload, uint64_t n,
                                     int32_t bits, int32_t* keys_out, int32_t* payload_out, uint32_t* offsets,
                                     gpudb_timing* t, const gpudb_exec* ex) {
  if (!ctx) return GPUDB_E_INVALID;
  if (bits < 0 || bits > kRadixMaxBits) return fail(ctx, GPUDB_E_INVALID, "radix: bits must be in 0..%d", kRadixMaxBits);
  if (!offsets || !keys_out || !payload_out || (n && !keys)) return fail(ctx, GPUDB_E_INVALID, "radix: NULL buffer");
  if (n >= (1ull << 32)) return fail(ctx, GPUDB_E_INVALID, "radix: at most 2^32-1 rows");
  Call call(ctx, ex, t);
  int rc = call.begin(16);
  if (rc) return rc;
  void* tmp = nullptr;
  rc = scratch(ctx, "radix.tmp", (2 * std::max<uint64_t>(n, 1) + 96) * sizeof(int32_t), &tmp);
  if (rc) return rc;
  int32_t* ktmp = static_cast<int32_t*>(tmp);
  int32_t* ptmp = ktmp + (std::max<uint64_t>(n, 1) + 16 + 31) / 32 * 32;   // 128-byte aligned
  rc = radix_partition_run<int32_t, true>(call, keys, payload, n, nullptr, bits, keys_out, payload_out, offsets, ktmp, ptmp);
  if (rc) return rc;
  return call.finish(16, [](const uint8_t*) { return GPUDB_OK; });
}

extern "C" int gpudb_radix_join_pairs(gpudb_ctx* ctx, const int32_t* build_keys, uint64_t n_build,
                                      const int32_t* probe_keys, uint64_t n_probe, int32_t* out_build_rows,
                                      int32_t* out_probe_rows, uint64_t capacity, uint64_t* n_pairs, gpudb_timing* t,
                                      const gpudb_exec* ex) {
  if (!ctx) return GPUDB_E_INVALID;
  if (!n_pairs || (n_build && !build_keys) || (n_probe && !probe_keys) ||
      (capacity && (!out_build_rows || !out_probe_rows)))
    return fail(ctx, GPUDB_E_INVALID, "radix join: NULL buffer");
  if (n_build >= (1ull << 31) || n_probe >= (1ull << 31)) return fail(ctx, GPUDB_E_INVALID, "radix join: at most 2^31-1 rows a side");
  Call call(ctx, ex, t);
  int rc = call.begin(16);
  if (rc) return rc;
  if (n_build && n_probe) {
    const int bits = radix_bits_for(n_build, kRowsPerPartition);
    Sides s;
    rc = partition_both(call, build_keys, n_build, probe_keys, n_probe, bits, true, &s);
    if (rc) return rc;
    GPUDB_LAUNCH(call, partition_pairs_kernel, 1u << bits, kPJThreads, 0, (const int32_t*)s.bk, (const int32_t*)s.brow,
                 (const uint32_t*)s.boff, (const int32_t*)s.pk, (const int32_t*)s.prow, (const uint32_t*)s.poff,
                 out_build_rows, out_probe_rows, capacity, call.result<unsigned long long>());
  }
  return call.finish(16, [n_pairs](const uint8_t* h) {
    std::memcpy(n_pairs, h, 8);
    return GPUDB_OK;
  });
}
