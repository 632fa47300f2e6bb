// Q13 (customer distribution): orders whose comment is NOT LIKE '%word1%word2%' are counted
// per customer, then customers are counted per order count (custdist), ordered by custdist
// desc, c_count desc.
// Reference: kernels/q13.metal:33-168 (pattern match into a qualifies byte, per-customer
// counts with device atomics, threadgroup-privatised histogram), src/q13.cpp:8-117 (driver),
// postProcessQ13 src/infra.h:778-800 (sort of the histogram).
//
// B200 design:
//  - q13_count_kernel: a warp takes 32 orders at a time, their 80-byte comment slots brought
//    to shared memory by bulk copies; each order is tested for a possible word1 (32-bit
//    compares), and only the orders that may hold it are queued and matched in full, 32 at a
//    time. Qualifying orders add 1 to their customer's count (L2-resident counter array, one
//    atomic per order).
//  - q13_hist_kernel: every customer row looks up its count and adds to a shared-memory
//    histogram of GPUDB_Q13_MAX_COUNT + 1 bins, flushed with one atomic per nonzero bin.
//  - q13_sort_kernel: one block ranks the nonzero bins (custdist desc, c_count desc).
#include <cstring>

#include "common.cuh"
#include "engine.h"
#include "join_common.cuh"
#include "tma.cuh"

namespace gpudb {
namespace {

constexpr int kQ13Threads = 256;
constexpr int kSlotWords = GPUDB_COMMENT_WIDTH / 4;   // 20
constexpr int kBins = GPUDB_Q13_MAX_COUNT + 1;

// The two words of the LIKE pattern, as bytes and as the 32-bit words the candidate tests use:
// LONG form (both words of kLongWord letters or more) p[j] = bytes j..j+3 of the word, else
// p[0] = its first min(4, length) bytes and `mask` which of them count. poly: the coefficients
// of (x - p[0])(x - p[1])(x - p[2])(x - p[3]) mod 2^32 (the LONG test of half the row words).
struct Q13Pattern {
  uint8_t w[2][16];   // NUL-padded
  int32_t len[2];
  uint32_t p[2][4];
  uint32_t mask[2];
  uint32_t poly[4];   // of word 0: x^4 + poly[3] x^3 + ... + poly[0]
};
constexpr int kLongWord = 7;

// Whether the word (its bytes at w) stands at byte `pos` of the row. vec: the row is 4-byte
// aligned and compared four letters at a time.
__device__ __forceinline__ bool word_at(const uint8_t* row, bool vec, int pos, const uint8_t* w, int len) {
  if (pos < 0 || pos + len > GPUDB_COMMENT_WIDTH) return false;
  if (vec) {
    const uint32_t* rw = reinterpret_cast<const uint32_t*>(row);
    const uint32_t* pw = reinterpret_cast<const uint32_t*>(w);
    const int k = pos >> 2;
    uint32_t x = __ldg(rw + k);
    for (int c = 0; c < len; c += 4) {
      const int i = k + (c >> 2) + 1;
      const uint32_t nx = i < kSlotWords ? __ldg(rw + i) : 0u;
      const uint32_t y = __funnelshift_r(x, nx, 8 * (pos & 3)) ^ pw[c >> 2];
      if (len - c >= 4 ? y : y << (8 * (4 - (len - c)))) return false;
      x = nx;
    }
    return true;
  }
  for (int c = 0; c < len; c++)
    if (row[pos + c] != w[c]) return false;
  return true;
}

// How the orders are tested, from the words' lengths:
//  kLong    both words of kLongWord letters or more (see candidates): queue the orders that may hold w0;
//  kBytes   w0 of three letters or more: the same with a compare at every byte;
//  kDirect  w0 of one or two letters, which most comments hold: a queue of nearly every order costs
//           more than it saves, so every order is matched at once (like2_short). 15M orders, whole
//           call: "s", "s" 332 us, queued 750; "ar", "ar" 517 us, queued 482 (few orders hold it);
//           "s ", " s" 504 us, queued 698.
enum Q13Form { kLong, kBytes, kDirect };

// High bit of every byte of x that is zero (exact per byte).
__device__ __forceinline__ uint32_t zero_bytes(uint32_t x) {
  const uint32_t y = (x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu;
  return ~(y | x | 0x7F7F7F7Fu);
}

// The positions of a row whose first two bytes (one letter: first byte) are those of word `w`:
// SWAR on the row word and the row word shifted by one byte. The flags of word k (bits 7, 15, 23,
// 31) land on bits (k & 7) + {0, 8, 16, 24} of c[k >> 3].
__device__ __forceinline__ void pair_flags(const uint32_t (&rw)[kSlotWords], const Q13Pattern& pat, int w, uint32_t (&c)[3]) {
  const uint32_t a = pat.w[w][0] * 0x01010101u, b = pat.w[w][1] * 0x01010101u;
  c[0] = c[1] = c[2] = 0;
  auto mark = [&](int k, uint32_t m) { c[k >> 3] |= (m >> (7 - (k & 7))) & (0x01010101u << (k & 7)); };
  if (pat.len[w] == 1) {
#pragma unroll
    for (int k = 0; k < kSlotWords; k++) mark(k, zero_bytes(rw[k] ^ a));
  } else {
#pragma unroll
    for (int k = 0; k < kSlotWords; k++) {
      const uint32_t x = rw[k], nx = k + 1 < kSlotWords ? rw[k + 1] : 0u;
      mark(k, zero_bytes(x ^ a) & zero_bytes(__funnelshift_r(x, nx, 8) ^ b));
    }
  }
}

// LIKE '%w0%w1%' on a row per lane, w0 of at most two letters, so that its flags are all of it and
// the first one decides; the positions of a longer w1 behind it are compared in full. Every lane
// of the warp calls it; w1 is not looked for when none of them has a w0.
__device__ __forceinline__ bool like2_short(const uint32_t (&rw)[kSlotWords], const uint8_t* row, bool vec, bool known,
                                            const Q13Pattern& pat, const uint8_t (&w)[2][16]) {
  uint32_t c0[3], c1[3];
  pair_flags(rw, pat, 0, c0);
  const int q = c0[0] ? 0 : c0[1] ? 1 : 2;
  const uint32_t c = q == 0 ? c0[0] : q == 1 ? c0[1] : c0[2];
  if (!__any_sync(FULL_MASK, known && c)) return false;
  pair_flags(rw, pat, 1, c1);
  if (!known || !c) return false;
  const int j = __ffs((c | c >> 8 | c >> 16 | c >> 24) & 0xFFu) - 1;   // the first word with a w0
  const int l1 = pat.len[1], start = 4 * (8 * q + j) + ((__ffs((c >> j) & 0x01010101u) - 1) >> 3) + pat.len[0];
#pragma unroll
  for (int q1 = 2; q1 >= 0; q1--) {
    uint32_t m = c1[q1];
    while (m) {
      const int b = __ffs(m) - 1;
      m &= m - 1;
      const int pos = 4 * (8 * q1 + (b & 7)) + (b >> 3);
      if (pos >= start && (l1 <= 2 || word_at(row, vec, pos, w[1], l1))) return true;
    }
  }
  return false;
}

// Calls f(hit, position) for the places where a word may start; every place where it does
// start has a hit. LONG: a word of 7 letters or more covers a whole aligned 32-bit word of the
// row wherever it starts, so each row word is compared with the four words that can stand
// there (80 compares a row, no shifts). Else the first four letters are compared at every byte.
template <bool LONG, class F>
__device__ __forceinline__ void candidates(const uint32_t (&rw)[kSlotWords], const uint32_t (&p)[4], uint32_t mask, F&& f) {
#pragma unroll
  for (int k = 0; k < kSlotWords; k++) {
    const uint32_t x = rw[k];
    if (LONG) {
#pragma unroll
      for (int j = 0; j < 4; j++) f(x == p[j], 4 * k - j);
    } else {
      const uint32_t nx = k + 1 < kSlotWords ? rw[k + 1] : 0u;
#pragma unroll
      for (int j = 0; j < 4; j++) f(((__funnelshift_r(x, nx, 8 * j) ^ p[0]) & mask) == 0u, 4 * k + j);
    }
  }
}

// Whether the row may hold word 0. The LONG compares run on the half-rate integer pipe and
// bind the kernel, so every other row word takes the polynomial instead, whose four multiplies
// run on the multiply pipe: it is 0 where the word equals one of the four, and for the few other
// words whose differences from the four multiply to 0 mod 2^32, which the full match turns away
// (more of them for a w0 that repeats letters: "aaaaaaa" 293 us a call, "special" 290).
template <bool LONG>
__device__ __forceinline__ bool may_hold(const uint32_t (&rw)[kSlotWords], const Q13Pattern& pat) {
  bool any = false;
  if (LONG) {
#pragma unroll
    for (int k = 0; k < kSlotWords; k++) {
      const uint32_t x = rw[k];
      if (k & 1)
        any |= (((x + pat.poly[3]) * x + pat.poly[2]) * x + pat.poly[1]) * x + pat.poly[0] == 0u;
      else
        any |= (x == pat.p[0][0]) | (x == pat.p[0][1]) | (x == pat.p[0][2]) | (x == pat.p[0][3]);
    }
  } else {
    candidates<LONG>(rw, pat.p[0], pat.mask[0], [&](bool hit, int) { any |= hit; });
  }
  return any;
}

// LIKE '%w0%w1%' on one row (its words in registers, its bytes at `row`): w1 has to start at
// or after the end of the first w0. The first candidate of w0 and the last of w1 decide when
// they verify, as they nearly always do; otherwise every position is compared.
template <bool LONG>
__device__ __forceinline__ bool like2(const uint32_t (&rw)[kSlotWords], const uint8_t* row, bool vec,
                                      const Q13Pattern& pat, const uint8_t (&w)[2][16]) {
  constexpr int kNone = 1 << 20;
  int first = kNone, last = -kNone;
  candidates<LONG>(rw, pat.p[0], pat.mask[0], [&](bool hit, int at) { if (hit) first = min(first, at); });
  if (first == kNone) return false;
  candidates<LONG>(rw, pat.p[1], pat.mask[1], [&](bool hit, int at) { if (hit) last = max(last, at); });
  const int l0 = pat.len[0], l1 = pat.len[1];
  if (last < first + l0) return false;   // no w1 starts after any w0
  bool found = word_at(row, vec, first, w[0], l0);
  if (!found) {
    for (first++; first <= GPUDB_COMMENT_WIDTH - l0 && !found; first++) found = word_at(row, vec, first, w[0], l0);
    if (!found) return false;
    first--;
  }
  if (last < first + l0) return false;
  if (word_at(row, vec, last, w[1], l1)) return true;
  for (int pos = first + l0; pos <= GPUDB_COMMENT_WIDTH - l1; pos++)
    if (word_at(row, vec, pos, w[1], l1)) return true;
  return false;
}

__device__ __forceinline__ void load_smem_slot(const unsigned char* slot, uint32_t (&rw)[kSlotWords]) {
#pragma unroll
  for (int q = 0; q < kSlotWords / 4; q++) {
    const uint4 v = reinterpret_cast<const uint4*>(slot)[q];
    rw[4 * q] = v.x; rw[4 * q + 1] = v.y; rw[4 * q + 2] = v.z; rw[4 * q + 3] = v.w;
  }
}

__device__ __forceinline__ void load_slot(const uint8_t* row, bool vec, uint32_t (&rw)[kSlotWords]) {
  if (vec) {
#pragma unroll
    for (int q = 0; q < kSlotWords / 4; q++) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(row) + q);
      rw[4 * q] = v.x; rw[4 * q + 1] = v.y; rw[4 * q + 2] = v.z; rw[4 * q + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < kSlotWords; k++)
      rw[k] = row[4 * k] | (uint32_t)row[4 * k + 1] << 8 | (uint32_t)row[4 * k + 2] << 16 | (uint32_t)row[4 * k + 3] << 24;
  }
}

// Warps are independent: each takes 32 orders at a time, whose comments (2560 contiguous bytes)
// and customer keys arrive by two bulk copies on the warp's own mbarrier, kQ13Stages tiles
// deep, so DRAM sees whole lines and no load waits in a register; a lane's slot is read back
// with five 16-byte loads at an 80-byte stride, which no two lanes of a phase conflict on.
// Per order only the test "may hold w0" runs; the orders that may (one in five with the
// generator's vocabulary) go to a warp queue and are matched 32 at a time with full lanes
// (rows re-read from L2), which keeps the rare work off the common path.
// 84 B per order bound it from below (193 us for 15M orders at the copy peak); above that the
// integer pipe does (half rate, about 65% busy). Whole call, 15M orders on one B200: 647 us with
// a SWAR test of every position of both words per order and 80-byte strided loads, 322 us with
// the tiles, compares and queue, 300 us with half of the compares as polynomials and four-letter
// verification; three stages a warp (fewer warps per SM) took 345 us.
constexpr int kQ13Warps = kQ13Threads / 32;
constexpr int kQ13Stages = 2;   // (the early exit waits for one other stage)
constexpr uint32_t kQ13StageBytes = 32 * (GPUDB_COMMENT_WIDTH + 4);

struct Q13Smem {
  unsigned char stage[kQ13Warps][kQ13Stages][kQ13StageBytes];   // 32 slots, then 32 customer keys
  uint2 queue[kQ13Warps][64];                                   // {the warp's step * 32 + lane, customer}
  uint64_t full[kQ13Warps][kQ13Stages];
  __align__(4) uint8_t w[2][16];
};

template <Q13Form FORM>
__global__ void __launch_bounds__(kQ13Threads, FORM != kBytes ? 4 : 3) q13_count_kernel(const char* __restrict__ comment,
                                                                    const int32_t* __restrict__ ocust, uint64_t n,
                                                                    int32_t cust_max,
                                                                    const __grid_constant__ Q13Pattern pat,
                                                                    uint32_t* counts,
                                                                    uint32_t* status) {
  extern __shared__ __align__(128) unsigned char q13_smem[];
  Q13Smem& S = *reinterpret_cast<Q13Smem*>(q13_smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < 32) S.w[threadIdx.x >> 4][threadIdx.x & 15] = pat.w[threadIdx.x >> 4][threadIdx.x & 15];
  if (lane == 0) {
    for (int q = 0; q < kQ13Stages; q++) mbar_init(&S.full[warp][q], 1);
    mbar_fence_init();
  }
  __syncthreads();
  const bool vec = (reinterpret_cast<uintptr_t>(comment) & 15u) == 0;
  const uint64_t whole = vec && (reinterpret_cast<uintptr_t>(ocust) & 15u) == 0 ? n / 32 : 0;   // tiles by bulk copy
  const uint64_t tiles = (n + 31) / 32, W = (uint64_t)gridDim.x * kQ13Warps;
  const uint64_t t0 = (uint64_t)blockIdx.x * kQ13Warps + warp;
  const uint8_t* text = reinterpret_cast<const uint8_t*>(comment);
  uint2* queue = S.queue[warp];
  auto issue = [&](uint64_t t, int q) {   // one lane
    unsigned char* st = S.stage[warp][q];
    mbar_arrive_expect_tx(&S.full[warp][q], kQ13StageBytes);
    bulk_copy_g2s(st, text + t * 32 * GPUDB_COMMENT_WIDTH, 32 * GPUDB_COMMENT_WIDTH, &S.full[warp][q]);
    bulk_copy_g2s(st + 32 * GPUDB_COMMENT_WIDTH, ocust + t * 32, 32 * 4, &S.full[warp][q]);
  };
  if (lane == 0)
    for (int q = 0; q < kQ13Stages; q++)
      if (t0 + q * W < whole) issue(t0 + q * W, q);
  uint32_t queued = 0, parity = 0;
  int q = 0;
  // The queue names an order by the warp's step and the lane: 32 bits of it last for any row
  // count, 32 bits of the row would not.
  uint32_t step = 0;
  for (uint64_t t = t0;; t += W, step++) {
    const bool more = t < tiles;
    if (more) {
      const uint64_t r = t * 32 + lane;
      const bool in = r < n;
      uint32_t rw[kSlotWords] = {};
      int32_t c = -1;
      if (t < whole) {
        if (!__all_sync(FULL_MASK, mbar_wait(&S.full[warp][q], parity, kMbarPollLimit))) {
          // gave up: report it, and leave once the copies still in flight have landed
          set_status(status, ST_TIMEOUT);
          if (t + W < whole)
            mbar_wait(&S.full[warp][(q + 1) % kQ13Stages], q + 1 == kQ13Stages ? parity ^ 1u : parity, kMbarPollLimit);
          return;
        }
        const unsigned char* st = S.stage[warp][q];
        load_smem_slot(st + lane * GPUDB_COMMENT_WIDTH, rw);
        c = reinterpret_cast<const int32_t*>(st + 32 * GPUDB_COMMENT_WIDTH)[lane];
        // every lane has its slot: refill the stage. The proxy fence is needed: without it the
        // loads above may still be outstanding (ptxas sinks them to their use) when the copy lands.
        fence_proxy_async();
        __syncwarp();
        if (lane == 0 && t + kQ13Stages * W < whole) issue(t + kQ13Stages * W, q);
        if (++q == kQ13Stages) { q = 0; parity ^= 1u; }
      } else if (in) {
        c = ld_stream(ocust + r);
        load_slot(text + r * GPUDB_COMMENT_WIDTH, vec, rw);
      }
      const bool known = in && c >= 0 && c <= cust_max;   // an order of no known customer counts for nobody
      if (FORM == kDirect) {
        if (!like2_short(rw, text + r * GPUDB_COMMENT_WIDTH, vec, known, pat, S.w) && known) atomicAdd(counts + c, 1u);
        __syncwarp();
        continue;
      }
      const bool maybe = known && may_hold<FORM == kLong>(rw, pat);
      if (known && !maybe) atomicAdd(counts + c, 1u);
      const uint32_t m = __ballot_sync(FULL_MASK, maybe);
      if (maybe) queue[queued + __popc(m & lanemask_lt())] = make_uint2(step * 32 + lane, (uint32_t)c);
      queued += __popc(m);
      __syncwarp();
    }
    if (queued >= 32 || !more) {   // match 32 queued orders (after the last tile, those left)
      const uint32_t take = min(queued, 32u);
      queued -= take;
      if ((uint32_t)lane < take) {
        const uint2 e = queue[queued + lane];
        const uint64_t r = (t0 + (uint64_t)(e.x >> 5) * W) * 32 + (e.x & 31u);
        const uint8_t* row = text + r * GPUDB_COMMENT_WIDTH;
        uint32_t rw[kSlotWords];
        load_slot(row, vec, rw);
        if (!like2<FORM == kLong>(rw, row, vec, pat, S.w)) atomicAdd(counts + e.y, 1u);
      }
      __syncwarp();
    }
    if (!more) break;
  }
}

__global__ void __launch_bounds__(256) q13_hist_kernel(const int32_t* __restrict__ ckey, uint64_t n, int32_t cust_max,
                                                       const uint32_t* __restrict__ counts, uint32_t* hist,
                                                       uint32_t* status) {
  __shared__ uint32_t sh[kBins];
  for (int i = threadIdx.x; i < kBins; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const int32_t k = ld_stream(ckey + i);
    if (k < 0 || k > cust_max) { set_status(status, ST_KEY_RANGE); continue; }
    const uint32_t c = counts[k];
    if (c >= (uint32_t)kBins) { set_status(status, ST_CAPACITY); continue; }
    atomicAdd(&sh[c], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kBins; i += blockDim.x)
    if (sh[i]) atomicAdd(hist + i, sh[i]);
}

// out = {u32 n, pad[3], rows[n] of (c_count, custdist)} ordered by custdist desc, c_count desc.
__global__ void __launch_bounds__(kBins) q13_sort_kernel(const uint32_t* __restrict__ hist, uint8_t* out) {
  __shared__ uint32_t h[kBins];
  const uint32_t b = threadIdx.x;
  h[b] = hist[b];
  const uint32_t cd = h[b];
  const int n = __syncthreads_count(cd != 0);
  if (cd) {
    uint32_t r = 0;
    for (uint32_t j = 0; j < (uint32_t)kBins; j++) {
      const uint32_t o = h[j];
      r += (o > cd) | ((o == cd) & (j > b));
    }
    reinterpret_cast<uint2*>(out + 16)[r] = make_uint2(b, cd);
  }
  if (b == 0) *reinterpret_cast<uint32_t*>(out) = (uint32_t)n;
}

}  // namespace
}  // namespace gpudb

using namespace gpudb;

extern "C" int gpudb_q13_distribution(gpudb_ctx* ctx, const gpudb_customer* cu, const gpudb_orders* od,
                                      const gpudb_q13_params* p, gpudb_q13_row* out, uint32_t capacity,
                                      uint32_t* n_rows, gpudb_timing* t, const gpudb_exec* ex) {
  if (!ctx) return GPUDB_E_INVALID;
  if (!cu || !od || !p || !n_rows || (capacity && !out))
    return fail(ctx, GPUDB_E_INVALID, "q13: customer, orders, params and n_rows are required");
  if (cu->n_rows && (!cu->cust_key || cu->key_max < 0))
    return fail(ctx, GPUDB_E_INVALID, "q13: customer.cust_key and key_max >= 0 are required");
  if (od->n_rows && (!od->cust_key || !od->comment))
    return fail(ctx, GPUDB_E_INVALID, "q13: orders.cust_key and orders.comment are required");
  Q13Pattern pat{};
  for (int i = 0; i < 2; i++) {
    const char* w = i ? p->word2 : p->word1;
    const size_t l = strnlen(w, 16);
    if (l < 1 || l > 15) return fail(ctx, GPUDB_E_INVALID, "q13: word%d must be 1..15 characters", i + 1);
    std::memcpy(pat.w[i], w, l);
    pat.len[i] = (int32_t)l;
    for (int j = 0; j < 4; j++) std::memcpy(&pat.p[i][j], pat.w[i] + j, 4);
    pat.mask[i] = l >= 4 ? ~0u : (1u << (8 * l)) - 1u;
  }
  uint32_t* c = pat.poly;   // multiply out (x - p0)(x - p1)(x - p2)(x - p3) mod 2^32
  const uint32_t* r = pat.p[0];
  const uint32_t s01 = 0u - r[0] - r[1], q01 = r[0] * r[1], s23 = 0u - r[2] - r[3], q23 = r[2] * r[3];
  c[3] = s01 + s23;
  c[2] = q01 + q23 + s01 * s23;
  c[1] = s01 * q23 + s23 * q01;
  c[0] = q01 * q23;
  Call call(ctx, ex, t);
  const size_t bytes = 16 + (size_t)kBins * sizeof(gpudb_q13_row);
  int rc = call.begin(bytes, true);
  if (rc) return rc;
  cudaStream_t s = call.stream();
  const int32_t cust_max = cu->n_rows ? cu->key_max : 0;
  void *counts = nullptr, *hist = nullptr;
  if ((rc = scratch(ctx, "q13.counts", ((size_t)cust_max + 1) * 4, &counts))) return rc;
  if ((rc = scratch(ctx, "q13.hist", (size_t)kBins * 4, &hist))) return rc;
  if ((rc = call.clear(counts, 0, ((size_t)cust_max + 1) * 4))) return rc;
  if ((rc = call.clear(hist, 0, (size_t)kBins * 4))) return rc;
  const int sms = ctx->sm_count;
  if (od->n_rows && cu->n_rows) {
    auto kern = pat.len[0] <= 2                                          ? q13_count_kernel<kDirect>
                : pat.len[0] >= kLongWord && pat.len[1] >= kLongWord ? q13_count_kernel<kLong>
                                                                     : q13_count_kernel<kBytes>;
    GPUDB_CUDA(ctx, kernel_smem(ctx, (const void*)kern, sizeof(Q13Smem)));
    const int per_sm = kernel_occupancy(ctx, (const void*)kern, kQ13Threads, sizeof(Q13Smem));
    const unsigned g = (unsigned)std::max<uint64_t>(
        1, std::min<uint64_t>((od->n_rows + kQ13Threads - 1) / kQ13Threads, (uint64_t)sms * std::max(1, per_sm)));
    GPUDB_LAUNCH(call, kern, g, kQ13Threads, sizeof(Q13Smem), od->comment, od->cust_key, od->n_rows, cust_max, pat,
                 (uint32_t*)counts, call.status());
  }
  if (cu->n_rows) {
    const unsigned g = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((cu->n_rows + 255) / 256, (uint64_t)sms * 4));
    GPUDB_LAUNCH(call, q13_hist_kernel, g, 256, 0, cu->cust_key, cu->n_rows, cust_max, (const uint32_t*)counts,
                 (uint32_t*)hist, call.status());
  }
  GPUDB_LAUNCH(call, q13_sort_kernel, 1, kBins, 0, (const uint32_t*)hist, call.result<uint8_t>());
  const uint32_t cap = capacity;
  return call.finish(bytes, [out, cap, n_rows](const uint8_t* h) {
    uint32_t n;
    std::memcpy(&n, h, 4);
    *n_rows = n;
    if (cap) std::memcpy(out, h + 16, (size_t)std::min(n, cap) * sizeof(gpudb_q13_row));
    return GPUDB_OK;
  });
}
