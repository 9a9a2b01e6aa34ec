// After the scan: result bitmaps to row ids, masked sums, and a fused
// scan-and-aggregate.
//
// The reference stops at the bitmap and its hit count; its query files name
// the step that follows in a query engine -- TPC-H Q6, a filtered sum of
// l_extendedprice * l_discount (test/scan_cmd_1e8-1c.txt:48-54).  These
// kernels are HBM-bound streaming passes:
//
//   * rts_bitmap_rows_async: ordered compaction of a bitmap into ascending
//     uint32 row ids.  Pass 1 counts the set bits of each block's tiles of
//     1024 words (one tile, four on large tables); pass 2 reloads them, sums
//     the counts before its block (past 2^30 rows a one-CTA scan does) and
//     expands the words.  Bytes: 2 x N/8 read + 4 per row id.
//   * rts_bitmap_sum_async: sum of a column, or of the product of two
//     columns, over the set rows (128-bit exact).  A warp takes 1024 rows:
//     its 32 bitmap words, then the values as 16-byte loads, each lane
//     fetching its four rows' bits from the owning lane.  Bytes: N/8 + 4·N
//     per column.
//   * rts_scan_aggregate_async: the conjunctive predicate and the sum in one
//     pass with no bitmap: terms are merged per column into one inclusive
//     range, a thread tests four rows per 16-byte load of every referenced
//     column once, and accumulates the count and the sum.  Bytes: 4·N per
//     referenced column (a column used by the predicate and the sum is read
//     once).
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "rts_internal.h"

namespace rts {
namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kCompactThreads = 256;
constexpr int kCompactRounds = 4;                                   // words per thread
constexpr int kCompactTileWords = kCompactThreads * kCompactRounds;  // 1024 words = 32768 rows
constexpr int kCompactGroup = 4;  // tiles of a block on large tables
constexpr int kScanThreads = 1024;
// Up to this many blocks (2^30 rows) every block of the write pass sums the
// counts of the blocks before it itself (at most 32 loads per thread, from
// L2); a scan launch of one block costs 3 us and more.
constexpr uint64_t kCompactSelfBlocks = 8192;
constexpr uint32_t kCompactDense = 3000;  // ids of a warp's 128 words, see compact_write_kernel

// The thread's kCompactRounds words of the tile: warp w's round r holds words
// 32 * (kCompactRounds * w + r) .. + 31 of it, one per lane.
__device__ __forceinline__ void compact_words(const uint32_t *__restrict__ bm, uint64_t words, uint32_t tail_mask,
                                              uint64_t tile, uint32_t (&x)[kCompactRounds]) {
  const uint64_t w0 = tile * kCompactTileWords + (threadIdx.x >> 5) * (32 * kCompactRounds) +
                      (threadIdx.x & 31);
#pragma unroll
  for (int r = 0; r < kCompactRounds; r++) {
    const uint64_t w = w0 + 32 * r;
    x[r] = w < words ? (w + 1 == words ? __ldg(bm + w) & tail_mask : __ldg(bm + w)) : 0u;
  }
}

// Set bits of every block's tiles.
template <int TILES>
__global__ void __launch_bounds__(kCompactThreads) compact_count_kernel(const uint32_t *__restrict__ bm,
                                                                        uint64_t words, uint32_t tail_mask,
                                                                        uint32_t *__restrict__ block_count) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t c = 0;
#pragma unroll
  for (int t = 0; t < TILES; t++) {
    uint32_t x[kCompactRounds];
    compact_words(bm, words, tail_mask, (uint64_t)blockIdx.x * TILES + t, x);
#pragma unroll
    for (int r = 0; r < kCompactRounds; r++) c += __popc(x[r]);
  }
  c = __reduce_add_sync(kFull, c);
  __shared__ uint32_t part[kCompactThreads / 32];
  if (lane == 0) part[warp] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t v = 0;
#pragma unroll
    for (int k = 0; k < kCompactThreads / 32; k++) v += part[k];
    block_count[blockIdx.x] = v;
  }
}

// One CTA: exclusive prefix of the block counts (as uint64) and the total.
__global__ void __launch_bounds__(kScanThreads) compact_scan_kernel(const uint32_t *__restrict__ block_count,
                                                                    uint64_t nblocks,
                                                                    unsigned long long *__restrict__ block_off,
                                                                    unsigned long long *__restrict__ total) {
  const uint64_t per = (nblocks + kScanThreads - 1) / kScanThreads;
  const uint64_t b = threadIdx.x * per, e = std::min<uint64_t>(nblocks, b + per);
  unsigned long long s = 0;
  for (uint64_t i = b; i < e; i++) s += block_count[i];
  // block-wide inclusive scan of the thread sums
  __shared__ unsigned long long warp_sum[kScanThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    unsigned long long v = warp_sum[lane], vi = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(kFull, vi, o);
      if (lane >= o) vi += y;
    }
    warp_sum[lane] = vi - v;  // exclusive prefix of the warp sums
  }
  __syncthreads();
  unsigned long long off = warp_sum[warp] + incl - s;
  for (uint64_t i = b; i < e; i++) {
    block_off[i] = off;
    off += block_count[i];
  }
  if (threadIdx.x == kScanThreads - 1) *total = off;
}

// A lane takes one word at a time, its ids go to the warp's buffer at the
// word's place, and the warp copies the buffer out as one run of consecutive
// addresses; where nearly every bit is set (kCompactDense) the warp takes a
// word at a time instead, a lane per bit.  (Every thread storing its ids of 16
// words straight to memory: 32 lines per store instruction; a lane per bit
// everywhere: 12 instructions per nonzero word, however few bits it has.)
// block_off null: the block sums the counts before its tiles, and the last
// block stores the total.
// Bound by issue, seven instructions per bit of a round's fullest word and
// five per 32 ids copied, then by the id writes.  Row ids of a bitmap, both
// passes (us; straight stores, a lane per bit, this): 2^25 rows at 3 % 23, 25,
// 13, at 50 % 107, 33, 27; 1e8 rows at 1 % 23, 37, 23, at 10 % 74, 80, 31, at
// 100 % 1253, 81, 82; 6e8 rows at 1 % 82, 184, 85, at 50 % 3078, 446, 358.
template <int TILES>
__global__ void __launch_bounds__(kCompactThreads) compact_write_kernel(
    const uint32_t *__restrict__ bm, uint64_t words, uint32_t tail_mask, const uint32_t *__restrict__ block_count,
    const unsigned long long *__restrict__ block_off, uint32_t *__restrict__ rows, uint64_t capacity,
    unsigned long long *__restrict__ total) {
  constexpr int kWarps = kCompactThreads / 32;
  __shared__ unsigned long long s_before[kWarps];
  __shared__ uint32_t s_warp[2][kWarps];
  __shared__ __align__(16) uint32_t s_ids[kWarps][33 * 32];  // a round's ids in order, the i-th at i + i / 32
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool last = blockIdx.x == gridDim.x - 1;
  const uint32_t tile0 = blockIdx.x * TILES;
  uint32_t next[kCompactRounds];
  compact_words(bm, words, tail_mask, tile0, next);
  if (TILES > 1 && !last && __ldg(block_count + blockIdx.x) == 0) return;  // (the last block may store the total)
  unsigned long long before = 0;
  if (!block_off)
    for (uint32_t i = threadIdx.x; i < blockIdx.x; i += kCompactThreads) before += __ldg(block_count + i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(kFull, before, o);
  if (lane == 0) s_before[warp] = before;
  unsigned long long base = block_off ? block_off[blockIdx.x] : 0ull;
  uint32_t *const ids = s_ids[warp];
#pragma unroll 1
  for (int t = 0; t < TILES; t++) {
    uint32_t x[kCompactRounds];
#pragma unroll
    for (int r = 0; r < kCompactRounds; r++) x[r] = next[r];
    if (t + 1 < TILES) compact_words(bm, words, tail_mask, tile0 + t + 1, next);
    // exclusive scans of the rounds' popcounts over the lanes, two rounds to a
    // word (a round has at most 1024 bits)
    static_assert(kCompactRounds == 4, "two packed scans");
    uint32_t c01 = __popc(x[0]) | __popc(x[1]) << 16, c23 = __popc(x[2]) | __popc(x[3]) << 16;
    const uint32_t own01 = c01, own23 = c23;
    if (__any_sync(kFull, (c01 | c23) != 0)) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y01 = __shfl_up_sync(kFull, c01, o), y23 = __shfl_up_sync(kFull, c23, o);
        if (lane >= o) {
          c01 += y01;
          c23 += y23;
        }
      }
    }
    const uint32_t all01 = __shfl_sync(kFull, c01, 31), all23 = __shfl_sync(kFull, c23, 31);
    c01 -= own01;
    c23 -= own23;
    const uint32_t sum[kCompactRounds] = {all01 & 0xFFFFu, all01 >> 16, all23 & 0xFFFFu, all23 >> 16};
    if (lane == 0) s_warp[t & 1][warp] = sum[0] + sum[1] + sum[2] + sum[3];
    __syncthreads();  // (the other buffer's readers are a barrier behind)
    if (t == 0) {
#pragma unroll
      for (int k = 0; k < kWarps; k++) base += s_before[k];
    }
    uint32_t start = 0, tile = 0;  // ids of the tile before this warp, in the tile
#pragma unroll
    for (int k = 0; k < kWarps; k++) {
      if (k < warp) start += s_warp[t & 1][k];
      tile += s_warp[t & 1][k];
    }
    if (base < capacity && (all01 | all23) != 0) {
      uint32_t *const dst = rows + base;
      const uint32_t room = (uint32_t)std::min<unsigned long long>(capacity - base, tile);
      const uint32_t row0 = (uint32_t)(((uint64_t)(tile0 + t) * kCompactTileWords + warp * (32 * kCompactRounds)) * 32);
      const uint32_t all = sum[0] + sum[1] + sum[2] + sum[3];
      if (all > kCompactDense && start + all <= room) {
        // the warp's nonzero words, each with its index and its ids' offset in
        // the tile; then a word at a time, a lane per bit
        uint2 *const list = reinterpret_cast<uint2 *>(ids);
        int n = 0;
#pragma unroll
        for (int r = 0; r < kCompactRounds; r++) {
          const uint32_t at =
              start + (r == 0 ? c01 & 0xFFFFu : r == 1 ? c01 >> 16 : r == 2 ? c23 & 0xFFFFu : c23 >> 16);
          const unsigned some = __ballot_sync(kFull, x[r] != 0);
          if (x[r]) list[n + __popc(some & ((1u << lane) - 1))] = make_uint2(x[r], at | (uint32_t)(32 * r + lane) << 16);
          n += __popc(some);
          start += sum[r];
        }
        __syncwarp();
        const uint32_t bit = 0x80000000u >> lane, above = ~(0xFFFFFFFFu >> lane);
#pragma unroll 4
        for (int k = 0; k < n; k++) {
          const uint2 w = list[k];
          if (w.x & bit) dst[(w.y & 0xFFFFu) + __popc(w.x & above)] = row0 + lane + ((w.y >> 16) << 5);
        }
        __syncwarp();
      } else {
        // through the buffer: all the rounds' ids at once where they fit it
        const bool together = all <= 32 * 32;
        uint32_t off = 0;
#pragma unroll
        for (int r = 0; r < kCompactRounds; r++) {
          uint32_t at = off + (r == 0 ? c01 & 0xFFFFu : r == 1 ? c01 >> 16 : r == 2 ? c23 & 0xFFFFu : c23 >> 16);
          const uint32_t row = row0 + 32 * (32 * r + lane);
          for (uint32_t w = x[r]; w; at++) {  // MSB-first: bit 31 is the word's first row
            const int b = __clz(w);
            ids[at + (at >> 5)] = row + b;
            w &= 0x7FFFFFFFu >> b;
          }
          off += sum[r];
          if (together && r + 1 < kCompactRounds) continue;
          __syncwarp();
          for (uint32_t i = lane; i < off; i += 32)
            if (start + i < room) dst[start + i] = ids[i + (i >> 5)];
          __syncwarp();
          start += off;
          off = 0;
        }
      }
    }
    base += tile;
  }
  if (!block_off && last && threadIdx.x == 0) *total = base;
}

// 128-bit accumulation: per-thread unsigned __int128, one pair of 64-bit
// atomics per CTA with the carry of the low half propagated.
__device__ __forceinline__ void add128(unsigned long long *res, unsigned __int128 v) {
  const unsigned long long lo = (unsigned long long)v, hi = (unsigned long long)(v >> 64);
  const unsigned long long old = atomicAdd(res, lo);
  const unsigned long long carry = old + lo < old ? 1ull : 0ull;
  if (hi + carry) atomicAdd(res + 1, hi + carry);
}

__device__ __forceinline__ unsigned __int128 block_sum128(unsigned __int128 v) {
  __shared__ unsigned long long part[2][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long lo = (unsigned long long)v, hi = (unsigned long long)(v >> 64);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long l2 = __shfl_xor_sync(kFull, lo, o), h2 = __shfl_xor_sync(kFull, hi, o);
    const unsigned long long nl = lo + l2;
    hi += h2 + (nl < lo ? 1ull : 0ull);
    lo = nl;
  }
  if (lane == 0) {
    part[0][warp] = lo;
    part[1][warp] = hi;
  }
  __syncthreads();
  unsigned __int128 t = 0;
  if (threadIdx.x == 0)
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += ((unsigned __int128)part[1][k] << 64) | part[0][k];
  return t;
}

// Sum of a (or a * b when b) over the set rows of bm; a warp takes 1024 rows.
template <bool PRODUCT>
__global__ void __launch_bounds__(256) bitmap_sum_kernel(const uint32_t *__restrict__ bm, const uint32_t *__restrict__ a,
                                                         const uint32_t *__restrict__ b, uint64_t nrows, int vec,
                                                         unsigned long long *__restrict__ res) {
  const int lane = threadIdx.x & 31;
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t ntiles = (nrows + 1023) / 1024, words = (nrows + 31) >> 5;
  unsigned __int128 acc = 0;
  for (uint64_t t = warp; t < ntiles; t += nwarps) {
    const uint64_t wi = t * 32 + lane;
    uint32_t myword = wi < words ? bm[wi] : 0u;
    if (wi + 1 == words && (nrows & 31)) myword &= ~(0xFFFFFFFFu >> (nrows & 31));  // bits past nrows
    const uint64_t row0 = t * 1024;
    const bool full = vec && row0 + 1024 <= nrows;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const uint32_t w = __shfl_sync(kFull, myword, j * 4 + (lane >> 3));
      const uint64_t r = row0 + j * 128 + lane * 4;
      uint32_t va[4], vb[4] = {1u, 1u, 1u, 1u};
      if (full) {
        const uint4 x = *reinterpret_cast<const uint4 *>(a + r);
        va[0] = x.x, va[1] = x.y, va[2] = x.z, va[3] = x.w;
        if (PRODUCT) {
          const uint4 y = *reinterpret_cast<const uint4 *>(b + r);
          vb[0] = y.x, vb[1] = y.y, vb[2] = y.z, vb[3] = y.w;
        }
      } else {
#pragma unroll
        for (int k = 0; k < 4; k++) {
          va[k] = r + k < nrows ? a[r + k] : 0u;
          if (PRODUCT) vb[k] = r + k < nrows ? b[r + k] : 0u;
        }
      }
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int bit = 31 - ((lane & 7) * 4 + k);
        if ((w >> bit) & 1u) acc += PRODUCT ? (unsigned __int128)((unsigned long long)va[k] * vb[k]) : va[k];
      }
    }
  }
  const unsigned __int128 t = block_sum128(acc);
  if (threadIdx.x == 0 && t) add128(res, t);
}

// Fused predicate + aggregate.  Column slot 0 is the first aggregate column
// and slot 1 the second (when MODE needs them); every slot carries the
// merged range of the terms on that column ((0, 2^32 - 1) when it has none).
struct AggParams {
  const uint32_t *col[8];
  uint32_t lo[8];
  uint32_t span[8];
  uint64_t nrows;
  unsigned long long *count;  // may be null
  unsigned long long *sum;    // two words (low, high); may be null
};

// MODE 0: count only; 1: sum of slot 0; 2: sum of slot 0 x slot 1;
// 3: sum of slot 0 squared.
// Row groups (four rows) that a thread loads before it tests any, 64 to 128
// bytes in flight.  Q6 on 6e7 rows x 4 columns (0.96 GB): one group a time and
// 8 blocks per SM 167 us, two groups and 16 blocks per SM 140, 1.05 of the
// copy rate.
constexpr int agg_groups(int nu) { return nu <= 1 ? 4 : nu <= 4 ? 2 : 1; }
template <int NU, int MODE, bool VEC>
__global__ void __launch_bounds__(256) scan_aggregate_kernel(const __grid_constant__ AggParams p) {
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (uint64_t)gridDim.x * blockDim.x;
  unsigned long long cnt = 0;
  unsigned __int128 acc = 0;
  auto one = [&](const uint32_t (&v)[NU]) {
    bool hit = true;
#pragma unroll
    for (int c = 0; c < NU; c++) hit = hit && (v[c] - p.lo[c] <= p.span[c]);
    cnt += hit;
    if (MODE == 1 && hit) acc += v[0];
    if (MODE == 2 && hit) acc += (unsigned __int128)((unsigned long long)v[0] * v[NU > 1 ? 1 : 0]);
    if (MODE == 3 && hit) acc += (unsigned __int128)((unsigned long long)v[0] * v[0]);
  };
  const uint64_t groups = VEC ? p.nrows / 4 : 0;
  constexpr int kG = agg_groups(NU);
  for (uint64_t g0 = (uint64_t)blockIdx.x * (256 * kG) + threadIdx.x; g0 < groups; g0 += nth * kG) {
    uint4 x[kG][NU];
#pragma unroll
    for (int j = 0; j < kG; j++)
      if (g0 + j * 256 < groups)
#pragma unroll
        for (int c = 0; c < NU; c++) x[j][c] = __ldg(reinterpret_cast<const uint4 *>(p.col[c]) + g0 + j * 256);
#pragma unroll
    for (int j = 0; j < kG; j++) {
      if (g0 + j * 256 >= groups) break;
      uint32_t v[NU];
#pragma unroll
      for (int c = 0; c < NU; c++) v[c] = x[j][c].x;
      one(v);
#pragma unroll
      for (int c = 0; c < NU; c++) v[c] = x[j][c].y;
      one(v);
#pragma unroll
      for (int c = 0; c < NU; c++) v[c] = x[j][c].z;
      one(v);
#pragma unroll
      for (int c = 0; c < NU; c++) v[c] = x[j][c].w;
      one(v);
    }
  }
  for (uint64_t r = groups * 4 + tid; r < p.nrows; r += nth) {
    uint32_t v[NU];
#pragma unroll
    for (int c = 0; c < NU; c++) v[c] = __ldg(p.col[c] + r);
    one(v);
  }
  // one addition per block to the count and to the sum: they all go to one
  // address, and with one per warp to the count their tail took 12 us of a
  // 1e8-row scan of one column (77 us, 67 without) and doubled 4e6 rows of
  // five (32 us, 16 without)
  __shared__ unsigned long long s_cnt[8];
  if (p.count) {
    unsigned long long c = cnt;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(kFull, c, o);
    if ((threadIdx.x & 31) == 0) s_cnt[threadIdx.x >> 5] = c;
  }
  unsigned __int128 sum = 0;
  if (MODE > 0 && p.sum) sum = block_sum128(acc);
  else __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long c = 0;
    if (p.count)
#pragma unroll
      for (int k = 0; k < 8; k++) c += s_cnt[k];
    if (c) atomicAdd(p.count, c);
    if (sum) add128(p.sum, sum);
  }
}

template <int NU, int MODE>
void launch_agg(const AggParams &p, bool vec, int sm_count, cudaStream_t s) {
  const uint64_t work = vec ? (p.nrows / 4 + agg_groups(NU) - 1) / agg_groups(NU) : p.nrows;
  // 16 blocks per SM (two waves, so that no SM idles through a last partial
  // one): within 2 % of the best of 8, 16 and 32 for one to eight columns of
  // 4e6 to 1e8 rows, where 8 loses up to 15 % (two columns) and 32 up to 30 %
  // (4e6 rows).  Four-byte loads: 8 (1e8 rows of three columns 228, 232 and
  // 234 us).
  const uint64_t most = (uint64_t)sm_count * (vec ? 16 : 8);
  const int grid = (int)std::max<uint64_t>(1, std::min<uint64_t>((work + 255) / 256, most));
  if (vec) scan_aggregate_kernel<NU, MODE, true><<<grid, 256, 0, s>>>(p);
  else scan_aggregate_kernel<NU, MODE, false><<<grid, 256, 0, s>>>(p);
}

template <int MODE>
void launch_agg_nu(int nu, const AggParams &p, bool vec, int sm_count, cudaStream_t s) {
  switch (nu) {
    case 1: launch_agg<1, MODE>(p, vec, sm_count, s); break;
    case 2: launch_agg<2, MODE>(p, vec, sm_count, s); break;
    case 3: launch_agg<3, MODE>(p, vec, sm_count, s); break;
    case 4: launch_agg<4, MODE>(p, vec, sm_count, s); break;
    case 5: launch_agg<5, MODE>(p, vec, sm_count, s); break;
    case 6: launch_agg<6, MODE>(p, vec, sm_count, s); break;
    case 7: launch_agg<7, MODE>(p, vec, sm_count, s); break;
    default: launch_agg<8, MODE>(p, vec, sm_count, s); break;
  }
}

// Device scratch for a compaction's block counts and offsets on stream s.  The
// context's calls share one buffer (grown as needed), each ordered after the
// one before, whatever their streams (agg_done).  A captured call runs when its
// graph is launched, so it gets a buffer of its own, which stays until the
// context goes.
struct AggScratch {
  rts_ctx *ctx;
  cudaStream_t s;
  void *dev = nullptr;
  bool captured = false;
  AggScratch(rts_ctx *c, size_t bytes, cudaStream_t stream) : ctx(c), s(stream) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &st) != cudaSuccess) cudaGetLastError();
    captured = st != cudaStreamCaptureStatusNone;
    if (captured) {
      ctx->agg_captured.reserve(ctx->agg_captured.size() + 1);
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // (an allocation is no part of the capture)
      RTS_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
      const bool ok = cudaMalloc(&dev, bytes) == cudaSuccess;
      RTS_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
      if (!ok) fail_alloc();
      ctx->agg_captured.push_back(dev);
      return;
    }
    if (!ctx->agg_done) RTS_CUDA(cudaEventCreateWithFlags(&ctx->agg_done, cudaEventDisableTiming));
    if (ctx->agg_bytes < bytes) {
      RTS_CUDA(cudaEventSynchronize(ctx->agg_done));
      if (ctx->agg_dev) cudaFree(ctx->agg_dev);
      ctx->agg_dev = nullptr;
      ctx->agg_bytes = 0;
      if (cudaMalloc(&ctx->agg_dev, bytes) != cudaSuccess) fail_alloc();
      ctx->agg_bytes = bytes;
    }
    dev = ctx->agg_dev;
    RTS_CUDA(cudaStreamWaitEvent(s, ctx->agg_done, 0));
  }
  // The call's last use of the buffer has been queued.
  void done() {
    if (!captured) RTS_CUDA(cudaEventRecord(ctx->agg_done, s));
  }
  static void fail_alloc() {
    cudaGetLastError();
    throw Error(RTS_ERR_NOMEM, "aggregate scratch allocation failed");
  }
};

rts_status fail(rts_ctx *ctx, const std::exception &e) {
  if (ctx) ctx->err = e.what();
  return set_thread_error(status_of(e), e.what());
}

}  // namespace
}  // namespace rts

extern "C" {

rts_status rts_bitmap_rows_async(rts_ctx *ctx, const uint32_t *dev_bitmap, uint64_t nrows, uint32_t *dev_rows,
                                 uint64_t capacity, uint64_t *dev_count, void *stream) {
  rts::Range nvtx_range_("rts_bitmap_rows_async");
  if (!ctx) return rts::set_thread_error(RTS_ERR_ARG, "null context");
  try {
    if (!dev_bitmap || !dev_count || (capacity && !dev_rows)) throw rts::Error(RTS_ERR_ARG, "null argument");
    if (nrows > 0xFFFFFFFFull) throw rts::Error(RTS_ERR_ARG, "row ids are uint32: at most 2^32 - 1 rows");
    rts::DeviceGuard g(ctx->device);
    cudaStream_t s = (cudaStream_t)stream;
    const uint64_t words = rts::words_for(nrows);
    if (words == 0) {
      RTS_CUDA(cudaMemsetAsync(dev_count, 0, 8, s));
      return RTS_OK;
    }
    const uint32_t tail_mask = (nrows & 31) ? ~(0xFFFFFFFFu >> (nrows & 31)) : 0xFFFFFFFFu;
    const uint64_t ntiles = (words + rts::kCompactTileWords - 1) / rts::kCompactTileWords;
    // four tiles per block once every SM has eight such blocks: 2.5e8 rows at
    // 1 % 39 us, a tile per block 52, but 1e8 rows at 50 % 88 and 66
    const bool group = ntiles >= (uint64_t)ctx->sm_count * 8 * rts::kCompactGroup;
    const uint64_t nblocks = group ? (ntiles + rts::kCompactGroup - 1) / rts::kCompactGroup : ntiles;
    const bool self = nblocks <= rts::kCompactSelfBlocks;
    rts::AggScratch buffer(ctx, nblocks * 12 + 16, s);
    char *scratch = static_cast<char *>(buffer.dev);
    auto *block_off = self ? nullptr : reinterpret_cast<unsigned long long *>(scratch);
    auto *block_count = reinterpret_cast<uint32_t *>(scratch + nblocks * 8);
    auto *total = reinterpret_cast<unsigned long long *>(dev_count);
    const auto count = group ? rts::compact_count_kernel<rts::kCompactGroup> : rts::compact_count_kernel<1>;
    const auto write = group ? rts::compact_write_kernel<rts::kCompactGroup> : rts::compact_write_kernel<1>;
    count<<<(unsigned)nblocks, rts::kCompactThreads, 0, s>>>(dev_bitmap, words, tail_mask, block_count);
    if (!self) rts::compact_scan_kernel<<<1, rts::kScanThreads, 0, s>>>(block_count, nblocks, block_off, total);
    write<<<(unsigned)nblocks, rts::kCompactThreads, 0, s>>>(dev_bitmap, words, tail_mask, block_count, block_off,
                                                             dev_rows, capacity, total);
    const cudaError_t launched = cudaGetLastError();
    buffer.done();
    RTS_CUDA(launched);
    ctx->launches += self ? 2 : 3;
    return RTS_OK;
  } catch (const std::exception &e) {
    return rts::fail(ctx, e);
  }
}

rts_status rts_bitmap_sum_async(rts_ctx *ctx, const uint32_t *dev_bitmap, int32_t col_a, int32_t col_b,
                                uint64_t *dev_sum, void *stream) {
  rts::Range nvtx_range_("rts_bitmap_sum_async");
  if (!ctx) return rts::set_thread_error(RTS_ERR_ARG, "null context");
  try {
    if (!dev_bitmap || !dev_sum) throw rts::Error(RTS_ERR_ARG, "null argument");
    const int nc = (int)ctx->cols.size();
    if (col_a < 0 || col_a >= nc || col_b < -1 || col_b >= nc) throw rts::Error(RTS_ERR_ARG, "column out of range");
    rts::DeviceGuard g(ctx->device);
    cudaStream_t s = (cudaStream_t)stream;
    const uint32_t *a = ctx->cols[col_a], *b = col_b >= 0 ? ctx->cols[col_b] : nullptr;
    const bool vec = (((uintptr_t)a | (uintptr_t)(b ? b : a)) & 15) == 0;
    const uint64_t ntiles = (ctx->nrows + 1023) / 1024;
    const int grid = (int)std::max<uint64_t>(1, std::min<uint64_t>((ntiles + 7) / 8, (uint64_t)ctx->sm_count * 8));
    RTS_CUDA(cudaMemsetAsync(dev_sum, 0, 16, s));
    auto *res = reinterpret_cast<unsigned long long *>(dev_sum);
    if (b) rts::bitmap_sum_kernel<true><<<grid, 256, 0, s>>>(dev_bitmap, a, b, ctx->nrows, vec ? 1 : 0, res);
    else rts::bitmap_sum_kernel<false><<<grid, 256, 0, s>>>(dev_bitmap, a, nullptr, ctx->nrows, vec ? 1 : 0, res);
    RTS_CUDA(cudaGetLastError());
    ctx->launches += 1;
    return RTS_OK;
  } catch (const std::exception &e) {
    return rts::fail(ctx, e);
  }
}

rts_status rts_scan_aggregate_async(rts_ctx *ctx, const rts_term *terms, int32_t nterms, int32_t col_a,
                                    int32_t col_b, uint64_t *dev_count, uint64_t *dev_sum, void *stream) {
  rts::Range nvtx_range_("rts_scan_aggregate_async");
  if (!ctx) return rts::set_thread_error(RTS_ERR_ARG, "null context");
  try {
    if (nterms < 0 || (nterms > 0 && !terms)) throw rts::Error(RTS_ERR_ARG, "bad terms");
    const int nc = (int)ctx->cols.size();
    if (nc == 0) throw rts::Error(RTS_ERR_STATE, "no columns loaded");
    if (col_a < -1 || col_a >= nc || col_b < -1 || col_b >= nc || (col_b >= 0 && col_a < 0))
      throw rts::Error(RTS_ERR_ARG, "aggregate column out of range");
    if (col_a >= 0 && !dev_sum) throw rts::Error(RTS_ERR_ARG, "a sum needs dev_sum");
    // slots: aggregate columns first, then the predicate's other columns
    std::vector<int> slot_col;
    std::vector<uint32_t> lo, hi;
    auto slot_of = [&](int col) {
      for (size_t i = 0; i < slot_col.size(); i++)
        if (slot_col[i] == col) return (int)i;
      slot_col.push_back(col);
      lo.push_back(0);
      hi.push_back(0xFFFFFFFFu);
      return (int)slot_col.size() - 1;
    };
    if (col_a >= 0) slot_of(col_a);
    if (col_b >= 0 && col_b != col_a) slot_of(col_b);
    bool empty = false;
    for (int i = 0; i < nterms; i++) {
      const rts_term &t = terms[i];
      if (t.column < 0 || t.column >= nc) throw rts::Error(RTS_ERR_ARG, "term column out of range");
      if (t.lo > t.hi) empty = true;
      const int k = slot_of(t.column);
      lo[k] = std::max(lo[k], t.lo);
      hi[k] = std::min(hi[k], t.hi);
      if (lo[k] > hi[k]) empty = true;
    }
    if (slot_col.size() > 8) throw rts::Error(RTS_ERR_ARG, "at most 8 distinct columns per aggregate scan");
    rts::DeviceGuard g(ctx->device);
    cudaStream_t s = (cudaStream_t)stream;
    if (dev_count) RTS_CUDA(cudaMemsetAsync(dev_count, 0, 8, s));
    if (dev_sum) RTS_CUDA(cudaMemsetAsync(dev_sum, 0, 16, s));
    if (empty || ctx->nrows == 0) return RTS_OK;
    if (slot_col.empty()) slot_of(0);  // no term and no aggregate: count every row
    rts::AggParams p{};
    bool vec = true;
    for (size_t i = 0; i < slot_col.size(); i++) {
      p.col[i] = ctx->cols[slot_col[i]];
      p.lo[i] = lo[i];
      p.span[i] = hi[i] - lo[i];
      vec = vec && ((uintptr_t)p.col[i] & 15) == 0;
    }
    p.nrows = ctx->nrows;
    p.count = reinterpret_cast<unsigned long long *>(dev_count);
    p.sum = reinterpret_cast<unsigned long long *>(dev_sum);
    const int nu = (int)slot_col.size();
    if (col_a < 0) {
      rts::launch_agg_nu<0>(nu, p, vec, ctx->sm_count, s);
    } else if (col_b < 0) {
      rts::launch_agg_nu<1>(nu, p, vec, ctx->sm_count, s);
    } else if (col_b == col_a) {
      rts::launch_agg_nu<3>(nu, p, vec, ctx->sm_count, s);
    } else {
      rts::launch_agg_nu<2>(nu, p, vec, ctx->sm_count, s);
    }
    RTS_CUDA(cudaGetLastError());
    ctx->launches += 1;
    return RTS_OK;
  } catch (const std::exception &e) {
    return rts::fail(ctx, e);
  }
}

}  // extern "C"
