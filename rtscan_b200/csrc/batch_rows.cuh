// Table passes with a thread per row (included by batch.cu inside its
// anonymous namespace; uses BatchPass and kFull from there).
//
// A pass has G groups of 32 query slots (16, 8 or 4).  A CTA of 8 warps
// answers a part of eight or four of them (see batch_rows_kernel) on blocks of
// 1024 rows (2048 for four groups), two CTAs per SM, in three phases over a
// 32 KiB buffer:
//   A. every thread ANDs the table rows of its rows, 16 bytes (four groups)
//      at a time, and writes the row masks to the buffer;
//   B. lane (tile, group) reads the 32 mask words of a 32-row tile for one
//      group, transposes them in registers (transpose_octets), counts their
//      bits and writes the 32 result words back to the buffer as one line of
//      32 words per query;
//   C. one TMA store per 128 queries takes the lines to the bitmaps (or,
//      where the bitmaps are in another order or not 16-byte aligned, eight
//      lanes store a line).
// One CTA's table loads (shared-memory bandwidth) overlap the other's
// transposes (integer pipes).
//
// What bounds it: the shared-memory pipe and the integer ALU pipe, and how
// far two CTAs' phases overlap.  Per row and 512 slots over C columns phase
// A reads 64 * C bytes of tables and writes 64, phase B reads and writes 64,
// so every access is laid out to run at 128 bytes a cycle:
//   * a table row is a part of a 128-byte line: a line has S slots of 128 / S
//     bytes, columns are put in groups of at most S (a power of two), a
//     column of a group owns S / size of the slots (copies), and position p
//     of every column of the group is in the group's line p.  Lane i of a
//     quarter-warp visits the slots and the 16-byte parts of a slot in the
//     order k ^ i, so its eight lanes are always in eight different 16-byte
//     parts of a line, whatever their positions are;
//   * the buffer's 16-byte pieces are swizzled by row and tile so that phase
//     A's 16-byte stores and phase B's 4-byte loads and stores meet 32 banks.
// A table position past the lines that fit (L.t_lines) has its row packed
// behind them instead, once: correct, with bank conflicts.  Two CTAs per SM
// hold about 648 lines each, so a column of a 512-slot pass that every
// second query constrains twice overflows by a few positions.
// Measured on 1e8 rows x 4 skewed columns, reading shared positions (the
// kernel before it had each lane AND 16 rows for two groups and stage 16-bit
// halves of the result words): 2.90 -> 2.35 ms for a 512-query pass, 1024
// queries with their pre-pass 6.43 -> 5.35 ms; 250 queries 2.09 -> 1.66 ms,
// 120 queries 1.46 -> 1.08 ms; 300 queries over 8 columns on 2^24 rows
// (searching their own positions before) 1.18 -> 0.65 ms.  At 2.1e7 rows a 448-query pass keeps the
// shared-memory pipe 58 % busy with 3.9 wavefronts per row (6.0 before) and
// issues 10.9 warp instructions per row (16.0 before).  The lines stored by
// 16-byte stores of eight lanes instead of TMA: 2.65 ms per 512-query pass;
// 4-byte stores straight from phase B's registers (32-byte sectors of four
// bitmaps per instruction): 4.7 ms.  All rows packed (no lines): 2.8 ms.
template <int KG>  // groups of a CTA
struct RowsShape {
  static_assert(KG == 8 || KG == 4, "256 or 128 slots per CTA");
  static constexpr int kQ = KG / 4;                      // 16-byte parts of a row's mask
  static constexpr int kLQ = kQ == 2 ? 1 : 0;
  static constexpr int kS = 8 / kQ;                      // table rows per 128-byte line
  static constexpr int kLS = 3 - kLQ;
  static constexpr int kRPT = 32 / KG;                   // rows per thread and block
  static constexpr int kRows = 256 * kRPT;               // rows per block
  static constexpr int kTiles = kRows / 32;
};
constexpr int kRowsBuffer = 32768;  // row masks, then result words


// Size and first column of the group that column c of C is in, with S slots
// per line: groups are the powers of two of C, largest first, at most S.
__host__ __device__ constexpr int rows_group_start(int C, int S, int c) {
  const int base = C / S * S, rem = C % S, q = c - base;
  return q < 0 ? c / S * S : q < (rem & 4) ? base : q < (rem & 6) ? base + (rem & 4) : base + (rem & 6);
}
__host__ __device__ constexpr int rows_group_size(int C, int S, int c) {
  const int base = C / S * S, rem = C % S, q = c - base;
  return q < 0 ? S : q < (rem & 4) ? 4 : q < (rem & 6) ? 2 : 1;
}
__host__ __device__ constexpr int rows_log2(int x) { return x >= 8 ? 3 : x >= 4 ? 2 : x >= 2 ? 1 : 0; }

// 32x32 bit transpose of the mask words of 32 rows: x[8 * o + r] holds row
// 8 * o + 7 - r; on return x[j] holds slot j's bits, row 0 the MSB.  Eight
// rows at a time: rotate row r left by r, merge bit columns across the rows
// with selects (out[i] takes bit p from word (i + p) % 8: three stages of one
// LOP3 per word, no shifts), rotate word i left by i; its byte b then holds
// the eight rows of slot (8b - i) % 32, and byte permutes gather the four
// octets' bytes.  216 integer instructions, against 304 for five delta-swap
// stages.
__device__ __forceinline__ void transpose_octets(uint32_t (&x)[32]) {
  uint32_t y[4][8];
#pragma unroll
  for (int o = 0; o < 4; o++) {
    uint32_t a[8], b[8];
#pragma unroll
    for (int r = 0; r < 8; r++) a[r] = r ? __funnelshift_l(x[8 * o + r], x[8 * o + r], r) : x[8 * o];
#pragma unroll
    for (int i = 0; i < 8; i++) b[i] = (a[i] & 0x55555555u) | (a[(i + 1) & 7] & 0xAAAAAAAAu);
#pragma unroll
    for (int i = 0; i < 8; i++) a[i] = (b[i] & 0x33333333u) | (b[(i + 2) & 7] & 0xCCCCCCCCu);
#pragma unroll
    for (int i = 0; i < 8; i++) b[i] = (a[i] & 0x0F0F0F0Fu) | (a[(i + 4) & 7] & 0xF0F0F0F0u);
#pragma unroll
    for (int i = 0; i < 8; i++) y[o][i] = i ? __funnelshift_l(b[i], b[i], i) : b[0];
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const uint32_t u0 = __byte_perm(y[1][i], y[0][i], 0x5140), u1 = __byte_perm(y[1][i], y[0][i], 0x7362);
    const uint32_t v0 = __byte_perm(y[3][i], y[2][i], 0x5140), v1 = __byte_perm(y[3][i], y[2][i], 0x7362);
    x[(32 - i) & 31] = __byte_perm(v0, u0, 0x5410);
    x[8 - i] = __byte_perm(v0, u0, 0x7632);
    x[16 - i] = __byte_perm(v1, u1, 0x5410);
    x[24 - i] = __byte_perm(v1, u1, 0x7632);
  }
}

__device__ __forceinline__ void rows_swap(uint32_t &a, uint32_t &b, bool yes) {
  const uint32_t x = yes ? b : a, y = yes ? a : b;
  a = x;
  b = y;
}

// Slot of the i-th query of a pass.  Phase B's result lines are in query
// order, and the order of slots is chosen so that its stores meet 32 banks:
// line 8 * (j / 2) + 2 * g + j % 2 of a quad of groups is group g's slot j.
__host__ __device__ inline int rows_slot(int i) {
  return (i & ~127) + 32 * ((i >> 1) & 3) + 2 * ((i & 127) >> 3) + (i & 1);
}

// One CTA's part of a pass: groups g0 .. g0 + KG - 1 on blocks bid, bid + nb,
// ... of the range, with the tables laid out as L says.  OVF: some column
// has positions past the lines.  TWO: with room for two buffers (p.nbuf) the
// blocks take turns in them, and a block's TMA stores read theirs while the
// next block fills the other (250 queries 1.74 -> 1.67 ms, 120 queries 1.13
// -> 1.09 ms on 1e8 rows).
template <int C, int KG, bool OVF, bool TWO>
__device__ __forceinline__ void batch_rows_part(const BatchPass &p, const RowsLayout &L, const CUtensorMap *tmap, int g0,
                                                uint32_t bid, uint32_t nb) {
  using R = RowsShape<KG>;
  constexpr int Q = R::kQ, S = R::kS;
  extern __shared__ __align__(1024) unsigned char rows_sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char *buf = rows_sm;
  const uint32_t nbuf = TWO ? p.nbuf : 1u;
  const unsigned char *tables = rows_sm + nbuf * kRowsBuffer;
  const uint64_t block_begin = p.row_begin / R::kRows, nblocks = (p.nrows + R::kRows - 1) / R::kRows;

  // the part's tables and their copies
  for (int c = 0; c < C; c++) {
    const uint32_t *src = p.blob + p.tab_off[c] + g0;
    const uint32_t n = (p.m[c] + 1) * Q;
    for (uint32_t k = tid; k < n; k += 256) {
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(src + (k / Q) * p.groups) + k % Q);
      const uint32_t pos = k / Q;
      unsigned char *dst = rows_sm + nbuf * kRowsBuffer + (k % Q) * 16;
      if (!OVF || pos < L.t_lines) {
        for (uint32_t r = 0; r < L.t_nrep[c]; r++)
          *reinterpret_cast<uint4 *>(dst + L.t_base[c] + pos * 128 + r * L.t_rep[c]) = v;
      } else {
        *reinterpret_cast<uint4 *>(dst + L.t_over[c] + (pos - L.t_lines) * (4 * KG)) = v;
      }
    }
  }
  __syncthreads();

  // phase A: the lane's k-th column of a group is its column k ^ sb; hx: its
  // first 16-byte part
  const uint32_t hx = lane & (Q - 1), sb = (lane & 7) >> R::kLQ;
  uint32_t lc[OVF ? 1 : Q][C];  // byte offset of table word offset 0 of the k-th column, part s ^ hx
  uint32_t lim[C], lo[C];       // OVF: word offset of its first position past the lines, offset of those rows
#pragma unroll
  for (int k = 0; k < C; k++) {
    const int size = rows_group_size(C, S, k);
    const int c = rows_group_start(C, S, k) + ((k - rows_group_start(C, S, k)) ^ (sb & (size - 1)));
#pragma unroll
    for (int s = 0; s < (OVF ? 1 : Q); s++)
      lc[s][k] = L.t_base[c] + L.t_rep[c] * (sb >> rows_log2(size)) - p.tab_off[c] * L.t_mul[0] + ((s ^ hx) << 4);
    lim[k] = p.tab_off[c] + L.t_lines * p.groups;
    lo[k] = L.t_over[c] - lim[k] * L.t_mul[1] + (hx << 4);
  }
  // a row's offsets come two to a word: the byte selector of the half of the
  // k-th column (the other half when sb is odd)
  const uint32_t sel[2] = {(sb & 1) ? 0x4432u : 0x4410u, (sb & 1) ? 0x4410u : 0x4432u};
  unsigned char *const mst = buf + (tid / S) * 128;
  const uint32_t mpos = (((tid & (S - 1)) * Q + (hx ^ ((tid >> R::kLS) & (Q - 1)))) ^ warp) << 4;
  // phase B: part h of tiles 8 * oct .. + 7
  const int h = warp & (Q - 1), oct = warp >> R::kLQ, tl = lane >> 2, gl = lane & 3;
  const unsigned char *const mld = buf + ((oct * 8 + tl) * 32 / S) * 128 + gl * 4;
  const uint32_t lx = (uint32_t)(h ^ tl) << 4;
  // result lines: 32 words (eight 16-byte chunks, chunk c of line i at c ^ (i % 8):
  // the 128-byte swizzle of a TMA tile) in two regions of 128 lines: one
  // per quad of groups, or, with one quad, one per 32 tiles
  const int chunk = (2 * oct + (tl >> 2)) & 7;
  unsigned char *const mwr = buf + (Q == 2 ? h : oct >> 2) * 16384 + gl * 256 + (tl & 3) * 4;
  unsigned char *const mw0 = mwr + ((chunk ^ (2 * gl)) << 4), *const mw1 = mwr + 128 + ((chunk ^ (2 * gl) ^ 1) << 4);
  const bool used = 32 * g0 + 128 * h < (int)p.nslots;
  uint32_t cnt[16];  // matches of the lane's 32 slots, two 16-bit counters each
#pragma unroll
  for (int j = 0; j < 16; j++) cnt[j] = 0;
  // add the lane's counters to `to` (indexed by slot)
  auto flush = [&](auto &&add) {
#pragma unroll
    for (int j = 0; j < 32; j++) {
      uint32_t c = (cnt[j >> 1] >> (16 * (j & 1))) & 0xFFFFu;
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) c += __shfl_xor_sync(kFull, c, o);
      if (tl == 0 && c) add(32 * (4 * h + gl) + j, c);
    }
#pragma unroll
    for (int j = 0; j < 16; j++) cnt[j] = 0;
  };

  // The rows' table word offsets, two per word.  Over up to four columns the
  // next block's are loaded behind phase A; over more (16 bytes a row, too
  // many registers to hold) they are only brought to L2 there.
  constexpr int kOffWords = C <= 4 ? 2 : 4;
  constexpr bool kHold = C <= 4;
  uint32_t off[R::kRPT][kOffWords];
  auto take = [&](int j, uint64_t i) {  // offsets of row pre_row0 + i
    if constexpr (kOffWords == 2) {
      const uint2 v = __ldg(p.pre + i);
      off[j][0] = v.x;
      off[j][1] = v.y;
    } else {
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p.pre) + i);
      off[j][0] = v.x;
      off[j][1] = v.y;
      off[j][2] = v.z;
      off[j][3] = v.w;
    }
  };
  auto load_offsets = [&](uint64_t b) {
    const uint64_t row0 = b * R::kRows;
    if (row0 + R::kRows <= p.nrows) {
      const uint64_t i = row0 - p.row_begin + tid;
#pragma unroll
      for (int j = 0; j < R::kRPT; j++) take(j, i + j * 256);
    } else {  // rows past the table take its last row's offsets (their masks are zeroed)
#pragma unroll
      for (int j = 0; j < R::kRPT; j++) take(j, min(row0 + tid + j * 256, p.nrows - 1) - p.row_begin);
    }
  };
  uint64_t blk = block_begin + bid;
  if (kHold && blk < nblocks) load_offsets(blk);
  uint32_t bo = 0;  // byte offset of the block's buffer
  for (uint32_t n = 1; blk < nblocks; blk += nb, n++, bo ^= (nbuf - 1) * kRowsBuffer) {
    const bool full = (blk + 1) * R::kRows <= p.nrows;
    auto piece = [&](int j, int s) {  // part s ^ hx of the thread's row j
      return reinterpret_cast<uint4 *>(mst + bo + j * (256 / S * 128) + (mpos ^ (s << 4)));
    };
    if (!kHold) load_offsets(blk);
    // ---- A ----
#pragma unroll
    for (int j = 0; j < R::kRPT; j++) {
      uint32_t w[kOffWords];
#pragma unroll
      for (int i = 0; i < kOffWords; i++) w[i] = off[j][i];
#pragma unroll
      for (int c = 0; c < C; c += 4) {  // groups of four and eight: columns k ^ 2, k ^ 4
        if (rows_group_size(C, S, c) >= 4) rows_swap(w[c / 2], w[c / 2 + 1], sb & 2);
      }
      if (C == 8 && S == 8) {
        rows_swap(w[0], w[kOffWords - 2], sb & 4);
        rows_swap(w[1], w[kOffWords - 1], sb & 4);
      }
      uint32_t o[C];
#pragma unroll
      for (int k = 0; k < C; k++)
        o[k] = __byte_perm(w[k / 2], 0u, rows_group_size(C, S, k) >= 2 ? sel[k & 1] : 0x4410u);
      if (OVF) {  // byte offsets of part hx; part s ^ hx is 16 * s away by XOR
#pragma unroll
        for (int k = 0; k < C; k++) o[k] = o[k] < lim[k] ? o[k] * L.t_mul[0] + lc[0][k] : o[k] * L.t_mul[1] + lo[k];
      }
      auto at = [&](int k, int s) { return OVF ? o[k] ^ (s << 4) : o[k] * L.t_mul[0] + lc[OVF ? 0 : s][k]; };
#pragma unroll
      for (int s = 0; s < Q; s++) {
        uint4 m = *reinterpret_cast<const uint4 *>(tables + at(0, s));
#pragma unroll
        for (int k = 1; k < C; k++) {
          const uint4 t = *reinterpret_cast<const uint4 *>(tables + at(k, s));
          m.x &= t.x;
          m.y &= t.y;
          m.z &= t.z;
          m.w &= t.w;
        }
        *piece(j, s) = m;
      }
    }
    if (!full) {
#pragma unroll
      for (int j = 0; j < R::kRPT; j++)
        if (blk * R::kRows + tid + j * 256 >= p.nrows)
#pragma unroll
          for (int s = 0; s < Q; s++) *piece(j, s) = make_uint4(0, 0, 0, 0);
    }
    if (blk + nb < nblocks) {  // in flight during B and C
      if (kHold) {
        load_offsets(blk + nb);
      } else {  // 16 bytes a row: a 128-byte line is eight rows
        const uint64_t row = (blk + nb) * R::kRows + (uint64_t)tid * 8;
        if (tid < R::kRows / 8 && row < p.nrows)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint4 *>(p.pre) + (row - p.row_begin)));
      }
    }
    __syncthreads();
    // ---- B ----
    uint32_t x[32];
    if (used) {
#pragma unroll
      for (int r = 0; r < 32; r++) {
        const uint32_t e = (uint32_t)((r & (S - 1)) * Q + ((r >> R::kLS) & (Q - 1))) << 4;
        x[(r & 24) | (7 - (r & 7))] = *reinterpret_cast<const uint32_t *>(mld + bo + (r / S) * 128 + (e ^ lx));
      }
    }
    __syncthreads();  // the masks are in registers
    if (used) {
      transpose_octets(x);
#pragma unroll
      for (int j = 0; j < 32; j++) {
        *reinterpret_cast<uint32_t *>(((j & 1) ? mw1 : mw0) + bo + (j >> 1) * 1024) = x[j];
        cnt[j >> 1] += (uint32_t)__popc(x[j]) * p.cnt_mul[j & 1];  // (run-time 1, 65536: on the FMA pipe)
      }
      if ((n & 1023) == 0)  // a block adds at most 32 to a 16-bit counter
        flush([&](int slot, uint32_t c) {
          const int32_t q = (int32_t)__ldg(p.blob + p.slot_off + 32 * g0 + slot);
          if (q >= 0) atomicAdd(p.counts + q, (unsigned long long)c);
        });
    }
    // ---- C ----
    const uint64_t word = blk * R::kTiles;
    if (p.tma && word + R::kTiles <= p.words) {  // (TMA clips a box at 16 bytes, not at the last word)
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncthreads();
      if (tid == 0) {
        const uint32_t src = (uint32_t)__cvta_generic_to_shared(buf) + bo;
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const int line0 = 32 * g0 + (Q == 2 ? 128 * i : 0);
          if (line0 < (int)p.nslots)
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                             tmap),
                         "r"((uint32_t)word + (Q == 2 ? 0 : 32 * i)), "r"(line0), "r"(src + 16384 * i)
                         : "memory");
        }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        // the buffer that the next block fills has been read
        if (nbuf == 2) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      }
    } else {  // bitmaps in any order or at any alignment: eight lanes per line
      __syncthreads();
      const int c = lane & 7;
      for (int i = tid >> 3; i < 256; i += 32) {
        const int32_t q = (int32_t)__ldg(p.blob + p.slot_off + 32 * g0 + rows_slot(Q == 2 ? i : i & 127));
        if (q < 0) continue;
        const uint4 v = *reinterpret_cast<const uint4 *>(buf + bo + i * 128 + ((c ^ (i & 7)) << 4));
        const uint64_t w = word + (Q == 2 ? 0 : 32 * (i >> 7)) + c * 4;
        uint32_t *dst = p.out + (uint64_t)q * p.stride_words + w;
        if (p.vec_store && w + 4 <= p.words) {
          *reinterpret_cast<uint4 *>(dst) = v;
        } else {
          const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int k = 0; k < 4; k++)
            if (w + k < p.words) dst[k] = w4[k];
        }
      }
    }
    __syncthreads();
  }
  if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  __syncthreads();  // (the buffers are free)
  // counts: the CTA's sum per slot, then one atomic each
  uint32_t *sum = reinterpret_cast<uint32_t *>(buf);
  sum[tid] = 0;
  __syncthreads();
  if (used) flush([&](int slot, uint32_t c) { atomicAdd(&sum[slot], c); });
  __syncthreads();
  if (tid < 32 * KG && sum[tid]) {
    const int32_t q = (int32_t)__ldg(p.blob + p.slot_off + 32 * g0 + tid);
    if (q >= 0) atomicAdd(p.counts + q, (unsigned long long)sum[tid]);
  }
}

// A pass of up to 32 * G queries: one part of 4 or 8 groups (G = 4, 8), one of 8
// and one of 4 (G = 12: up to 384 queries), or two of 8 (G = 16).  The first
// p.split CTAs take the first part.
template <int C, int G, bool OVF>
__global__ void __launch_bounds__(256, 2) batch_rows_kernel(const __grid_constant__ BatchPass p,
                                                            const __grid_constant__ CUtensorMap tmap) {
  static_assert(G == 4 || G == 8 || G == 12 || G == 16, "parts of four and eight groups");
  if (G <= 8) {
    batch_rows_part<C, G == 4 ? 4 : 8, OVF, true>(p, p.lay[0], &tmap, 0, blockIdx.x, gridDim.x);
  } else if (G == 16) {
    const bool second = blockIdx.x >= p.split;
    batch_rows_part<C, 8, OVF, false>(p, p.lay[0], &tmap, second ? 8 : 0, blockIdx.x - (second ? p.split : 0),
                               second ? gridDim.x - p.split : p.split);
  } else if (blockIdx.x < p.split) {
    batch_rows_part<C, 8, OVF, false>(p, p.lay[0], &tmap, 0, blockIdx.x, p.split);
  } else {
    batch_rows_part<C, 4, OVF, false>(p, p.lay[1], &tmap, 8, blockIdx.x - p.split, gridDim.x - p.split);
  }
}

// Tensor map of a pass's bitmaps: nslots rows of p.words words from the
// pass's first bitmap on, boxes of 32 words x 128 rows; false when TMA
// cannot write them.
inline bool rows_tensor_map(const BatchPass &bp, uint32_t *first, CUtensorMap *map) {
  static const auto encode = []() -> PFN_cuTensorMapEncodeTiled {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult got;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &got) !=
            cudaSuccess ||
        got != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled>(fn);
  }();
  const cuuint64_t stride = bp.stride_words * 4;
  if (!encode || ((uintptr_t)first & 15) || stride % 16 || stride >= (1ull << 40) || bp.words >= (1ull << 31))
    return false;
  const cuuint64_t dim[2] = {bp.words, bp.nslots};
  const cuuint32_t box[2] = {32, 128}, step[2] = {1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, first, dim, &stride, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Table layout in shared memory of a part of kg groups of a pass of `groups`
// groups: as many lines as `limit` bytes hold beside the buffer, the
// positions past them packed behind.
inline RowsLayout rows_layout(const BatchPass &bp, int groups, int kg, size_t limit) {
  RowsLayout L;
  const int S = 32 / kg, C = bp.ncols;
  const uint32_t row = 4 * kg;  // bytes of a table row
  auto bytes = [&](uint32_t lines) {
    uint64_t at = 0;
    for (int c = 0; c < C; c++) {
      const int start = rows_group_start(C, S, c), size = rows_group_size(C, S, c);
      if (c == start) {
        uint32_t m = 0;
        for (int k = 0; k < size; k++) m = std::max(m, bp.m[c + k]);
        for (int k = 0; k < size; k++) {
          L.t_base[c + k] = (uint32_t)(at + k * row);
          L.t_rep[c + k] = size * row;
          L.t_nrep[c + k] = S / size;
        }
        at += (uint64_t)std::min(m + 1, lines) * 128;
      }
    }
    for (int c = 0; c < C; c++) {
      L.t_over[c] = (uint32_t)at;
      if (bp.m[c] + 1 > lines) at += (uint64_t)(bp.m[c] + 1 - lines) * row;
    }
    return at;
  };
  memset(&L, 0, sizeof L);
  uint32_t lo = 0, hi = 0;  // the most lines that fit
  for (int c = 0; c < C; c++) hi = std::max(hi, bp.m[c] + 1);
  L.t_ovf = bytes(hi) + kRowsBuffer > limit;
  while (L.t_ovf && hi - lo > 1) {
    const uint32_t mid = (lo + hi) / 2;
    (bytes(mid) + kRowsBuffer > limit ? hi : lo) = mid;
  }
  L.t_lines = L.t_ovf ? lo : hi;
  L.t_bytes = (uint32_t)bytes(L.t_lines);
  L.t_mul[0] = 128 / groups;
  L.t_mul[1] = row / groups;
  return L;
}
