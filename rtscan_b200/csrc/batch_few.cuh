// Batched kernel for passes of few queries (at most 31: included by batch.cu
// inside its anonymous namespace; uses kFull, kMaxCols, PreCol, pre_bucket(),
// transpose_octets() from there).
//
// Every row's verdict on a column, for all queries of the pass, is one word
// (bit j: query j), constant between the column's sorted distinct bounds.  A
// CTA builds, per column, a table of value buckets (the bucket shapes of the
// shared positions) whose entry is that word itself, or, for a bucket with a
// bound inside, where to search.  So a row costs a bucket number, one
// shared-memory load and an AND per column, whatever the number of queries; a
// warp gathers the words of its tile, each lane transposes 32 of them in
// registers (transpose_octets), and a query's words for the tile leave as one
// line straight from registers.  Passes of very few queries test their terms
// instead (few_direct).
//
// What bounds it: the column reads (HBM), then integer issue: about 12
// instructions per row and column, the transpose 7 per row; on small tables
// the latency of one tile (launch_few).  The bounds and verdicts travel in
// the kernel parameters, so a call uploads nothing.
//
// Measured on one 2^23-row segment of 4 columns (us; before: a term-by-term
// test of every row, one ballot per query and 32 rows, up to 20 queries, then
// a 128-slot table pass): 4 queries 54 -> 33, 8 queries 86 -> 43, 16 queries
// 131 -> 54, 31 queries 137 -> 58; the columns take 21 at the copy rate; on
// 2e5 rows 14.5 -> 8.6, 21 -> 10.6, 35 -> 12.6 and 19 -> 14.6.  A pass of 40
// queries takes 107 in the 128-slot table shape, hence as many queries here
// as a word holds.  At 16 queries: 3700 warp instructions per 1024 rows (12200
// before), issue 67 % busy, DRAM 134 MB.
constexpr int kFewSlots = 32;
// Bit 31 of a bucket entry marks a bucket to search, so 31 queries.
constexpr int kFewMaxQueries = 31;
constexpr int kFewBounds = 2 * kFewMaxQueries;
constexpr int kFewMaxWarps = 32;
constexpr int kFewSmWarps = 16;  // see launch_few
constexpr int kFewTileWords = 36 * 32;  // a warp's 1024 row words, 4 of padding per 32

// Most buckets per column of a pass over `ncols` columns of a table of nrows
// rows: a bucket with a bound inside is searched (20 bounds on a uniform
// column: 0.5 % of the rows with 4096 buckets), filling the table costs
// every CTA about 1 us per 4096 buckets and column.
constexpr uint32_t few_buckets(int ncols, uint64_t nrows) {
  return (nrows >= (1u << 22) ? 4096u : 1024u) / (ncols <= 4 ? 1 : 2);
}

// A column as the kernel sees it: its bucket shape (as in PreCol), its m
// bounds at tab[at], the verdicts at its m + 1 positions behind them.
struct FewCol {
  uint32_t origin, nbk;
  uint16_t at, m;
  uint8_t M, L, pad[2];
};
__host__ __device__ __forceinline__ PreCol few_shape(const FewCol &c) {
  PreCol pc{};
  pc.origin = c.origin;
  pc.nbk = c.nbk;
  pc.M = c.M;
  pc.L = c.L;
  pc.m = c.m;
  return pc;
}

// The kernel's parameters, packed and in the order of use: every CTA reads
// them through the constant cache, a miss per 64 bytes, before its first row
// (terms and bounds at fixed strides took 2-4 us a pass of four queries).
struct FewParams {
  const uint32_t *col[kMaxCols];
  uint32_t *out;
  unsigned long long *counts;
  uint64_t stride_words;
  uint64_t nrows;
  uint64_t words;
  uint64_t tile_begin;  // first tile of the range
  uint64_t ntiles;      // end of the range, in tiles
  int nq;
  int vec;              // every column 16-byte aligned
  int tile_groups;      // 128-row groups of a tile: 1, 2, 4 or 8
  FewCol shape[kMaxCols];
  int32_t slot_query[kFewSlots];  // bitmap index of slot s, -1 when unused
  uint32_t tab[kMaxCols * (2 * kFewBounds + 1)];
};

// A pass as it was planned.
struct FewPass {
  const uint32_t *col[kMaxCols];
  uint2 term[kFewSlots][kMaxCols];  // (lo, hi - lo) of slot s on pass column c; (0, 2^32 - 1) if unconstrained
  int32_t slot_query[kFewSlots];    // bitmap index of slot s, -1 when unused
  int nq;
  int ncols;
};

// Column c of a pass into the kernel's parameters (at word `at` of its
// tables; returns the word behind it): sorted distinct bounds B, bucket
// shape pc, and the verdicts.  A query's bit changes where its range begins
// and ends, so the verdicts are a running XOR.
inline uint32_t few_column(FewParams &fk, const FewPass &fp, int c, const std::vector<uint32_t> &B, const PreCol &pc,
                           uint32_t at) {
  FewCol &col = fk.shape[c];
  col.origin = pc.origin;
  col.nbk = pc.nbk;
  col.M = (uint8_t)pc.M;
  col.L = (uint8_t)pc.L;
  col.at = (uint16_t)at;
  col.m = (uint16_t)B.size();
  uint32_t *const bnd = fk.tab + at, *const verdict = bnd + B.size();
  std::copy(B.begin(), B.end(), bnd);
  std::fill(verdict, verdict + B.size() + 1, 0u);
  auto position = [&](uint32_t x) { return std::upper_bound(B.begin(), B.end(), x) - B.begin(); };
  for (int j = 0; j < fp.nq; j++) {
    const uint32_t lo = fp.term[j][c].x, hi = lo + fp.term[j][c].y;
    verdict[position(lo)] ^= 1u << j;
    if (hi < 0xFFFFFFFFu) verdict[position(hi + 1)] ^= 1u << j;
  }
  for (size_t k = 1; k <= B.size(); k++) verdict[k] ^= verdict[k - 1];
  return at + 2 * (uint32_t)B.size() + 1;
}

// Passes of at most this many queries test their terms directly: two
// instructions per term, fewer than a bucket's, and no tables to fill first.
// On 2^23 rows x 4 columns four queries take 33 us, through buckets 42 (58-69
// where the bounds crowd into one); over six columns four slots would take 66
// us (their terms do not fit the registers), two 50, buckets 52.
constexpr int few_direct_max(int ncols) { return ncols <= 4 ? 4 : 2; }

// Words of shared memory: per column its buckets, bounds, masks and the
// bounds' buckets, then the tile buffers and the counts.
constexpr uint32_t kFewColWords = 3 * 64;
inline size_t few_smem(const FewParams &p, int ncols, int tiles) {
  size_t w = (size_t)ncols * kFewColWords + tiles * kFewTileWords + 2 * kFewSlots;
  for (int c = 0; c < ncols; c++) w += p.shape[c].nbk;
  return w * 4;
}

// Fill the tables (every thread of the block): per column its bounds (at S),
// the verdicts at every position (at S + 64) and the bounds' buckets (at
// S + 128), S = cols_sm + c * kFewColWords; then the bucket entries: the
// verdicts when no bound lies above the bucket's first value, else bit 31 |
// their number << 16 | position of the first value (a thread fills a run of
// one column's buckets).
template <int C>
__device__ __forceinline__ void few_tables(const FewParams &p, uint32_t *cols_sm, uint32_t *bkt_sm) {
  const int tid = threadIdx.x;
  for (int i = tid; i < C * 64; i += blockDim.x) {
    const int c = i >> 6, k = i & 63;
    uint32_t *S = cols_sm + c * kFewColWords;
    const int m = p.shape[c].m;
    const uint32_t *tab = p.tab + p.shape[c].at;
    if (k < m) {
      const uint32_t b = tab[k];
      S[k] = b;
      S[128 + k] = pre_bucket(few_shape(p.shape[c]), b);
    }
    if (k <= m) S[64 + k] = tab[m + k];
  }
  __syncthreads();
  const int tpc = blockDim.x / C, c = min(tid / tpc, C - 1), t = tid - c * tpc;
  const int threads = c < C - 1 ? tpc : (int)blockDim.x - c * tpc;
  uint32_t *dst = bkt_sm;
  for (int i = 0; i < c; i++) dst += p.shape[i].nbk;
  const PreCol pc = few_shape(p.shape[c]);
  const uint32_t *S = cols_sm + c * kFewColWords;
  const uint32_t m = pc.m, per = (pc.nbk + threads - 1) / threads;
  const uint32_t k0 = min(t * per, pc.nbk), k1 = min(k0 + per, pc.nbk);
  if (k0 < k1) {
    uint32_t lo = 0;  // first bound whose bucket is >= k
    for (uint32_t n = m; n;) {
      const uint32_t h = n >> 1;
      if (S[128 + lo + h] < k0) {
        lo += h + 1;
        n -= h + 1;
      } else {
        n = h;
      }
    }
    uint32_t next = lo < m ? S[128 + lo] : kFull, pure = S[64 + lo];
    for (uint32_t k = k0; k < k1; k++) {
      uint32_t e = pure;
      if (next == k) {
        const bool at_start = (uint64_t)S[lo] == (uint64_t)pc.origin + pre_bucket_start(pc.M, pc.L, k);
        const uint32_t base = lo + at_start;
        do lo++;
        while (lo < m && S[128 + lo] == k);
        next = lo < m ? S[128 + lo] : kFull;
        pure = S[64 + lo];
        e = lo > base ? 0x80000000u | (lo - base) << 16 | base : pure;
      }
      dst[k] = e;
    }
  }
  __syncthreads();
}

// m[i]: the verdicts of four rows with column values x[c][i].
template <int C>
__device__ __forceinline__ void few_verdicts(const FewParams &p, const uint32_t *cols_sm,
                                             const uint32_t *bkt_sm, const uint32_t (&x)[C][4], uint32_t (&m)[4]) {
#pragma unroll
  for (int i = 0; i < 4; i++) m[i] = kFull;
  const uint32_t *bkt = bkt_sm;
#pragma unroll
  for (int c = 0; c < C; c++) {
    const FewCol &pc = p.shape[c];
    const uint32_t *S = cols_sm + c * kFewColWords;
    uint32_t e[4];
    {
      const uint32_t last = pc.nbk - 1;
      if (pc.M == 31) {  // linear buckets
#pragma unroll
        for (int i = 0; i < 4; i++) e[i] = bkt[min((max(x[c][i], pc.origin) - pc.origin) >> pc.L, last)];
      } else {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const uint32_t v = max(x[c][i], pc.origin) - pc.origin;
          const int s = max(31 - (int)pc.M - __clz(v), (int)pc.L);
          e[i] = bkt[min((((uint32_t)s - pc.L) << pc.M) + (v >> s), last)];
        }
      }
      bkt += pc.nbk;
      if ((e[0] | e[1] | e[2] | e[3]) >> 31) {
#pragma unroll
        for (int i = 0; i < 4; i++)
          if (e[i] >> 31) {
            uint32_t pos = e[i] & 0xFFFFu, n = (e[i] >> 16) & 0x7FFFu;
            while (n) {  // nearly always one bound, but a column's rows may crowd where its bounds do
              const uint32_t h = n >> 1;
              const bool up = S[pos + h] <= x[c][i];
              pos += up ? h + 1 : 0;
              n = up ? n - h - 1 : h;
            }
            e[i] = S[64 + pos];
          }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) m[i] &= e[i];
  }
}

// The same by the terms: slot j's term on column c is (tab[2 * (j * C + c)],
// its span behind it), always true for slots past the queries.
template <int C>
__device__ __forceinline__ void few_direct(const FewParams &p, const uint32_t (&x)[C][4], uint32_t (&m)[4]) {
#pragma unroll
  for (int i = 0; i < 4; i++) {
    m[i] = 0;
#pragma unroll
    for (int j = 0; j < few_direct_max(C); j++) {
      bool hit = true;
#pragma unroll
      for (int c = 0; c < C; c++) hit = hit && x[c][i] - p.tab[2 * (j * C + c)] <= p.tab[2 * (j * C + c) + 1];
      m[i] |= hit ? 1u << j : 0u;
    }
  }
}

// Column values of rows 4 * lane + i (vec) or 32 * i + lane (i < 4) of the
// 128 rows from row0 on.
template <int C>
__device__ __forceinline__ void few_load(const FewParams &p, uint64_t row0, bool vec, int lane, uint32_t (&x)[C][4]) {
  if (vec) {
#pragma unroll
    for (int c = 0; c < C; c++) {
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p.col[c] + row0) + lane);
      x[c][0] = v.x;
      x[c][1] = v.y;
      x[c][2] = v.z;
      x[c][3] = v.w;
    }
  } else {
#pragma unroll
    for (int c = 0; c < C; c++)
#pragma unroll
      for (int i = 0; i < 4; i++) x[c][i] = __ldg(p.col[c] + min(row0 + 32 * i + lane, p.nrows - 1));
  }
}

// The verdicts of those rows to the tile buffer (rows past the table: none).
__device__ __forceinline__ void few_store(const FewParams &p, uint32_t *tile_sm, uint64_t row0, int g, bool vec, int lane,
                                          const uint32_t (&m)[4]) {
  if (vec) {
    *reinterpret_cast<uint4 *>(tile_sm + (4 * g + (lane >> 3)) * 36 + 4 * (lane & 7)) =
        make_uint4(m[0], m[1], m[2], m[3]);
  } else {
#pragma unroll
    for (int i = 0; i < 4; i++) tile_sm[(4 * g + i) * 36 + lane] = row0 + 32 * i + lane < p.nrows ? m[i] : 0u;
  }
}

// The lane's 32 rows of a tile's verdicts, transposed: x[j] is query j's word.
__device__ __forceinline__ void few_words(const uint32_t *tile_sm, int lane, uint32_t (&x)[32]) {
#pragma unroll
  for (int r = 0; r < 32; r += 4) {
    const uint4 v = *reinterpret_cast<const uint4 *>(tile_sm + lane * 36 + r);
    x[(r & 24) | (7 - (r & 7))] = v.x;
    x[(r & 24) | (6 - (r & 7))] = v.y;
    x[(r & 24) | (5 - (r & 7))] = v.z;
    x[(r & 24) | (4 - (r & 7))] = v.w;
  }
  transpose_octets(x);
}

// A warp per tile of G * 128 rows, one CTA per SM.  SMALL: G as the launch
// chose it, else 8.  DIRECT: at most
// few_direct_max(C) queries, no tables.
template <int C, bool SMALL, bool DIRECT>
__global__ void __launch_bounds__(kFewMaxWarps * 32, 1) batch_few_kernel(const __grid_constant__ FewParams p) {
  extern __shared__ __align__(16) uint32_t few_sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
  uint32_t *tile_sm = few_sm + warp * kFewTileWords;
  unsigned long long *cnt = reinterpret_cast<unsigned long long *>(few_sm + warps * kFewTileWords);
  uint32_t *cols_sm = few_sm + warps * kFewTileWords + 2 * kFewSlots;
  uint32_t *bkt_sm = cols_sm + C * kFewColWords;
  const int nq = p.nq, G = SMALL ? p.tile_groups : 8;
  if (tid < kFewSlots) cnt[tid] = 0;
  if (DIRECT) __syncthreads();
  else few_tables<C>(p, cols_sm, bkt_sm);

  const uint64_t gw = (uint64_t)blockIdx.x * warps + warp, nw = (uint64_t)gridDim.x * warps;
  unsigned long long mine = 0;  // lane j: matches of query j in this warp's tiles
  for (uint64_t tile = p.tile_begin + gw; tile < p.ntiles; tile += nw) {
    const uint64_t row0 = tile * (128 * G), word = tile * (4 * G) + lane;
    const bool vec = p.vec && row0 + 128 * G <= p.nrows;
    uint32_t nxt[C][4];
    if (C <= 4) few_load<C>(p, row0, vec, lane, nxt);  // (over more columns two steps' values do not fit the registers)
    for (int g = 0; g < G; g++) {
      if (C > 4) few_load<C>(p, row0 + 128 * g, vec, lane, nxt);
      uint32_t x[C][4], m[4];
#pragma unroll
      for (int c = 0; c < C; c++)
#pragma unroll
        for (int i = 0; i < 4; i++) x[c][i] = nxt[c][i];
      if (C <= 4 && g < G - 1) few_load<C>(p, row0 + 128 * (g + 1), vec, lane, nxt);
      if (DIRECT) few_direct<C>(p, x, m);
      else few_verdicts<C>(p, cols_sm, bkt_sm, x, m);
      few_store(p, tile_sm, row0 + 128 * g, g, vec, lane, m);
    }
    __syncwarp();
    uint32_t x[32];
    few_words(tile_sm, lane, x);
    __syncwarp();
    const bool own = lane < 4 * G;
#pragma unroll
    for (int j = 0; j < (DIRECT ? few_direct_max(C) : kFewMaxQueries); j++) {
      if (j < nq) {
        const int32_t sq = p.slot_query[j];
        if (sq >= 0 && own && word < p.words) p.out[(uint64_t)sq * p.stride_words + word] = x[j];
        const uint32_t total = __reduce_add_sync(kFull, own ? (uint32_t)__popc(x[j]) : 0u);
        if (lane == j) mine += total;
      }
    }
  }
  if (lane < nq && mine) atomicAdd(&cnt[lane], mine);
  __syncthreads();
  if (tid < nq && cnt[tid] && p.slot_query[tid] >= 0) atomicAdd(p.counts + p.slot_query[tid], cnt[tid]);
}

template <int C, bool SMALL, bool DIRECT>
void launch_few_shape(const FewParams &fp, int sm_count, cudaStream_t s) {
  static std::atomic<uint64_t> raised{0};
  raise_smem_limit(batch_few_kernel<C, SMALL, DIRECT>, raised, 227 * 1024);
  const uint64_t tiles = fp.ntiles - fp.tile_begin, sms = (uint64_t)sm_count;
  // (at least eight warps to fill the tables)
  const int warps = (int)std::max<uint64_t>(8, std::min<uint64_t>(kFewMaxWarps, (tiles + sms - 1) / sms));
  const int grid = (int)std::max<uint64_t>(1, std::min<uint64_t>((tiles + warps - 1) / warps, sms));
  batch_few_kernel<C, SMALL, DIRECT><<<grid, warps * 32, few_smem(fp, C, warps), s>>>(fp);
}

// Rows [row_begin, fp.nrows).  Tiles of 1024 rows, of half, a quarter or an
// eighth of that while an SM has no more than kFewSmWarps of them: a warp
// goes through its tile 128 rows at a time, one load latency after another.
// (2e5 rows x 4 columns: tiles of 1024 rows take 31 queries 29 us, of 128
// rows 14.7; 1e6 rows 29 and 20.9; 2e6 rows of 512 or 1024 rows the same.)
template <int C>
void launch_few(FewParams &fp, uint64_t row_begin, int sm_count, cudaStream_t s) {
  const uint64_t rows = fp.nrows - row_begin, most = (uint64_t)sm_count * kFewSmWarps;
  fp.tile_groups = 1;
  while (fp.tile_groups < 8 && rows > most * 128 * fp.tile_groups) fp.tile_groups *= 2;
  const uint64_t tile_rows = 128 * (uint64_t)fp.tile_groups;
  fp.tile_begin = row_begin / tile_rows;
  fp.ntiles = (fp.nrows + tile_rows - 1) / tile_rows;
  if (fp.nq <= few_direct_max(C)) launch_few_shape<C, true, true>(fp, sm_count, s);
  else if (fp.tile_groups < 8) launch_few_shape<C, true, false>(fp, sm_count, s);
  else launch_few_shape<C, false, false>(fp, sm_count, s);
}
