// Batched kernel for passes of few queries (at most 31: included by batch.cu
// inside its anonymous namespace; uses kFull, kMaxCols, PreCol, pre_bucket(),
// transpose_octets() from there).
//
// Every row's verdict on a column, for all queries of the pass, is one word
// (bit j: query j), constant between the column's sorted distinct bounds.  A
// CTA builds, per column, a table of up to kFewBuckets value buckets (the
// bucket shapes of the shared positions) whose entry is that word itself, or,
// for a bucket with a bound inside, where to search.  So a row costs a bucket
// number, one shared-memory load and an AND per column, whatever the number
// of queries; a warp gathers the words of 1024 rows, each lane transposes 32
// of them in registers (transpose_octets), and a query's 32 words for the
// tile leave as one 128-byte line.
//
// What bounds it: the column reads (HBM), then integer issue: about 12
// instructions per row and column, the transpose 7 per row.  The terms
// travel in the kernel parameters, so a call uploads nothing.
//
// Measured on one 2^23-row segment of 4 columns (us; before: a term-by-term
// test of every row, one ballot per query and 32 rows, up to 20 queries, then
// a 128-slot table pass): 4 queries 57 -> 43, 8 queries 86 -> 45, 16 queries
// 133 -> 54, 31 queries 147 -> 63; the columns take 21 at the copy rate.  A
// pass of 40 queries takes 124 in the 128-slot table shape, hence as many
// queries here as a word holds.  At 16 queries: 3700 warp instructions per
// 1024 rows (12200 before), issue 67 % busy, DRAM 134 MB.
constexpr int kFewSlots = 32;
// Bit 31 of a bucket entry marks a bucket to search, so 31 queries.
constexpr int kFewMaxQueries = 31;
constexpr int kFewBounds = 2 * kFewMaxQueries;
constexpr int kFewMaxWarps = 32;
constexpr int kFewTileWords = 36 * 32;  // a warp's 1024 row words, 4 of padding per 32

// Most buckets per column of a pass over `ncols` columns of a table of nrows
// rows: a bucket with a bound inside is searched (20 bounds on a uniform
// column: 0.5 % of the rows with 4096 buckets), filling the table costs
// every CTA about 1 us per 4096 buckets and column.
constexpr uint32_t few_buckets(int ncols, uint64_t nrows) {
  return (nrows >= (1u << 22) ? 4096u : 1024u) / (ncols <= 4 ? 1 : 2);
}

struct FewPass {
  const uint32_t *col[kMaxCols];
  uint2 term[kFewSlots][kMaxCols];  // (lo, hi - lo) of slot s on pass column c; (0, 2^32 - 1) if unconstrained
  int32_t slot_query[kFewSlots];    // bitmap index of slot s, -1 when unused
  uint32_t bnd[kMaxCols][kFewBounds];  // sorted distinct bounds (lo and hi + 1) of column c
  PreCol shape[kMaxCols];           // its bucket shape (origin, M, L, nbk, m)
  int nq;
  int ncols;
  uint32_t *out;
  uint64_t stride_words;
  unsigned long long *counts;
  uint64_t nrows;
  uint64_t words;
  uint64_t tile_begin;  // first 1024-row tile of the range
  uint64_t ntiles;      // end of the range, in tiles
  int vec;              // every column 16-byte aligned
};

// Words of shared memory: per column its buckets, bounds, masks and the
// bounds' buckets, then the warps' tiles and the counts.
constexpr uint32_t kFewColWords = 3 * 64;
inline size_t few_smem(const FewPass &p, int warps) {
  size_t w = (size_t)p.ncols * kFewColWords + warps * kFewTileWords + 2 * kFewSlots;
  for (int c = 0; c < p.ncols; c++) w += p.shape[c].nbk;
  return w * 4;
}

template <int C>
__global__ void __launch_bounds__(kFewMaxWarps * 32, 1) batch_few_kernel(const __grid_constant__ FewPass p) {
  extern __shared__ __align__(16) uint32_t few_sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
  uint32_t *tile_sm = few_sm + warp * kFewTileWords;
  unsigned long long *cnt = reinterpret_cast<unsigned long long *>(few_sm + warps * kFewTileWords);
  uint32_t *cols_sm = few_sm + warps * kFewTileWords + 2 * kFewSlots;  // per column: bounds, masks, their buckets
  uint32_t *bkt_sm = cols_sm + C * kFewColWords;
  const int nq = p.nq;

  // per column: bounds, the mask of every position (its first value's), the bounds' buckets
  if (tid < kFewSlots) cnt[tid] = 0;
  for (int i = tid; i < C * 64; i += blockDim.x) {
    const int c = i >> 6, k = i & 63;
    uint32_t *S = cols_sm + c * kFewColWords;
    const int m = (int)p.shape[c].m;
    if (k < m) {
      S[k] = p.bnd[c][k];
      S[128 + k] = pre_bucket(p.shape[c], p.bnd[c][k]);
    }
    if (k <= m) {
      const uint32_t v = k ? p.bnd[c][k - 1] : 0u;
      uint32_t mask = 0;
      for (int j = 0; j < nq; j++) mask |= (v - p.term[j][c].x <= p.term[j][c].y ? 1u : 0u) << j;
      S[64 + k] = mask;
    }
  }
  __syncthreads();
  // bucket entries: the mask when no bound lies above the bucket's first
  // value, else bit 31 | their number << 16 | position of the first value
  // (a thread fills a run of one column's buckets)
  {
    const int tpc = blockDim.x / C, c = min(tid / tpc, C - 1), t = tid - c * tpc;
    const int threads = c < C - 1 ? tpc : (int)blockDim.x - c * tpc;
    uint32_t *dst = bkt_sm;
    for (int i = 0; i < c; i++) dst += p.shape[i].nbk;
    const PreCol &pc = p.shape[c];
    const uint32_t *S = cols_sm + c * kFewColWords;
    const uint32_t m = pc.m, per = (pc.nbk + threads - 1) / threads;
    const uint32_t k0 = min(t * per, pc.nbk), k1 = min(k0 + per, pc.nbk);
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

  const uint64_t gw = (uint64_t)blockIdx.x * warps + warp, nw = (uint64_t)gridDim.x * warps;
  unsigned long long mine = 0;  // lane j: matches of query j in this warp's tiles
  for (uint64_t tile = p.tile_begin + gw; tile < p.ntiles; tile += nw) {
    const uint64_t row0 = tile * 1024, word = tile * 32 + lane;
    const bool vec = p.vec && row0 + 1024 <= p.nrows;
    uint32_t nxt[C][4];
    // rows 4 * lane + i of 128 rows (vec), or 32 * i + lane
    auto load = [&](int g) {
      if (vec) {
#pragma unroll
        for (int c = 0; c < C; c++) {
          const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p.col[c] + row0 + 128 * g) + lane);
          nxt[c][0] = v.x;
          nxt[c][1] = v.y;
          nxt[c][2] = v.z;
          nxt[c][3] = v.w;
        }
      } else {
#pragma unroll
        for (int c = 0; c < C; c++)
#pragma unroll
          for (int i = 0; i < 4; i++)
            nxt[c][i] = __ldg(p.col[c] + min(row0 + 128 * g + 32 * i + lane, p.nrows - 1));
      }
    };
    if (C <= 4) load(0);  // (over more columns two steps' values do not fit the registers)
    for (int g = 0; g < 8; g++) {
      if (C > 4) load(g);
      uint32_t x[C][4];
#pragma unroll
      for (int c = 0; c < C; c++)
#pragma unroll
        for (int i = 0; i < 4; i++) x[c][i] = nxt[c][i];
      if (C <= 4 && g < 7) load(g + 1);
      uint32_t m[4] = {kFull, kFull, kFull, kFull};
      const uint32_t *bkt = bkt_sm;
#pragma unroll
      for (int c = 0; c < C; c++) {
        const PreCol &pc = p.shape[c];
        const uint32_t last = pc.nbk - 1;
        uint32_t e[4];
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
          const uint32_t *S = cols_sm + c * kFewColWords;
#pragma unroll
          for (int i = 0; i < 4; i++)
            if (e[i] >> 31) {
              uint32_t pos = e[i] & 0xFFFFu, n = (e[i] >> 16) & 0x7FFFu;
              while (n && S[pos] <= x[c][i]) {  // nearly always one bound
                pos++;
                n--;
              }
              e[i] = S[64 + pos];
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) m[i] &= e[i];
      }
      if (vec) {
        *reinterpret_cast<uint4 *>(tile_sm + (4 * g + (lane >> 3)) * 36 + 4 * (lane & 7)) =
            make_uint4(m[0], m[1], m[2], m[3]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; i++)
          tile_sm[(4 * g + i) * 36 + lane] = row0 + 128 * g + 32 * i + lane < p.nrows ? m[i] : 0u;
      }
    }
    __syncwarp();
    uint32_t x[32];
#pragma unroll
    for (int r = 0; r < 32; r += 4) {
      const uint4 v = *reinterpret_cast<const uint4 *>(tile_sm + lane * 36 + r);
      x[(r & 24) | (7 - (r & 7))] = v.x;
      x[(r & 24) | (6 - (r & 7))] = v.y;
      x[(r & 24) | (5 - (r & 7))] = v.z;
      x[(r & 24) | (4 - (r & 7))] = v.w;
    }
    __syncwarp();
    transpose_octets(x);
#pragma unroll
    for (int j = 0; j < kFewMaxQueries; j++) {
      if (j < nq) {
        const int32_t sq = p.slot_query[j];
        if (sq >= 0 && word < p.words) p.out[(uint64_t)sq * p.stride_words + word] = x[j];
        const uint32_t total = __reduce_add_sync(kFull, (uint32_t)__popc(x[j]));
        if (lane == j) mine += total;
      }
    }
  }
  if (lane < nq && mine) atomicAdd(&cnt[lane], mine);
  __syncthreads();
  if (tid < nq && cnt[tid] && p.slot_query[tid] >= 0) atomicAdd(p.counts + p.slot_query[tid], cnt[tid]);
}

// One CTA per SM; few tiles are spread over all SMs first.
template <int C>
void launch_few(const FewPass &fp, int sm_count, cudaStream_t s) {
  static std::atomic<uint64_t> raised{0};
  raise_smem_limit(batch_few_kernel<C>, raised, 227 * 1024);
  const uint64_t tiles = fp.ntiles - fp.tile_begin;
  const int warps =
      (int)std::max<uint64_t>(4, std::min<uint64_t>(kFewMaxWarps, (tiles + sm_count - 1) / (uint64_t)sm_count));
  const int grid =
      (int)std::max<uint64_t>(1, std::min<uint64_t>((tiles + warps - 1) / warps, (uint64_t)sm_count));
  batch_few_kernel<C><<<grid, warps * 32, few_smem(fp, warps), s>>>(fp);
}
