// GPU check of the table passes that search their own positions
// (batch4_kernel; compiled and run by tests/test_gpu_search_passes.py).  A
// plan's passes run that way when the device has no room for its shared
// positions; here every plan is launched without scratch, whole and in two
// row ranges, with a query dropped, and compared with the terms row by row.
// Usage: search_passes_check SEED; exit status 0 when every result is right.
#include "../rtscan_b200/csrc/batch.cu"

#include <cstdio>
#include <random>

namespace {

#define CU(call)                                                                    \
  do {                                                                              \
    const cudaError_t e_ = (call);                                                  \
    if (e_ != cudaSuccess) {                                                        \
      std::fprintf(stderr, "%s: %s\n", #call, cudaGetErrorString(e_));              \
      std::exit(2);                                                                 \
    }                                                                               \
  } while (0)

int g_fails = 0;

uint32_t draw(std::mt19937_64 &rng, int kind) {
  return kind == 0 ? (uint32_t)rng() : kind == 1 ? (uint32_t)(rng() % 100) : (uint32_t)rng() >> (rng() % 32);
}

void run(std::mt19937_64 &rng, int ncols, int nq, int warps, uint64_t n) {
  std::vector<std::vector<uint32_t>> cols(ncols, std::vector<uint32_t>(n));
  auto *ctx = new rts_ctx();  // (its columns are freed below)
  cudaDeviceProp prop;
  CU(cudaGetDeviceProperties(&prop, 0));
  ctx->sm_count = prop.multiProcessorCount;
  ctx->nrows = n;
  ctx->batch_cfg.warps_per_cta = warps;
  std::vector<uint32_t *> dev(ncols);
  for (int c = 0; c < ncols; c++) {
    for (auto &v : cols[c]) v = draw(rng, c % 3);
    CU(cudaMalloc(&dev[c], n * 4));
    CU(cudaMemcpy(dev[c], cols[c].data(), n * 4, cudaMemcpyHostToDevice));
    ctx->cols.push_back(dev[c]);
  }
  std::vector<rts_term> terms;
  std::vector<int32_t> offsets = {0};
  for (int q = 0; q < nq; q++) {
    const int k = 1 + (int)(rng() % std::min(ncols, 4));
    for (int i = 0; i < k; i++) {
      const int c = (int)((q + i) % ncols);
      uint32_t a = draw(rng, c % 3), b = draw(rng, c % 3);
      if (a > b) std::swap(a, b);
      terms.push_back({c, rng() % 4 ? a : 0u, b});
    }
    offsets.push_back((int32_t)terms.size());
  }
  std::vector<rts::NormQuery> norm = rts::normalize_all(ctx, terms.data(), offsets.data(), nq);
  std::vector<int> inside;
  for (int q = 0; q < nq; q++)
    if (rts::runs_in_kernel(norm[q])) inside.push_back(q);
  rts::BatchPlanPtr plan = rts::make_batch_plan(ctx, norm, inside, nullptr, ctx->batch_cfg.table_budget, true);
  const uint64_t words = rts::words_for(n), stride = (words + 3) / 4 * 4;
  uint32_t *blob, *out;
  unsigned long long *counts;
  CU(cudaMalloc(&out, (size_t)nq * stride * 4));
  CU(cudaMalloc(&counts, nq * 8));
  std::vector<uint32_t> got((size_t)nq * stride), want(stride);
  std::vector<unsigned long long> cnt(nq);
  CU(cudaMalloc(&blob, plan->blob.size() * 4));
  for (int round = 0; round < 2; round++) {  // the whole table; then two row ranges without the query in the middle
    const int dropped = round ? inside[inside.size() / 2] : -1;
    std::vector<uint32_t> changed;
    if (round) rts::batch_plan_drop(*plan, dropped, changed);
    CU(cudaMemcpy(blob, plan->blob.data(), plan->blob.size() * 4, cudaMemcpyHostToDevice));
    CU(cudaMemset(out, 0xAB, (size_t)nq * stride * 4));
    CU(cudaMemset(counts, 0, nq * 8));
    const uint64_t cut = round ? std::min<uint64_t>(n, 4096) : n;
    rts::launch_batch_plan(ctx, *plan, blob, out, stride, counts, 0, cut, nullptr, 0, nullptr);
    if (cut < n) rts::launch_batch_plan(ctx, *plan, blob, out, stride, counts, cut, n, nullptr, 0, nullptr);
    CU(cudaDeviceSynchronize());
    CU(cudaMemcpy(got.data(), out, got.size() * 4, cudaMemcpyDeviceToHost));
    CU(cudaMemcpy(cnt.data(), counts, nq * 8, cudaMemcpyDeviceToHost));
    for (int q : inside) {
      std::fill(want.begin(), want.end(), 0u);
      unsigned long long c = 0;
      for (uint64_t r = 0; r < n; r++) {
        bool hit = true;
        for (size_t k = 0; k < norm[q].cols.size() && hit; k++) {
          const uint32_t v = cols[norm[q].cols[k]][r];
          hit = norm[q].lo[k] <= v && v <= norm[q].hi[k];
        }
        if (hit) want[r / 32] |= 0x80000000u >> (r % 32), c++;
      }
      bool same = cnt[q] == (q == dropped ? 0 : c);
      for (uint64_t w = 0; w < words && same; w++) same = got[q * stride + w] == (q == dropped ? 0xABABABABu : want[w]);
      if (!same && g_fails++ < 10)
        std::fprintf(stderr, "%d columns, %d queries, %d warps, %llu rows, round %d: query %d differs\n", ncols, nq, warps,
                     (unsigned long long)n, round, q);
    }
  }
  CU(cudaFree(blob));
  CU(cudaFree(out));
  CU(cudaFree(counts));
  for (auto *d : dev) CU(cudaFree(d));
  ctx->cols.clear();
}

}  // namespace

int main(int argc, char **argv) {
  std::mt19937_64 rng(argc > 1 ? std::strtoull(argv[1], nullptr, 10) : 1);
  int cases = 0;
  for (int ncols : {1, 3, 4, 5, 8})
    for (int nq : {40, 129, 200, 257, 500})
      for (int warps : {8, 16})
        for (uint64_t n : {(uint64_t)31, (uint64_t)4096 + 1025, (uint64_t)33000}) {
          run(rng, ncols, nq, warps, n);
          cases++;
        }
  if (g_fails) {
    std::fprintf(stderr, "%d results differ\n", g_fails);
    return 1;
  }
  std::printf("search passes ok: %d cases\n", cases);
  return 0;
}
