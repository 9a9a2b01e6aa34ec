// CPU check of the parts of a batch plan that planner_check.cu does not look
// at (compiled and run by tests/test_planner_groups_cpu.py; no GPU needed):
//   * every group of passes sharing positions, of up to eight columns: union
//     positions and map entries against each pass's own boundaries;
//   * few-query passes as their kernel reads them: terms where they are
//     tested directly, else bounds, verdicts at every position, and the
//     bucket entries made from the shape, for values around every bound;
//   * first_bitmap: set only when the pass's queries write consecutive
//     bitmaps, and given up when one of them is dropped;
//   * a plan asked not to share positions has no trace of them.
// Usage: planner_groups_check SEED TRIALS; exit status 0 when every check holds.
#include "../rtscan_b200/csrc/batch.cu"

#include <cstdio>
#include <random>

namespace {

int g_fails = 0;
uint64_t g_groups = 0, g_wide = 0, g_lookups = 0, g_direct = 0, g_tables = 0, g_in_order = 0, g_given_up = 0;
#define CHECK(cond, ...)                     \
  do {                                       \
    if (!(cond)) {                           \
      std::fprintf(stderr, __VA_ARGS__);     \
      std::fprintf(stderr, "\n");            \
      if (++g_fails > 20) std::exit(1);      \
    }                                        \
  } while (0)

constexpr uintptr_t kColStride = 0x100000;
constexpr uint32_t kMax = 0xFFFFFFFFu;

std::vector<uint32_t> probes(const uint32_t *B, uint32_t m, std::mt19937_64 &rng) {
  std::vector<uint32_t> xs = {0u, 1u, kMax - 1, kMax};
  for (uint32_t i = 0; i < m; i++)
    for (int d = -1; d <= 1; d++) xs.push_back(B[i] + (uint32_t)d);
  for (int r = 0; r < 32; r++) xs.push_back((uint32_t)rng() >> (rng() % 32));
  return xs;
}

uint32_t position(const uint32_t *B, uint32_t m, uint32_t x) { return (uint32_t)(std::upper_bound(B, B + m, x) - B); }

template <class F>
void check_group(const rts::BatchPlan &plan, const rts::PreParams &P, size_t off, F &&slot_of, std::mt19937_64 &rng) {
  g_groups++;
  if (P.ncols > 4) g_wide++;
  CHECK(P.npass >= 1 && P.npass <= (P.ncols <= 4 ? rts::kMaxPrePasses : 2), "%d passes over %d columns share", P.npass,
        P.ncols);
  CHECK(P.blob_words * 4 <= 200 * 1024 && off + P.blob_words <= plan.blob.size(), "union blob of %u words", P.blob_words);
  const uint32_t *ub = plan.blob.data() + off;
  const int NW = (P.npass + 1) / 2;
  int fed = 0;
  for (const auto &b : plan.passes) {
    const int q = slot_of(b);
    if (q < 0) continue;
    fed++;
    CHECK(!b.few && b.variant == 4 && b.bp.ncols == P.ncols && q < P.npass, "a pass of %d columns in slot %d", b.bp.ncols, q);
    const uint32_t *pblob = plan.blob.data() + b.off;
    for (int c = 0; c < P.ncols; c++) {
      const rts::PreCol &pc = P.c[c];
      CHECK(pc.col == b.bp.col[c], "pass column %d is not union column %d", c, c);
      const uint32_t *Bu = ub + pc.bnd_off, *Bp = pblob + b.bp.bnd_off[c];
      for (uint32_t x : probes(Bu, pc.m, rng)) {
        const uint32_t upos = rts::pre_position(pc, ub, x);
        CHECK(upos == position(Bu, pc.m, x), "union column %d value %u: position %u", c, x, upos);
        const uint32_t want = b.bp.tab_off[c] + position(Bp, b.bp.m[c], x) * (uint32_t)b.groups;
        const uint32_t got = (ub[pc.map_off + upos * NW + q / 2] >> (16 * (q & 1))) & 0xFFFFu;
        CHECK(got == want, "column %d value %u: offset %u, want %u", c, x, got, want);
        g_lookups++;
      }
    }
  }
  CHECK(fed == P.npass, "%d passes fed, %d planned", fed, P.npass);
}

// The verdicts of value x on column c, as the kernel finds them: its bucket's
// entry, made from the bounds of the column, or a search among those inside.
uint32_t few_lookup(const rts::FewParams &f, int c, uint32_t x) {
  const rts::FewCol &col = f.shape[c];
  const rts::PreCol pc = rts::few_shape(col);
  const uint32_t *B = f.tab + col.at, *verdict = B + col.m;
  const uint32_t k = rts::pre_bucket(pc, x);
  CHECK(k < pc.nbk, "bucket %u of %u", k, pc.nbk);
  uint32_t lo = 0;
  while (lo < col.m && rts::pre_bucket(pc, B[lo]) < k) lo++;
  uint32_t hi = lo;
  while (hi < col.m && rts::pre_bucket(pc, B[hi]) == k) hi++;
  uint32_t pos = lo;
  if (hi > lo) {
    if (B[lo] == (uint64_t)pc.origin + rts::pre_bucket_start(pc.M, pc.L, k)) pos++;
    while (pos < hi && B[pos] <= x) pos++;
  }
  return verdict[pos];
}

void check_few(const rts::BatchPlan::Pass &b, std::mt19937_64 &rng) {
  const rts::FewPass &p = b.fp;
  const rts::FewParams &f = b.fk;
  CHECK(f.nq == p.nq, "%d queries, %d in the parameters", p.nq, f.nq);
  auto hits = [&](int j, int c, uint32_t x) { return x - p.term[j][c].x <= p.term[j][c].y; };
  const int direct = rts::few_direct_max(p.ncols);
  for (int c = 0; c < p.ncols; c++) {
    CHECK(f.col[c] == p.col[c], "column %d", c);
    if (p.nq <= direct) {
      for (int j = 0; j < direct; j++) {
        const uint32_t *t = f.tab + 2 * (j * p.ncols + c);
        CHECK(t[0] == p.term[j][c].x && t[1] == p.term[j][c].y, "slot %d column %d: term", j, c);
      }
      g_direct++;
      continue;
    }
    const rts::FewCol &col = f.shape[c];
    CHECK(col.m <= rts::kFewBounds && col.nbk <= 4096, "%u bounds, %u buckets", col.m, col.nbk);
    const uint32_t *B = f.tab + col.at;
    for (uint32_t i = 1; i < col.m; i++) CHECK(B[i - 1] < B[i], "bounds not increasing");
    for (uint32_t x : probes(B, col.m, rng)) {
      uint32_t want = 0;
      for (int j = 0; j < p.nq; j++) want |= hits(j, c, x) ? 1u << j : 0u;
      const uint32_t got = few_lookup(f, c, x);
      CHECK(got == want, "column %d value %u: verdicts %08x, want %08x", c, x, got, want);
      g_lookups++;
    }
    g_tables++;
  }
}

// The bitmaps of a table pass's queries, in the order of its result lines.
std::vector<int> bitmaps_of(const rts::BatchPlan &plan, const rts::BatchPlan::Pass &b) {
  std::vector<int> o;
  for (uint32_t i = 0; i < b.bp.nslots; i++)
    o.push_back((int)plan.blob[b.off + b.bp.slot_off + (b.variant == 4 ? rts::rows_slot((int)i) : (int)i)]);
  return o;
}

void check_first_bitmaps(rts::BatchPlan &plan, std::mt19937_64 &rng) {
  for (const auto &b : plan.passes) {
    if (b.few) continue;
    const std::vector<int> o = bitmaps_of(plan, b);
    bool run = true;
    for (size_t i = 0; i < o.size(); i++) run = run && o[i] == o[0] + (int)i;
    CHECK(b.bp.first_bitmap == (run ? o[0] : -1), "first bitmap %d of a pass starting at %d", b.bp.first_bitmap, o[0]);
    g_in_order += run;
  }
  std::vector<uint32_t> words;
  for (size_t i = 0; i < plan.passes.size(); i++) {
    if (plan.passes[i].few || rng() % 2) continue;
    const std::vector<int> o = bitmaps_of(plan, plan.passes[i]);
    std::vector<int> before;
    for (const auto &b : plan.passes) before.push_back(b.few ? -1 : b.bp.first_bitmap);
    rts::batch_plan_drop(plan, o[rng() % o.size()], words);
    for (size_t k = 0; k < plan.passes.size(); k++)
      if (!plan.passes[k].few)
        CHECK(plan.passes[k].bp.first_bitmap == (k == i ? -1 : before[k]), "pass %zu's first bitmap after a drop in pass %zu",
              k, i);
    g_given_up++;
  }
}

}  // namespace

int main(int argc, char **argv) {
  const uint64_t seed = argc > 1 ? std::strtoull(argv[1], nullptr, 10) : 1;
  const int trials = argc > 2 ? std::atoi(argv[2]) : 20;
  std::mt19937_64 rng(seed);
  const int counts[] = {2, 3, 4, 5, 6, 20, 31, 32, 64, 128, 129, 256, 300, 512, 700, 1400};
  for (int t = 0; t < trials; t++) {
    auto *ctx = new rts_ctx();  // never destroyed: it owns no device memory
    const int ncols = 1 + t % 8;
    for (int c = 0; c < ncols; c++) ctx->cols.push_back(reinterpret_cast<const uint32_t *>(kColStride * (c + 1)));
    ctx->nrows = rng() % 2 ? 1 << 20 : 1 << 23;
    ctx->sm_count = 148;
    const int nq = counts[rng() % (sizeof counts / sizeof counts[0])];
    // bounds at random, from a few values, or crowded near 3e9
    const int kind = (int)(rng() % 3);
    auto bound = [&]() -> uint32_t {
      if (kind == 0) return (uint32_t)rng() >> (rng() % 32);
      if (kind == 1) return (uint32_t)(rng() % 40) * 1000u;
      return rng() % 8 ? 3000000000u + (uint32_t)(rng() % 100) : (uint32_t)(rng() % 100);
    };
    std::vector<rts_term> terms;
    std::vector<int32_t> offsets = {0};
    for (int q = 0; q < nq; q++) {
      const int k = 1 + (int)(rng() % ncols);
      for (int i = 0; i < k; i++) {
        uint32_t a = bound(), b = bound();
        if (a > b) std::swap(a, b);
        terms.push_back({(int32_t)(rng() % ncols), rng() % 8 ? a : 0u, rng() % 8 ? b : kMax});
      }
      offsets.push_back((int32_t)terms.size());
    }
    std::vector<rts::NormQuery> norm = rts::normalize_all(ctx, terms.data(), offsets.data(), nq);
    std::vector<int> inside;
    for (int q = 0; q < nq; q++)
      if (rts::runs_in_kernel(norm[q])) inside.push_back(q);
    if (inside.empty()) continue;
    rts::BatchPlanPtr plan = rts::make_batch_plan(ctx, norm, inside, nullptr, ctx->batch_cfg.table_budget, true);
    if (plan->pre.npass)
      check_group(*plan, plan->pre, plan->pre_off, [](const rts::BatchPlan::Pass &b) { return b.pre_slot; }, rng);
    for (size_t g = 0; g < plan->groups.size(); g++)
      check_group(*plan, plan->groups[g].pre, plan->groups[g].off,
                  [g](const rts::BatchPlan::Pass &b) { return b.group == (int)g ? b.group_slot : -1; }, rng);
    for (const auto &b : plan->passes) {
      CHECK(b.few || b.pre_slot >= 0 || b.group >= 0, "a table pass that shares no positions");
      if (b.few) check_few(b, rng);
    }
    check_first_bitmaps(*plan, rng);
    // junk where the next plan will be made: members that nothing sets show up
    const size_t junk = sizeof(rts::BatchPlan);
    void *p = ::operator new(junk);
    memset(p, 0x5A, junk);
    ::operator delete(p);
    rts::BatchPlanPtr alone = rts::make_batch_plan(ctx, norm, inside, nullptr, ctx->batch_cfg.table_budget, false);
    CHECK(alone->pre.npass == 0 && alone->groups.empty(), "%d passes share positions in a plan asked not to",
          alone->pre.npass);
    for (const auto &b : alone->passes) CHECK(b.pre_slot < 0 && b.group < 0, "a pass has a slot for shared positions");
    CHECK(rts::batch_plan_scratch_bytes(*alone, ctx->nrows) == 0, "scratch for no shared positions");
  }
  if (g_fails) {
    std::fprintf(stderr, "%d checks failed\n", g_fails);
    return 1;
  }
  std::printf("plans ok: %llu groups, %llu over more than four columns, %llu lookups, %llu direct columns, %llu table columns, "
              "%llu passes in order, %llu given up\n",
              (unsigned long long)g_groups, (unsigned long long)g_wide, (unsigned long long)g_lookups,
              (unsigned long long)g_direct, (unsigned long long)g_tables, (unsigned long long)g_in_order,
              (unsigned long long)g_given_up);
  return 0;
}
