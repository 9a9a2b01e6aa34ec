// CPU check of the server's error paths under threads (compiled and run by
// tests/test_server_errors_cpu.py; no GPU needed).  It includes the server's
// translation unit and calls a server that has no worker from many threads
// at once: producers refused by a full queue or for a bad term, waits that
// time out, polls, fetches and cancels of tickets that do not exist, and
// readers of the context's last message.  Every call's status and its
// thread's message are the call's own, and the context's message is always
// one of those messages, whole.
// Usage: server_errors_check ROUNDS; exit status 0 when every check holds.
#include "../rtscan_b200/csrc/serve.cpp"

#include <cstdio>
#include <cstdlib>
#include <set>

namespace {

std::atomic<int> g_fails{0};

void expect(bool ok, const char *what, const char *got) {
  if (!ok && g_fails++ < 20) std::fprintf(stderr, "%s: got \"%s\"\n", what, got);
}

// The calling thread's call returned rc; it must have failed as stated.
void refused(rts_status rc, rts_status want, const char *message) {
  expect(rc == want, message, std::to_string(rc).c_str());
  expect(std::string(rts_last_error(nullptr)) == message, message, rts_last_error(nullptr));
}

}  // namespace

int main(int argc, char **argv) {
  const int rounds = argc > 1 ? std::atoi(argv[1]) : 1000;
  auto *ctx = new rts_ctx();  // never destroyed: it owns no device memory
  ctx->cols.push_back(reinterpret_cast<const uint32_t *>(0x1000));
  ctx->nrows = 1 << 20;
  auto *srv = new rts_server();
  srv->ctx = ctx;
  srv->cfg.max_queue = 2;
  const rts_term good{0, 1, 2}, bad{7, 1, 2};
  uint64_t first = 0, ticket = 0;
  if (rts_server_submit(srv, &good, 1, &first) != RTS_OK || rts_server_submit(srv, &good, 1, &ticket) != RTS_OK) {
    std::fprintf(stderr, "an empty queue refused a request: %s\n", rts_last_error(nullptr));
    return 1;
  }
  const char *const messages[] = {"request queue full",    "term column out of range",
                                  "request not done within the timeout", "unknown ticket",
                                  "unknown or unfinished ticket", "bad submit arguments"};
  const std::set<std::string> known(messages, messages + 6);
  std::atomic<bool> go{false};
  std::vector<std::thread> threads;
  auto start = [&](auto &&body) {
    threads.emplace_back([&go, rounds, body] {
      while (!go.load()) std::this_thread::yield();
      for (int i = 0; i < rounds; i++) body();
    });
  };
  for (int k = 0; k < 2; k++) {
    start([&] {
      uint64_t t = 0;
      refused(rts_server_submit(srv, &good, 1, &t), RTS_ERR_FULL, messages[0]);
    });
    start([&] { refused(rts_server_wait(srv, first, 0, nullptr), RTS_ERR_TIMEOUT, messages[2]); });
  }
  start([&] {
    uint64_t t = 0;
    refused(rts_server_submit(srv, &bad, 1, &t), RTS_ERR_ARG, messages[1]);
    refused(rts_server_submit(srv, &good, 1, nullptr), RTS_ERR_ARG, messages[5]);
  });
  start([&] {
    int32_t done = 0;
    refused(rts_server_poll(srv, 99, &done, nullptr), RTS_ERR_ARG, messages[3]);
    refused(rts_server_fetch(srv, 99, nullptr, nullptr), RTS_ERR_ARG, messages[4]);
    refused(rts_server_cancel(srv, 99), RTS_ERR_ARG, messages[3]);
    rts_server_stats st;
    expect(rts_server_get_stats(srv, &st) == RTS_OK && st.queued == 2 && st.submitted == 2, "stats", "");
  });
  for (int k = 0; k < 2; k++)
    start([&] {
      const std::string m = rts_last_error(ctx);
      expect(m.empty() || known.count(m), "the context's message", m.c_str());
    });
  go = true;
  for (auto &t : threads) t.join();
  rts_server_stats st;
  expect(rts_server_get_stats(srv, &st) == RTS_OK && st.rejected == (uint64_t)(2 * rounds), "rejected requests",
         std::to_string(st.rejected).c_str());
  expect(known.count(rts_last_error(ctx)) == 1, "the context's last message", rts_last_error(ctx));
  if (g_fails) {
    std::fprintf(stderr, "%d checks failed\n", g_fails.load());
    return 1;
  }
  std::printf("server errors ok: %d rounds\n", rounds);
  return 0;
}
