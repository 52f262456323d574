// Host model of the exchanges between the CTAs of a cluster (cuda_b200/csrc/cluster_exchange.h,
// lnt_cluster.cu) under random schedules and delays: one CTA quits, the others give up at
// waits that cannot end (or, at random, at one that could).  A barrier is never armed while its phase
// is open, its byte count stays within the 2^20 - 1 it can hold, and after the missing bytes are taken
// off, every phase completes exactly when the last word on its way has landed.
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>
#include "../../cuda_b200/csrc/cluster_exchange.h"

using namespace lnt;

struct Barrier {
  int64_t tx = 0;    // bytes expected less bytes landed, of the open phase
  bool armed = false;
  uint64_t phase = 0;
  void settle() {
    if (armed && tx == 0) {
      armed = false;
      phase++;
    }
  }
};
struct Cta {
  Barrier bar[3];
  uint64_t sent = 0, passed = 0;
  bool left = false, lost = false;
};
struct Word {
  uint32_t to;
  int b;
  uint32_t bytes;
};

static int fails = 0;
#define CHECK(c, ...) \
  do { if (!(c) && fails++ < 5) { std::printf(__VA_ARGS__); std::printf("\n"); } } while (0)

static void run(std::mt19937_64& rng, uint32_t C, uint32_t m, uint64_t squarings, uint64_t quit_at, bool impatient) {
  std::vector<Cta> cta(C);
  std::vector<Word> flying;
  auto expect = [&](uint32_t c, int b) {
    uint32_t bytes = 0;
    for (uint32_t f = 0; f < C; ++f) bytes += cluster::bytes_sent(b, f, c, C, m);
    Barrier& k = cta[c].bar[b];
    CHECK(!k.armed, "armed twice");
    k.armed = true;
    k.tx += bytes;
    k.settle();
  };
  for (uint32_t c = 0; c < C; ++c)
    for (int b = 0; b < 3; ++b) expect(c, b);
  auto land = [&](size_t i) {
    const Word w = flying[i];
    flying[i] = flying.back();
    flying.pop_back();
    Barrier& k = cta[w.to].bar[w.b];
    k.tx -= w.bytes;
    CHECK(k.tx > -(1 << 20) && k.tx < (1 << 20), "count out of range");
    k.settle();
  };
  auto leave = [&](Cta& x, bool lost) {
    x.left = true;
    x.lost = lost;
  };
  for (;;) {
    bool moved = false;
    for (uint32_t step = 0; step < 4 * C; ++step) {
      if (!flying.empty() && rng() % 3) {
        land(rng() % flying.size());
        moved = true;
        continue;
      }
      const uint32_t c = (uint32_t)(rng() % C);
      Cta& x = cta[c];
      if (x.left) continue;
      if (x.sent == x.passed) {  // between exchanges
        if (x.passed == 3 * squarings) leave(x, false);
        else if (c == 0 && x.passed == 3 * quit_at) leave(x, true);
        else {
          const int b = (int)(x.sent % 3);
          for (uint32_t to = 0; to < C; ++to)
            for (uint32_t left = cluster::bytes_sent(b, c, to, C, m); left;) {
              const uint32_t piece = left > 64 ? left / 2 / 8 * 8 : left;
              flying.push_back({to, b, piece});
              left -= piece;
            }
          x.sent++;
        }
        moved = true;
        continue;
      }
      const int b = (int)(x.passed % 3);
      const bool arrived = x.bar[b].phase > x.passed / 3;
      if (impatient && rng() % 200 == 0) {  // some thread gave up, others may have seen the phase end
        leave(x, true);
        moved = true;
      } else if (arrived) {
        expect(c, b);
        x.passed++;
        moved = true;
      }
    }
    if (moved || !flying.empty()) continue;
    bool waiting = false;
    for (Cta& x : cta)
      if (!x.left) {
        waiting = true;
        leave(x, true);  // nothing can arrive: the wait runs out
        break;
      }
    if (!waiting) break;
  }
  std::vector<uint64_t> sent(C);
  for (uint32_t c = 0; c < C; ++c) sent[c] = cta[c].sent;
  for (uint32_t c = 0; c < C; ++c) {
    Cta& x = cta[c];
    if (!x.lost) {
      CHECK(x.passed == 3 * squarings && x.sent == x.passed, "left early");
      continue;
    }
    for (int b = 0; b < 3; ++b) {
      Barrier& k = x.bar[b];
      const uint64_t phase = cluster::armed(x.passed, b) - 1;
      const uint32_t missing = cluster::bytes_missing(b, x.passed, sent.data(), c, C, m);
      if (k.armed) {
        CHECK(k.phase == phase, "phase %llu open, %llu armed", (unsigned long long)k.phase, (unsigned long long)phase);
        CHECK(k.tx == (int64_t)missing, "C %u barrier %d: %lld bytes open, %u missing", C, b, (long long)k.tx, missing);
      } else {
        CHECK(k.phase == phase + 1 && k.tx == 0 && missing == 0, "a phase not re-armed holds words");
      }
    }
  }
}

int main() {
  std::mt19937_64 rng(5);
  for (uint32_t C : {4u, 8u, 16u})
    for (int rep = 0; rep < 400; ++rep) {
      const uint64_t squarings = 1 + rng() % 6;
      const uint32_t m = 64u << (rng() % 6);
      if (8 * C > m) continue;
      run(rng, C, m, squarings, rep % 4 == 3 ? squarings : rng() % squarings, rep % 2 == 0);
    }
  if (fails) {
    std::printf("FAILED %d\n", fails);
    return 1;
  }
  std::printf("ok\n");
  return 0;
}
