// The alpha-beta schedule's host side (csrc/ab_order.h) on the CPU:
//   ab_order jobs  what a job throws on another thread reaches the caller
//   ab_order order the ordered steps of small batches hold every single once,
//                  with the y slots of a window disjoint
// Exits 0 when all checks hold; built with the undefined-behaviour sanitizer.
#include "ab_order.h"

#include <cstdio>
#include <cstring>
#include <map>
#include <new>
#include <random>
#include <stdexcept>
#include <string>

using namespace sbdx;

#define CHECK(x) \
  do { \
    if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } \
  } while (0)

static int jobs_case() {
  for (size_t threads : {1, 2, 8}) {
    std::vector<std::atomic<int>> ran(1000);
    run_jobs(ran.size(), threads, [&](size_t j) { ++ran[j]; });
    for (auto& x : ran) CHECK(x.load() == 1);
    // the first job holds its thread until another one has thrown
    for (int kind = 0; kind < 2; ++kind) {
      std::atomic<bool> thrown{false};
      std::atomic<int> after{0};
      bool caught = false;
      try {
        run_jobs(1000, threads, [&](size_t j) {
          if (threads > 1 && j == 0)
            for (int k = 0; k < 2000 && !thrown.load(); ++k) std::this_thread::sleep_for(std::chrono::milliseconds(1));
          if (j == (threads > 1 ? 1u : 0u)) {
            thrown = true;
            if (kind == 0) throw std::bad_alloc();
            throw std::runtime_error("job");
          }
          if (j > 1 && thrown.load()) ++after;
        });
      } catch (const std::bad_alloc&) {
        caught = kind == 0;
      } catch (const std::runtime_error& e) {
        caught = kind == 1 && std::string(e.what()) == "job";
      }
      CHECK(caught);
      CHECK(after.load() < 900);  // the remaining jobs are given up
    }
  }
  return 0;
}

static int order_case() {
  std::mt19937 rng(7);
  auto pick = [&](uint32_t m) { return (uint32_t)(rng() % m); };
  for (int nt : {32, 256})
    for (int n : {0, 1, 7, 8, 9, 15, 16, 17, 31, 32})
      for (int most : {0, 1, 5, 40})
        for (int nmain : {1, 4, 60})
          for (double effort : {0.0, 3.0}) {
            AbBatch B;
            B.n = n;
            B.beg.assign(1, 0);
            std::vector<uint32_t> deg(nmain, 0);
            for (int i = 0; i < n; ++i) {
              const uint32_t len = most ? pick(most + 1) : 0;
              for (uint32_t k = 0; k < len; ++k) {
                B.list.push_back({pick(nmain), (uint16_t)pick(300), (uint8_t)pick(2)});
                ++deg[B.list.back().slot0];
              }
              B.beg.push_back((uint32_t)B.list.size());
              B.maxlen = std::max(B.maxlen, len);
            }
            std::vector<uint32_t> s0(nmain + 1, 0);
            for (int i = 0; i < nmain; ++i) s0[i + 1] = s0[i] + deg[i] / 16;
            const int ny = nmain + (int)s0[nmain];
            const AbOrder o{nt, ny, s0, nmain, effort};
            o.run(B, 11);
            CHECK(B.steps >= (int)B.maxlen);
            CHECK(B.rec.size() == (size_t)((B.steps + 3) / 4) * nt * 4);
            CHECK(B.wsteps.size() == (size_t)(nt + 31) / 32);
            auto bra_of = [&](uint32_t y) {
              if (y < (uint32_t)nmain) return y;
              uint32_t i = 0;
              while (s0[i + 1] <= y - nmain) ++i;
              return i;
            };
            using Key = std::pair<uint32_t, std::pair<uint32_t, uint32_t>>;  // bra, pair, sign
            for (int i = 0; i < nt; ++i) {
              std::map<Key, int> left;
              if (i < n)
                for (uint32_t k = B.beg[i]; k < B.beg[i + 1]; ++k) ++left[{B.list[k].slot0, {B.list[k].pq, B.list[k].neg}}];
              for (int m = 0; m < B.steps; ++m) {
                const uint32_t r = B.rec[((size_t)(m >> 2) * nt + i) * 4 + (m & 3)];
                if (r & kAbPad) continue;
                CHECK((uint32_t)m < B.wsteps[i >> 5]);
                const Key k{bra_of((r >> 12) & 0xffffu), {r & 0xfffu, r >> 31}};
                CHECK(left.count(k) && left[k] > 0);
                if (--left[k] == 0) left.erase(k);
              }
              CHECK(left.empty());
            }
            for (int w = 0; w < B.steps; w += kAbWindow) {
              std::vector<int> used(ny, 0);
              for (int m = w; m < std::min(B.steps, w + kAbWindow); ++m)
                for (int i = 0; i < nt; ++i) {
                  const uint32_t r = B.rec[((size_t)(m >> 2) * nt + i) * 4 + (m & 3)];
                  if (r & kAbPad) continue;
                  const uint32_t y = (r >> 12) & 0xffffu;
                  CHECK(y < (uint32_t)ny);
                  CHECK(used[y]++ == 0);
                }
            }
          }
  return 0;
}

int main(int argc, char** argv) {
  if (argc == 2 && !std::strcmp(argv[1], "jobs")) return jobs_case();
  if (argc == 2 && !std::strcmp(argv[1], "order")) return order_case();
  return 2;
}
