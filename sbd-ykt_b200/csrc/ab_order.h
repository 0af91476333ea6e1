// Ordering of one batch of the packed alpha-beta kernel's schedule (see
// ab_plan.cu), and the threads that order the batches. Host code without CUDA,
// so that the CPU tests compile it.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <exception>
#include <thread>
#include <utility>
#include <vector>

namespace sbdx {

// A record of the schedule: bits 0-11 pair index, 12-27 y slot, 31 same-spin
// sign, kAbPad: no single.
constexpr uint32_t kAbPad = 1u << 30;
constexpr int kAbWindow = 2;  // steps whose updates of y are disjoint (divides 4)

// job(j) for every j < jobs on up to `threads` threads, the caller's among
// them. What a job throws ends the remaining ones and is thrown again here,
// once every thread has been joined; threads that cannot be created are done
// without.
template <typename F>
void run_jobs(size_t jobs, size_t threads, F&& job) {
  std::atomic<size_t> next{0};
  std::atomic<bool> failed{false};
  std::exception_ptr first;
  auto work = [&]() noexcept {
    try {
      for (size_t j; !failed.load() && (j = next.fetch_add(1)) < jobs;) job(j);
    } catch (...) {
      if (!failed.exchange(true)) first = std::current_exception();
    }
  };
  struct Joined {
    std::vector<std::thread> th;
    ~Joined() {
      for (auto& t : th) t.join();
    }
  };
  {
    Joined g;
    try {
      if (threads > 1) g.th.reserve(threads - 1);
      for (size_t t = 1; t < threads; ++t) g.th.emplace_back(work);
    } catch (...) {  // no memory for or no permission to start another thread
    }
    work();
  }
  if (first) std::rethrow_exception(first);
}

constexpr uint16_t kNoPair = 0xffff;

struct AbSingle {
  uint32_t slot0;  // first y slot candidate list entry: local bra
  uint16_t pq;
  uint8_t neg;
};

// Work of one (panel, batch): lanes' lists in, ordered steps out.
struct AbBatch {
  int n = 0;                    // lanes in use
  std::vector<uint32_t> beg;    // [n + 1] into list
  std::vector<AbSingle> list;     // slot0 = local bra index
  uint32_t maxlen = 0;
  // out
  int steps = 0;
  std::vector<uint32_t> wsteps;   // per warp: last step with a record, plus one
  std::vector<uint32_t> rec;      // [ceil(steps / 4)][threads][4]
};

struct AbOrder {
  int nt, ny;
  const std::vector<uint32_t>& s0;  // y slots of local bra i: main i, extras nmain + s0[i] .. nmain + s0[i + 1]
  int nmain;
  double effort;  // descent moves per record

  int slots_of(uint32_t i) const { return 1 + (int)(s0[i + 1] - s0[i]); }
  uint32_t slot(uint32_t i, int k) const { return k == 0 ? i : (uint32_t)nmain + s0[i] + (uint32_t)(k - 1); }

  void run(AbBatch& B, uint64_t seed) const {
    if (B.list.empty()) {  // no lane, or none with a single: no step
      B.steps = 0;
      B.wsteps.assign((nt + 31) / 32, 0);
      B.rec.clear();
      return;
    }
    const int n = B.n, nq = (n + 7) / 8, nh = (n + 15) / 16;
    uint64_t rs = seed * 0x9e3779b97f4a7c15ull + 0x1234567ull;
    auto rnd = [&](uint32_t m) -> uint32_t {  // xorshift64*
      rs ^= rs >> 12; rs ^= rs << 25; rs ^= rs >> 27;
      return (uint32_t)(((rs * 0x2545f4914f6cdd1dull) >> 32) * (uint64_t)m >> 32);
    };
    const int n8 = (n + 15) & ~15;   // row stride: whole half-warps
    std::vector<uint16_t> gp;  // [step][lane] pair, kNoPair when idle
    std::vector<uint32_t> gy;  // y slot (bit 31: sign)
    std::vector<uint32_t> gb;  // local bra
    // singles per bank slot, one byte each: distinct pairs of a quarter-warp's
    // step by pair mod 8, y slots of a half-warp's step by slot mod 16
    std::vector<uint64_t> vc, yc;
    std::vector<uint8_t> used;
    std::vector<uint32_t> len(n), deg;
    std::vector<AbSingle> left = B.list;
    size_t rem = left.size();
    for (int i = 0; i < n; ++i) len[i] = B.beg[i + 1] - B.beg[i];
    deg.assign(nmain, 0);
    for (const AbSingle& s : left) ++deg[s.slot0];
    int T = 0;
    auto grow = [&]() {
      gp.resize((size_t)(T + 1) * n8, kNoPair);
      gy.resize((size_t)(T + 1) * n8, 0);
      gb.resize((size_t)(T + 1) * n8, 0);
      vc.resize((size_t)(T + 1) * nq, 0);
      yc.resize((size_t)(T + 1) * nh * 2, 0);
      used.resize((size_t)(T / kAbWindow + 1) * ny, 0);
    };
    auto one = [](uint32_t x) { return 1ull << (8 * x); };
    // whether another lane of lane i's quarter-warp takes the same pair in step m
    auto dup = [&](int m, int i, uint16_t pq) {
      const uint16_t* g = &gp[(size_t)m * n8 + (i & ~7)];
      int c = 0;
      for (int z = 0; z < 8; ++z) c += g[z] == pq;
      return c > (g[i & 7] == pq ? 1 : 0);
    };
    auto ybank = [&](int m, int i, uint32_t y) -> uint64_t& { return yc[((size_t)m * nh + (i >> 4)) * 2 + ((y >> 3) & 1)]; };
    auto put = [&](int m, int i, uint16_t pq, uint32_t y, uint32_t bra) {
      if (!dup(m, i, pq)) vc[(size_t)m * nq + (i >> 3)] += one(pq & 7);
      ybank(m, i, y) += one(y & 7);
      used[(size_t)(m / kAbWindow) * ny + (y & 0x7fffffffu)] = 1;
      gp[(size_t)m * n8 + i] = pq;
      gy[(size_t)m * n8 + i] = y;
      gb[(size_t)m * n8 + i] = bra;
    };
    // greedy: per step, lanes with the most singles left choose first
    std::vector<int> ord(n), bucket;
    while (rem) {
      grow();
      const int m = T++;
      uint32_t mx = 0;
      for (int i = 0; i < n; ++i) mx = std::max(mx, len[i]);
      bucket.assign(mx + 2, 0);
      for (int i = 0; i < n; ++i) ++bucket[mx - len[i] + 1];
      for (uint32_t k = 0; k <= mx; ++k) bucket[k + 1] += bucket[k];
      const int rot = (int)rnd((uint32_t)n);
      for (int j = 0; j < n; ++j) {
        const int i = j + rot < n ? j + rot : j + rot - n;
        ord[bucket[mx - len[i]]++] = i;
      }
      for (int j = 0; j < n; ++j) {
        const int i = ord[j];
        if (len[i] == 0) break;  // the rest are empty too
        AbSingle* l = left.data() + B.beg[i];
        const uint64_t cv = vc[(size_t)m * nq + (i >> 3)];
        const uint64_t* cy = &yc[((size_t)m * nh + (i >> 4)) * 2];
        int best = -1;
        uint32_t by = 0;
        float bc = 1e30f;
        for (uint32_t t = 0; t < len[i]; ++t) {
          const int ns = slots_of(l[t].slot0);
          const float pref = 0.02f * (float)deg[l[t].slot0] / (float)ns;  // crowded bra strings early
          const float cvv = 5.0f * (float)(dup(m, i, l[t].pq) ? 0 : (int)((cv >> (8 * (l[t].pq & 7))) & 0xff));
          if (cvv - pref >= bc) continue;
          for (int k = 0; k < ns; ++k) {
            const uint32_t s = slot(l[t].slot0, k);
            if (used[(size_t)(m / kAbWindow) * ny + s]) continue;
            const float cost = cvv + 2.0f * (float)((cy[(s >> 3) & 1] >> (8 * (s & 7))) & 0xff) - pref;
            if (cost < bc) { bc = cost; best = (int)t; by = s; }
          }
        }
        if (best < 0) continue;
        const AbSingle s = l[best];
        put(m, i, s.pq, by | ((uint32_t)s.neg << 31), s.slot0);
        --deg[s.slot0];
        l[best] = l[--len[i]];
        --rem;
      }
    }
    // descent: exchange two steps of one lane when the estimate does not grow
    const int nw = (nt + 31) / 32;
    B.wsteps.assign(nw, 0);
    for (int m = 0; m < T; ++m)
      for (int i = 0; i < n; ++i)
        if (gp[(size_t)m * n8 + i] != kNoPair) B.wsteps[i >> 5] = (uint32_t)(m + 1);
    // the largest byte of v (0 and 1 both cost one wavefront)
    auto most = [](uint64_t v) {
      int k = 1;
      while ((v + (uint64_t)(127 - k) * 0x0101010101010101ull) & 0x8080808080808080ull) ++k;
      return k;
    };
    auto cost = [&](uint64_t v, uint64_t y0, uint64_t y1) { return 5 * most(v) + 2 * std::max(most(y0), most(y1)); };
    // half-warp by half-warp (their steps stay in cache), kPasses times over
    constexpr int kPasses = 3;
    const long long moves = (long long)(effort * (double)B.list.size() / (kPasses * nh)) * kPasses * nh;
    for (long long it = 0; it < moves; ++it) {
      const int h0 = 16 * (int)(it / (moves / (kPasses * nh)) % nh);
      const int i = h0 + (int)rnd((uint32_t)std::min(16, n - h0));
      const uint32_t tw = B.wsteps[i >> 5];
      if (tw < 2) continue;
      const int m1 = (int)rnd(tw), m2 = (int)rnd(tw);
      const size_t p1 = (size_t)m1 * n8 + i, p2 = (size_t)m2 * n8 + i;
      const uint16_t pa = gp[p1], pb = gp[p2];
      if (m1 == m2 || pa == pb) continue;
      const uint32_t ya = gy[p1], yb = gy[p2];
      uint64_t &v1 = vc[(size_t)m1 * nq + (i >> 3)], &v2 = vc[(size_t)m2 * nq + (i >> 3)];
      if ((it & 7) != 0 && most(v1) == 1) continue;  // mostly steps with a conflict to resolve
      uint64_t *y1 = &yc[((size_t)m1 * nh + (i >> 4)) * 2], *y2 = &yc[((size_t)m2 * nh + (i >> 4)) * 2];
      uint64_t n1 = v1, n2 = v2, a1[2] = {y1[0], y1[1]}, a2[2] = {y2[0], y2[1]};
      const int w1 = m1 / kAbWindow, w2 = m2 / kAbWindow;
      // slots in the other window (the two singles vacate theirs)
      auto pick = [&](uint32_t bra, uint32_t y, int w, uint32_t vacant, bool has, uint32_t& out) {
        if (w1 == w2) { out = y; return true; }
        const int ns = slots_of(bra), st = ns > 1 ? (int)rnd((uint32_t)ns) : 0;
        for (int k = 0; k < ns; ++k) {
          const uint32_t s = slot(bra, ns > 1 ? (st + k) % ns : 0);
          if (!used[(size_t)w * ny + s] || (has && s == (vacant & 0x7fffffffu))) {
            out = s | (y & 0x80000000u);
            return true;
          }
        }
        return false;
      };
      uint32_t na = 0, nb = 0;
      if (pa != kNoPair && !pick(gb[p1], ya, w2, yb, pb != kNoPair, na)) continue;
      if (pb != kNoPair && !pick(gb[p2], yb, w1, ya, pa != kNoPair, nb)) continue;
      if (pa != kNoPair) {
        if (!dup(m1, i, pa)) n1 -= one(pa & 7);
        if (!dup(m2, i, pa)) n2 += one(pa & 7);
        a1[(ya >> 3) & 1] -= one(ya & 7);
        a2[(na >> 3) & 1] += one(na & 7);
      }
      if (pb != kNoPair) {
        if (!dup(m2, i, pb)) n2 -= one(pb & 7);
        if (!dup(m1, i, pb)) n1 += one(pb & 7);
        a2[(yb >> 3) & 1] -= one(yb & 7);
        a1[(nb >> 3) & 1] += one(nb & 7);
      }
      if (cost(n1, a1[0], a1[1]) + cost(n2, a2[0], a2[1]) > cost(v1, y1[0], y1[1]) + cost(v2, y2[0], y2[1])) continue;
      v1 = n1; v2 = n2;
      y1[0] = a1[0]; y1[1] = a1[1];
      y2[0] = a2[0]; y2[1] = a2[1];
      if (w1 != w2) {
        if (pa != kNoPair) used[(size_t)w1 * ny + (ya & 0x7fffffffu)] = 0;
        if (pb != kNoPair) used[(size_t)w2 * ny + (yb & 0x7fffffffu)] = 0;
        if (pa != kNoPair) used[(size_t)w2 * ny + (na & 0x7fffffffu)] = 1;
        if (pb != kNoPair) used[(size_t)w1 * ny + (nb & 0x7fffffffu)] = 1;
      }
      gp[p1] = pb; gp[p2] = pa;
      gy[p1] = nb; gy[p2] = na;
      std::swap(gb[p1], gb[p2]);
    }
    // records; an idle lane repeats a gather address of its quarter-warp (a broadcast)
    B.steps = T;
    const size_t nblk = ((size_t)T + 3) / 4;
    B.rec.assign(nblk * nt * 4, kAbPad);
    for (int m = 0; m < T; ++m)
      for (int i = 0; i < nt; ++i) {
        uint32_t r = kAbPad;
        if (i < n && gp[(size_t)m * n8 + i] != kNoPair) {
          const uint32_t y = gy[(size_t)m * n8 + i];
          r = (uint32_t)gp[(size_t)m * n8 + i] | ((y & 0xffffu) << 12) | (y & 0x80000000u);
        } else {
          const int q0 = i & ~7, q1 = std::min(n, q0 + 8);
          for (int z = q0; z < q1; ++z)
            if (gp[(size_t)m * n8 + z] != kNoPair) { r = kAbPad | gp[(size_t)m * n8 + z]; break; }
        }
        B.rec[((size_t)(m >> 2) * nt + i) * 4 + (m & 3)] = r;
      }
  }
};

}  // namespace sbdx
