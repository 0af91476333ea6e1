// The schedule of the packed alpha-beta kernel (sigma_ab_kernel, sigma.cu).
//
// For one group of alpha singles (ia; ja_r, pq_r, s_r) the kernel evaluates
//   y[ib] += s_b * sum_r s_r (pq_r|rs) C'[ja_r, jb]
// over the beta singles (ib <- jb, pair rs, sign s_b). A lane owns a ket string
// jb: the group's C'[ja_r, jb] sit in its registers, and each of its singles
// costs the gather of the group's integrals of the pair rs from shared memory
// and one read-add-write of y[ib], also in shared memory. This file arranges
// the singles of all kets into steps:
//   - a ket with many singles is split over several lanes, lanes are ordered
//     longest list first and cut into batches of one lane per thread;
//   - in a step every lane of the batch takes one of its singles (or none);
//     in a window of kAbWindow steps no two singles update the same y slot, so
//     the updates need no atomics and one synchronisation per window, and
//     every sum has one order; a bra string that a batch reaches more often
//     than it has windows gets several slots, added in slot order at the end;
//   - a quarter-warp's 128-bit integral gathers take one wavefront per distinct
//     pair in its most used 16-byte bank slot (pair mod 8), a half-warp's
//     64-bit y accesses one per lane in its most used bank pair (slot mod 16):
//     a greedy choice per step, then a seeded descent that exchanges two steps
//     of one lane, keep both near one. The descent's budget follows the pairs
//     that one product evaluates, so a problem whose product takes
//     microseconds is not given milliseconds of ordering.
// The restatement of the reference's task loop that these sums come from is
// chemistry/tpb/mult.h:453-489 (task type 0).
#include "sbdx_internal.cuh"

#include <algorithm>
#include <atomic>
#include <thread>

namespace sbdx {

namespace {

constexpr uint16_t kNone = 0xffff;

struct Single {
  uint32_t slot0;  // first y slot candidate list entry: local bra
  uint16_t pq;
  uint8_t neg;
};

// Work of one (panel, batch): lanes' lists in, ordered steps out.
struct Batch {
  int n = 0;                    // lanes in use
  std::vector<uint32_t> beg;    // [n + 1] into list
  std::vector<Single> list;     // slot0 = local bra index
  uint32_t maxlen = 0;
  // out
  int steps = 0;
  std::vector<uint32_t> wsteps;   // per warp: last step with a record, plus one
  std::vector<uint32_t> rec;      // [ceil(steps / 4)][threads][4]
};

struct Order {
  int nt, ny;
  const std::vector<uint32_t>& s0;  // y slots of local bra i: main i, extras nmain + s0[i] .. nmain + s0[i + 1]
  int nmain;
  double effort;  // descent moves per record

  int slots_of(uint32_t i) const { return 1 + (int)(s0[i + 1] - s0[i]); }
  uint32_t slot(uint32_t i, int k) const { return k == 0 ? i : (uint32_t)nmain + s0[i] + (uint32_t)(k - 1); }

  void run(Batch& B, uint64_t seed) const {
    const int n = B.n, nq = (n + 7) / 8, nh = (n + 15) / 16;
    uint64_t rs = seed * 0x9e3779b97f4a7c15ull + 0x1234567ull;
    auto rnd = [&](uint32_t m) -> uint32_t {  // xorshift64*
      rs ^= rs >> 12; rs ^= rs << 25; rs ^= rs >> 27;
      return (uint32_t)(((rs * 0x2545f4914f6cdd1dull) >> 32) * (uint64_t)m >> 32);
    };
    const int n8 = (n + 15) & ~15;   // row stride: whole half-warps
    std::vector<uint16_t> gp;  // [step][lane] pair, kNone when idle
    std::vector<uint32_t> gy;  // y slot (bit 31: sign)
    std::vector<uint32_t> gb;  // local bra
    // singles per bank slot, one byte each: distinct pairs of a quarter-warp's
    // step by pair mod 8, y slots of a half-warp's step by slot mod 16
    std::vector<uint64_t> vc, yc;
    std::vector<uint8_t> used;
    std::vector<uint32_t> len(n), deg;
    std::vector<Single> left = B.list;
    size_t rem = left.size();
    for (int i = 0; i < n; ++i) len[i] = B.beg[i + 1] - B.beg[i];
    deg.assign(nmain, 0);
    for (const Single& s : left) ++deg[s.slot0];
    int T = 0;
    auto grow = [&]() {
      gp.resize((size_t)(T + 1) * n8, kNone);
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
        Single* l = left.data() + B.beg[i];
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
        const Single s = l[best];
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
        if (gp[(size_t)m * n8 + i] != kNone) B.wsteps[i >> 5] = (uint32_t)(m + 1);
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
      if (pa != kNone && !pick(gb[p1], ya, w2, yb, pb != kNone, na)) continue;
      if (pb != kNone && !pick(gb[p2], yb, w1, ya, pa != kNone, nb)) continue;
      if (pa != kNone) {
        if (!dup(m1, i, pa)) n1 -= one(pa & 7);
        if (!dup(m2, i, pa)) n2 += one(pa & 7);
        a1[(ya >> 3) & 1] -= one(ya & 7);
        a2[(na >> 3) & 1] += one(na & 7);
      }
      if (pb != kNone) {
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
        if (pa != kNone) used[(size_t)w1 * ny + (ya & 0x7fffffffu)] = 0;
        if (pb != kNone) used[(size_t)w2 * ny + (yb & 0x7fffffffu)] = 0;
        if (pa != kNone) used[(size_t)w2 * ny + (na & 0x7fffffffu)] = 1;
        if (pb != kNone) used[(size_t)w1 * ny + (nb & 0x7fffffffu)] = 1;
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
        if (i < n && gp[(size_t)m * n8 + i] != kNone) {
          const uint32_t y = gy[(size_t)m * n8 + i];
          r = (uint32_t)gp[(size_t)m * n8 + i] | ((y & 0xffffu) << 12) | (y & 0x80000000u);
        } else {
          const int q0 = i & ~7, q1 = std::min(n, q0 + 8);
          for (int z = q0; z < q1; ++z)
            if (gp[(size_t)m * n8 + z] != kNone) { r = kAbPad | gp[(size_t)m * n8 + z]; break; }
        }
        B.rec[((size_t)(m >> 2) * nt + i) * 4 + (m & 3)] = r;
      }
  }
};

}  // namespace

void free_ab_plan(Ctx* c, AbPlan& P) {
  dev_free(c, P.vket);
  for (AbPanel& q : P.panels) {
    dev_free(c, q.rec); dev_free(c, q.boff); dev_free(c, q.bsteps); dev_free(c, q.wsteps);
    dev_free(c, q.ex_row); dev_free(c, q.ex_off);
  }
  P = AbPlan{};
}

// hs, off, rec: the beta singles by string (a string's list serves as bra
// and as ket list: pair and sign of a single are symmetric); alpha_singles:
// all alpha singles, for the ordering budget.
int build_ab_plan(Ctx* c, size_t n, const std::vector<uint32_t>& hs, const std::vector<uint64_t>& off,
                  const std::vector<uint64_t>& rec, uint64_t alpha_singles) {
  AbPlan& P = c->ab;
  free_ab_plan(c, P);
  uint64_t total = 0;
  for (size_t r = 0; r < n; ++r) total += hs[r];
  P.vstr = (uint32_t)((c->npair + 7) & ~(size_t)7);
  // lanes: (ket, part of its list); lists above 1.5 times the mean are split
  struct VKet { uint32_t ket, part, parts, len; };
  const uint32_t cap = std::max<uint32_t>(16, (uint32_t)((3 * total + 2 * n - 1) / (2 * std::max<size_t>(n, 1))));
  std::vector<VKet> vk;
  for (size_t k = 0; k < n; ++k) {
    if (hs[k] == 0) continue;
    const uint32_t p = (hs[k] + cap - 1) / cap;
    for (uint32_t j = 0; j < p; ++j) vk.push_back({(uint32_t)k, j, p, hs[k] / p + (j < hs[k] % p ? 1u : 0u)});
  }
  std::stable_sort(vk.begin(), vk.end(), [](const VKet& a, const VKet& b) { return a.len > b.len; });
  // Panels of bra strings whose y slots fit in shared memory beside the
  // integrals of kAbPacks packs (or one less, when that saves a panel); groups
  // of 4 consecutive columns go to the panels in turn, so that every panel
  // gets its share of each list. Slots: the panel's strings plus extras; their
  // room is estimated and checked below.
  auto fits = [&](int packs, size_t slots) {
    return 16 * (size_t)packs * P.vstr + sizeof(double) * slots + kAbStaticSmem <= kAbSmemBudget;
  };
  size_t np = 1;
  for (;; ++np) {
    const size_t per = (n + np - 1) / np + 4, est = per + per / 8 + 512;
    if (fits(kAbPacks, est) || (fits(kAbPacks - 1, est) && kAbPacks > 1)) break;
    if (per <= 8) break;
  }
  for (;; ++np) {
    const size_t per = (n + np - 1) / np + 4;
    const bool small = 16 * (size_t)kAbPacks * P.vstr + sizeof(double) * (per + per / 8 + 512) + kAbStaticSmem <=
                       kAbSmemBudget / 2;
    const int nt = small ? (vk.size() <= 256 ? 256 : 512) : (vk.size() <= 512 ? 512 : 1024);
    const size_t nbatch = std::max<size_t>(1, (vk.size() + nt - 1) / nt);
    const double effort =
        std::min(120.0, (double)alpha_singles * (double)total / 2e8);  // 2.4e10 pairs: 120 moves per record
    struct PanelWork {
      int nmain = 0, nex = 0, ny = 0;
      std::vector<uint32_t> s0, ex_row, ex_off;
      std::vector<Batch> b;
    };
    std::vector<PanelWork> W(np);
    bool ok = true;
    for (size_t q = 0; q < np; ++q) {
      PanelWork& w = W[q];
      for (size_t ib = 0; ib < n; ++ib) w.nmain += (ib / 4) % np == q;
      w.b.resize(nbatch);
      std::vector<uint32_t> need(w.nmain, 1), deg(w.nmain, 0);
      for (size_t b = 0; b < nbatch; ++b) {
        Batch& B = w.b[b];
        const size_t i0 = b * nt, i1 = std::min(vk.size(), i0 + nt);
        B.n = i1 > i0 ? (int)(i1 - i0) : 0;
        B.beg.assign(1, 0);
        for (size_t i = i0; i < i1; ++i) {
          const uint64_t* r = rec.data() + off[vk[i].ket];
          uint32_t m = 0, in = 0;
          for (uint32_t e = 0; e < hs[vk[i].ket]; ++e) in += np == 1 || (rec_ket(r[e]) / 4) % np == q;
          for (uint32_t e = 0; e < hs[vk[i].ket]; ++e) {
            const uint32_t ib = rec_ket(r[e]);
            if (np > 1 && (ib / 4) % np != q) continue;
            // this part's share of the panel's sub-list
            if ((uint64_t)m * vk[i].parts / in == vk[i].part) {
              const uint32_t loc = (uint32_t)(ib / (4 * np) * 4 + ib % 4);
              B.list.push_back({loc, (uint16_t)((r[e] >> 16) & 0xfffu), (uint8_t)((r[e] >> 40) & 1u)});
            }
            ++m;
          }
          B.beg.push_back((uint32_t)B.list.size());
          B.maxlen = std::max(B.maxlen, B.beg[B.beg.size() - 1] - B.beg[B.beg.size() - 2]);
        }
        for (const Single& s : B.list) ++deg[s.slot0];
        for (const Single& s : B.list) {
          if (deg[s.slot0] == 0) continue;
          // strings reached in nearly every window of the batch get more slots
          const double win = 0.85 * ((B.maxlen + kAbWindow - 1) / kAbWindow);
          const uint32_t x = (uint32_t)((deg[s.slot0] + win - 1e-9) / win);
          need[s.slot0] = std::max(need[s.slot0], x);
          deg[s.slot0] = 0;
        }
      }
      w.s0.assign(w.nmain + 1, 0);
      w.ex_off.assign(1, 0);
      for (int i = 0; i < w.nmain; ++i) {
        w.s0[i + 1] = w.s0[i] + need[i] - 1;
        if (need[i] > 1) {
          w.ex_row.push_back((uint32_t)i);
          w.ex_off.push_back(w.s0[i + 1]);
        }
      }
      w.nex = (int)w.ex_row.size();
      w.ny = w.nmain + (int)w.s0[w.nmain];
      int packs = 0;
      for (int k = 1; k <= kAbPacks; ++k)
        if (fits(k, w.ny)) packs = k;
      if (w.ny > 0xffff || packs < std::min(kAbPacks, 4)) { ok = false; break; }
    }
    if (!ok && np < n / 4 + 1) continue;
    if (!ok) {
      c->err = "build_connectivity: the alpha-beta schedule does not fit in shared memory";
      return SBDX_ERR_ARG;
    }
    // order the batches on several host threads (a batch's seed is its place, so the
    // result does not depend on the thread count)
    const size_t jobs = np * nbatch;
    std::atomic<size_t> next{0};
    auto work = [&]() {
      for (size_t j; (j = next.fetch_add(1)) < jobs;) {
        PanelWork& w = W[j / nbatch];
        const Order o{nt, w.ny, w.s0, w.nmain, effort};
        o.run(w.b[j % nbatch], j + 1);
      }
    };
    {
      const size_t hw = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
      const size_t nth = std::min({hw, jobs, (size_t)(total / 4096 + 1)});
      std::vector<std::thread> th;
      for (size_t t = 1; t < nth; ++t) th.emplace_back(work);
      work();
      for (auto& x : th) x.join();
    }
    // upload
    P.threads = nt;
    P.nbatch = (int)nbatch;
    P.np = (int)np;
    P.xs = nbatch * nt;
    std::vector<uint32_t> vket(P.xs, 0);
    for (size_t i = 0; i < vk.size(); ++i) vket[i] = vk[i].ket;
    auto up = [&](const auto& h, auto** d) -> int {
      using E = typename std::decay<decltype(h[0])>::type;
      SBDX_CUDA(c, dev_alloc(c, d, sizeof(E) * std::max<size_t>(1, h.size())));
      if (!h.empty()) SBDX_CUDA(c, cudaMemcpyAsync(*d, h.data(), sizeof(E) * h.size(), cudaMemcpyHostToDevice, c->stream));
      return 0;
    };
    int rc = up(vket, &P.vket);
    if (rc) return rc;
    P.panels.resize(np);
    for (size_t q = 0; q < np; ++q) {
      PanelWork& w = W[q];
      AbPanel& A = P.panels[q];
      A.nmain = w.nmain;
      A.nex = w.nex;
      A.ny = w.ny;
      std::vector<uint32_t> all, bsteps, wsteps;
      std::vector<uint64_t> boff;
      for (Batch& B : w.b) {
        boff.push_back(all.size() / 4);
        bsteps.push_back((uint32_t)B.steps);
        B.wsteps.resize(nt / 32, 0);
        wsteps.insert(wsteps.end(), B.wsteps.begin(), B.wsteps.end());
        all.insert(all.end(), B.rec.begin(), B.rec.end());
      }
      if ((rc = up(all, &A.rec)) || (rc = up(boff, &A.boff)) || (rc = up(bsteps, &A.bsteps)) ||
          (rc = up(wsteps, &A.wsteps)) || (rc = up(w.ex_row, &A.ex_row)) || (rc = up(w.ex_off, &A.ex_off)))
        return rc;
      SBDX_CUDA(c, cudaStreamSynchronize(c->stream));  // host vectors die here
    }
    return 0;
  }
}

}  // namespace sbdx
