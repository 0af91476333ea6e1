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
#include <thread>

namespace sbdx {

void free_ab_plan(Ctx* c, AbPlan& P) {
  dev_free(c, P.vket); dev_free(c, P.pairs); dev_free(c, P.V); dev_free(c, P.V32);
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
  // The pairs in use. A sample of 150 strings has singles for a few of the 1711
  // pairs of 58 orbitals, and staging the integrals of all of them took longer
  // than using them: alpha-beta time of 8000 x 150 strings (7 electrons) 1549 us
  // FP64 and 1073 us FP32 with all pairs, 406 and 291 us with these; 5000 x 200
  // 991 and 677, 516 and 345 us; 8000 x 8000, where nearly all are used, the same.
  std::vector<uint32_t> pairs, pair_at(c->npair, 0);
  for (size_t r = 0; r < n; ++r)
    for (uint32_t e = 0; e < hs[r]; ++e) pair_at[(rec[off[r] + e] >> 16) & 0xfffu] = 1;
  for (size_t t = 0; t < c->npair; ++t)
    if (pair_at[t]) {
      pair_at[t] = (uint32_t)pairs.size();
      pairs.push_back((uint32_t)t);
    }
  P.npu = (int)pairs.size();
  P.vstride = (pairs.size() + 1) / 2 * 2;
  P.vstride32 = (pairs.size() + 3) / 4 * 4;
  P.vstr = (uint32_t)((pairs.size() + 7) & ~(size_t)7);
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
  auto fits = [&](int packs, size_t slots, size_t budget = kAbSmemBudget) {
    return 16 * (size_t)packs * P.vstr + sizeof(double) * slots + kAbStaticSmem <= budget;
  };
  // Two CTAs of 512 threads share an SM where three packs fit in half of it: one
  // stages integrals while the other one uses its own. Alpha-beta time with one
  // CTA and five packs / two CTAs and three or four, 7 electrons in 58 orbitals,
  // us: 8000 x 440 strings FP64 2499 / 1863, FP32 1709 / 1215; 3000 x 500 879 /
  // 743 and 593 / 479; 2000 x 2000 980 / 952 and 648 / 583; with a single pack,
  // 300 x 8000, 514 / 967.
  constexpr int kHalfPacks = 3;
  bool halves = true;
  size_t np = 1;
  for (;; ++np) {
    const size_t per = (n + np - 1) / np + 4, est = per + per / 8 + 512;
    if (fits(kAbPacks, est) || (fits(kAbPacks - 1, est) && kAbPacks > 1)) break;
    if (per <= 8) break;
  }
  for (;;) {
    const size_t per = (n + np - 1) / np + 4;
    halves = halves && fits(kHalfPacks, per + per / 8 + 512, kAbSmemBudget / 2);
    const bool quarters = vk.size() <= 256 && fits(kAbPacks, per + per / 8 + 512, kAbSmemBudget / 2);
    P.smem = halves ? kAbSmemBudget / 2 : kAbSmemBudget;
    const int nt = quarters ? 256 : halves || vk.size() <= 512 ? 512 : 1024;
    const size_t nbatch = std::max<size_t>(1, (vk.size() + nt - 1) / nt);
    const double effort =
        std::min(120.0, (double)alpha_singles * (double)total / 2e8);  // 2.4e10 pairs: 120 moves per record
    struct PanelWork {
      int nmain = 0, nex = 0, ny = 0;
      std::vector<uint32_t> s0, ex_row, ex_off;
      std::vector<AbBatch> b;
    };
    std::vector<PanelWork> W(np);
    bool ok = true;
    for (size_t q = 0; q < np; ++q) {
      PanelWork& w = W[q];
      for (size_t ib = 0; ib < n; ++ib) w.nmain += (ib / 4) % np == q;
      w.b.resize(nbatch);
      std::vector<uint32_t> need(w.nmain, 1), deg(w.nmain, 0);
      for (size_t b = 0; b < nbatch; ++b) {
        AbBatch& B = w.b[b];
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
              B.list.push_back({loc, (uint16_t)pair_at[(r[e] >> 16) & 0xfffu], (uint8_t)((r[e] >> 40) & 1u)});
            }
            ++m;
          }
          B.beg.push_back((uint32_t)B.list.size());
          B.maxlen = std::max(B.maxlen, B.beg[B.beg.size() - 1] - B.beg[B.beg.size() - 2]);
        }
        for (const AbSingle& s : B.list) ++deg[s.slot0];
        for (const AbSingle& s : B.list) {
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
      if (w.ny > 0xffff || !fits(halves ? kHalfPacks : kAbPacks - 1, w.ny, P.smem)) { ok = false; break; }
    }
    if (!ok && halves) {  // the extra slots need more room than half an SM
      halves = false;
      continue;
    }
    if (!ok && np < n / 4 + 1) {
      ++np;
      continue;
    }
    if (!ok) {
      c->err = "build_connectivity: the alpha-beta schedule does not fit in shared memory";
      return SBDX_ERR_ARG;
    }
    // order the batches on several host threads (a batch's seed is its place, so the
    // result does not depend on the thread count)
    const size_t jobs = np * nbatch;
    const size_t hw = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    run_jobs(jobs, std::min({hw, jobs, (size_t)(total / 4096 + 1)}), [&](size_t j) {
      PanelWork& w = W[j / nbatch];
      const AbOrder o{nt, w.ny, w.s0, w.nmain, effort};
      o.run(w.b[j % nbatch], j + 1);
    });
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
    if (rc || (rc = up(pairs, &P.pairs))) return rc;
    P.panels.resize(np);
    P.steps.assign(nbatch, 0);
    P.packs = kAbPacks;
    for (const PanelWork& w : W)
      while (P.packs > 1 && !fits(P.packs, w.ny, P.smem)) --P.packs;
    for (size_t q = 0; q < np; ++q) {
      PanelWork& w = W[q];
      AbPanel& A = P.panels[q];
      A.nmain = w.nmain;
      A.nex = w.nex;
      A.ny = w.ny;
      std::vector<uint32_t> all, bsteps, wsteps;
      std::vector<uint64_t> boff;
      for (AbBatch& B : w.b) {
        boff.push_back(all.size() / 4);
        bsteps.push_back((uint32_t)B.steps);
        P.steps[bsteps.size() - 1] += (uint64_t)B.steps;
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
