// Stored Hamiltonian: the reference's method 1 (chemistry/tpb/sbdiag.h:275-330).
// The reference builds every non-zero H_IJ of its bra block as (ih, jh, hij)
// triplets per task and thread (makeQCham, chemistry/tpb/qcham.h:10-312) and
// multiplies with them (mult, chemistry/tpb/mult.h:13-123): Wb[ih] += hij *
// T[jh] after Wb += hii * T. Here the elements lie in blocks that share their
// column lists:
//   - a block is one alpha string ia and a slice of G = 32 beta strings ib, the
//     strings with the most single excitations first so that the lists of a
//     slice have like lengths; lane l of a warp owns row (ia, ib_l). Where the
//     padding would be more than a quarter of the elements (few beta strings,
//     lists of very different lengths) G is the largest power of two below that,
//     and a warp takes 32 / G entries of the block at a time (at G = 1 nothing is
//     padded);
//   - its values, G per entry and one per row: the alpha same-spin entries of
//     ia (columns (ja, ib_l): consecutive in the permuted vector), the beta
//     singles and doubles of the slice (columns (ia, jb)), and the pairs of an
//     alpha single of ia and a beta single (columns (ja, jb)), the same elements
//     the on-the-fly sigma evaluates; shorter lists are padded with zeros;
//   - the column lists are per slice (jb) and per alpha string (ja), so an
//     element costs its 8 bytes;
//   - the values carry the determinant phases, H_IJ = phi_I phi_J H'_IJ with
//     H' the alpha-first-basis matrix of the sigma kernels; the diagonal stays
//     in the context's hii vector.
// The product permutes the vector's columns, then a CTA per alpha string and
// group of slices streams the values, with the vector row that the current
// entries gather from in shared memory. Deterministic (a lane sums its row in
// one order). Bound: HBM, 8 bytes per element, and the latency of a warp's
// stream. 1000 x 1000 strings, 575 M elements: 1.12 ms (4.1 TB/s); as CSR, 12 bytes
// per element, a warp per row and 32 gather wavefronts per 32 elements, 1.62 ms.
// Tighter register bounds spill (1.7 to 2.8 ms at 4 values in flight), 16 values
// in flight took 1.24 ms, several slices per warp 2.0 ms: the warp with the
// longest lists holds up the others at every staged row.
#include "sbdx.h"
#include "sbdx_internal.cuh"

#include <algorithm>
#include <string>
#include <vector>

namespace sbdx {
namespace {

constexpr int kStoredThreads = 256;  // 8 warps
constexpr int kStoredBatch = 8;      // values a lane has in flight

// Same-spin element of entry e (first `ns` entries of the row are singles):
// sign * (value + opposite-spin Coulomb term of a single, table row pq).
__device__ __forceinline__ double same_element(uint32_t inf, double v, bool single, const double* __restrict__ Dt,
                                               size_t dstride, size_t col) {
  if (single) v += Dt[(size_t)((inf >> 12) & 0xfffu) * dstride + col];
  return (inf >> 31) ? -v : v;
}

// First value of block (ia, s), in entries of G values from rowbase: the blocks
// of ia follow each other, the entries of ia (ne of them, nas singles) per slice
// plus the slices' own lists.
__device__ __forceinline__ uint64_t block_entry(uint64_t ne, uint64_t nas, int s, const uint32_t* __restrict__ psd,
                                                const uint32_t* __restrict__ ps) {
  return ne * s + psd[s] + nas * ps[s];
}

// A warp per block.
__global__ void __launch_bounds__(kStoredThreads)
stored_fill_kernel(const uint64_t* __restrict__ astr, const uint64_t* __restrict__ bstr,
                   const uint64_t* __restrict__ a_off, const uint32_t* __restrict__ a_ns,
                   const uint32_t* __restrict__ a_ket, const double* __restrict__ a_val,
                   const uint32_t* __restrict__ a_info, const uint64_t* __restrict__ b_off,
                   const uint32_t* __restrict__ b_ns, const uint32_t* __restrict__ b_ket,
                   const double* __restrict__ b_val, const uint32_t* __restrict__ b_info,
                   const double* __restrict__ Da, size_t da_stride, const double* __restrict__ Db, size_t db_stride,
                   const double* __restrict__ V, size_t vstride, const uint64_t* __restrict__ rowbase,
                   const uint32_t* __restrict__ perm, const uint32_t* __restrict__ psd,
                   const uint32_t* __restrict__ ps, int nslice, int G, double* __restrict__ val) {
  const uint32_t lane = threadIdx.x & 31, col = lane & (G - 1), sub = lane / G, step = 32 / G;
  const size_t ia = blockIdx.x;
  const uint64_t a0 = a_off[ia], ne = a_off[ia + 1] - a0, nas = a_ns[ia];
  const uint64_t ppa = prefix_parity(astr[ia]);
  for (int s = blockIdx.y * (kStoredThreads / 32) + (threadIdx.x >> 5); s < nslice;
       s += gridDim.y * (kStoredThreads / 32)) {
    double* out = val + rowbase[ia] + G * block_entry(ne, nas, s, psd, ps) + col;
    const uint32_t ib = perm[G * s + col];
    const bool in = ib != kNoRow;
    const uint64_t bI = in ? bstr[ib] : 0ull;
    const uint32_t phI = basis_phase(ppa, bI);
    // alpha same-spin: (ja, ib)
    for (uint64_t k = sub; k < ne; k += step) {
      const uint64_t e = a0 + k;
      double v = in ? same_element(a_info[e], a_val[e], k < nas, Db, db_stride, ib) : 0.0;
      if (phI ^ basis_phase(prefix_parity(astr[a_ket[e]]), bI)) v = -v;
      out[G * k] = v;
    }
    out += G * ne;
    // beta same-spin: (ia, jb), singles then doubles, each padded to the slice's longest list
    const uint64_t b0 = in ? b_off[ib] : 0, nbs = in ? b_ns[ib] : 0, nbd = in ? b_off[ib + 1] - b0 - nbs : 0;
    const uint32_t ls = ps[s + 1] - ps[s], ld = psd[s + 1] - psd[s] - ls;
    for (uint32_t m = sub; m < ls + ld; m += step) {
      const bool single = m < ls, has = single ? m < nbs : m - ls < nbd;
      double v = 0.0;
      if (has) {
        const uint64_t e = b0 + (single ? m : nbs + m - ls);
        v = same_element(b_info[e], b_val[e], single, Da, da_stride, ia);
        if (phI ^ basis_phase(ppa, bstr[b_ket[e]])) v = -v;
      }
      out[G * (size_t)m] = v;
    }
    out += G * (size_t)(ls + ld);
    // alpha single x beta single: (ja, jb), s_a s_b (a i|b j)
    for (uint64_t ka = 0; ka < nas; ++ka, out += G * (size_t)ls) {
      const uint32_t inf = a_info[a0 + ka];
      const double* row = V + (size_t)((inf >> 12) & 0xfffu) * vstride;
      const uint64_t ppj = prefix_parity(astr[a_ket[a0 + ka]]);
      for (uint32_t m = sub; m < ls; m += step) {
        double v = 0.0;
        if (m < nbs) {
          const uint32_t ib_inf = b_info[b0 + m];
          v = row[(ib_inf >> 12) & 0xfffu];
          if ((inf >> 31) ^ (ib_inf >> 31) ^ phI ^ basis_phase(ppj, bstr[b_ket[b0 + m]])) v = -v;
        }
        out[G * (size_t)m] = v;
      }
    }
  }
}

// Xq[ia, t] = X[ia, perm[t]], rows of stride xs (zero beyond nb).
__global__ void permute_columns_kernel(const double* __restrict__ X, size_t nb, const uint32_t* __restrict__ perm,
                                       size_t xs, double* __restrict__ Xq) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= xs) return;
  Xq[blockIdx.y * xs + t] = t < nb ? X[blockIdx.y * nb + perm[t]] : 0.0;
}

// S = hii o X + H_offdiag X: CTA = work item (alpha string, up to 8 slices, one per
// warp; or a range of the alpha singles of that, the partial rows added in item
// order by the last of them to finish), longest first. Xq: X
// with permuted columns. A block's values are one stream that the warp reads in
// batches, the next batch (of the next section too) loaded before the current
// one is used. The vector row that the entries gather from is staged with
// cp.async while the row before it is in use (kStaged), two buffers of xs
// doubles; without room it is read from global memory.
template <bool kStaged, int G>
__global__ void __launch_bounds__(kStoredThreads, 3)
stored_product_kernel(size_t nb, size_t xs, const uint64_t* __restrict__ a_off, const uint32_t* __restrict__ a_ns,
                      const uint32_t* __restrict__ a_ket, const uint64_t* __restrict__ rowbase,
                      const uint32_t* __restrict__ perm, const uint32_t* __restrict__ idx,
                      const uint32_t* __restrict__ psd, const uint32_t* __restrict__ ps, int nslice,
                      const double* __restrict__ val, const double* __restrict__ hii, const double* __restrict__ X,
                      const double* __restrict__ Xq, double* __restrict__ S, const uint4* __restrict__ items,
                      const uint2* __restrict__ split, const uint32_t* __restrict__ slot_split,
                      uint32_t* __restrict__ done, double* __restrict__ part) {
  extern __shared__ __align__(16) double rows[];  // [2][xs] when staged
  constexpr int kB = kStoredBatch, P = 32 / G;  // P entries per warp and load
  const int lane = threadIdx.x & 31, col = lane & (G - 1), sub = lane / G;
  const uint4 item = items[blockIdx.x];  // ia, slice group, alpha singles [z & 0xffff, z >> 16), slot
  const size_t ia = item.x;
  const int j0 = (int)(item.z & 0xffffu), j1 = (int)(item.z >> 16);
  const bool first = j0 == 0;  // the item with the same-spin entries
  const uint64_t a0 = a_off[ia];
  const int ne = (int)(a_off[ia + 1] - a0), nas = (int)a_ns[ia];
  auto stage = [&](int buf, size_t row) {
    if constexpr (kStaged) {
      for (size_t t = 2 * threadIdx.x; t < xs; t += 2 * blockDim.x) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(rows + buf * xs + t);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(Xq + row * xs + t) : "memory");
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
  };
  if (first) stage(0, ia);
  else stage((j0 + 1) & 1, a_ket[a0 + j0]);
  const int s = (int)item.y * (int)(blockDim.x >> 5) + (threadIdx.x >> 5);
  const bool active = s < nslice;
  const int lb = active ? (int)(psd[s + 1] - psd[s]) : 0, ls = active ? (int)(ps[s + 1] - ps[s]) : 0;
  const int na_e = active ? ne : 0;
  // sections: -2 alpha same-spin entries, -1 beta same-spin, j >= 0 alpha single j with the beta singles
  auto size = [&](int j) { return j == -2 ? na_e : j == -1 ? lb : j < j1 ? ls : 0; };
  const double* p = active ? val + rowbase[ia] + G * block_entry((uint64_t)ne, (uint64_t)nas, s, psd, ps) + lane : val;
  const uint32_t* ix = idx + (active ? (uint64_t)G * psd[s] : 0ull) + lane;
  const double* xcol = Xq + min((size_t)G * (active ? s : 0) + col, xs - 1);  // values beyond nb are zero
  if (!first) p += G * ((int64_t)ne + lb + (int64_t)j0 * ls);
  double cur[kB], acc = 0.0;
  auto load = [&](double (&o)[kB], int n) {
#pragma unroll
    for (int u = 0; u < kB; ++u) o[u] = P * u + sub < n ? __ldcs(p + 32 * u) : 0.0;
    p += G * (int64_t)n;
  };
  load(cur, min(kB * P, !first ? ls : na_e > 0 ? na_e : lb));  // without beta entries there are no pairs either
  for (int j = first ? -2 : j0; j < j1; ++j) {
    const double* r = nullptr;
    if (j >= -1) {
      const int buf = (j + 1) & 1;
      if constexpr (kStaged) {
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();  // the row is in, and the other buffer's row is no longer read
        if (j + 1 < j1) stage(buf ^ 1, a_ket[a0 + j + 1]);
        r = rows + buf * xs;
      } else {
        r = Xq + (j < 0 ? ia : (size_t)a_ket[a0 + j]) * xs;
      }
    }
    const int n = size(j);
    for (int m = 0; m < n; m += kB * P) {
      const int cnt = n - m - sub;  // entries of the lane's from here: those of P * u < cnt
      double nxt[kB];
      load(nxt, min(kB * P, m + kB * P < n ? n - m - kB * P : size(j + 1)));
      if (j == -2) {
        double x[kB];
#pragma unroll
        for (int u = 0; u < kB; ++u) x[u] = P * u < cnt ? __ldg(xcol + (size_t)__ldg(a_ket + a0 + m + sub + P * u) * xs) : 0.0;
#pragma unroll
        for (int u = 0; u < kB; ++u) acc = fma(cur[u], x[u], acc);
      } else {
        uint32_t t[kB];
#pragma unroll
        for (int u = 0; u < kB; ++u) t[u] = P * u < cnt ? __ldg(ix + G * m + 32 * u) : kNoRow;
#pragma unroll
        for (int u = 0; u < kB; ++u)
          if (t[u] != kNoRow) acc = fma(cur[u], r[t[u]], acc);
      }
#pragma unroll
      for (int u = 0; u < kB; ++u) cur[u] = nxt[u];
    }
  }
#pragma unroll
  for (int o = 16; o >= G; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  const uint32_t ib = active && sub == 0 ? perm[G * s + col] : kNoRow;
  if (item.w != 0) {
    __shared__ bool s_last;
    const uint32_t slot = item.w - 1, id = slot_split[slot];
    const uint2 sp = split[id];  // first slot, number of slots
    part[(size_t)slot * kStoredThreads + threadIdx.x] = acc;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      s_last = atomicAdd(done + id, 1u) + 1 == sp.y;
      if (s_last) done[id] = 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    acc = 0.0;
    for (uint32_t k = 0; k < sp.y; ++k) acc += __ldcg(part + (size_t)(sp.x + k) * kStoredThreads + threadIdx.x);
  }
  if (ib == kNoRow) return;
  const size_t I = ia * nb + ib;
  S[I] = fma(hii[I], X[I], acc);
}

}  // namespace

void release_stored(Ctx* c) {
  StoredH& H = c->stored;
  for (void* p : {(void*)H.val, (void*)H.rowbase, (void*)H.perm, (void*)H.idx, (void*)H.psd, (void*)H.ps,
                  (void*)H.item, (void*)H.split, (void*)H.slot_split, (void*)H.done, (void*)H.part})
    dev_free(c, p);
  H = StoredH{};
}

int build_stored(Ctx* c) {
  if (!c->have_conn) { int rc = build_connectivity(c); if (rc) return rc; }
  if (!c->have_hii) { int rc = diag_terms(c); if (rc) return rc; }
  if (int rc = ensure_coulomb_a(c)) return rc;
  release_stored(c);
  const size_t na = c->na, nb = c->nb, D = na * nb;
  if (D > (size_t)UINT32_MAX) {  // a limit that callers can rely on, whatever the layout
    c->err = "build_hamiltonian: " + std::to_string(D) +
             " determinants exceed the stored matrix's 4294967295";
    return SBDX_ERR_ARG;
  }
  const Conn& ca = c->conn[0];
  const Conn& cb = c->conn[1];
  std::vector<uint32_t> as(na), bs(nb), bd(nb), bket(std::max<size_t>(1, cb.total));
  std::vector<uint64_t> aoff(na + 1), boff(nb + 1);
  auto down = [&](void* h, const void* d, size_t bytes) {
    return cudaMemcpyAsync(h, d, bytes, cudaMemcpyDeviceToHost, c->stream);
  };
  SBDX_CUDA(c, down(as.data(), ca.nsing, sizeof(uint32_t) * na));
  SBDX_CUDA(c, down(bs.data(), cb.nsing, sizeof(uint32_t) * nb));
  SBDX_CUDA(c, down(bd.data(), cb.ndoub, sizeof(uint32_t) * nb));
  SBDX_CUDA(c, down(aoff.data(), ca.off, sizeof(uint64_t) * (na + 1)));
  SBDX_CUDA(c, down(boff.data(), cb.off, sizeof(uint64_t) * (nb + 1)));
  if (cb.total) SBDX_CUDA(c, down(bket.data(), cb.ket, sizeof(uint32_t) * cb.total));
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
  // beta strings with the most singles, then doubles, first
  uint64_t sa = 0, sb = 0;
  for (uint32_t x : as) sa += x;
  for (uint32_t x : bs) sb += x;
  const uint64_t nnz = ca.total * nb + na * (uint64_t)cb.total + sa * sb;
  std::vector<uint32_t> perm(nb + 32, kNoRow), pos(nb), psd, ps;
  for (size_t t = 0; t < nb; ++t) perm[t] = (uint32_t)t;
  std::sort(perm.begin(), perm.begin() + nb, [&](uint32_t x, uint32_t y) {
    return bs[x] != bs[y] ? bs[x] > bs[y] : bd[x] != bd[y] ? bd[x] > bd[y] : x < y;
  });
  for (size_t t = 0; t < nb; ++t) pos[perm[t]] = (uint32_t)t;
  size_t G = 32, ns = 0;
  uint64_t total = 0;
  for (;; G /= 2) {
    ns = (nb + G - 1) / G;
    ps.assign(ns + 1, 0);
    psd.assign(ns + 1, 0);
    for (size_t s = 0; s < ns; ++s) {
      uint32_t ls = 0, ld = 0;
      for (size_t t = G * s; t < std::min(nb, G * s + G); ++t) {
        ls = std::max(ls, bs[perm[t]]);
        ld = std::max(ld, bd[perm[t]]);
      }
      ps[s + 1] = ps[s] + ls;
      psd[s + 1] = psd[s] + ls + ld;
    }
    total = G * (ca.total * ns + na * (uint64_t)psd[ns] + sa * ps[ns]);
    if (G == 1 || total <= nnz + nnz / 4) break;
  }
  std::vector<uint32_t> idx(std::max<size_t>(1, G * psd[ns]), kNoRow);
  for (size_t t = 0; t < nb; ++t) {
    const size_t s = t / G, ls = ps[s + 1] - ps[s];
    const uint32_t b = perm[t];
    uint32_t* o = idx.data() + G * psd[s] + t % G;
    // the kernel skips the padding, so that an infinity stays where the matrix
    // puts it (zero times it is NaN)
    for (uint32_t m = 0; m < psd[s + 1] - psd[s]; ++m) o[G * m] = kNoRow;
    for (uint32_t m = 0; m < bs[b] + bd[b]; ++m)
      o[G * (m < bs[b] ? (size_t)m : ls + m - bs[b])] = pos[bket[boff[b] + m]];
  }
  std::vector<uint64_t> rowbase(na);
  uint64_t base = 0;
  for (size_t a = 0; a < na; ++a) {
    rowbase[a] = base;
    base += G * ((aoff[a + 1] - aoff[a]) * ns + psd[ns] + (uint64_t)as[a] * ps[ns]);
  }
  // work items: a CTA walks its entries batch by batch, so the strings with the
  // most excitations would be a serial chain much longer than the rest (1000 x 150
  // strings, L = 24: 417 us without the split, 204 with it); items above a quarter of an SM slot's share are
  // split over their alpha singles
  constexpr size_t kMinCap = 48, kMaxWarps = kStoredThreads / 32;  // cap in batches
  const size_t ng = (ns + kMaxWarps - 1) / kMaxWarps, warps = (ns + ng - 1) / ng;  // few idle warps
  const auto batches = [&](uint64_t n) { return (n * G + 32 * kStoredBatch - 1) / (32 * kStoredBatch); };
  std::vector<uint64_t> mls(ng, 0), mlb(ng, 0);
  for (size_t s = 0; s < ns; ++s) {
    mls[s / warps] = std::max<uint64_t>(mls[s / warps], ps[s + 1] - ps[s]);
    mlb[s / warps] = std::max<uint64_t>(mlb[s / warps], psd[s + 1] - psd[s]);
  }
  auto fixed = [&](size_t a, size_t g) { return batches(aoff[a + 1] - aoff[a]) + batches(mlb[g]) + 1; };
  auto per = [&](size_t g) { return batches(mls[g]) + 1; };
  uint64_t cost = 0;
  for (size_t a = 0; a < na; ++a)
    for (size_t g = 0; g < ng; ++g) cost += fixed(a, g) + as[a] * per(g);
  int nsm = 0;
  SBDX_CUDA(c, cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device));
  const uint64_t cap = std::max<uint64_t>(kMinCap, cost / (4 * 3 * (uint64_t)nsm));
  struct Item { uint64_t cost; uint4 v; };
  std::vector<Item> list;
  std::vector<uint2> split;
  std::vector<uint32_t> slot_split;
  for (size_t a = 0; a < na; ++a)
    for (size_t g = 0; g < ng; ++g) {
      const uint64_t f = fixed(a, g), q = per(g), t = f + as[a] * q;
      const uint32_t n = as[a];
      const uint32_t parts = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((t + cap - 1) / cap, n));
      if (parts == 1) {
        list.push_back({t, make_uint4((uint32_t)a, (uint32_t)g, n << 16, 0)});
        continue;
      }
      split.push_back(make_uint2((uint32_t)slot_split.size(), parts));
      // the first part holds the same-spin entries and fewer singles (one at least)
      const uint64_t share = t / parts;
      uint32_t j = (uint32_t)std::min<uint64_t>(n - (parts - 1), std::max<uint64_t>(1, share > f ? (share - f) / q : 1));
      for (uint32_t k = 0, lo = 0; k < parts; ++k) {
        list.push_back({(k == 0 ? f : 0) + (j - lo) * q,
                        make_uint4((uint32_t)a, (uint32_t)g, lo | (j << 16), 1 + (uint32_t)slot_split.size())});
        slot_split.push_back((uint32_t)split.size() - 1);
        lo = j;
        if (k + 1 < parts) j = lo + (n - lo) / (parts - 1 - k);
      }
    }
  std::stable_sort(list.begin(), list.end(), [](const Item& x, const Item& y) { return x.cost > y.cost; });
  std::vector<uint4> item(list.size());
  for (size_t k = 0; k < list.size(); ++k) item[k] = list[k].v;
  const size_t nslot = slot_split.size();
  if (split.empty()) { split.resize(1); slot_split.resize(1); }
  std::vector<uint32_t> done(split.size(), 0);
  StoredH& H = c->stored;
  auto up = [&](auto** d, const auto& h) -> cudaError_t {
    const size_t bytes = sizeof(h[0]) * h.size();
    const cudaError_t e = dev_alloc(c, d, bytes);
    return e != cudaSuccess ? e : cudaMemcpyAsync(*d, h.data(), bytes, cudaMemcpyHostToDevice, c->stream);
  };
  H.nslice = (int)ns;
  H.width = (int)G;
  H.warps = (int)warps;
  H.nitem = (uint32_t)item.size();
  if (direct_alloc(c, reinterpret_cast<void**>(&H.val), sizeof(double) * std::max<uint64_t>(1, total)) != cudaSuccess ||
      up(&H.rowbase, rowbase) != cudaSuccess || up(&H.perm, perm) != cudaSuccess || up(&H.idx, idx) != cudaSuccess ||
      up(&H.psd, psd) != cudaSuccess || up(&H.ps, ps) != cudaSuccess || up(&H.item, item) != cudaSuccess ||
      up(&H.split, split) != cudaSuccess || up(&H.slot_split, slot_split) != cudaSuccess ||
      up(&H.done, done) != cudaSuccess ||
      dev_alloc(c, &H.part, sizeof(double) * kStoredThreads * std::max<size_t>(1, nslot)) != cudaSuccess) {
    cudaGetLastError();
    cudaStreamSynchronize(c->stream);
    release_stored(c);
    c->err = "build_hamiltonian: the stored matrix (" + std::to_string(nnz) + " elements, " +
             std::to_string(8.0 * (double)total / 1e9) + " GB) does not fit in device memory";
    return SBDX_ERR_NOMEM;
  }
  const dim3 grid((unsigned)na, (unsigned)std::min<size_t>((ns + 7) / 8, 65535));
  stored_fill_kernel<<<grid, kStoredThreads, 0, c->stream>>>(
      c->d_a, c->d_b, ca.off, ca.nsing, ca.ket, ca.val, ca.info, cb.off, cb.nsing, cb.ket, cb.val, cb.info, c->d_Da,
      c->da_stride, c->d_Db, c->db_stride, c->d_V, c->vstride, H.rowbase, H.perm, H.psd, H.ps, (int)ns, (int)G, H.val);
  SBDX_LAUNCHED(c);
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));  // host vectors die at return
  H.nnz = nnz;
  clear_sigma_graphs(c);
  return 0;
}

// The permuted vector lies in the sigma's scratch (d_xp, row stride xsa).
int stored_sigma(Ctx* c, const double* X, double* S) {
  const StoredH& H = c->stored;
  const size_t xs = c->xsa, smem = 2 * sizeof(double) * xs;
  double* Xq = reinterpret_cast<double*>(c->d_xp);
  // alpha rows in launches of at most 65535 (the y extent of a grid)
  for (size_t a = 0; a < c->na; a += 65535) {
    const dim3 grid((unsigned)((xs + 255) / 256), (unsigned)std::min<size_t>(65535, c->na - a));
    permute_columns_kernel<<<grid, 256, 0, c->stream>>>(X + a * c->nb, c->nb, H.perm, xs, Xq + a * xs);
    SBDX_LAUNCHED(c);
  }
  const Conn& ca = c->conn[0];
  auto launch = [&](auto kernel, size_t bytes) -> int {
    SBDX_CUDA(c, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAbSmemBudget));
    kernel<<<H.nitem, 32 * H.warps, bytes, c->stream>>>(c->nb, xs, ca.off, ca.nsing, ca.ket, H.rowbase, H.perm, H.idx,
                                                       H.psd, H.ps, H.nslice, H.val, c->d_hii, X, Xq, S, H.item,
                                                       H.split, H.slot_split, H.done, H.part);
    SBDX_LAUNCHED(c);
    return 0;
  };
  // a CTA's rows gather from the staged one about as many elements as it has,
  // or more; narrow slices of many strings use too little of it
  const bool staged = smem <= kAbSmemBudget && (H.width == 32 || c->nb <= 64 * (size_t)H.width);
  auto pick = [&](auto st, auto unst) -> int { return staged ? launch(st, smem) : launch(unst, 0); };
  switch (H.width) {
    case 32: return pick(stored_product_kernel<true, 32>, stored_product_kernel<false, 32>);
    case 16: return pick(stored_product_kernel<true, 16>, stored_product_kernel<false, 16>);
    case 8: return pick(stored_product_kernel<true, 8>, stored_product_kernel<false, 8>);
    case 4: return pick(stored_product_kernel<true, 4>, stored_product_kernel<false, 4>);
    case 2: return pick(stored_product_kernel<true, 2>, stored_product_kernel<false, 2>);
    default: return pick(stored_product_kernel<true, 1>, stored_product_kernel<false, 1>);
  }
}

}  // namespace sbdx
