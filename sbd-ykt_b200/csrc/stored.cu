// Stored Hamiltonian: the reference's method 1 (chemistry/tpb/sbdiag.h:275-330).
// The reference builds every non-zero H_IJ of its bra block as (ih, jh, hij)
// triplets per task and thread (makeQCham, chemistry/tpb/qcham.h:10-312) and
// multiplies with them (mult, chemistry/tpb/mult.h:13-123): Wb[ih] += hij *
// T[jh] after Wb += hii * T. Here the elements lie in blocks that share their
// column lists:
//   - a block is one string r of the spin with fewer strings and a slice of G =
//     32 strings of the other, the strings with the most single excitations
//     first so that the lists of a slice have like lengths; lane l of a warp owns
//     row (r, s_l). Where the padding would be more than a tenth of the elements
//     (few strings, lists of very different lengths) G is the largest power of
//     two below that, and a warp takes 32 / G entries of the block at a time (at
//     G = 1 nothing is padded). A quarter instead of a tenth is slower on nearly
//     every shape: 150 x 1000 strings, 7 electrons in 58 orbitals, 231 us against
//     181, 600 x 1000, 6 in 32, 646 against 572, 1000 x 1000, 5 in 24, 1077
//     against 1054 (300 x 300, 7 in 58, 138 against 144); a twenty-fifth 191, 768
//     and 1126. Only the smallest problems, short of warps for narrow slices' long
//     chains, keep a quarter (150 x 150, 5 in 24: 24.7 us against 27.0);
//   - its values, G per entry and one per row: the same-spin entries of r
//     (columns (r', s_l): consecutive in the permuted vector), the singles and
//     doubles of the slice (columns (r, s')), and the pairs of a single of r and
//     one of the slice (columns (r', s')), the same elements the on-the-fly sigma
//     evaluates; shorter lists are padded with zeros, which the product skips;
//   - the column lists are per slice (s') and per row string (r'), so an element
//     costs its 8 bytes;
//   - the values carry the determinant phases, H_IJ = phi_I phi_J H'_IJ with
//     H' the alpha-first-basis matrix of the sigma kernels; the diagonal stays
//     in the context's hii vector.
// The product permutes the vector (the slices' spin innermost), then a CTA per
// row string and group of slices streams the values, with the vector row that
// the current entries gather from in shared memory. Deterministic (a lane sums
// its row in one order). Bound: HBM, 8 bytes per element, and the latency of a
// warp's stream. 1000 x 1000 strings, 575 M elements: 0.99 ms (4.6 TB/s); as CSR,
// 12 bytes per element, a warp per row and 32 gather wavefronts per 32 elements,
// 1.62 ms. 1000 x 150 strings: 130 us, with the slices over the spin with fewer
// strings 205, as CSR 163. 150 x 150, where two launches and short streams are all,
// 24.7 us, as CSR 22.2. Tighter register bounds spill (1.7 to 2.8 ms at 4
// values in flight), 16 values in flight took 1.24 ms, several slices per warp
// 2.0 ms: the warp with the longest lists holds up the others at every staged row.
#include "sbdx.h"
#include "sbdx_internal.cuh"

#include <algorithm>
#include <string>
#include <vector>

namespace sbdx {
namespace {

constexpr int kStoredThreads = 256;  // 8 warps
constexpr int kStoredBatch = 8;      // values a lane has in flight
constexpr size_t kDirectDets = size_t(1) << 15;  // up to here the product reads the vector itself

// Same-spin element of entry e (first `ns` entries of the row are singles):
// sign * (value + opposite-spin Coulomb term of a single, table row pq).
__device__ __forceinline__ double same_element(uint32_t inf, double v, bool single, const double* __restrict__ Dt,
                                               size_t dstride, size_t col) {
  if (single) v += Dt[(size_t)((inf >> 12) & 0xfffu) * dstride + col];
  return (inf >> 31) ? -v : v;
}

// First value of block (r, s), in entries of G values from rowbase: the blocks
// of r follow each other, the entries of r (ne of them, ns singles) per slice
// plus the slices' own lists.
__device__ __forceinline__ uint64_t block_entry(uint64_t ne, uint64_t ns, int s, const uint32_t* __restrict__ psd,
                                                const uint32_t* __restrict__ ps) {
  return ne * s + psd[s] + ns * ps[s];
}

// The phase of the determinant of a row and a slice string.
__device__ __forceinline__ uint32_t block_phase(int rows, uint64_t r, uint64_t s) {
  return rows == 0 ? basis_phase(prefix_parity(r), s) : basis_phase(prefix_parity(s), r);
}

// The lists of one spin, and its singles' Coulomb terms with each string of the
// other one.
struct SpinLists {
  const uint64_t* str;
  const uint64_t* off;
  const uint32_t *ns, *ket, *info;
  const double *val, *Dt;
  size_t dstride;
};

// A warp per block.
__global__ void __launch_bounds__(kStoredThreads)
stored_fill_kernel(const SpinLists R, const SpinLists S, int rows, const double* __restrict__ V, size_t vstride,
                   const uint64_t* __restrict__ rowbase, const uint32_t* __restrict__ perm,
                   const uint32_t* __restrict__ psd, const uint32_t* __restrict__ ps, int nslice, int G,
                   double* __restrict__ val) {
  const uint32_t lane = threadIdx.x & 31, col = lane & (G - 1), sub = lane / G, step = 32 / G;
  const size_t r = blockIdx.x;
  const uint64_t a0 = R.off[r], ne = R.off[r + 1] - a0, nas = R.ns[r], rI = R.str[r];
  for (int s = blockIdx.y * (kStoredThreads / 32) + (threadIdx.x >> 5); s < nslice;
       s += gridDim.y * (kStoredThreads / 32)) {
    double* out = val + rowbase[r] + G * block_entry(ne, nas, s, psd, ps) + col;
    const uint32_t is = perm[G * s + col];
    const bool in = is != kNoRow;
    const uint64_t sI = in ? S.str[is] : 0ull;
    const uint32_t phI = block_phase(rows, rI, sI);
    // same-spin entries of r: (r', s)
    for (uint64_t k = sub; k < ne; k += step) {
      const uint64_t e = a0 + k;
      double v = in ? same_element(R.info[e], R.val[e], k < nas, R.Dt, R.dstride, is) : 0.0;
      if (phI ^ block_phase(rows, R.str[R.ket[e]], sI)) v = -v;
      out[G * k] = v;
    }
    out += G * ne;
    // those of the slice: (r, s'), singles then doubles, each padded to the slice's longest list
    const uint64_t b0 = in ? S.off[is] : 0, nbs = in ? S.ns[is] : 0, nbd = in ? S.off[is + 1] - b0 - nbs : 0;
    const uint32_t ls = ps[s + 1] - ps[s], ld = psd[s + 1] - psd[s] - ls;
    for (uint32_t m = sub; m < ls + ld; m += step) {
      const bool single = m < ls, has = single ? m < nbs : m - ls < nbd;
      double v = 0.0;
      if (has) {
        const uint64_t e = b0 + (single ? m : nbs + m - ls);
        v = same_element(S.info[e], S.val[e], single, S.Dt, S.dstride, r);
        if (phI ^ block_phase(rows, rI, S.str[S.ket[e]])) v = -v;
      }
      out[G * (size_t)m] = v;
    }
    out += G * (size_t)(ls + ld);
    // single of r x single of the slice: (r', s'), the two signs times (pair|pair)
    for (uint64_t ka = 0; ka < nas; ++ka, out += G * (size_t)ls) {
      const uint32_t inf = R.info[a0 + ka];
      const double* row = V + (size_t)((inf >> 12) & 0xfffu) * vstride;
      const uint64_t rJ = R.str[R.ket[a0 + ka]];
      for (uint32_t m = sub; m < ls; m += step) {
        double v = 0.0;
        if (m < nbs) {
          const uint32_t s_inf = S.info[b0 + m];
          v = row[(s_inf >> 12) & 0xfffu];
          if ((inf >> 31) ^ (s_inf >> 31) ^ phI ^ block_phase(rows, rJ, S.str[S.ket[b0 + m]])) v = -v;
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

// The same with the alpha strings in the slices: Xq[ib, t] = X[perm[t], ib], one
// 32 x 32 tile per CTA.
__global__ void __launch_bounds__(256)
permute_rows_kernel(const double* __restrict__ X, size_t na, size_t nb, const uint32_t* __restrict__ perm, size_t xs,
                    double* __restrict__ Xq) {
  __shared__ double tile[32][33];
  const size_t t0 = (size_t)blockIdx.x * 32, b0 = (size_t)blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const size_t t = t0 + k, ib = b0 + threadIdx.x;
    tile[k][threadIdx.x] = t < na && ib < nb ? X[(size_t)perm[t] * nb + ib] : 0.0;
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const size_t ib = b0 + k, t = t0 + threadIdx.x;
    if (ib < nb && t < xs) Xq[ib * xs + t] = tile[threadIdx.x][k];
  }
}

// S = hii o X + H_offdiag X: CTA = work item (row string, up to 8 slices, one per
// warp; or a range of the singles of that, the partial rows added in item
// order by the last of them to finish), longest first. Xq: the permuted vector.
// A block's values are one stream that the warp reads in
// batches, the next batch (of the next section too) loaded before the current
// one is used. The vector row that the entries gather from is staged with
// cp.async while the row before it is in use (kStaged), two buffers of xs
// doubles; without room it is read from global memory. kDirect: Xq is X itself,
// rows of nb doubles (8-byte copies, and a gather for the entries of r: a launch
// less for small problems).
template <bool kStaged, bool kDirect, int G>
__global__ void __launch_bounds__(kStoredThreads, 3)
stored_product_kernel(int row_spin, size_t nb, size_t nsl, size_t xs, const uint64_t* __restrict__ a_off, const uint32_t* __restrict__ a_ns,
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
  const uint4 item = items[blockIdx.x];  // row string, slice group, its singles [z & 0xffff, z >> 16), slot
  const size_t ia = item.x;
  const int j0 = (int)(item.z & 0xffffu), j1 = (int)(item.z >> 16);
  const bool first = j0 == 0;  // the item with the same-spin entries
  const uint64_t a0 = a_off[ia];
  const int ne = (int)(a_off[ia + 1] - a0), nas = (int)a_ns[ia];
  const size_t stride = kDirect ? nb : xs;
  auto stage = [&](int buf, size_t row) {
    if constexpr (kStaged) {
      constexpr int kStep = kDirect ? 1 : 2;
      for (size_t t = kStep * threadIdx.x; t < (kDirect ? nb : xs); t += kStep * blockDim.x) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(rows + buf * xs + t);
        if constexpr (kDirect)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(Xq + row * stride + t) : "memory");
        else
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(Xq + row * stride + t) : "memory");
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
  // sections: -2 same-spin entries of the row, -1 of the slice, j >= 0 single j with the slice's singles
  auto size = [&](int j) { return j == -2 ? na_e : j == -1 ? lb : j < j1 ? ls : 0; };
  const double* p = active ? val + rowbase[ia] + G * block_entry((uint64_t)ne, (uint64_t)nas, s, psd, ps) + lane : val;
  const uint32_t* ix = idx + (active ? (uint64_t)G * psd[s] : 0ull) + lane;
  const size_t at = (size_t)G * (active ? s : 0) + col;  // values beyond the strings are zero
  const double* xcol = Xq + (kDirect ? (size_t)perm[min(at, nsl - 1)] : min(at, xs - 1));
  if (!first) p += G * ((int64_t)ne + lb + (int64_t)j0 * ls);
  double cur[kB], acc = 0.0;
  auto load = [&](double (&o)[kB], int n) {
#pragma unroll
    for (int u = 0; u < kB; ++u) o[u] = P * u + sub < n ? __ldcs(p + 32 * u) : 0.0;
    p += G * (int64_t)n;
  };
  load(cur, min(kB * P, !first ? ls : na_e > 0 ? na_e : lb));  // without slice entries there are no pairs either
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
        r = Xq + (j < 0 ? ia : (size_t)a_ket[a0 + j]) * stride;
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
        for (int u = 0; u < kB; ++u) x[u] = P * u < cnt ? __ldg(xcol + (size_t)__ldg(a_ket + a0 + m + sub + P * u) * stride) : 0.0;
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
  const size_t I = row_spin == 0 ? ia * nb + ib : ib * nb + ia;
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
  const size_t D = c->na * c->nb;
  if (D > (size_t)UINT32_MAX) {  // a limit that callers can rely on, whatever the layout
    c->err = "build_hamiltonian: " + std::to_string(D) +
             " determinants exceed the stored matrix's 4294967295";
    return SBDX_ERR_ARG;
  }
  // the slices run over the spin with more strings (below: b), the rows over the other (a)
  const int rows = c->na > c->nb ? 1 : 0;
  const Conn& ca = c->conn[rows];
  const Conn& cb = c->conn[1 - rows];
  const size_t na = ca.n, nb = cb.n;
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
  const bool direct = rows == 0 && D <= kDirectDets && 2 * sizeof(double) * pad8(nb) <= kAbSmemBudget;
  // slice strings with the most singles, then doubles, first
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
    if (G == 1 || total <= nnz + nnz / (D <= kDirectDets ? 4 : 10)) break;
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
      o[G * (m < bs[b] ? (size_t)m : ls + m - bs[b])] = direct ? bket[boff[b] + m] : pos[bket[boff[b] + m]];
  }
  std::vector<uint64_t> rowbase(na);
  uint64_t base = 0;
  for (size_t a = 0; a < na; ++a) {
    rowbase[a] = base;
    base += G * ((aoff[a + 1] - aoff[a]) * ns + psd[ns] + (uint64_t)as[a] * ps[ns]);
  }
  // work items: a CTA walks its entries batch by batch, so the strings with the
  // most excitations would be a serial chain much longer than the rest; items
  // above a quarter of an SM slot's share are split over their row's singles,
  // down to 48 batches (24 and 96: 150 x 200 strings 30.5 us against 34.9 and
  // 41.3)
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
  H.rows = rows;
  H.direct = direct;
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
  auto lists = [&](int spin) {
    const Conn& cn = c->conn[spin];
    return SpinLists{spin == 0 ? c->d_a : c->d_b, cn.off, cn.nsing, cn.ket, cn.info, cn.val, spin == 0 ? c->d_Db : c->d_Da,
                     spin == 0 ? c->db_stride : c->da_stride};
  };
  stored_fill_kernel<<<grid, kStoredThreads, 0, c->stream>>>(lists(rows), lists(1 - rows), rows, c->d_V, c->vstride,
                                                             H.rowbase, H.perm, H.psd, H.ps, (int)ns, (int)G, H.val);
  SBDX_LAUNCHED(c);
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));  // host vectors die at return
  H.nnz = nnz;
  clear_sigma_graphs(c);
  return 0;
}

// The permuted vector lies in the sigma's scratch (d_xp, row stride xsa or,
// with the alpha strings in the slices, xsb).
int stored_sigma(Ctx* c, const double* X, double* S) {
  const StoredH& H = c->stored;
  const size_t nrow = H.rows == 0 ? c->na : c->nb, nsl = H.rows == 0 ? c->nb : c->na;
  const size_t xs = H.rows == 0 ? c->xsa : c->xsb, smem = 2 * sizeof(double) * xs;
  double* Xq = reinterpret_cast<double*>(c->d_xp);
  // rows in launches of at most 65535 blocks (the y extent of a grid)
  if (H.rows == 1) {
    const dim3 grid((unsigned)((xs + 31) / 32), (unsigned)((c->nb + 31) / 32));  // at most 65,536 beta strings here
    permute_rows_kernel<<<grid, dim3(32, 8), 0, c->stream>>>(X, c->na, c->nb, H.perm, xs, Xq);
    SBDX_LAUNCHED(c);
  } else if (!H.direct) {
    for (size_t a = 0; a < c->na; a += 65535) {
      const dim3 grid((unsigned)((xs + 255) / 256), (unsigned)std::min<size_t>(65535, c->na - a));
      permute_columns_kernel<<<grid, 256, 0, c->stream>>>(X + a * c->nb, c->nb, H.perm, xs, Xq + a * xs);
      SBDX_LAUNCHED(c);
    }
  }
  const Conn& cr = c->conn[H.rows];
  auto launch = [&](auto kernel, size_t bytes) -> int {
    SBDX_CUDA(c, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAbSmemBudget));
    kernel<<<H.nitem, 32 * H.warps, bytes, c->stream>>>(H.rows, c->nb, nsl, xs, cr.off, cr.nsing, cr.ket, H.rowbase, H.perm,
                                                       H.idx, H.psd, H.ps, H.nslice, H.val, c->d_hii, X,
                                                       H.direct ? X : Xq, S, H.item, H.split, H.slot_split, H.done, H.part);
    SBDX_LAUNCHED(c);
    return 0;
  };
  // a CTA's rows gather from the staged one about as many elements as it has,
  // or more; narrow slices of many strings use too little of it
  const bool staged = H.direct || (smem <= kAbSmemBudget && (H.width == 32 || nsl <= 64 * (size_t)H.width));
  auto pick = [&](auto st, auto unst, auto dir) -> int {
    return H.direct ? launch(dir, smem) : staged ? launch(st, smem) : launch(unst, 0);
  };
  switch (H.width) {
    case 32: return pick(stored_product_kernel<true, false, 32>, stored_product_kernel<false, false, 32>, stored_product_kernel<true, true, 32>);
    case 16: return pick(stored_product_kernel<true, false, 16>, stored_product_kernel<false, false, 16>, stored_product_kernel<true, true, 16>);
    case 8: return pick(stored_product_kernel<true, false, 8>, stored_product_kernel<false, false, 8>, stored_product_kernel<true, true, 8>);
    case 4: return pick(stored_product_kernel<true, false, 4>, stored_product_kernel<false, false, 4>, stored_product_kernel<true, true, 4>);
    case 2: return pick(stored_product_kernel<true, false, 2>, stored_product_kernel<false, false, 2>, stored_product_kernel<true, true, 2>);
    default: return pick(stored_product_kernel<true, false, 1>, stored_product_kernel<false, false, 1>, stored_product_kernel<true, true, 1>);
  }
}

}  // namespace sbdx
