// Excitation-connectivity builder.
//
// Restates GenerateExcitation (reference chemistry/tpb/helper.h:132-197): for
// every bra string r of one spin, the ket strings k with popcount(s_r ^ s_k)
// == 2 (single) or == 4 (double), in ascending k, singles then doubles per
// row (the flattened layout of MakeSmartHelper, helper.h:367-437).
//
// B200 form: one CTA per bra row; pass 1 counts with an XOR-popcount scan, the
// host scans the counts into row offsets, pass 2 re-scans and compacts with a
// warp-ballot prefix so the output order is the ascending scan order. Pass 2
// also evaluates, once per entry, everything of the matrix element that does
// not depend on the opposite-spin string:
//   - the same-spin part of the fermionic sign and the opposite-spin parity
//     mask (the two halves of the reference parity(), determinants.h:228-279,
//     on the interleaved layout alpha p -> 2p, beta p -> 2p+1);
//   - the same-spin part of the value: OneExcite (determinants.h:423-445)
//     without the opposite-spin Coulomb sum, or TwoExcite (:447-465).
// The sigma kernels combine these with the opposite-spin string of each
// determinant in O(1) (a popcount) per pair.
#include "sbdx_internal.cuh"
#include "sbdx.h"

#include <algorithm>
#include <array>
#include <cstdint>
#include <random>
#include <thread>
#include <vector>

namespace sbdx {

namespace {

constexpr int kConnThreads = 256;

__global__ void __launch_bounds__(kConnThreads)
conn_count_kernel(const uint64_t* __restrict__ s, size_t n, uint32_t* __restrict__ nsing,
                  uint32_t* __restrict__ ndoub) {
  const size_t r = blockIdx.x;
  const uint64_t sr = s[r];
  uint32_t cs = 0, cd = 0;
  for (size_t k = threadIdx.x; k < n; k += blockDim.x) {
    int d = popc64(sr ^ s[k]);
    cs += (d == 2);
    cd += (d == 4);
  }
  for (int o = 16; o > 0; o >>= 1) {
    cs += __shfl_down_sync(0xffffffffu, cs, o);
    cd += __shfl_down_sync(0xffffffffu, cd, o);
  }
  __shared__ uint32_t ws[kConnThreads / 32], wd[kConnThreads / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { ws[warp] = cs; wd[warp] = cd; }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t ts = 0, td = 0;
    for (int w = 0; w < kConnThreads / 32; ++w) { ts += ws[w]; td += wd[w]; }
    nsing[r] = ts;
    ndoub[r] = td;
  }
}

// Same-spin part of <bra|H|ket> for bra string sr, ket string sk of spin `spin`.
__device__ void make_entry(int spin, uint64_t sr, uint64_t sk, int L, const double* __restrict__ h,
                           const double* __restrict__ eri, double& val, uint64_t& om, uint32_t& info) {
  const uint64_t hole = sk & ~sr;  // occupied in ket only
  const uint64_t part = sr & ~sk;  // occupied in bra only
  if (popc64(hole) == 1) {
    const int i = __ffsll((long long)hole) - 1, a = __ffsll((long long)part) - 1;
    const int lo = i < a ? i : a, hi = i < a ? a : i;
    // parity(ket, 2lo+s, 2hi+s): same-spin bits strictly between (the start
    // bit and the [start,end) count cancel on the occupied end), plus the
    // opposite-spin bits of the range.
    const uint32_t neg = (uint32_t)(popc64(sk & range_mask(lo + 1, hi)) & 1);
    om = other_range(spin, lo, hi);
    double v = h[(size_t)a * L + i];
    uint64_t bits = sk;
    while (bits) {
      const int q = __ffsll((long long)bits) - 1;
      v += eri[eri_index(a, i, q, q)] - eri[eri_index(a, q, q, i)];
      bits &= bits - 1;
    }
    val = v;
    info = (neg << 31) | kInfoSingle | (uint32_t)i | ((uint32_t)a << 6) |
           ((uint32_t)pair_index(a, i) << 12);
  } else {
    const int i = __ffsll((long long)hole) - 1;
    const int j = __ffsll((long long)(hole & (hole - 1))) - 1;
    const int a = __ffsll((long long)part) - 1;
    const int b = __ffsll((long long)(part & (part - 1))) - 1;
    int par = 0;
    uint64_t m = 0;
    {
      const int lo = i < a ? i : a, hi = i < a ? a : i;
      par += popc64(sk & range_mask(lo, hi)) + (int)((sk >> lo) & 1ull);
      m ^= other_range(spin, lo, hi);
    }
    {
      const int lo = j < b ? j : b, hi = j < b ? b : j;
      par += popc64(sk & range_mask(lo, hi)) + (int)((sk >> lo) & 1ull);
      m ^= other_range(spin, lo, hi);
    }
    if (a > j || b < i) par += 1;
    om = m;
    val = eri[eri_index(a, i, b, j)] - eri[eri_index(a, j, b, i)];
    info = ((uint32_t)(par & 1) << 31) | (uint32_t)i | ((uint32_t)j << 6) | ((uint32_t)a << 12) |
           ((uint32_t)b << 18);
  }
}

__global__ void __launch_bounds__(kConnThreads)
conn_fill_kernel(int spin, const uint64_t* __restrict__ s, size_t n, const uint64_t* __restrict__ off,
                 const uint32_t* __restrict__ nsing, int L, const double* __restrict__ h,
                 const double* __restrict__ eri, uint32_t* __restrict__ ket, double* __restrict__ val,
                 float* __restrict__ val32, uint64_t* __restrict__ omask, uint32_t* __restrict__ info,
                 uint64_t* __restrict__ srec, uint32_t* __restrict__ spos) {
  const size_t r = blockIdx.x;
  const uint64_t sr = s[r];
  const uint64_t sbase0 = off[r];
  const uint64_t dbase0 = off[r] + nsing[r];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  __shared__ uint32_t ws[kConnThreads / 32], wd[kConnThreads / 32];
  __shared__ uint32_t s_run, d_run;
  if (threadIdx.x == 0) { s_run = 0; d_run = 0; }
  __syncthreads();
  for (size_t k0 = 0; k0 < n; k0 += kConnThreads) {
    const size_t k = k0 + threadIdx.x;
    uint64_t sk = 0;
    int d = 0;
    if (k < n) { sk = s[k]; d = popc64(sr ^ sk); }
    const bool is_s = (k < n) && d == 2, is_d = (k < n) && d == 4;
    const unsigned bs = __ballot_sync(0xffffffffu, is_s), bd = __ballot_sync(0xffffffffu, is_d);
    if (lane == 0) { ws[warp] = __popc(bs); wd[warp] = __popc(bd); }
    __syncthreads();
    uint32_t sp = 0, dp = 0, st = 0, dt = 0;
    for (int w = 0; w < kConnThreads / 32; ++w) {
      if (w < warp) { sp += ws[w]; dp += wd[w]; }
      st += ws[w];
      dt += wd[w];
    }
    if (is_s || is_d) {
      const uint64_t pos = is_s ? sbase0 + s_run + sp + __popc(bs & lt)
                                : dbase0 + d_run + dp + __popc(bd & lt);
      double v;
      uint64_t m;
      uint32_t inf;
      make_entry(spin, sr, sk, L, h, eri, v, m, inf);
      ket[pos] = (uint32_t)k;
      val[pos] = v;
      val32[pos] = (float)v;
      omask[pos] = m;
      info[pos] = inf;
      {
        // boundaries of the opposite-spin ranges: [lo,hi) for alpha
        // excitations, (lo,hi] = [lo+1,hi+1) for beta excitations
        uint32_t p[4] = {0, 0, 0, 0};
        const uint32_t sh = (uint32_t)spin;
        if (is_s) {
          const uint32_t i = inf & 63u, a = (inf >> 6) & 63u;
          p[0] = (i < a ? i : a) + sh;
          p[1] = (i < a ? a : i) + sh;
        } else {
          const uint32_t i = inf & 63u, j = (inf >> 6) & 63u, a = (inf >> 12) & 63u, b = (inf >> 18) & 63u;
          p[0] = (i < a ? i : a) + sh;
          p[1] = (i < a ? a : i) + sh;
          p[2] = (j < b ? j : b) + sh;
          p[3] = (j < b ? b : j) + sh;
        }
        spos[pos] = p[0] | (p[1] << 7) | (p[2] << 14) | (p[3] << 21) | (inf & (kInfoNeg | kInfoSingle));
      }
      if (is_s) {
        const uint32_t i = inf & 63u, a = (inf >> 6) & 63u;
        const uint64_t lo = i < a ? i : a, hi = i < a ? a : i;
        srec[pos] = rec_ket_bits(k) | ((uint64_t)((inf >> 12) & 0xfffu) << 16) | (lo << 28) | (hi << 34) |
                    ((uint64_t)(inf >> 31) << 40);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) { s_run += st; d_run += dt; }
    __syncthreads();
  }
}

void free_ab_items(Ctx* c, AbItems (&ab)[2]) {
  dev_free(c, ab[0].ypart);  // both precisions'
  for (AbItems& a : ab) {
    dev_free(c, a.item); dev_free(c, a.split); dev_free(c, a.slot); dev_free(c, a.done);
    a = AbItems{};
  }
}

void free_conn(Ctx* c, Conn& cn) {
  dev_free(c, cn.nsing); dev_free(c, cn.ndoub); dev_free(c, cn.off); dev_free(c, cn.ket);
  dev_free(c, cn.val); dev_free(c, cn.val32); dev_free(c, cn.omask); dev_free(c, cn.info);
  dev_free(c, cn.srec); dev_free(c, cn.order); dev_free(c, cn.spos);
  dev_free(c, cn.sell); dev_free(c, cn.soff); dev_free(c, cn.slen);
  SellPanel& p = cn.bal;
  dev_free(c, p.sell); dev_free(c, p.soff); dev_free(c, p.slen); dev_free(c, p.vrow); dev_free(c, p.vslot);
  dev_free(c, p.split_row); dev_free(c, p.split_slot);
  free_ab_items(c, cn.ab);
  dev_free(c, cn.same_item); dev_free(c, cn.same_split); dev_free(c, cn.same_slot); dev_free(c, cn.same_done); dev_free(c, cn.same_ypart);
  for (SameBlocks& b : cn.blk) free_blocks(c, b);
  cn = Conn{};
}

// Splits rows of `len` work units longer than cap into items: {row, first
// unit, one past the last, 1 + slot or 0},
// longest first; split rows as {row, first slot, parts, 0}. Empty rows get an
// item only with keep_empty (a kernel that assigns its output row).
// Rows are numbered from row0 (len[i] belongs to row row0 + i).
void split_rows(const std::vector<uint32_t>& len, uint32_t cap, bool keep_empty, std::vector<uint4>& items,
                std::vector<uint4>& split, int& nslot, size_t row0 = 0) {
  items.clear();
  split.clear();
  nslot = 0;
  for (size_t i = 0; i < len.size(); ++i) {
    const uint32_t r = (uint32_t)(row0 + i);
    if (len[i] <= cap) {
      if (len[i] || keep_empty) items.push_back(make_uint4(r, 0u, len[i], 0u));
      continue;
    }
    const uint32_t parts = (len[i] + cap - 1) / cap;
    split.push_back(make_uint4(r, (uint32_t)nslot, parts, 0u));
    for (uint32_t q = 0; q < parts; ++q)
      items.push_back(make_uint4(r, q * cap, std::min(len[i], (q + 1) * cap), (uint32_t)(nslot + q + 1)));
    nslot += (int)parts;
  }
  std::stable_sort(items.begin(), items.end(), [](const uint4& x, const uint4& y) { return x.z - x.y > y.z - y.y; });
}

int upload_items(Ctx* c, const std::vector<uint4>& items, const std::vector<uint4>& split, int nslot, size_t ncol,
                 uint4** d_items, uint4** d_split, double** d_part) {
  SBDX_CUDA(c, dev_alloc(c, d_items, sizeof(uint4) * std::max<size_t>(1, items.size())));
  SBDX_CUDA(c, dev_alloc(c, d_split, sizeof(uint4) * std::max<size_t>(1, split.size())));
  if (!items.empty())
    SBDX_CUDA(c, cudaMemcpyAsync(*d_items, items.data(), sizeof(uint4) * items.size(), cudaMemcpyHostToDevice,
                                 c->stream));
  if (!split.empty()) {
    SBDX_CUDA(c, cudaMemcpyAsync(*d_split, split.data(), sizeof(uint4) * split.size(), cudaMemcpyHostToDevice,
                                 c->stream));
    if (d_part) SBDX_CUDA(c, dev_alloc(c, d_part, sizeof(double) * (size_t)nslot * std::max<size_t>(8, pad8(ncol))));
  }
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));  // host vectors die at return
  return 0;
}

// The last-to-finish bookkeeping of split rows: per partial slot its split
// entry, and zeroed counters, `strips` per split entry.
int upload_slots(Ctx* c, const std::vector<uint4>& split, int nslot, size_t strips, uint32_t** d_slot, uint32_t** d_done) {
  if (split.empty()) return 0;
  std::vector<uint32_t> of(nslot);
  for (size_t q = 0; q < split.size(); ++q)
    for (uint32_t k = 0; k < split[q].z; ++k) of[split[q].y + k] = (uint32_t)q;
  SBDX_CUDA(c, dev_alloc(c, d_slot, sizeof(uint32_t) * of.size()));
  SBDX_CUDA(c, dev_alloc(c, d_done, sizeof(uint32_t) * split.size() * strips));
  SBDX_CUDA(c, cudaMemcpyAsync(*d_slot, of.data(), sizeof(uint32_t) * of.size(), cudaMemcpyHostToDevice, c->stream));
  SBDX_CUDA(c, cudaMemsetAsync(*d_done, 0, sizeof(uint32_t) * split.size() * strips, c->stream));
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
  return 0;
}

int sm_count(Ctx* c) {
  int nsm = 0;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device) != cudaSuccess || nsm < 1) nsm = 148;
  return nsm;
}

// Same-spin work items (see Conn::same_item). A CTA handles one item and one
// strip of 1024 columns (4 per thread); an item longer than the mean work of
// a CTA slot (8 resident CTAs per SM) would set the kernel's duration, so
// rows with more entries are split (at least 64 entries per item).
// Rows row0 .. row0 + hs.size() - 1 (all rows, or one shard of them).
int build_same_items(Ctx* c, Conn& cn, const std::vector<uint32_t>& hs, const std::vector<uint32_t>& hd, size_t ncol,
                     size_t row0 = 0) {
  std::vector<uint32_t> len(hs.size());
  uint64_t total = 0;
  for (size_t r = 0; r < hs.size(); ++r) total += (len[r] = hs[r] + hd[r]);
  const uint64_t strips = std::max<uint64_t>(1, (ncol + 1023) / 1024);
  const uint64_t slots = 8ull * sm_count(c);
  const uint32_t cap = (uint32_t)std::max<uint64_t>(64, (total * strips + slots - 1) / slots);
  std::vector<uint4> items, split;
  int nslot = 0;
  split_rows(len, cap, true, items, split, nslot, row0);  // every row's output is assigned
  cn.same_cap = (int)cap;
  cn.n_same_item = items.size();
  cn.n_same_split = (int)split.size();
  cn.n_same_part = nslot;
  const int rc = upload_slots(c, split, nslot, (ncol + 255) / 256, &cn.same_slot, &cn.same_done);
  if (rc) return rc;
  return upload_items(c, items, split, nslot, ncol, &cn.same_item, &cn.same_split, &cn.same_ypart);
}

uint64_t bit_reverse64(uint64_t x) {
  x = ((x >> 1) & 0x5555555555555555ull) | ((x & 0x5555555555555555ull) << 1);
  x = ((x >> 2) & 0x3333333333333333ull) | ((x & 0x3333333333333333ull) << 2);
  x = ((x >> 4) & 0x0f0f0f0f0f0f0f0full) | ((x & 0x0f0f0f0f0f0f0f0full) << 4);
  x = ((x >> 8) & 0x00ff00ff00ff00ffull) | ((x & 0x00ff00ff00ff00ffull) << 8);
  x = ((x >> 16) & 0x0000ffff0000ffffull) | ((x & 0x0000ffff0000ffffull) << 16);
  return (x >> 32) | (x << 32);
}

// The union of a block's excitation kets as a bitmap over windows of the ket
// range, kUnionWords words of shared memory at a time. Pass 1 (ucnt) counts
// it; pass 2 writes the ascending kets and, per entry of the block's strings,
// its signed value at the ket's rank (the values, FP64 or FP32, start at zero).
constexpr int kUnionWords = 4096;  // 131,072 kets per window
__global__ void __launch_bounds__(256)
union_kernel(const uint32_t* __restrict__ rows, size_t n, const uint64_t* __restrict__ off,
             const uint32_t* __restrict__ ket, const double* __restrict__ val, const float* __restrict__ val32,
             const uint32_t* __restrict__ info, int width, uint32_t* __restrict__ ucnt, const uint64_t* __restrict__ uoff,
             uint32_t* __restrict__ uket, double* __restrict__ uval, float* __restrict__ uval32) {
  __shared__ uint32_t bits[kUnionWords], pre[kUnionWords];
  __shared__ uint32_t wsum[8], run;
  const size_t b = blockIdx.x;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  if (t == 0) run = 0;
  uint32_t last = 0;
  for (size_t w0 = 0; w0 < n; w0 += (size_t)kUnionWords * 32) {
    const size_t kets = min(n - w0, (size_t)kUnionWords * 32);
    const int words = (int)((kets + 31) / 32), per = (words + 255) / 256;
    __syncthreads();
    for (int i = t; i < words; i += 256) bits[i] = 0;
    __syncthreads();
    for (int k = 0; k < width; ++k) {
      const uint32_t r = rows[b * width + k];
      if (r == kNoRow) continue;
      for (uint64_t e = off[r] + t; e < off[r + 1]; e += 256) {
        const uint32_t x = ket[e];
        if (x >= w0 && x < w0 + kets) atomicOr(&bits[(x - w0) >> 5], 1u << ((x - w0) & 31));
      }
    }
    __syncthreads();
    // exclusive prefix of the words' counts: per thread a run of words
    uint32_t c = 0;
    for (int i = t * per; i < min(words, (t + 1) * per); ++i) c += __popc(bits[i]);
    uint32_t inc = c;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    uint32_t base = run + inc - c, all = 0;
    for (int w = 0; w < 8; ++w) {
      if (w < warp) base += wsum[w];
      all += wsum[w];
    }
    if (uket != nullptr) {
      for (int i = t * per; i < min(words, (t + 1) * per); ++i) {
        pre[i] = base;
        uint32_t m = bits[i];
        while (m) {
          const int x = __ffs((int)m) - 1;
          m &= m - 1;
          uket[uoff[b] + base++] = (uint32_t)(w0 + (size_t)i * 32 + x);
        }
      }
      __syncthreads();
      for (int k = 0; k < width; ++k) {
        const uint32_t r = rows[b * width + k];
        if (r == kNoRow) continue;
        for (uint64_t e = off[r] + t; e < off[r + 1]; e += 256) {
          const uint32_t x = ket[e];
          if (x < w0 || x >= w0 + kets) continue;
          const uint32_t wd = (uint32_t)((x - w0) >> 5), bit = (uint32_t)((x - w0) & 31);
          const uint64_t at = uoff[b] + pre[wd] + __popc(bits[wd] & ((1u << bit) - 1u));
          const bool neg = (info[e] & kInfoNeg) != 0;
          if (uval != nullptr) uval[(at >> 2) * (4 * width) + k * 4 + (at & 3)] = neg ? -val[e] : val[e];
          else uval32[at * width + k] = neg ? -val32[e] : val32[e];
        }
      }
    }
    last += all;
    __syncthreads();
    if (t == 0) run += all;
  }
  if (uket == nullptr) {
    if (t == 0) ucnt[b] = last;
  } else {
    // padding entries repeat a ket of the block (their values are zero)
    __syncthreads();
    const uint64_t end = uoff[b + 1];
    for (uint64_t u = uoff[b] + last + t; u < end; u += 256) uket[u] = last ? uket[uoff[b] + last - 1] : 0u;
  }
}

// Blocks of the blocked same-spin kernels (see SameBlocks) over the bra
// strings row0 .. row0 + n - 1 of connectivity cn, built on the device;
// `strings` all strings of the spin, ncol the other spin's string count
// (partial rows have stride pad8(ncol)).
int build_same_blocks(Ctx* c, const Conn& cn, const std::vector<uint64_t>& strings, size_t row0, size_t n, size_t ncol,
                      int width, SameBlocks& B) {
  free_blocks(c, B);
  if (n == 0) return 0;
  // rows in bit-reversed string order, cut into blocks
  std::vector<std::pair<uint64_t, uint32_t>> rkey(n);
  for (size_t i = 0; i < n; ++i) rkey[i] = {bit_reverse64(strings[row0 + i]), (uint32_t)i};
  std::sort(rkey.begin(), rkey.end());
  const size_t nblk = (n + width - 1) / width;
  std::vector<uint32_t> rows(nblk * width, kNoRow);
  for (size_t i = 0; i < n; ++i) rows[i] = (uint32_t)(row0 + rkey[i].second);
  SBDX_CUDA(c, dev_alloc(c, &B.rows, sizeof(uint32_t) * rows.size()));
  SBDX_CUDA(c, dev_alloc(c, &B.uoff, sizeof(uint64_t) * (nblk + 1)));
  SBDX_CUDA(c, cudaMemcpyAsync(B.rows, rows.data(), sizeof(uint32_t) * rows.size(), cudaMemcpyHostToDevice, c->stream));
  uint32_t* d_cnt = nullptr;
  SBDX_CUDA(c, dev_alloc(c, &d_cnt, sizeof(uint32_t) * nblk));
  union_kernel<<<(unsigned)nblk, 256, 0, c->stream>>>(B.rows, cn.n, cn.off, cn.ket, cn.val, cn.val32, cn.info, width,
                                                      d_cnt, nullptr, nullptr, nullptr, nullptr);
  ++c->launches;
  std::vector<uint32_t> cnt(nblk);
  cudaError_t e = cudaMemcpyAsync(cnt.data(), d_cnt, sizeof(uint32_t) * nblk, cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  dev_free(c, d_cnt);
  SBDX_CUDA(c, e);
  std::vector<uint64_t> uoff(nblk + 1, 0);
  for (size_t b = 0; b < nblk; ++b) uoff[b + 1] = uoff[b] + ((cnt[b] + 7) & ~7u);
  const uint64_t nu = uoff[nblk];
  // work items: blocks above the cap are split (see build_same_items; a CTA
  // handles an item and a strip of up to 1024 columns; four per SM)
  const uint64_t strips = std::max<uint64_t>(1, (ncol + 1023) / 1024);
  const uint64_t slots = 4ull * sm_count(c);
  const uint32_t cap = (uint32_t)std::max<uint64_t>(64, ((nu * strips + slots - 1) / slots + 7) & ~7ull);
  std::vector<uint32_t> len(nblk);
  for (size_t b = 0; b < nblk; ++b) len[b] = (uint32_t)(uoff[b + 1] - uoff[b]);
  std::vector<uint4> items, split;
  int nslot = 0;
  split_rows(len, cap, true, items, split, nslot);
  const size_t nu1 = nu ? nu : 1;
  B.width = width;
  B.nblk = nblk;
  B.nu = nu;
  B.cap = (int)cap;
  B.n_item = items.size();
  B.n_split = (int)split.size();
  B.n_part = nslot;
  SBDX_CUDA(c, dev_alloc(c, &B.uket, sizeof(uint32_t) * nu1));
  const bool f64 = width == kBlkRows64;
  const size_t vbytes = (f64 ? sizeof(double) : sizeof(float)) * width * nu1;
  SBDX_CUDA(c, dev_alloc(c, f64 ? (void**)&B.uval : (void**)&B.uval32, vbytes));
  SBDX_CUDA(c, cudaMemsetAsync(f64 ? (void*)B.uval : (void*)B.uval32, 0, vbytes, c->stream));
  SBDX_CUDA(c, cudaMemcpyAsync(B.uoff, uoff.data(), sizeof(uint64_t) * (nblk + 1), cudaMemcpyHostToDevice, c->stream));
  union_kernel<<<(unsigned)nblk, 256, 0, c->stream>>>(B.rows, cn.n, cn.off, cn.ket, cn.val, cn.val32, cn.info, width,
                                                      nullptr, B.uoff, B.uket, B.uval, B.uval32);
  SBDX_LAUNCHED(c);
  const int rc = upload_slots(c, split, nslot, (ncol + 255) / 256, &B.slot, &B.done);
  if (rc) return rc;
  // upload_items synchronises the stream before the host vectors die
  return upload_items(c, items, split, nslot * width, ncol, &B.item, &B.split, &B.ypart);
}

// Work items of the packed alpha-beta kernel (see AbItems; partial rows have
// the padded stride pad8(nb) of the sigma's alpha-major vectors). A CTA
// handles one item and the kernel lasts about as long as the busiest SM, so
// a few strings with many singles (near-Aufbau strings of a small sample
// connect to ten times the mean) would set its duration: strings are split
// into items of at most cap singles, cap = a quarter of the mean work per SM
// rounded up to whole groups of the kernel (up to 10 singles in FP64, 20 with
// FP32 storage; two groups in FP64 where single ones are short and more than the CTAs
// that the GPU holds: 400 x 400 strings, 45 against 39 us), and items run longest
// first. Large samples have many strings per SM and split nothing. Where the items are fewer than the CTAs that the GPU
// holds, they are split over the schedule's batches too, into ranges of like
// numbers of steps, from four batches on (below, the partial rows cost what the
// split saves: 400 x 400 strings, two batches, 39 -> 45 us). Alpha-beta time
// with groups of 20 and whole batches / with both (us, FP64): 100 x 20000
// strings (7 electrons in 58 orbitals) 1265 / 553; 3 x 9000 (5 in 24) 204 / 58;
// 150 x 4000 240 / 158; 200 x 5000 (8 in 40) 189 / 153; two and four items per
// resident CTA 165 and 182.
int build_ab_items(Ctx* c, AbItems (&out)[2], std::vector<uint32_t> hs, size_t nb, size_t row0 = 0) {
  const AbPlan& P = c->ab;
  const uint64_t nsm = (uint64_t)sm_count(c);
  const uint64_t resident = nsm * (P.threads == 256 ? 4 : P.smem < kAbSmemBudget ? 2 : 1);
  uint64_t total = 0;
  for (uint32_t& h : hs) total += ++h;  // the string itself counts as one more
  const uint64_t quarter = (total + 4 * nsm - 1) / (4 * nsm);
  for (int q = 0; q < 2; ++q) {
    const uint64_t group = (uint64_t)P.packs * (q == 0 ? 2 : 4);
    uint32_t cap = 0;
    uint64_t whole = 0;
    auto set_cap = [&](uint64_t unit) {
      cap = (uint32_t)std::max<uint64_t>(unit, (quarter + unit - 1) / unit * unit);
      whole = 0;
      for (uint32_t h : hs) whole += (h + cap - 1) / cap;
    };
    set_cap(group);
    if (q == 0 && P.nbatch < 4 && whole > resident) set_cap(2 * group);
    const uint64_t want = whole && P.nbatch >= 4 ? (resident + whole - 1) / whole : 1;
    const int ways = (int)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)P.nbatch));
    // batch ranges of like numbers of steps
    std::vector<uint32_t> cut(1, 0);
    std::vector<uint64_t> sum(P.steps.size() + 1, 0);
    for (size_t b = 0; b < P.steps.size(); ++b) sum[b + 1] = sum[b] + P.steps[b];
    for (int w = 1; w < ways; ++w) {
      uint32_t b = cut.back() + 1;
      while (b + (uint32_t)(ways - w) < (uint32_t)P.nbatch && sum[b] * ways < sum.back() * w) ++b;
      cut.push_back(b);
    }
    cut.push_back((uint32_t)P.nbatch);
    struct Item { uint64_t cost; uint4 v; };
    std::vector<Item> list;
    std::vector<uint4> split;
    int slot = 0;
    for (size_t i = 0; i < hs.size(); ++i) {
      const uint32_t r = (uint32_t)(row0 + i), parts = (hs[i] + cap - 1) / cap;
      const bool many = parts * (uint32_t)ways > 1;
      if (many) split.push_back(make_uint4(r, (uint32_t)slot, parts * (uint32_t)ways, 0u));
      for (uint32_t k = 0; k < parts; ++k)
        for (int w = 0; w < ways; ++w) {
          const uint32_t s0 = k * cap, s1 = std::min(hs[i], s0 + cap);
          list.push_back({(s1 - s0) * (sum[cut[w + 1]] - sum[cut[w]] + 1),
                          make_uint4(r, s0 | (s1 << 16), cut[w] | (cut[w + 1] << 16), many ? (uint32_t)++slot : 0u)});
        }
    }
    std::stable_sort(list.begin(), list.end(), [](const Item& x, const Item& y) { return x.cost > y.cost; });
    std::vector<uint4> items(list.size());
    for (size_t k = 0; k < list.size(); ++k) items[k] = list[k].v;
    AbItems& A = out[q];
    A.n = items.size();
    A.n_split = (int)split.size();
    A.n_part = slot;
    int rc = upload_slots(c, split, slot, 1, &A.slot, &A.done);
    if (rc || (rc = upload_items(c, items, split, slot, nb, &A.item, &A.split, nullptr))) return rc;
  }
  if (const int most = std::max(out[0].n_part, out[1].n_part)) {  // one product runs at a time
    SBDX_CUDA(c, dev_alloc(c, &out[0].ypart, sizeof(double) * (size_t)most * std::max<size_t>(8, pad8(nb))));
    out[1].ypart = out[0].ypart;
  }
  return 0;
}

// Balanced SELL-32 of the single records (see SellPanel). The cap starts at
// twice the mean list length (at least 16), so that no lane of a warp walks a
// list much longer than the others, and doubles until the partial-sum slots
// fit the kernel's shared-memory budget. The slices per warp are the smallest
// of 8, 12, 16 that cover the virtual rows in the fewest CTAs.
int build_balanced_sell(Ctx* c, SellPanel& P, size_t n, const std::vector<uint32_t>& hs,
                        const std::vector<uint64_t>& off, const std::vector<uint64_t>& rec) {
  std::vector<uint32_t> order(n);
  for (size_t r = 0; r < n; ++r) order[r] = (uint32_t)r;
  std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return hs[x] > hs[y]; });
  uint64_t total = 0;
  uint32_t mx = 0;
  for (size_t r = 0; r < n; ++r) { total += hs[r]; mx = std::max(mx, hs[r]); }
  uint32_t cap = std::max<uint32_t>(16, 2 * (uint32_t)((total + n - 1) / n));
  std::vector<uint32_t> parts(n);
  int nslot = 0;
  for (;;) {
    nslot = 0;
    for (size_t r = 0; r < n; ++r) {
      parts[r] = hs[r] == 0 ? 0 : (hs[r] + cap - 1) / cap;
      if (parts[r] > 1) nslot += (int)parts[r];
    }
    if (nslot <= kMaxSplitSlots || cap >= mx) break;
    cap *= 2;
  }
  if (nslot > kMaxSplitSlots) {
    c->err = "build_connectivity: too many split beta lists";
    return SBDX_ERR_ARG;
  }
  // virtual rows: (bra string, first record, length, slot + 1 or 0)
  struct VRow { uint32_t r; uint64_t beg; uint32_t len; uint32_t slot1; };
  std::vector<VRow> vr;
  std::vector<uint32_t> split_row, split_slot(1, 0);
  for (uint32_t r : order) {
    if (parts[r] <= 1) continue;
    const uint32_t p = parts[r], base = hs[r] / p, rem = hs[r] % p;
    uint64_t beg = off[r];
    for (uint32_t j = 0; j < p; ++j) {
      const uint32_t len = base + (j < rem ? 1u : 0u);
      vr.push_back({r, beg, len, split_slot.back() + j + 1});
      beg += len;
    }
    split_row.push_back(r);
    split_slot.push_back(split_slot.back() + p);
  }
  for (uint32_t r : order)  // longest first
    if (parts[r] == 1) vr.push_back({r, off[r], hs[r], 0});
  const size_t nv = vr.size();
  int ks = 8;
  {
    size_t best = SIZE_MAX;
    for (int cand : {8, 12, 16}) {
      const size_t chunks = (nv + 1024 * (size_t)cand - 1) / (1024 * (size_t)cand);
      if (chunks < best) { best = chunks; ks = cand; }
    }
  }
  const size_t ns = (nv + 31) / 32;
  std::vector<uint64_t> soff(ns + 1, 0);
  std::vector<uint32_t> slen(ns ? ns : 1, 0);
  for (size_t sl = 0; sl < ns; ++sl) {
    uint32_t m = 0;
    for (size_t l = 0; l < 32 && sl * 32 + l < nv; ++l) m = std::max(m, vr[sl * 32 + l].len);
    slen[sl] = m;
    soff[sl + 1] = soff[sl] + 32ull * m;
  }
  // padding records contribute nothing (bit 41) and point at ket index 0, so
  // the kernel's shared-memory index stays in range
  const uint64_t kPad = 1ull << 41;
  std::vector<uint64_t> sell(soff[ns] ? soff[ns] : 1, kPad);
  std::vector<uint32_t> vrow(nv ? nv : 1, 0), vslot(nv ? nv : 1, 0);
  for (size_t v = 0; v < nv; ++v) {
    vrow[v] = vr[v].r;
    vslot[v] = vr[v].slot1;
    for (uint32_t m = 0; m < vr[v].len; ++m) sell[soff[v / 32] + 32ull * m + v % 32] = rec[vr[v].beg + m];
  }
  P.nslice = ns;
  P.nv = nv;
  P.nsplit = (int)split_row.size();
  P.nslot = (int)split_slot.back();
  P.cap = (int)cap;
  P.slices_per_warp = ks;
  if (split_row.empty()) split_row.push_back(0);
  SBDX_CUDA(c, dev_alloc(c, &P.sell, sizeof(uint64_t) * sell.size()));
  SBDX_CUDA(c, dev_alloc(c, &P.soff, sizeof(uint64_t) * (ns + 1)));
  SBDX_CUDA(c, dev_alloc(c, &P.slen, sizeof(uint32_t) * slen.size()));
  SBDX_CUDA(c, dev_alloc(c, &P.vrow, sizeof(uint32_t) * vrow.size()));
  SBDX_CUDA(c, dev_alloc(c, &P.vslot, sizeof(uint32_t) * vslot.size()));
  SBDX_CUDA(c, dev_alloc(c, &P.split_row, sizeof(uint32_t) * split_row.size()));
  SBDX_CUDA(c, dev_alloc(c, &P.split_slot, sizeof(uint32_t) * split_slot.size()));
  SBDX_CUDA(c, cudaMemcpyAsync(P.sell, sell.data(), sizeof(uint64_t) * sell.size(), cudaMemcpyHostToDevice, c->stream));
  SBDX_CUDA(c, cudaMemcpyAsync(P.soff, soff.data(), sizeof(uint64_t) * (ns + 1), cudaMemcpyHostToDevice, c->stream));
  SBDX_CUDA(c, cudaMemcpyAsync(P.slen, slen.data(), sizeof(uint32_t) * slen.size(), cudaMemcpyHostToDevice, c->stream));
  SBDX_CUDA(c, cudaMemcpyAsync(P.vrow, vrow.data(), sizeof(uint32_t) * vrow.size(), cudaMemcpyHostToDevice, c->stream));
  SBDX_CUDA(c, cudaMemcpyAsync(P.vslot, vslot.data(), sizeof(uint32_t) * vslot.size(), cudaMemcpyHostToDevice,
                               c->stream));
  SBDX_CUDA(c, cudaMemcpyAsync(P.split_row, split_row.data(), sizeof(uint32_t) * split_row.size(),
                               cudaMemcpyHostToDevice, c->stream));
  SBDX_CUDA(c, cudaMemcpyAsync(P.split_slot, split_slot.data(), sizeof(uint32_t) * split_slot.size(),
                               cudaMemcpyHostToDevice, c->stream));
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));  // host vectors die at return
  return 0;
}

// The compact records of all entries (singles slots valid).
int single_records(Ctx* c, const Conn& cn, std::vector<uint64_t>& rec) {
  rec.resize(cn.total ? cn.total : 1);
  if (cn.total)
    SBDX_CUDA(c, cudaMemcpyAsync(rec.data(), cn.srec, sizeof(uint64_t) * cn.total, cudaMemcpyDeviceToHost, c->stream));
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
  return 0;
}

// full = false: the lists only (CSR, per-entry values, masks and records),
// without the sigma's work items, SELL layouts, ket positions and blocks.
int build_one(Ctx* c, int spin, bool full) {
  Conn& cn = c->conn[spin];
  free_conn(c, cn);
  const size_t n = spin == 0 ? c->na : c->nb;
  const uint64_t* s = spin == 0 ? c->d_a : c->d_b;
  cn.n = n;
  SBDX_CUDA(c, dev_alloc(c, &cn.nsing, sizeof(uint32_t) * n));
  SBDX_CUDA(c, dev_alloc(c, &cn.ndoub, sizeof(uint32_t) * n));
  SBDX_CUDA(c, dev_alloc(c, &cn.off, sizeof(uint64_t) * (n + 1)));
  conn_count_kernel<<<(unsigned)n, kConnThreads, 0, c->stream>>>(s, n, cn.nsing, cn.ndoub);
  SBDX_LAUNCHED(c);
  std::vector<uint32_t> hs(n), hd(n);
  SBDX_CUDA(c, cudaMemcpyAsync(hs.data(), cn.nsing, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost, c->stream));
  SBDX_CUDA(c, cudaMemcpyAsync(hd.data(), cn.ndoub, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost, c->stream));
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
  std::vector<uint64_t> off(n + 1, 0);
  for (size_t r = 0; r < n; ++r) off[r + 1] = off[r] + hs[r] + hd[r];
  cn.total = off[n];
  SBDX_CUDA(c, cudaMemcpyAsync(cn.off, off.data(), sizeof(uint64_t) * (n + 1), cudaMemcpyHostToDevice, c->stream));
  const size_t t = cn.total ? cn.total : 1;
  SBDX_CUDA(c, dev_alloc(c, &cn.ket, sizeof(uint32_t) * t));
  SBDX_CUDA(c, dev_alloc(c, &cn.val, sizeof(double) * t));
  SBDX_CUDA(c, dev_alloc(c, &cn.val32, sizeof(float) * t));
  SBDX_CUDA(c, dev_alloc(c, &cn.omask, sizeof(uint64_t) * t));
  SBDX_CUDA(c, dev_alloc(c, &cn.info, sizeof(uint32_t) * t));
  SBDX_CUDA(c, dev_alloc(c, &cn.srec, sizeof(uint64_t) * t));
  SBDX_CUDA(c, dev_alloc(c, &cn.spos, sizeof(uint32_t) * t));
  SBDX_CUDA(c, dev_alloc(c, &cn.order, sizeof(uint32_t) * n));
  conn_fill_kernel<<<(unsigned)n, kConnThreads, 0, c->stream>>>(spin, s, n, cn.off, cn.nsing, c->L, c->d_h,
                                                                 c->d_eri, cn.ket, cn.val, cn.val32,
                                                                 cn.omask, cn.info, cn.srec, cn.spos);
  SBDX_LAUNCHED(c);
  if (!full) {
    SBDX_CUDA(c, cudaStreamSynchronize(c->stream));  // the host copy of `off` dies at return
    return 0;
  }
  // bra strings ordered by their number of singles (longest first), so the
  // threads of one warp in the alpha-beta kernels walk lists of similar length
  std::vector<uint32_t> order(n);
  for (size_t r = 0; r < n; ++r) order[r] = (uint32_t)r;
  std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return hs[x] > hs[y]; });
  SBDX_CUDA(c, cudaMemcpyAsync(cn.order, order.data(), sizeof(uint32_t) * n, cudaMemcpyHostToDevice, c->stream));
  {
    int rc = build_same_items(c, cn, hs, hd, spin == 0 ? c->nb : c->na);
    if (rc) return rc;
    for (int q = 0; q < 2; ++q)
      if ((rc = build_same_blocks(c, cn, spin == 0 ? c->h_a : c->h_b, 0, n, spin == 0 ? c->nb : c->na,
                                  q == 0 ? kBlkRows64 : kBlkRows32, cn.blk[q])))
        return rc;
  }
  if (spin == 1) {
    std::vector<uint64_t> rec;
    int rc = single_records(c, cn, rec);
    if (rc) return rc;
    uint64_t alpha_singles = 0;
    std::vector<uint32_t> ha(c->na);
    SBDX_CUDA(c, cudaMemcpyAsync(ha.data(), c->conn[0].nsing, sizeof(uint32_t) * c->na, cudaMemcpyDeviceToHost, c->stream));
    SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
    for (uint32_t h : ha) alpha_singles += h;
    if ((rc = build_ab_plan(c, n, hs, off, rec, alpha_singles)) || (rc = build_ab_items(c, c->conn[0].ab, ha, c->nb)))
      return rc;
  }
  // the host copy of `off` must stay alive until the async copy ran
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
  return 0;
}

}  // namespace

void free_blocks(Ctx* c, SameBlocks& b) {
  dev_free(c, b.rows); dev_free(c, b.uoff); dev_free(c, b.uket); dev_free(c, b.uval); dev_free(c, b.uval32);
  dev_free(c, b.item); dev_free(c, b.split); dev_free(c, b.slot); dev_free(c, b.done); dev_free(c, b.ypart);
  b = SameBlocks{};
}

// The SELL layouts: a plain SELL-32 of either spin's singles over `order`
// and the balanced one of the beta singles.
int ensure_sell(Ctx* c) {
  if (c->have_sell) return 0;
  for (int spin = 0; spin < 2; ++spin) {
    Conn& cn = c->conn[spin];
    const size_t n = cn.n;
    std::vector<uint32_t> hs(n), order(n);
    std::vector<uint64_t> off(n + 1), rec;
    SBDX_CUDA(c, cudaMemcpyAsync(hs.data(), cn.nsing, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost, c->stream));
    SBDX_CUDA(c, cudaMemcpyAsync(order.data(), cn.order, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost, c->stream));
    SBDX_CUDA(c, cudaMemcpyAsync(off.data(), cn.off, sizeof(uint64_t) * (n + 1), cudaMemcpyDeviceToHost, c->stream));
    int rc = single_records(c, cn, rec);
    if (rc) return rc;
    const size_t ns = (n + 31) / 32;
    std::vector<uint64_t> soff(ns + 1, 0);
    std::vector<uint32_t> slen(ns, 0);
    for (size_t sl = 0; sl < ns; ++sl) {
      uint32_t mx = 0;
      for (size_t l = 0; l < 32 && sl * 32 + l < n; ++l) mx = std::max(mx, hs[order[sl * 32 + l]]);
      slen[sl] = mx;
      soff[sl + 1] = soff[sl] + 32ull * mx;
    }
    const uint64_t kPad = 1ull << 41;
    std::vector<uint64_t> sell(soff[ns] ? soff[ns] : 1, kPad);
    for (size_t sl = 0; sl < ns; ++sl)
      for (size_t l = 0; l < 32 && sl * 32 + l < n; ++l) {
        const uint32_t r = order[sl * 32 + l];
        for (uint32_t m = 0; m < hs[r]; ++m) sell[soff[sl] + 32ull * m + l] = rec[off[r] + m];
      }
    dev_free(c, cn.sell); dev_free(c, cn.soff); dev_free(c, cn.slen);
    cn.sell = nullptr; cn.soff = nullptr; cn.slen = nullptr;
    cn.nslice = ns;
    SBDX_CUDA(c, dev_alloc(c, &cn.sell, sizeof(uint64_t) * sell.size()));
    SBDX_CUDA(c, dev_alloc(c, &cn.soff, sizeof(uint64_t) * (ns + 1)));
    SBDX_CUDA(c, dev_alloc(c, &cn.slen, sizeof(uint32_t) * (ns ? ns : 1)));
    SBDX_CUDA(c, cudaMemcpyAsync(cn.sell, sell.data(), sizeof(uint64_t) * sell.size(), cudaMemcpyHostToDevice, c->stream));
    SBDX_CUDA(c, cudaMemcpyAsync(cn.soff, soff.data(), sizeof(uint64_t) * (ns + 1), cudaMemcpyHostToDevice, c->stream));
    if (ns) SBDX_CUDA(c, cudaMemcpyAsync(cn.slen, slen.data(), sizeof(uint32_t) * ns, cudaMemcpyHostToDevice, c->stream));
    SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
    if (spin == 1 && (rc = build_balanced_sell(c, cn.bal, n, hs, off, rec))) return rc;
  }
  c->have_sell = true;
  return 0;
}

void free_range_items(Ctx* c, Conn& r) {
  for (SameBlocks& b : r.blk) free_blocks(c, b);
  dev_free(c, r.same_item); dev_free(c, r.same_split); dev_free(c, r.same_slot); dev_free(c, r.same_done); dev_free(c, r.same_ypart);
  r.same_slot = r.same_done = nullptr;
  free_ab_items(c, r.ab);
  r.same_item = r.same_split = nullptr;
  r.same_ypart = nullptr;
  r.n_same_item = 0;
  r.n_same_split = r.n_same_part = 0;
}

void free_row_range(Ctx* c) {
  free_range_items(c, c->range_conn);
  c->range_a0 = c->range_a1 = 0;
  c->have_range = false;
}

// Work items of the alpha rows [a0, a1) only, for a sigma that writes those
// output rows: the same-spin and alpha-beta items over that range, their caps
// derived from the range's own work (one shard of the alpha strings), or the
// FP64 same-spin items alone (one chunk of a pipelined product, which evaluates
// the alpha-beta product of all rows in one launch).
int build_range_items(Ctx* c, size_t a0, size_t a1, Conn& r, bool chunk) {
  free_range_items(c, r);
  const Conn& ca = c->conn[0];
  const size_t n = a1 - a0;
  std::vector<uint32_t> hs(n ? n : 1), hd(n ? n : 1);
  if (n) {
    SBDX_CUDA(c, cudaMemcpyAsync(hs.data(), ca.nsing + a0, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost, c->stream));
    SBDX_CUDA(c, cudaMemcpyAsync(hd.data(), ca.ndoub + a0, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost, c->stream));
    SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  hs.resize(n);
  hd.resize(n);
  int rc = build_same_items(c, r, hs, hd, c->nb, a0);
  if (rc) return rc;
  for (int q = 0; q < (chunk ? 1 : 2); ++q)
    if ((rc = build_same_blocks(c, ca, c->h_a, a0, n, c->nb, q == 0 ? kBlkRows64 : kBlkRows32, r.blk[q]))) return rc;
  return chunk ? 0 : build_ab_items(c, r.ab, hs, c->nb, a0);
}

int build_row_range(Ctx* c, size_t a0, size_t a1) {
  free_row_range(c);
  const int rc = build_range_items(c, a0, a1, c->range_conn, false);
  if (rc) return rc;
  c->range_a0 = a0;
  c->range_a1 = a1;
  c->have_range = true;
  return 0;
}

void free_connectivity(Ctx* c) {
  clear_sigma_graphs(c);
  release_stored(c);  // its elements come from the connectivity
  free_row_range(c);
  free_io_chunks(c);
  free_conn(c, c->conn[0]);
  free_conn(c, c->conn[1]);
  free_ab_plan(c, c->ab);
  dev_free(c, c->d_Dr); dev_free(c, c->d_Dr32);
  c->d_Dr = nullptr;
  c->d_Dr32 = nullptr;
  c->have_sell = false;
  dev_free(c, c->d_Da); dev_free(c, c->d_Db); dev_free(c, c->d_Da32); dev_free(c, c->d_Db32);
  c->d_Da = c->d_Db = nullptr;
  c->d_Da32 = c->d_Db32 = nullptr;
  c->have_conn = false;
  c->have_lists = false;
}

int build_connectivity(Ctx* c, bool full) {
  if (!c->have_strings || !c->have_integrals) {
    c->err = "build_connectivity: set integrals and strings first";
    return 3;
  }
  free_connectivity(c);
  int rc = build_one(c, 0, full);
  if (rc) return rc;
  rc = build_one(c, 1, full);
  if (rc) return rc;
  c->have_lists = true;
  if (!full) {
    pool_trim(c);
    return 0;
  }
  rc = build_coulomb_tables(c);
  if (rc) return rc;
  c->have_conn = true;
  return 0;
}

}  // namespace sbdx
