// 1-/2-particle reduced density matrices, occupation density, alpha-string
// weights and the energy adjoint.
//
// Restates Correlation (reference chemistry/tpb/correlation.h:194-444) with
// ZeroDiffCorrelation (:15-44), OneDiffCorrelation (:49-86) and
// TwoDiffCorrelation (:91-130): the same element indices and signs, summed in
// a different order. The reference accumulates every (bra, ket) pair into a
// per-thread copy of the 4*L^4 array; here the sums are regrouped, without
// atomics, so that every output element has one writer and one order:
//   - the vector is taken to the alpha-first basis, W' = phi o W (basis_phase):
//     the opposite-spin parities of all terms are then 1, and an entry's sign
//     is its same-spin sign;
//   - diagonal: per bra row, the row weight sum_c W^2 and the opposite-spin
//     occupation profile sum_c W^2 n_q(c) (one CTA per row), then an L x L
//     finalize;
//   - same-spin singles and doubles (r <- k): sum_c W'[r,c] W'[k,c], an element
//     of the Gram matrix W' W'^T, which is evaluated densely on the FP64 tensor
//     pipe (gram_kernel) unless the strings connect too sparsely;
//   - alpha single x beta single, and the singles of one spin x the
//     occupations of the other: per chunk of alpha singles of one pattern,
//     W'[ia, :] and W'[ja, :] in shared memory and one lane per beta pattern
//     (rdm_ab_chunk_kernel).
// Layout: one[s*L^2 + p + L q], two[(s + 2t)*L^4 + i + L j + L^2 k + L^3 l].
#include "sbdx_internal.cuh"

#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <vector>

namespace sbdx {

int ensure_sigma_scratch(Ctx* c);

namespace {


// Reference parity(det, start, end) (determinants.h:228-279) on the
// interleaved determinant of (alpha, beta): returns the sign bit (1 = -1).
__device__ __forceinline__ uint32_t ref_parity_bit(uint64_t a, uint64_t b, int start, int end) {
  const uint64_t ma = range_mask((start + 1) >> 1, (end + 1) >> 1);
  const uint64_t mb = range_mask(start >> 1, end >> 1);
  const uint64_t sw = (start & 1) ? b : a;
  return (uint32_t)(popc64(a & ma) + popc64(b & mb) + (int)((sw >> (start >> 1)) & 1ull)) & 1u;
}

// Row weights and occupation profiles of one orientation of W (rows x cols),
// without atomics: wrow[r] = sum_c W[r,c]^2 (lane-strided sums, a fixed
// shuffle tree, warps added in order) and, when vq is not null, the row's
// opposite-spin occupation profile vq[r*L + q] = sum_c W[r,c]^2 n_q(s_col[c])
// (per-thread shared accumulators of L doubles, added in thread order).
constexpr int kRowWeightThreads = 64;
__global__ void __launch_bounds__(kRowWeightThreads)
row_weight_kernel(const double* __restrict__ W, size_t cols, size_t ldw, const uint64_t* __restrict__ s_col, int L,
                  double* __restrict__ wrow, double* __restrict__ vq) {
  extern __shared__ double acc_q[];  // [thread][L] when vq != null
  __shared__ double red[kRowWeightThreads / 32];
  const size_t r = blockIdx.x;
  double* mine = acc_q + (size_t)threadIdx.x * L;
  if (vq != nullptr)
    for (int q = 0; q < L; ++q) mine[q] = 0.0;
  double s = 0.0;
  for (size_t c = threadIdx.x; c < cols; c += blockDim.x) {
    const double w = W[r * ldw + c];
    const double w2 = w * w;
    s += w2;
    if (vq != nullptr && w2 != 0.0) {
      uint64_t bits = s_col[c];
      while (bits) {
        const int q = __ffsll((long long)bits) - 1;
        bits &= bits - 1;
        mine[q] += w2;
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kRowWeightThreads / 32; ++w) t += red[w];
    wrow[r] = t;
  }
  if (vq != nullptr)
    for (int q = threadIdx.x; q < L; q += blockDim.x) {
      double v = 0.0;
      for (int t = 0; t < kRowWeightThreads; ++t) v += acc_q[(size_t)t * L + q];
      vq[r * L + q] = v;
    }
}

// P[p][q] = sum_r wrow[r] over the rows whose string holds p and q, and (if X
// is not null) X[p][q] = sum_r vq[r][q] over the rows whose string holds p.
// CTA p; thread (q, part) adds the rows part, part + kOccParts, ... in order,
// and the parts are added in order. (One thread per element over all rows
// took 220 us for 2000 rows of 32 orbitals; 64 x 16 threads per orbital p take
// a sixteenth of its serial length.)
constexpr int kOccParts = 16;
__global__ void __launch_bounds__(64 * kOccParts)
occupation_sums_kernel(size_t rows, const uint64_t* __restrict__ s_row, int L, const double* __restrict__ wrow,
                       const double* __restrict__ vq, double* __restrict__ P, double* __restrict__ X) {
  __shared__ double sa[kOccParts][64], sb[kOccParts][64];
  const int p = blockIdx.x, q = threadIdx.x, part = threadIdx.y;
  double a = 0.0, b = 0.0;
#pragma unroll 4
  for (size_t r = part; r < rows; r += kOccParts) {
    const uint64_t own = s_row[r];
    if (!((own >> p) & 1ull)) continue;
    if ((own >> q) & 1ull) a += wrow[r];
    if (X != nullptr && q < L) b += vq[r * L + q];
  }
  sa[part][q] = a;
  sb[part][q] = b;
  __syncthreads();
  if (part != 0 || q >= L) return;
  for (int k = 1; k < kOccParts; ++k) {
    a += sa[k][q];
    b += sb[k][q];
  }
  P[p * L + q] = a;
  if (X != nullptr) X[p * L + q] = b;
}

// Diagonal (ZeroDiffCorrelation) contributions from P_alpha, P_beta, X.
__global__ void diag_finalize_kernel(int L, const double* __restrict__ Pa, const double* __restrict__ Pb,
                                     const double* __restrict__ X, double* __restrict__ one, double* __restrict__ two) {
  const size_t L2 = (size_t)L * L, L3 = L2 * L, L4 = L3 * L;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= L * L) return;
  const int p = t / L, q = t % L;
  const size_t d = (size_t)p + L * q + L2 * p + L3 * q;   // [p, q, p, q]
  const size_t x = (size_t)p + L * q + L2 * q + L3 * p;   // [p, q, q, p]
  if (p == q) {
    one[(size_t)p + L * p] += Pa[t];
    one[L2 + (size_t)p + L * p] += Pb[t];
  }
  if (two == nullptr) return;  // the 1-RDM alone
  if (p != q) {
    two[0 * L4 + d] += Pa[t];
    two[0 * L4 + x] -= Pa[t];
    two[3 * L4 + d] += Pb[t];
    two[3 * L4 + x] -= Pb[t];
  }
  // opposite spins: alpha p, beta q -> block 2 at [p,q,p,q], block 1 at [q,p,q,p]
  const double v = X[t];
  two[2 * L4 + d] += v;
  two[1 * L4 + (size_t)q + L * p + L2 * q + L3 * p] += v;
}

// G = A A^T of the n rows of A (K columns, row stride lda), lower tiles only,
// from tile t0 on, row r at G + r n (the caller's panel starts there: an offset
// taken off at the stores costs 40 registers and a CTA per SM): CTA = one 64 x 64
// tile, four warps of 32 x 32, m8n8k4 on the FP64 tensor pipe. The operands pass
// through shared memory in two stages of 16 columns (cp.async, zero beyond n and
// K); a lane reads two consecutive columns per 16-byte load and uses them as the
// k-slots of two steps, the same ones in A and B. Rows are padded to 24 doubles, so
// that the 8 lanes of a quarter-warp (two rows) read 128 different bytes.
constexpr int kGramTile = 64, kGramK = 16, kGramPad = 24;
__device__ __forceinline__ void dmma_m8n8k4(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}
__global__ void __launch_bounds__(128)
gram_kernel(const double* __restrict__ A, size_t n, size_t K, size_t lda, double* __restrict__ G, size_t t0) {
  __shared__ __align__(16) double sm[2][2][kGramTile][kGramPad];  // [stage][operand]
  // tile t -> (bi, bj), bj <= bi
  const size_t t = blockIdx.x + t0;
  size_t bi = (size_t)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
  while (bi * (bi + 1) / 2 > t) --bi;
  while ((bi + 1) * (bi + 2) / 2 <= t) ++bi;
  const size_t bj = t - bi * (bi + 1) / 2;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const int wr = (warp >> 1) * 32, wc = (warp & 1) * 32;
  auto stage = [&](size_t k0, int s) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {  // 2 operands x 64 rows x 8 pieces of 16 bytes
      const int x = tid + 128 * u, op = x >> 9, row = (x >> 3) & 63, pc = x & 7;
      const size_t r = (op ? bj : bi) * kGramTile + row, k = k0 + 2 * pc;
      const int bytes = r < n && k < K ? (k + 1 < K ? 16 : 8) : 0;
      const double* src = bytes ? A + r * lda + k : A;
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&sm[s][op][row][2 * pc]);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  double acc[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  stage(0, 0);
  int s = 0;
  for (size_t k0 = 0; k0 < K; k0 += kGramK, s ^= 1) {
    if (k0 + kGramK < K) {
      stage(k0 + kGramK, s ^ 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kGramK; kk += 8) {
      double2 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i] = *reinterpret_cast<const double2*>(&sm[s][0][wr + 8 * i + g][kk + 2 * q]);
        b[i] = *reinterpret_cast<const double2*>(&sm[s][1][wc + 8 * i + g][kk + 2 * q]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma_m8n8k4(acc[i][j], a[i].x, b[j].x);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma_m8n8k4(acc[i][j], a[i].y, b[j].y);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const size_t r = bi * kGramTile + wr + 8 * i + g;
    if (r >= n) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const size_t c = bj * kGramTile + wc + 8 * j + 2 * q;
      if (c < n) G[r * n + c] = acc[i][j][0];
      if (c + 1 < n) G[r * n + c + 1] = acc[i][j][1];
    }
  }
}

// Packed single of the RDM: bits 0-23 bra, 24-47 ket, 48-59 pattern (hole |
// particle << 6, the info word's bits 0-11), 63 same-spin sign.
__host__ __device__ __forceinline__ uint32_t ps_bra(uint64_t r) { return (uint32_t)r & 0xffffffu; }
__host__ __device__ __forceinline__ uint32_t ps_ket(uint64_t r) { return (uint32_t)(r >> 24) & 0xffffffu; }
__host__ __device__ __forceinline__ uint32_t ps_pat(uint64_t r) { return (uint32_t)(r >> 48) & 0xfffu; }

// Values of one spin's same-spin entries, CTA = bra row: singles packed to
// srec[soff[r] + k] with value sval, doubles (when dkey is given) to position
// off[r] - soff[r] + k with pattern key dkey (info bits 0-23) and value dval.
// value = sign * sum_c W'[r,c] W'[k,c], from rows [r0, r1) of the Gram
// matrix's lower triangle (kDense: the entries whose larger string lies there)
// or by a warp per entry. Signs as in OneDiffCorrelation
// and TwoDiffCorrelation (correlation.h:49-130).
template <bool kDense>
__global__ void __launch_bounds__(128)
rdm_entries_kernel(const double* __restrict__ W, size_t cols, size_t ldw, const double* __restrict__ G, size_t n, size_t r0,
                   size_t r1,
                   const uint64_t* __restrict__ s_row, const uint64_t* __restrict__ off,
                   const uint64_t* __restrict__ soff, const uint32_t* __restrict__ ket,
                   const uint32_t* __restrict__ info, uint64_t* __restrict__ srec, double* __restrict__ sval,
                   uint32_t* __restrict__ dkey, double* __restrict__ dval) {
  const size_t r = blockIdx.x;
  const uint64_t e0 = off[r], s0 = soff[r];
  const uint32_t ns = (uint32_t)(soff[r + 1] - s0), ne = (uint32_t)(off[r + 1] - e0);
  const uint32_t todo = dkey != nullptr ? ne : ns;
  const uint64_t sr = s_row[r];
  const int lane = threadIdx.x & 31;
  const uint32_t first = kDense ? threadIdx.x : threadIdx.x >> 5, step = kDense ? blockDim.x : blockDim.x >> 5;
  for (uint32_t k = first; k < todo; k += step) {
    const uint32_t kt = ket[e0 + k], inf = info[e0 + k];
    double v = 0.0;
    if constexpr (kDense) {
      const size_t hi = max(r, (size_t)kt), lo = min(r, (size_t)kt);
      if (hi < r0 || hi >= r1) continue;
      v = G[(hi - r0) * n + lo];
    } else {
      const double* wr = W + r * ldw;
      const double* wk = W + (size_t)kt * ldw;
      double p[4] = {0.0, 0.0, 0.0, 0.0};  // eight loads in flight
      size_t c = lane;
      for (; c + 96 < cols; c += 128) {
#pragma unroll
        for (int u = 0; u < 4; ++u) p[u] = fma(__ldg(wr + c + 32 * u), __ldg(wk + c + 32 * u), p[u]);
      }
      for (; c < cols; c += 32) p[0] = fma(__ldg(wr + c), __ldg(wk + c), p[0]);
      v = (p[0] + p[1]) + (p[2] + p[3]);
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane != 0) continue;
    }
    if (k < ns) {
      if (inf >> 31) v = -v;
      srec[s0 + k] = (uint64_t)r | ((uint64_t)kt << 24) | ((uint64_t)(inf & 0xfffu) << 48) | ((uint64_t)(inf >> 31) << 63);
      sval[s0 + k] = v;
    } else {
      const int i_e = (int)(inf & 63u), j_e = (int)((inf >> 6) & 63u);
      const int a_e = (int)((inf >> 12) & 63u), b_e = (int)((inf >> 18) & 63u);
      // TwoDiffCorrelation sign on the bra: I = a_e, J = b_e (bra-only), A = i_e, B = j_e (ket-only)
      int par = 0;
      {
        const int lo = a_e < i_e ? a_e : i_e, hi = a_e < i_e ? i_e : a_e;
        par += popc64(sr & range_mask(lo, hi)) + (int)((sr >> lo) & 1ull);
      }
      {
        const int lo = b_e < j_e ? b_e : j_e, hi = b_e < j_e ? j_e : b_e;
        par += popc64(sr & range_mask(lo, hi)) + (int)((sr >> lo) & 1ull);
      }
      if (i_e > b_e || j_e < a_e) par += 1;
      const uint64_t d = e0 - s0 + (k - ns);
      dkey[d] = inf & 0xffffffu;
      dval[d] = (par & 1) ? -v : v;
    }
  }
}

// Singles of spin `spin`, one thread per (group, x), the group's singles in
// ascending bra then ket order (sidx: positions in srec): x = 0 the 1-RDM element
// gamma[particle + L hole]; x = 1 + oj (oj < L) the four same-spin 2-RDM
// elements of the bra orbital oj (oj = the particle: they cancel, skipped);
// x = 1 + L + q the two opposite-spin elements of the other spin's orbital q
// (prof[group * pstride + q]).
__global__ void rdm_singles_finalize_kernel(int spin, int L, const uint32_t* __restrict__ gkey,
                                            const uint32_t* __restrict__ goff, size_t ngroups,
                                            const uint32_t* __restrict__ sidx, const uint64_t* __restrict__ srec,
                                            const uint64_t* __restrict__ s_row, const double* __restrict__ sval,
                                            const double* __restrict__ prof, size_t pstride, double* __restrict__ one,
                                            double* __restrict__ two) {
  const int nx = two ? 1 + 2 * L : 1;
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ngroups * nx) return;
  const size_t g = t / nx;
  const int x = (int)(t % nx);
  const uint32_t key = gkey[g];
  const int oa = (int)(key & 63u), oi = (int)((key >> 6) & 63u);  // hole (ket-only), particle (bra-only)
  const size_t L2 = (size_t)L * L, L3 = L2 * L, L4 = L3 * L;
  if (x == 0) {
    double v = 0.0;
    for (uint32_t q = goff[g]; q < goff[g + 1]; ++q) v += sval[sidx[q]];
    one[(size_t)spin * L2 + oi + (size_t)L * oa] += v;
    return;
  }
  const int ss = 3 * spin;
  if (x <= L) {
    const int oj = x - 1;
    if (oj == oi) return;
    double v = 0.0;
    for (uint32_t q = goff[g]; q < goff[g + 1]; ++q)
      if ((s_row[ps_bra(srec[sidx[q]])] >> oj) & 1ull) v += sval[sidx[q]];
    if (v == 0.0) return;
    two[ss * L4 + oa + (size_t)L * oj + L2 * oi + L3 * oj] += v;
    two[ss * L4 + oj + (size_t)L * oa + L2 * oj + L3 * oi] += v;
    two[ss * L4 + oa + (size_t)L * oj + L2 * oj + L3 * oi] -= v;
    two[ss * L4 + oj + (size_t)L * oa + L2 * oi + L3 * oj] -= v;
    return;
  }
  const int qo = x - 1 - L;
  const double v = prof[g * pstride + qo];
  if (v == 0.0) return;
  const int so = spin + 2 * (1 - spin), os = (1 - spin) + 2 * spin;
  two[so * L4 + oa + (size_t)L * qo + L2 * oi + L3 * qo] += v;
  two[os * L4 + qo + (size_t)L * oa + L2 * qo + L3 * oi] += v;
}

// Doubles of spin `spin` (i, j ket-only; a, b bra-only), sorted stably by
// pattern key; the thread at a pattern's first entry adds all of them.
__global__ void rdm_doubles_finalize_kernel(int spin, int L, const uint32_t* __restrict__ key,
                                            const uint32_t* __restrict__ idx, size_t nd,
                                            const double* __restrict__ dval, double* __restrict__ two) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nd) return;
  const uint32_t k = key[t];
  if (t > 0 && key[t - 1] == k) return;
  double s = 0.0;
  for (size_t q = t; q < nd && key[q] == k; ++q) s += dval[idx[q]];
  if (s == 0.0) return;
  const size_t i_e = k & 63u, j_e = (k >> 6) & 63u, a_e = (k >> 12) & 63u, b_e = (k >> 18) & 63u;
  const size_t L2 = (size_t)L * L, L4 = L2 * L2;
  const int ss = 3 * spin;
  two[ss * L4 + i_e + (size_t)L * j_e + L2 * (a_e + (size_t)L * b_e)] += s;
  two[ss * L4 + j_e + (size_t)L * i_e + L2 * (b_e + (size_t)L * a_e)] += s;
  two[ss * L4 + i_e + (size_t)L * j_e + L2 * (b_e + (size_t)L * a_e)] -= s;
  two[ss * L4 + j_e + (size_t)L * i_e + L2 * (a_e + (size_t)L * b_e)] -= s;
}
__global__ void iota_kernel(uint32_t* p, size_t n) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) p[t] = (uint32_t)t;
}

// Alpha single x beta single pairs (task type 0). One CTA per bra alpha row.
__global__ void __launch_bounds__(512)
rdm_ab_kernel(const double* __restrict__ W, size_t nb, const uint64_t* __restrict__ astr,
              const uint64_t* __restrict__ bstr, const uint64_t* __restrict__ a_off,
              const uint32_t* __restrict__ a_nsing, const uint32_t* __restrict__ a_ket,
              const uint32_t* __restrict__ a_info, const uint64_t* __restrict__ b_off,
              const uint32_t* __restrict__ b_nsing, const uint32_t* __restrict__ b_ket,
              const uint32_t* __restrict__ b_info, int L, double* __restrict__ two, int staged) {
  extern __shared__ __align__(16) unsigned char smem[];
  double* acc = reinterpret_cast<double*>(smem);  // [L*L] by (i_b, a_b)
  double* ws = acc + (size_t)L * L;               // [nb] when staged
  const size_t ia = blockIdx.x;
  const uint64_t alpha_bra = astr[ia];
  const double* wbra = W + ia * nb;
  const size_t L2 = (size_t)L * L, L3 = L2 * L, L4 = L3 * L;
  const uint32_t ns = a_nsing[ia];
  for (uint32_t k = 0; k < ns; ++k) {
    const uint64_t e = a_off[ia] + k;
    const size_t ja = a_ket[e];
    const uint32_t inf = a_info[e];
    const int ia_h = (int)(inf & 63u);          // alpha ket-only orbital i_a
    const int ia_p = (int)((inf >> 6) & 63u);   // alpha bra-only orbital a_a
    __syncthreads();
    for (int t = threadIdx.x; t < L * L; t += blockDim.x) acc[t] = 0.0;
    // the ket row W[ja, :] in shared memory, or read from global memory
    // (L2) when a beta row does not fit
    const double* wket = staged ? ws : W + ja * nb;
    if (staged)
      for (size_t t = threadIdx.x; t < nb; t += blockDim.x) ws[t] = W[ja * nb + t];
    __syncthreads();
    for (size_t ib = threadIdx.x; ib < nb; ib += blockDim.x) {
      const double wi = wbra[ib];
      if (wi == 0.0) continue;
      const uint64_t beta_bra = bstr[ib];
      const uint64_t m0 = b_off[ib], m1 = m0 + b_nsing[ib];
      for (uint64_t m = m0; m < m1; ++m) {
        const double wj = wket[b_ket[m]];
        if (wj == 0.0) continue;
        const uint32_t i2 = b_info[m];
        const int ib_h = (int)(i2 & 63u), ib_p = (int)((i2 >> 6) & 63u);
        // c = bra-only {2 a_a, 2 a_b + 1}, d = ket-only {2 i_a, 2 i_b + 1}
        const int c0 = 2 * ia_p, c1 = 2 * ib_p + 1, d0 = 2 * ia_h, d1 = 2 * ib_h + 1;
        const int I = c0 < c1 ? c0 : c1, J = c0 < c1 ? c1 : c0;
        const int A = d0 < d1 ? d0 : d1, B = d0 < d1 ? d1 : d0;
        const uint32_t par = ref_parity_bit(alpha_bra, beta_bra, I < A ? I : A, I < A ? A : I) ^
                             ref_parity_bit(alpha_bra, beta_bra, J < B ? J : B, J < B ? B : J);
        const double v = wi * wj;
        atomicAdd(&acc[ib_h * L + ib_p], par ? -v : v);
      }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < L * L; t += blockDim.x) {
      const double v0 = acc[t];
      if (v0 == 0.0) continue;
      const int ib_h = t / L, ib_p = t % L;
      const int c0 = 2 * ia_p, c1 = 2 * ib_p + 1, d0 = 2 * ia_h, d1 = 2 * ib_h + 1;
      const int I = c0 < c1 ? c0 : c1, J = c0 < c1 ? c1 : c0;
      const int A = d0 < d1 ? d0 : d1, B = d0 < d1 ? d1 : d0;
      const double sg = (A > J || B < I) ? -v0 : v0;
      const int oi = I >> 1, si = I & 1, oa = A >> 1, sa = A & 1, oj = J >> 1, sj = J & 1, ob = B >> 1;
      if (si == sa) {
        atomicAdd(&two[(si + 2 * sj) * L4 + oa + (size_t)L * ob + L2 * (oi + (size_t)L * oj)], sg);
        atomicAdd(&two[(sj + 2 * si) * L4 + ob + (size_t)L * oa + L2 * (oj + (size_t)L * oi)], sg);
      } else {
        atomicAdd(&two[(si + 2 * sj) * L4 + oa + (size_t)L * ob + L2 * (oj + (size_t)L * oi)], -sg);
        atomicAdd(&two[(sj + 2 * si) * L4 + ob + (size_t)L * oa + L2 * (oi + (size_t)L * oj)], -sg);
      }
    }
  }
}

// Singles of the row spin x (singles and occupations of the column spin),
// without atomics. A CTA takes a chunk of at most kAbChunk singles of one row
// pattern, R at a time: the rows s W'[bra, :] and W'[ket, :] go to shared
// memory, interleaved in pairs of singles (R > 1) so that one 16-byte gather
// serves two. A lane owns one (part of a) column pattern and walks its singles
// (ib <- jb, sign): sum_r s W'[bra_r, ib] W'[ket_r, jb], kept in a register
// over the whole chunk: no reduction between lanes, one order; it goes to
// partial[chunk][part].
// Bound by the shared-memory pipe (two gathers per pair of singles and
// record); staging R singles at once costs the record load once for all.
constexpr int kAbChunk = 32;
constexpr int kAbDetThreads = 1024;
constexpr int kAbPerThread = 4;  // column pattern parts per thread
template <int R>
__global__ void __launch_bounds__(kAbDetThreads)
rdm_ab_chunk_kernel(const double* __restrict__ W, size_t cols, size_t ldw, const uint2* __restrict__ chunks, const uint64_t* __restrict__ arec,
                    const uint32_t* __restrict__ vlen, const uint64_t* __restrict__ voff,
                    const uint64_t* __restrict__ brec, int nvp, double* __restrict__ partial) {
  constexpr int H = R > 1 ? R / 2 : 1, E = R > 1 ? 2 : 1;  // packs, singles per pack
  extern __shared__ __align__(16) unsigned char smem[];
  double* wi = reinterpret_cast<double*>(smem);  // [H][cols][E]
  double* wj = wi + (size_t)H * cols * E;
  const uint2 ch = chunks[blockIdx.x];   // {first single, count}
  const int t = threadIdx.x;
  double acc[kAbPerThread];
#pragma unroll
  for (int u = 0; u < kAbPerThread; ++u) acc[u] = 0.0;
  for (uint32_t q0 = 0; q0 < ch.y; q0 += R) {
    const int nr = min((uint32_t)R, ch.y - q0);
    __syncthreads();
    for (size_t c = t; c < cols; c += kAbDetThreads) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        double a = 0.0, b = 0.0;
        if (r < nr) {
          const uint64_t ar = __ldg(arec + ch.x + q0 + r);
          a = __ldg(W + (size_t)ps_bra(ar) * ldw + c);
          b = __ldg(W + (size_t)ps_ket(ar) * ldw + c);
          if (ar >> 63) a = -a;
        }
        wi[((size_t)(r / E) * cols + c) * E + r % E] = a;
        wj[((size_t)(r / E) * cols + c) * E + r % E] = b;
      }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kAbPerThread; ++u) {
      const int v = t + u * kAbDetThreads;
      if (u * kAbDetThreads >= nvp) break;  // uniform
      const uint32_t len = v < nvp ? vlen[v] : 0;
      const uint64_t* rp = brec + voff[(size_t)(v < nvp ? v : 0) >> 5] + (v & 31);
      double s = acc[u];
#pragma unroll 2
      for (uint32_t m = 0; m < len; ++m) {
        const uint64_t br = __ldg(rp + 32ull * m);
        const uint32_t ib = ps_bra(br), jb = ps_ket(br);
        double d = 0.0;
#pragma unroll
        for (int h = 0; h < H; ++h) {
          if constexpr (E == 2) {
            const double2 x = *reinterpret_cast<const double2*>(wi + ((size_t)h * cols + ib) * 2);
            const double2 y = *reinterpret_cast<const double2*>(wj + ((size_t)h * cols + jb) * 2);
            d = fma(x.x, y.x, fma(x.y, y.y, d));
          } else {
            d = fma(wi[ib], wj[jb], d);
          }
        }
        s += (br >> 63) ? -d : d;
      }
      acc[u] = s;
    }
  }
  double* out = partial + (size_t)blockIdx.x * nvp;
#pragma unroll
  for (int u = 0; u < kAbPerThread; ++u)
    if (t + u * kAbDetThreads < nvp) out[t + u * kAbDetThreads] = acc[u];
}

// The same chunks x the occupations of the column spin: part[chunk][q] = sum
// over the columns c whose string holds q of z[c] = sum over the chunk's
// singles of s W'[bra, c] W'[ket, c], kOccCols columns of z at a time in shared
// memory; warp w adds the orbitals w, w + 8, ....
constexpr int kOccCols = 2048;
__global__ void __launch_bounds__(256)
rdm_occ_chunk_kernel(const double* __restrict__ W, size_t cols, size_t ldw, const uint64_t* __restrict__ s_col, int L,
                     const uint2* __restrict__ chunks, const uint64_t* __restrict__ arec, double* __restrict__ part) {
  __shared__ double zs[kOccCols];
  __shared__ uint64_t ar[kAbChunk];
  const uint2 ch = chunks[blockIdx.x];  // {first single, count}
  const int t = threadIdx.x, lane = t & 31;
  if (t < (int)ch.y) ar[t] = arec[ch.x + t];
  double acc[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) acc[u] = 0.0;
  for (size_t c0 = 0; c0 < cols; c0 += kOccCols) {
    const int n = (int)min(cols - c0, (size_t)kOccCols);
    __syncthreads();
    for (int c = t; c < n; c += 256) {
      double z = 0.0;
#pragma unroll 4
      for (uint32_t q = 0; q < ch.y; ++q) {
        const double a = __ldg(W + (size_t)ps_bra(ar[q]) * ldw + c0 + c), b = __ldg(W + (size_t)ps_ket(ar[q]) * ldw + c0 + c);
        z = fma(ar[q] >> 63 ? -a : a, b, z);
      }
      zs[c] = z;
    }
    __syncthreads();
    for (int c = lane; c < n; c += 32) {
      const double z = zs[c];
      const uint64_t bits = s_col[c0 + c] >> (t >> 5);
#pragma unroll
      for (int u = 0; u < 8; ++u) acc[u] += (bits >> (8 * u)) & 1ull ? z : 0.0;
    }
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    double s = acc[u];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    const int q = (t >> 5) + 8 * u;
    if (lane == 0 && q < L) part[(size_t)blockIdx.x * L + q] = s;
  }
}

// Per row pattern, the sums over its chunks (in chunk order) of every column's
// parts [vfirst[p], vfirst[p + 1]) (part p itself when vfirst is null):
// G[row pattern][column], ncol columns from partial rows of nvp parts, the
// first of them that of chunk `chunk0`.
__global__ void rdm_chunk_sum_kernel(const uint2* __restrict__ apat, int npa, uint32_t chunk0, int ncol,
                                     const uint32_t* __restrict__ vfirst, int nvp, const double* __restrict__ partial,
                                     double* __restrict__ G) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (size_t)npa * ncol) return;
  const int pa = (int)(t / ncol), p = (int)(t % ncol);
  const uint2 ap = apat[pa];  // {first chunk, chunks}
  const int v0 = vfirst ? (int)vfirst[p] : p, v1 = vfirst ? (int)vfirst[p + 1] : p + 1;
  double v = 0.0;
  for (uint32_t q = 0; q < ap.y; ++q)
    for (int x = v0; x < v1; ++x) v += partial[(size_t)(ap.x - chunk0 + q) * nvp + x];
  G[t] = v;
}

// The two 2-RDM elements of the pattern pair (alpha hole h1, particle p1;
// beta hole h2, particle p2): the indices of TwoDiffCorrelation
// (correlation.h:91-130). Its operator-order sign cancels against the
// reference parities: in the alpha-first basis both elements take the sum of
// s_alpha s_beta W' W' as it is.
__device__ __forceinline__ void ab_targets(int h1, int p1, int h2, int p2, int L, size_t (&e)[2]) {
  const size_t L2 = (size_t)L * L, L3 = L2 * L, L4 = L3 * L;
  const int c0 = 2 * p1, c1 = 2 * p2 + 1, d0 = 2 * h1, d1 = 2 * h2 + 1;
  const int I = c0 < c1 ? c0 : c1, J = c0 < c1 ? c1 : c0;
  const int A = d0 < d1 ? d0 : d1, B = d0 < d1 ? d1 : d0;
  const int oi = I >> 1, si = I & 1, oa = A >> 1, sa = A & 1, oj = J >> 1, sj = J & 1, ob = B >> 1;
  if (si == sa) {
    e[0] = (si + 2 * sj) * L4 + oa + (size_t)L * ob + L2 * (oi + (size_t)L * oj);
    e[1] = (sj + 2 * si) * L4 + ob + (size_t)L * oa + L2 * (oj + (size_t)L * oi);
  } else {
    e[0] = (si + 2 * sj) * L4 + oa + (size_t)L * ob + L2 * (oj + (size_t)L * oi);
    e[1] = (sj + 2 * si) * L4 + ob + (size_t)L * oa + L2 * (oi + (size_t)L * oj);
  }
}

// Writes the alpha-beta 2-RDM elements, one thread per pattern pair. Two
// pattern pairs reach the same element exactly when they differ by exchanging
// the particles (equal holes) or the holes (equal particles) of the two
// spins; the element is then written once, by the pair that comes first in
// (h1, p1, h2, p2) order, as its own term followed by its partner's, so every
// element has one writer and one summation order. amap, bmap: pattern index
// of (hole << 6 | particle), -1 when no single has that pattern.
__global__ void rdm_ab_write_kernel(const uint32_t* __restrict__ akey, int npa, const uint32_t* __restrict__ bkey,
                                    int npb, const int* __restrict__ amap, const int* __restrict__ bmap,
                                    const double* __restrict__ G, int L, double* __restrict__ two) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (size_t)npa * npb) return;
  const int pa = (int)(t / npb), p = (int)(t % npb);
  const int h1 = (int)(akey[pa] >> 6), p1 = (int)(akey[pa] & 63u);
  const int h2 = (int)(bkey[p] >> 6), p2 = (int)(bkey[p] & 63u);
  const double v = G[t];
  size_t e[2], ep[2] = {~(size_t)0, ~(size_t)0};
  ab_targets(h1, p1, h2, p2, L, e);
  int q1 = -1, q2 = -1, x1 = 0, y1 = 0, x2 = 0, y2 = 0;  // partner (alpha x1 -> y1, beta x2 -> y2)
  if (h1 == h2 && p1 != p2) { x1 = h1; y1 = p2; x2 = h2; y2 = p1; }
  else if (p1 == p2 && h1 != h2) { x1 = h2; y1 = p1; x2 = h1; y2 = p2; }
  else x1 = -1;
  double vp = 0.0;
  bool partner_first = false;
  if (x1 >= 0) {
    q1 = amap[(x1 << 6) | y1];
    q2 = bmap[(x2 << 6) | y2];
    if (q1 >= 0 && q2 >= 0) {
      vp = G[(size_t)q1 * npb + q2];
      ab_targets(x1, y1, x2, y2, L, ep);
      partner_first = x1 < h1 || (x1 == h1 && (y1 < p1 || (y1 == p1 && (x2 < h2 || (x2 == h2 && y2 < p2)))));
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    double val = v;
    bool skip = false;
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (ep[j] == e[i]) {
        if (partner_first) skip = true;
        else val += vp;
      }
    if (!skip && val != 0.0) two[e[i]] += val;
  }
}

template <typename T>
__global__ void transpose_d_kernel(const T* __restrict__ in, size_t rows, size_t cols, T* __restrict__ out) {
  __shared__ T tile[32][33];
  const size_t c0 = (size_t)blockIdx.x * 32, r0 = (size_t)blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const size_t r = r0 + k, c = c0 + threadIdx.x;
    if (r < rows && c < cols) tile[k][threadIdx.x] = in[r * cols + c];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const size_t c = c0 + k, r = r0 + threadIdx.x;
    if (r < rows && c < cols) out[c * rows + r] = tile[threadIdx.x][k];
  }
}

// dE/dh and dE/d(pq|rs) from the RDMs: E = I0 + sum_pq h_pq g_pq
//   + 1/2 sum_{io,jo,ia,ja} (io ia|jo ja) sum_s G_s[io + L jo + L^2 ia + L^3 ja]
// (sample main.cc:166-216). One thread per 8-fold class sums its distinct
// index permutations.
__global__ void backward_eri_kernel(int L, const double* __restrict__ two, double* __restrict__ g) {
  const size_t npair = (size_t)L * (L + 1) / 2;
  const size_t neri = npair * (npair + 1) / 2;
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= neri) return;
  // decode t -> (pq, rs) with pq >= rs, then pq -> (p >= q), rs -> (r >= s)
  size_t pq = (size_t)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
  while (pq * (pq + 1) / 2 > t) --pq;
  while ((pq + 1) * (pq + 2) / 2 <= t) ++pq;
  const size_t rs = t - pq * (pq + 1) / 2;
  auto split = [](size_t x, int& a, int& b) {
    size_t p = (size_t)((sqrt(8.0 * (double)x + 1.0) - 1.0) * 0.5);
    while (p * (p + 1) / 2 > x) --p;
    while ((p + 1) * (p + 2) / 2 <= x) ++p;
    a = (int)p;
    b = (int)(x - p * (p + 1) / 2);
  };
  int p, q, r, s;
  split(pq, p, q);
  split(rs, r, s);
  const size_t L2 = (size_t)L * L, L3 = L2 * L, L4 = L3 * L;
  // the 8 index orders (io, ia | jo, ja); keep distinct ones
  int cand[8][4] = {{p, q, r, s}, {q, p, r, s}, {p, q, s, r}, {q, p, s, r},
                    {r, s, p, q}, {s, r, p, q}, {r, s, q, p}, {s, r, q, p}};
  double sum = 0.0;
  for (int k = 0; k < 8; ++k) {
    bool dup = false;
    for (int m = 0; m < k; ++m)
      if (cand[m][0] == cand[k][0] && cand[m][1] == cand[k][1] && cand[m][2] == cand[k][2] && cand[m][3] == cand[k][3])
        dup = true;
    if (dup) continue;
    const int io = cand[k][0], ia = cand[k][1], jo = cand[k][2], ja = cand[k][3];
    const size_t idx = (size_t)io + L * (size_t)jo + L2 * ia + L3 * ja;
    sum += 0.5 * (two[idx] + two[L4 + idx] + two[2 * L4 + idx] + two[3 * L4 + idx]);
  }
  g[t] = sum;
}

// Device scratch of one call, released on the context's stream; after more than
// kTrimBytes of it the pool gives back what it does not keep.
struct Scratch {
  static constexpr size_t kTrimBytes = size_t(128) << 20;
  Ctx* c;
  std::vector<void*> p;
  size_t bytes = 0;
  explicit Scratch(Ctx* ctx) : c(ctx) {}
  ~Scratch() {
    for (void* q : p) dev_free(c, q);
    if (bytes > kTrimBytes) pool_trim(c);
  }
  template <typename T>
  cudaError_t get(T** d, size_t n) {
    const cudaError_t e = temp_alloc(c, d, sizeof(T) * std::max<size_t>(1, n));
    if (e == cudaSuccess) {
      p.push_back(*d);
      bytes += sizeof(T) * n;
    }
    return e;
  }
  // a copy of a host array; the array must stay until the stream has run
  template <typename T>
  cudaError_t put(T** d, const std::vector<T>& h) {
    const cudaError_t e = get(d, h.size());
    if (e != cudaSuccess || h.empty()) return e;
    return cudaMemcpyAsync(*d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice, c->stream);
  }
};

constexpr size_t kMaxPartials = size_t(256) << 20;  // bytes of chunk partials at a time

}  // namespace

// Row weights of both orientations: wa[na], wb[nb]; P_a, P_b, X (L*L each), from
// W (row stride ldw) and, for wb and P_b, its transpose Wt (row stride ldt).
// (P and X are written, not accumulated; the sums have a fixed order.)
static int weights(Ctx* c, const double* dW, size_t ldw, double* wa, double* wb, double* Pa, double* Pb, double* X,
                   const double* Wt, size_t ldt) {
  const size_t na = c->na, nb = c->nb;
  const int L = c->L;
  Scratch sc(c);
  double* vq = nullptr;
  if (X) SBDX_CUDA(c, sc.get(&vq, na * (size_t)L));
  const size_t smem = X ? sizeof(double) * kRowWeightThreads * (size_t)L : 0;
  row_weight_kernel<<<(unsigned)na, kRowWeightThreads, smem, c->stream>>>(dW, nb, ldw, c->d_b, L, wa, vq);
  SBDX_LAUNCHED(c);
  if (Pa) {
    occupation_sums_kernel<<<(unsigned)L, dim3(64, kOccParts), 0, c->stream>>>(na, c->d_a, L, wa, vq, Pa, X);
    SBDX_LAUNCHED(c);
  }
  if (wb) {
    row_weight_kernel<<<(unsigned)nb, kRowWeightThreads, 0, c->stream>>>(Wt, na, ldt, c->d_a, L, wb, nullptr);
    SBDX_LAUNCHED(c);
    occupation_sums_kernel<<<(unsigned)L, dim3(64, kOccParts), 0, c->stream>>>(nb, c->d_b, L, wb, nullptr, Pb, nullptr);
    SBDX_LAUNCHED(c);
  }
  return 0;
}

// One spin's singles grouped by pattern (info bits 0-11: hole, particle), each
// group in ascending bra then ket order.
struct SingleGroups {
  std::vector<uint32_t> pat, off, idx;  // patterns, group offsets, positions in srec
  std::vector<uint64_t> rec;            // the packed singles in group order
  uint32_t* d_key = nullptr;
  uint32_t* d_off = nullptr;
  uint32_t* d_idx = nullptr;
  uint64_t* d_rec = nullptr;            // in group order
  uint64_t* d_srec = nullptr;           // in CSR order
  double* d_sval = nullptr;
  // chunks of at most kAbChunk singles of one pattern, and each pattern's chunks
  std::vector<uint2> chunks, cpat;
  uint2 *d_chunks = nullptr, *d_cpat = nullptr;
};

// The same-spin entries' values of one spin; the doubles' contributions to the
// 2-RDM (two may be null: singles only); the singles' values and groups.
static int rdm_same(Ctx* c, Scratch& sc, int spin, const double* Wm, size_t ldw, double* two, SingleGroups& S,
                    std::vector<uint64_t>& keep) {
  const Conn& cn = c->conn[spin];
  const size_t n = cn.n, cols = spin == 0 ? c->nb : c->na;
  const uint64_t* s_row = spin == 0 ? c->d_a : c->d_b;
  std::vector<uint32_t> ns(n);
  SBDX_CUDA(c, cudaMemcpyAsync(ns.data(), cn.nsing, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost, c->stream));
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
  keep.assign(n + 1, 0);
  for (size_t r = 0; r < n; ++r) keep[r + 1] = keep[r] + ns[r];
  const size_t nsing = keep[n], nd = cn.total - nsing;
  uint64_t* d_soff = nullptr;
  SBDX_CUDA(c, sc.put(&d_soff, keep));
  SBDX_CUDA(c, sc.get(&S.d_srec, nsing));
  SBDX_CUDA(c, sc.get(&S.d_sval, nsing));
  Scratch own(c);  // of this spin only
  uint32_t *d_key = nullptr, *d_key2 = nullptr, *d_idx = nullptr, *d_idx2 = nullptr;
  double* d_dval = nullptr;
  if (two && nd) {
    SBDX_CUDA(c, own.get(&d_key, nd));
    SBDX_CUDA(c, own.get(&d_key2, nd));
    SBDX_CUDA(c, own.get(&d_idx, nd));
    SBDX_CUDA(c, own.get(&d_idx2, nd));
    SBDX_CUDA(c, own.get(&d_dval, nd));
  }
  // The Gram matrix costs n^2 cols flops at about 25 TFLOP/s, a dot per entry
  // reads 16 cols bytes at about 10 TB/s: dense from 1 entry in 40 pairs (the
  // sampled sets hold 4 to 15%), while there is room. Above kGramElems elements
  // it comes in panels of rows (20000 x 200 strings, 3.2 GB of it: 24 ms a call; in
  // one piece and given back each time 57 ms).
  constexpr size_t kGramElems = size_t(1) << 26;
  double* G = nullptr;
  const size_t prow = n * n > kGramElems ? std::max<size_t>(kGramTile, kGramElems / n / kGramTile * kGramTile) : n;
  if (two && (double)cn.total * 40.0 >= (double)n * (double)n && own.get(&G, prow * n) != cudaSuccess) {
    cudaGetLastError();
    G = nullptr;
  }
  for (size_t r0 = 0; r0 < n; r0 += G ? prow : n) {
    const size_t r1 = G ? std::min(n, r0 + prow) : n;
    if (G) {
      const size_t b0 = r0 / kGramTile, b1 = (r1 + kGramTile - 1) / kGramTile;
      gram_kernel<<<(unsigned)((b1 * (b1 + 1) - b0 * (b0 + 1)) / 2), 128, 0, c->stream>>>(Wm, n, cols, ldw, G - r0 * n,
                                                                                         b0 * (b0 + 1) / 2);
      SBDX_LAUNCHED(c);
    }
    auto entries = [&](auto kernel) {
      kernel<<<(unsigned)n, 128, 0, c->stream>>>(Wm, cols, ldw, G, n, r0, r1, s_row, cn.off, d_soff, cn.ket, cn.info, S.d_srec,
                                                 S.d_sval, d_key, d_dval);
    };
    if (G) entries(rdm_entries_kernel<true>);
    else entries(rdm_entries_kernel<false>);
    SBDX_LAUNCHED(c);
  }
  if (d_key) {
    iota_kernel<<<(unsigned)((nd + 255) / 256), 256, 0, c->stream>>>(d_idx, nd);
    SBDX_LAUNCHED(c);
    size_t tmp = 0;
    SBDX_CUDA(c, cub::DeviceRadixSort::SortPairs(nullptr, tmp, d_key, d_key2, d_idx, d_idx2, nd, 0, 24, c->stream));
    unsigned char* d_tmp = nullptr;
    SBDX_CUDA(c, own.get(&d_tmp, tmp));
    SBDX_CUDA(c, cub::DeviceRadixSort::SortPairs(d_tmp, tmp, d_key, d_key2, d_idx, d_idx2, nd, 0, 24, c->stream));
    rdm_doubles_finalize_kernel<<<(unsigned)((nd + 255) / 256), 256, 0, c->stream>>>(spin, c->L, d_key2, d_idx2, nd,
                                                                                     d_dval, two);
    SBDX_LAUNCHED(c);
  }
  // the singles by pattern: a stable counting sort of the packed records
  std::vector<uint64_t> rec(nsing);
  if (nsing)
    SBDX_CUDA(c, cudaMemcpyAsync(rec.data(), S.d_srec, sizeof(uint64_t) * nsing, cudaMemcpyDeviceToHost, c->stream));
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
  std::vector<uint32_t> start(4097, 0);
  for (uint64_t r : rec) ++start[ps_pat(r) + 1];
  S.off.assign(1, 0);
  for (uint32_t k = 0; k < 4096; ++k) {
    if (start[k + 1]) {
      S.pat.push_back(k);
      S.off.push_back(S.off.back() + start[k + 1]);
    }
    start[k + 1] += start[k];
  }
  S.idx.resize(nsing);
  S.rec.resize(nsing);
  for (size_t t = 0; t < nsing; ++t) {
    const uint32_t at = start[ps_pat(rec[t])]++;
    S.idx[at] = (uint32_t)t;
    S.rec[at] = rec[t];
  }
  for (size_t g = 0; g < S.pat.size(); ++g) {
    const uint32_t first = (uint32_t)S.chunks.size();
    for (uint32_t b = S.off[g]; b < S.off[g + 1]; b += kAbChunk)
      S.chunks.push_back(make_uint2(b, std::min<uint32_t>(kAbChunk, S.off[g + 1] - b)));
    S.cpat.push_back(make_uint2(first, (uint32_t)S.chunks.size() - first));
  }
  SBDX_CUDA(c, sc.put(&S.d_key, S.pat));
  SBDX_CUDA(c, sc.put(&S.d_off, S.off));
  SBDX_CUDA(c, sc.put(&S.d_idx, S.idx));
  SBDX_CUDA(c, sc.put(&S.d_rec, S.rec));
  SBDX_CUDA(c, sc.put(&S.d_chunks, S.chunks));
  SBDX_CUDA(c, sc.put(&S.d_cpat, S.cpat));
  return 0;
}

// The singles' contributions: 1-RDM, same-spin 2-RDM and the opposite-spin
// 2-RDM elements with an occupation of the other spin.
static int rdm_singles(Ctx* c, Scratch& sc, int spin, const double* Wm, size_t ldw, const SingleGroups& S, double* one,
                       double* two) {
  const size_t ng = S.pat.size();
  if (ng == 0) return 0;
  const int L = c->L;
  const size_t cols = spin == 0 ? c->nb : c->na;
  const uint64_t* s_row = spin == 0 ? c->d_a : c->d_b;
  const uint64_t* s_col = spin == 0 ? c->d_b : c->d_a;
  double *part = nullptr, *prof = nullptr;
  if (two) {
    SBDX_CUDA(c, sc.get(&part, S.chunks.size() * (size_t)L));
    SBDX_CUDA(c, sc.get(&prof, ng * (size_t)L));
    rdm_occ_chunk_kernel<<<(unsigned)S.chunks.size(), 256, 0, c->stream>>>(Wm, cols, ldw, s_col, L, S.d_chunks, S.d_rec,
                                                                          part);
    SBDX_LAUNCHED(c);
    rdm_chunk_sum_kernel<<<(unsigned)((ng * L + 255) / 256), 256, 0, c->stream>>>(S.d_cpat, (int)ng, 0u, L, nullptr, L, part,
                                                                                  prof);
    SBDX_LAUNCHED(c);
  }
  const size_t nt = ng * (two ? 1 + 2 * (size_t)L : 1);
  rdm_singles_finalize_kernel<<<(unsigned)((nt + 255) / 256), 256, 0, c->stream>>>(
      spin, L, S.d_key, S.d_off, ng, S.d_idx, S.d_srec, s_row, S.d_sval, prof, (size_t)L, one, two);
  SBDX_LAUNCHED(c);
  return 0;
}

template <int R>
static int launch_ab_chunks(Ctx* c, const double* W, const SingleGroups& A, uint32_t chunk0, uint32_t chunks,
                            const uint32_t* vlen, const uint64_t* voff, const uint64_t* brec, int nvp, double* part) {
  SBDX_CUDA(c, cudaFuncSetAttribute(rdm_ab_chunk_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAbSmemBudget));
  rdm_ab_chunk_kernel<R><<<chunks, kAbDetThreads, 2 * sizeof(double) * R * c->nb, c->stream>>>(
      W, c->nb, c->xsa, A.d_chunks + chunk0, A.d_rec, vlen, voff, brec, nvp, part);
  SBDX_LAUNCHED(c);
  return 0;
}

// The alpha-single x beta-single 2-RDM contributions (W' in d_xp). `done` stays
// false when the staged rows or the beta patterns do not fit (the caller then
// uses rdm_ab_kernel).
static int rdm_ab_chunks(Ctx* c, Scratch& sc, const SingleGroups& A, const SingleGroups& B, double* two, bool& done) {
  done = false;
  const size_t nb = c->nb;
  if (2 * sizeof(double) * nb > kAbSmemBudget) return 0;
  const int npa = (int)A.pat.size(), npb = (int)B.pat.size();
  if (npa == 0 || npb == 0) {
    done = true;
    return 0;
  }
  // parts of the beta patterns: lists above twice the mean split (more if the
  // parts exceed a lane each), longest first in slices of 32 lanes
  struct Part { uint32_t p, b, e; };
  std::vector<Part> parts;
  std::vector<uint32_t> vfirst, slot;
  uint32_t cap = std::max<uint32_t>(8, (uint32_t)(2 * B.rec.size() / npb));
  for (;; cap *= 2) {
    parts.clear();
    for (int p = 0; p < npb; ++p) {
      const uint32_t n = B.off[p + 1] - B.off[p], k = (n + cap - 1) / cap;
      for (uint32_t j = 0; j < k; ++j)
        parts.push_back({(uint32_t)p, B.off[p] + (uint32_t)((uint64_t)n * j / k), B.off[p] + (uint32_t)((uint64_t)n * (j + 1) / k)});
    }
    if (parts.size() <= (size_t)kAbPerThread * kAbDetThreads || cap > B.rec.size()) break;
  }
  const int nvp = (int)parts.size();
  if (nvp > kAbPerThread * kAbDetThreads) return 0;
  done = true;
  // part v of the kernel is parts[v] (pattern order, so a pattern's parts are
  // adjacent and summed in order); its records in slices of 32 lanes
  vfirst.assign(npb + 1, 0);
  for (const Part& x : parts) ++vfirst[x.p + 1];
  for (int p = 0; p < npb; ++p) vfirst[p + 1] += vfirst[p];
  std::vector<uint32_t> vlen(nvp);
  std::vector<uint64_t> voff((nvp + 31) / 32 + 1, 0);
  for (int v = 0; v < nvp; ++v) vlen[v] = parts[v].e - parts[v].b;
  for (size_t s = 0; s + 1 < voff.size(); ++s) {
    uint32_t m = 0;
    for (int v = (int)s * 32; v < std::min(nvp, (int)s * 32 + 32); ++v) m = std::max(m, vlen[v]);
    voff[s + 1] = voff[s] + 32ull * m;
  }
  std::vector<uint64_t> brec(voff.back() + 32, 0);
  for (int v = 0; v < nvp; ++v)
    for (uint32_t m = 0; m < vlen[v]; ++m) brec[voff[v >> 5] + 32ull * m + (v & 31)] = B.rec[parts[v].b + m];
  std::vector<int> amap(64 * 64, -1), bmap(64 * 64, -1);
  auto key_of = [](uint32_t pat) { return ((pat & 63u) << 6) | (pat >> 6); };  // hole << 6 | particle
  std::vector<uint32_t> akey(npa), bkey(npb);
  for (int q = 0; q < npa; ++q) amap[akey[q] = key_of(A.pat[q])] = q;
  for (int q = 0; q < npb; ++q) bmap[bkey[q] = key_of(B.pat[q])] = q;
  uint32_t *d_vlen = nullptr, *d_vfirst = nullptr, *d_akey = nullptr, *d_bkey = nullptr;
  uint64_t *d_voff = nullptr, *d_brec = nullptr;
  int *d_amap = nullptr, *d_bmap = nullptr;
  double *part = nullptr, *G = nullptr;
  SBDX_CUDA(c, sc.put(&d_vlen, vlen));
  SBDX_CUDA(c, sc.put(&d_vfirst, vfirst));
  SBDX_CUDA(c, sc.put(&d_voff, voff));
  SBDX_CUDA(c, sc.put(&d_brec, brec));
  SBDX_CUDA(c, sc.put(&d_akey, akey));
  SBDX_CUDA(c, sc.put(&d_bkey, bkey));
  SBDX_CUDA(c, sc.put(&d_amap, amap));
  SBDX_CUDA(c, sc.put(&d_bmap, bmap));
  // ranges of alpha patterns whose chunk partials fit in kMaxPartials (one
  // pattern at least)
  std::vector<int> range(1, 0);
  size_t most = 0;
  for (int q = 0; q < npa;) {
    size_t n = A.cpat[q].y;
    int e = q + 1;
    while (e < npa && (n + A.cpat[e].y) * nvp * sizeof(double) <= kMaxPartials) n += A.cpat[e++].y;
    most = std::max(most, n);
    range.push_back(q = e);
  }
  SBDX_CUDA(c, sc.get(&part, most * (size_t)nvp));
  SBDX_CUDA(c, sc.get(&G, (size_t)npa * npb));
  const double* W = reinterpret_cast<const double*>(c->d_xp);
  const size_t row = 2 * sizeof(double) * nb;
  for (size_t k = 0; k + 1 < range.size(); ++k) {
    const int q0 = range[k], q1 = range[k + 1];
    const uint32_t c0 = A.cpat[q0].x, nc = A.cpat[q1 - 1].x + A.cpat[q1 - 1].y - c0;
    int rc;
    if (8 * row <= kAbSmemBudget / 2) rc = launch_ab_chunks<8>(c, W, A, c0, nc, d_vlen, d_voff, d_brec, nvp, part);
    else if (6 * row <= kAbSmemBudget) rc = launch_ab_chunks<6>(c, W, A, c0, nc, d_vlen, d_voff, d_brec, nvp, part);
    else if (4 * row <= kAbSmemBudget) rc = launch_ab_chunks<4>(c, W, A, c0, nc, d_vlen, d_voff, d_brec, nvp, part);
    else if (2 * row <= kAbSmemBudget) rc = launch_ab_chunks<2>(c, W, A, c0, nc, d_vlen, d_voff, d_brec, nvp, part);
    else rc = launch_ab_chunks<1>(c, W, A, c0, nc, d_vlen, d_voff, d_brec, nvp, part);
    if (rc) return rc;
    const size_t sums = (size_t)(q1 - q0) * npb;
    rdm_chunk_sum_kernel<<<(unsigned)((sums + 255) / 256), 256, 0, c->stream>>>(A.d_cpat + q0, q1 - q0, c0, npb, d_vfirst,
                                                                               nvp, part, G + (size_t)q0 * npb);
    SBDX_LAUNCHED(c);
  }
  const size_t npairs = (size_t)npa * npb;
  rdm_ab_write_kernel<<<(unsigned)((npairs + 255) / 256), 256, 0, c->stream>>>(d_akey, npa, d_bkey, npb, d_amap, d_bmap,
                                                                               G, c->L, two);
  SBDX_LAUNCHED(c);
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));  // the host vectors die at return
  return 0;
}

int rdm_device(Ctx* c, const double* dW, double* d_one, double* d_two) {
  if (!c->have_lists) { int rc = build_connectivity(c, false); if (rc) return rc; }
  int rc = ensure_sigma_scratch(c);
  if (rc) return rc;
  const size_t na = c->na, nb = c->nb, L = (size_t)c->L, L2 = L * L, L4 = L2 * L2;
  SingleGroups S[2];
  std::vector<uint64_t> keep[2];  // host sources of copies, alive until the last synchronisation
  Scratch sc(c);
  double* wa = nullptr;
  SBDX_CUDA(c, sc.get(&wa, na + nb + 3 * L2));
  double* wb = wa + na;
  double* Pa = wb + nb;
  double* Pb = Pa + L2;
  double* X = Pb + L2;
  double* two = d_two;  // null: the 1-RDM alone
  SBDX_CUDA(c, cudaMemsetAsync(d_one, 0, sizeof(double) * 2 * L2, c->stream));
  if (two) SBDX_CUDA(c, cudaMemsetAsync(two, 0, sizeof(double) * 4 * L4, c->stream));
  if ((rc = phase_vectors(c, dW))) return rc;
  const double* Wm[2] = {reinterpret_cast<const double*>(c->d_xp), reinterpret_cast<const double*>(c->d_xt)};
  const size_t ld[2] = {c->xsa, c->xsb};
  if ((rc = weights(c, Wm[0], ld[0], wa, wb, Pa, Pb, X, Wm[1], ld[1]))) return rc;
  diag_finalize_kernel<<<(unsigned)((L2 + 255) / 256), 256, 0, c->stream>>>(c->L, Pa, Pb, X, d_one, two);
  SBDX_LAUNCHED(c);
  for (int spin = 0; spin < 2; ++spin) {
    if ((rc = rdm_same(c, sc, spin, Wm[spin], ld[spin], two, S[spin], keep[spin]))) return rc;
    if ((rc = rdm_singles(c, sc, spin, Wm[spin], ld[spin], S[spin], d_one, two))) return rc;
  }
  bool done = two == nullptr;  // the alpha-beta pairs only add to the 2-RDM
  if (!done && (rc = rdm_ab_chunks(c, sc, S[0], S[1], two, done))) return rc;
  if (!done) {
    const int staged = sizeof(double) * (L2 + nb) <= kAbSmemBudget;
    const size_t smem = sizeof(double) * (L2 + (staged ? nb : 0));
    if (smem > kAbSmemBudget) { c->err = "rdm: too many orbitals for the shared-memory accumulator"; return 1; }
    SBDX_CUDA(c, cudaFuncSetAttribute(rdm_ab_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAbSmemBudget));
    const Conn& ca = c->conn[0];
    const Conn& cb = c->conn[1];
    rdm_ab_kernel<<<(unsigned)na, 512, smem, c->stream>>>(dW, nb, c->d_a, c->d_b, ca.off, ca.nsing, ca.ket, ca.info,
                                                           cb.off, cb.nsing, cb.ket, cb.info, c->L, two, staged);
    SBDX_LAUNCHED(c);
  }
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
  return 0;
}

int occupation_device(Ctx* c, const double* dW, double* d_density) {
  int rc = ensure_sigma_scratch(c);
  if (rc) return rc;
  const size_t na = c->na, nb = c->nb, L = (size_t)c->L, L2 = L * L;
  Scratch sc(c);
  double* wa = nullptr;
  SBDX_CUDA(c, sc.get(&wa, na + nb + 2 * L2));
  double *wb = wa + na, *Pa = wb + nb, *Pb = Pa + L2;
  double* Wt = reinterpret_cast<double*>(c->d_xt);
  const dim3 grid((unsigned)((nb + 31) / 32), (unsigned)((na + 31) / 32));
  transpose_d_kernel<double><<<grid, dim3(32, 8), 0, c->stream>>>(dW, na, nb, Wt);
  SBDX_LAUNCHED(c);
  if ((rc = weights(c, dW, nb, wa, wb, Pa, Pb, nullptr, Wt, na))) return rc;
  // density[2p] = Pa[p][p], density[2p+1] = Pb[p][p]
  std::vector<double> pab(2 * L2), dens(2 * L);
  SBDX_CUDA(c, cudaMemcpyAsync(pab.data(), Pa, sizeof(double) * 2 * L2, cudaMemcpyDeviceToHost, c->stream));
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
  for (size_t p = 0; p < L; ++p) { dens[2 * p] = pab[p * L + p]; dens[2 * p + 1] = pab[L2 + p * L + p]; }
  SBDX_CUDA(c, cudaMemcpyAsync(d_density, dens.data(), sizeof(double) * 2 * L, cudaMemcpyHostToDevice, c->stream));
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
  return 0;
}

int alpha_weights_device(Ctx* c, const double* dW, double* d_w) {
  const int rc = weights(c, dW, c->nb, d_w, nullptr, nullptr, nullptr, nullptr, nullptr, 0);
  if (rc) return rc;
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
  return 0;
}

int backward_device(Ctx* c, const double* dW, double* dE_dh, double* dE_deri) {
  // the excitation lists are rebuilt from the strings; nothing of the forward
  // solve is kept (the sigma's layouts are not needed and not built: a later
  // sigma rebuilds the full connectivity)
  int rc = build_connectivity(c, false);
  if (rc) return rc;
  const size_t L = (size_t)c->L, L2 = L * L, L4 = L2 * L2;
  Scratch sc(c);
  double* one = nullptr;
  SBDX_CUDA(c, sc.get(&one, 2 * L2 + 4 * L4 + c->neri));
  double *two = one + 2 * L2, *g = two + 4 * L4;
  if ((rc = rdm_device(c, dW, one, two))) return rc;
  backward_eri_kernel<<<(unsigned)((c->neri + 255) / 256), 256, 0, c->stream>>>(c->L, two, g);
  SBDX_LAUNCHED(c);
  std::vector<double> h1(2 * L2);
  SBDX_CUDA(c, cudaMemcpyAsync(h1.data(), one, sizeof(double) * 2 * L2, cudaMemcpyDeviceToHost, c->stream));
  SBDX_CUDA(c, cudaMemcpyAsync(dE_deri, g, sizeof(double) * c->neri, cudaMemcpyDeviceToHost, c->stream));
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
  // one FCIDUMP entry (p, q) sets h[p][q] and h[q][p] (makeintegrals.h:108-112)
  for (size_t p = 0; p < L; ++p)
    for (size_t q = 0; q < L; ++q) {
      const double gpq = h1[p + L * q] + h1[L2 + p + L * q];
      const double gqp = h1[q + L * p] + h1[L2 + q + L * p];
      dE_dh[p * L + q] = p == q ? gpq : gpq + gqp;
    }
  return 0;
}

}  // namespace sbdx
