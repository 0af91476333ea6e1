// Sigma = H * C on the fly (Slater-Condon rules), the hot kernel of the path.
//
// Restates mult (reference chemistry/tpb/mult.h:376-632) at world size 1:
//   S = hii o C                                  (diagonal, :439-444)
//     + sum over alpha singles/doubles, same ib  (task type 2, :484-520)
//     + sum over beta singles/doubles, same ia   (task type 1, :522-556)
//     + sum over alpha single x beta single      (task type 0, :558-578)
// with every matrix element recomputed from the strings, as Hij does
// (chemistry/basic/determinants.h:467-526).
//
// B200 form: the alpha-first kernels (below, "the alpha-first sigma"), which
// evaluate the product in the alpha-before-beta determinant ordering. The
// kernels of the interleaved ordering (launch codes 1 to 49) are kept for
// comparison; one such sigma is 5 launches:
//   1. same-spin kernel over alpha rows of C: a CTA owns one bra alpha row ia
//      and a strip of beta columns; it walks the connectivity list of ia
//      (staged in shared memory) and streams the ket rows C[ja, strip]
//      coalesced, so every pair costs one 8/4-byte load, one popcount (the
//      beta-dependent sign) and one FMA; hii o C initialises the accumulator.
//   2. transpose C -> C^T (tiled through shared memory)
//   3. the same kernel over beta rows of C^T (beta excitations become row
//      streams too), writing S^T
//   4. alpha-beta kernel: a CTA owns one bra alpha row ia; for each alpha
//      single ja of ia it stages the whole ket row C[ja, :] and the integral
//      row (ai|..) in shared memory, then every thread sums its bra beta
//      strings' beta singles as shared-memory gathers; the sign splits into an
//      alpha factor (once per thread and ja) and a beta factor (per pair)
//   5. S = S_alpha + S_ab + (S^T)^T, converted to the output precision.
// Accumulation is FP64 in every precision mode ("FP64 per-row accumulation");
// FP32 mode reads FP32 vectors and FP32 matrix elements.
#include "sbdx_internal.cuh"

#include <cstdint>
#include <type_traits>
#include <vector>

namespace sbdx {

namespace {

constexpr int kSameThreads = 256;

// D += A B on the FP64 tensor pipe: A 8 x 4 (lane: row lane >> 2, k lane & 3),
// B 4 x 8 (k lane & 3, column lane >> 2), D row lane >> 2, columns 2 (lane & 3)
// + {0, 1}.
__device__ __forceinline__ void dmma_m8n8k4(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

template <typename T> struct Prec;
template <> struct Prec<double> { using V = double; };
template <> struct Prec<float> { using V = float; };

// ---- v2 kernels ----------------------------------------------------------------

template <typename T, int VEC> struct VecIO;
template <> struct VecIO<double, 1> {
  static __device__ __forceinline__ void load(const double* p, double* o) { o[0] = __ldg(p); }
};
template <> struct VecIO<double, 2> {
  static __device__ __forceinline__ void load(const double* p, double* o) {
    const double2 v = __ldg(reinterpret_cast<const double2*>(p));
    o[0] = v.x; o[1] = v.y;
  }
};
template <> struct VecIO<double, 4> {
  static __device__ __forceinline__ void load(const double* p, double* o) {
    const double2 v = __ldg(reinterpret_cast<const double2*>(p));
    const double2 w = __ldg(reinterpret_cast<const double2*>(p) + 1);
    o[0] = v.x; o[1] = v.y; o[2] = w.x; o[3] = w.y;
  }
};
template <> struct VecIO<float, 1> {
  static __device__ __forceinline__ void load(const float* p, double* o) { o[0] = (double)__ldg(p); }
};
template <> struct VecIO<float, 2> {
  static __device__ __forceinline__ void load(const float* p, double* o) {
    const float2 v = __ldg(reinterpret_cast<const float2*>(p));
    o[0] = v.x; o[1] = v.y;
  }
};
template <> struct VecIO<float, 4> {
  static __device__ __forceinline__ void load(const float* p, double* o) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  }
};

// Same-spin excitations, VEC consecutive columns per thread. Grid: x = bra
// row (fastest, so the CTAs resident at one time share one column strip of the
// ket rows and the strip stays in L2), y = column strip of kSameThreads*VEC.
// Requires ncol % VEC == 0 (the host picks VEC accordingly).
template <typename T, int VEC>
__global__ void __launch_bounds__(kSameThreads)
sigma_same_v2_kernel(const T* __restrict__ X, size_t ncol, const uint64_t* __restrict__ other,
                     const uint64_t* __restrict__ off, const uint32_t* __restrict__ nsing,
                     const uint32_t* __restrict__ ket, const typename Prec<T>::V* __restrict__ val,
                     const uint64_t* __restrict__ omask, const uint32_t* __restrict__ info,
                     const typename Prec<T>::V* __restrict__ G, int L, const double* __restrict__ hii,
                     double* __restrict__ Y) {
  using V = typename Prec<T>::V;
  const size_t r = blockIdx.x;
  const size_t c0 = ((size_t)blockIdx.y * kSameThreads + threadIdx.x) * VEC;
  const bool active = c0 < ncol;
  uint64_t o[VEC];
  uint32_t olo[VEC], ohi[VEC];
  double acc[VEC];
#pragma unroll
  for (int v = 0; v < VEC; ++v) {
    o[v] = active ? other[c0 + v] : 0ull;
    olo[v] = (uint32_t)o[v];
    ohi[v] = (uint32_t)(o[v] >> 32);
    acc[v] = 0.0;
  }
  if (hii != nullptr && active) {
    double x[VEC];
    VecIO<T, VEC>::load(X + r * ncol + c0, x);
#pragma unroll
    for (int v = 0; v < VEC; ++v) acc[v] = hii[r * ncol + c0 + v] * x[v];
  }
  __shared__ uint32_t s_ket[kSameThreads], s_info[kSameThreads];
  __shared__ uint64_t s_om[kSameThreads];
  __shared__ V s_val[kSameThreads];
  const uint64_t beg = off[r], end = off[r + 1], send = beg + nsing[r];
  for (uint64_t base = beg; base < end; base += kSameThreads) {
    const int cnt = (int)min((uint64_t)kSameThreads, end - base);
    const int nsb = send > base ? (int)min((uint64_t)cnt, send - base) : 0;
    __syncthreads();
    if ((int)threadIdx.x < cnt) {
      const uint64_t e = base + threadIdx.x;
      s_ket[threadIdx.x] = ket[e];
      s_info[threadIdx.x] = info[e];
      s_om[threadIdx.x] = omask[e];
      s_val[threadIdx.x] = val[e];
    }
    __syncthreads();
    if (!active) continue;
    // singles: value + opposite-spin Coulomb sum_{q in other} (ai|qq)
    for (int e = 0; e < nsb; ++e) {
      const uint32_t inf = s_info[e];
      const double hv0 = (double)s_val[e];
      const uint64_t om = s_om[e];
      const V* g = G + (size_t)((inf >> 12) & 0xfffu) * L;
      double x[VEC];
      VecIO<T, VEC>::load(X + (size_t)s_ket[e] * ncol + c0, x);
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        double hv = hv0;
        uint64_t bits = o[v];
        while (bits) {
          const int q = __ffsll((long long)bits) - 1;
          bits &= bits - 1;
          hv += (double)g[q];
        }
        const uint32_t neg = (uint32_t)popc64(o[v] & om) ^ (inf >> 31);
        acc[v] = fma(flip_sign(hv, neg), x[v], acc[v]);
      }
    }
    // doubles: one popcount per pair
#pragma unroll 2
    for (int e = nsb; e < cnt; ++e) {
      const uint32_t sgn = s_info[e] >> 31;
      const double hv = (double)s_val[e];
      const uint64_t om = s_om[e];
      const uint32_t omlo = (uint32_t)om, omhi = (uint32_t)(om >> 32);
      double x[VEC];
      VecIO<T, VEC>::load(X + (size_t)s_ket[e] * ncol + c0, x);
#pragma unroll
      for (int v = 0; v < VEC; ++v)
        acc[v] = fma(flip_sign(hv, and_parity(olo[v], ohi[v], omlo, omhi) + sgn), x[v], acc[v]);
    }
  }
  if (active) {
#pragma unroll
    for (int v = 0; v < VEC; ++v) Y[r * ncol + c0 + v] = acc[v];
  }
}

template <> struct VecIO<double, 8> {
  static __device__ __forceinline__ void load(const double* p, double* o) {
    const double2* q = reinterpret_cast<const double2*>(p);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double2 v = __ldg(q + k);
      o[2 * k] = v.x; o[2 * k + 1] = v.y;
    }
  }
};
template <> struct VecIO<float, 8> {
  static __device__ __forceinline__ void load(const float* p, double* o) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    const float4 w = __ldg(reinterpret_cast<const float4*>(p) + 1);
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; o[4] = w.x; o[5] = w.y; o[6] = w.z; o[7] = w.w;
  }
};

constexpr int kParityRows = 65;  // prefix-parity positions 0..64

// Same-spin excitations, v4. As v2 (VEC consecutive columns per thread,
// rows-fastest grid) but the opposite-spin sign of an entry is read from a
// per-thread table of prefix parities in shared memory: tab[x][t] bit v =
// parity(other[c0+v] & bits[0,x)); an entry's sign for all VEC columns is the
// xor of four table bytes at its boundary positions (spos). No popcount in
// the inner loop.
template <typename T, int VEC>
__global__ void __launch_bounds__(kSameThreads)
sigma_same_v4_kernel(const T* __restrict__ X, size_t ncol, const uint64_t* __restrict__ other,
                     const uint64_t* __restrict__ off, const uint32_t* __restrict__ nsing,
                     const uint32_t* __restrict__ ket, const typename Prec<T>::V* __restrict__ val,
                     const uint32_t* __restrict__ spos, const uint32_t* __restrict__ info,
                     const typename Prec<T>::V* __restrict__ G, int L, const double* __restrict__ hii,
                     double* __restrict__ Y) {
  static_assert(VEC <= 8, "one byte of parity bits per thread");
  using V = typename Prec<T>::V;
  __shared__ uint8_t tab[kParityRows][kSameThreads];
  __shared__ uint32_t s_ket[kSameThreads], s_pos[kSameThreads];
  __shared__ V s_val[kSameThreads];
  const size_t r = blockIdx.x;
  const size_t c0 = ((size_t)blockIdx.y * kSameThreads + threadIdx.x) * VEC;
  const bool active = c0 < ncol;
  uint64_t o[VEC];
  double acc[VEC];
  {
    uint64_t P[VEC];
#pragma unroll
    for (int v = 0; v < VEC; ++v) {
      o[v] = active ? other[c0 + v] : 0ull;
      P[v] = prefix_parity(o[v]);
      acc[v] = 0.0;
    }
    tab[0][threadIdx.x] = 0;
    for (int x = 1; x < kParityRows; ++x) {
      uint32_t b = 0;
#pragma unroll
      for (int v = 0; v < VEC; ++v) b |= (uint32_t)((P[v] >> (x - 1)) & 1ull) << v;
      tab[x][threadIdx.x] = (uint8_t)b;
    }
  }
  if (hii != nullptr && active) {
    double x[VEC];
    VecIO<T, VEC>::load(X + r * ncol + c0, x);
#pragma unroll
    for (int v = 0; v < VEC; ++v) acc[v] = hii[r * ncol + c0 + v] * x[v];
  }
  const uint64_t beg = off[r], end = off[r + 1], send = beg + nsing[r];
  const unsigned t = threadIdx.x;
  for (uint64_t base = beg; base < end; base += kSameThreads) {
    const int cnt = (int)min((uint64_t)kSameThreads, end - base);
    const int nsb = send > base ? (int)min((uint64_t)cnt, send - base) : 0;
    __syncthreads();
    if ((int)t < cnt) {
      const uint64_t e = base + t;
      s_ket[t] = ket[e];
      s_pos[t] = spos[e];
      s_val[t] = val[e];
    }
    __syncthreads();
    if (!active) continue;
    for (int e = 0; e < nsb; ++e) {
      const uint32_t ps = s_pos[e];
      const uint32_t neg = (uint32_t)tab[ps & 127u][t] ^ (uint32_t)tab[(ps >> 7) & 127u][t] ^ ((ps >> 31) ? 0xffu : 0u);
      const uint32_t inf = info[base + e];
      const V* g = G + (size_t)((inf >> 12) & 0xfffu) * L;
      const double hv0 = (double)s_val[e];
      double x[VEC];
      VecIO<T, VEC>::load(X + (size_t)s_ket[e] * ncol + c0, x);
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        double hv = hv0;
        uint64_t bits = o[v];
        while (bits) {
          const int q = __ffsll((long long)bits) - 1;
          bits &= bits - 1;
          hv += (double)g[q];
        }
        acc[v] = fma(flip_sign(hv, neg >> v), x[v], acc[v]);
      }
    }
#pragma unroll 2
    for (int e = nsb; e < cnt; ++e) {
      const uint32_t ps = s_pos[e];
      const uint32_t neg = (uint32_t)tab[ps & 127u][t] ^ (uint32_t)tab[(ps >> 7) & 127u][t] ^
                           (uint32_t)tab[(ps >> 14) & 127u][t] ^ (uint32_t)tab[(ps >> 21) & 127u][t] ^
                           ((ps >> 31) ? 0xffu : 0u);
      const double hv = (double)s_val[e];
      double x[VEC];
      VecIO<T, VEC>::load(X + (size_t)s_ket[e] * ncol + c0, x);
#pragma unroll
      for (int v = 0; v < VEC; ++v) acc[v] = fma(flip_sign(hv, neg >> v), x[v], acc[v]);
    }
  }
  if (active) {
#pragma unroll
    for (int v = 0; v < VEC; ++v) Y[r * ncol + c0 + v] = acc[v];
  }
}

constexpr int kAb2Threads = 1024;
constexpr int kAb2Slots = 8;  // beta strings per thread per CTA (register accumulators)

// Slot k of thread t takes position k*nthreads + t of the list-length order on
// even k and k*nthreads + (nthreads-1-t) on odd k, so every thread's lists add
// up to about the same length (a plain stride gives warp 0 the longest list of
// every slot).
__device__ __forceinline__ size_t snake_index(size_t chunk0, int k, int nthreads, int t) {
  return chunk0 + (size_t)k * nthreads + (size_t)((k & 1) ? (nthreads - 1 - t) : t);
}

// Alpha single x beta single, v2. One CTA per (bra alpha row ia, chunk of the
// beta order). R ket rows C[ja, :] of the alpha singles of ia and their
// integral rows (ai|..) are staged in shared memory per pass; each thread owns
// up to kAb2Slots bra beta strings (taken from the list-length order) and
// walks their beta-single records once per pass, applying each record to all
// R staged rows. Sign: alpha factor s_a (-1)^{|beta(ib) & [lo_a,hi_a)|} per
// (thread, row) and beta factor s_b (-1)^{|alpha(ja) & (lo_b,hi_b]|} per pair,
// the latter from the prefix-parity word of alpha(ja).
template <typename T, int R, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT)
sigma_ab_v2_kernel(const T* __restrict__ X, size_t nb, const uint64_t* __restrict__ astr,
                   const uint64_t* __restrict__ bstr, const uint64_t* __restrict__ a_off,
                   const uint32_t* __restrict__ a_nsing, const uint32_t* __restrict__ a_ket,
                   const uint32_t* __restrict__ a_info, const uint64_t* __restrict__ a_omask,
                   const uint64_t* __restrict__ b_off, const uint32_t* __restrict__ b_nsing,
                   const uint64_t* __restrict__ b_rec, const uint32_t* __restrict__ b_order,
                   const typename Prec<T>::V* __restrict__ eri, int npair, size_t xstride,
                   double* __restrict__ Y) {
  using V = typename Prec<T>::V;
  constexpr int kSlots = 8192 / NT;
  extern __shared__ __align__(16) unsigned char smem[];
  T* xs = reinterpret_cast<T*>(smem);                                  // [R][xstride]
  V* erow = reinterpret_cast<V*>(smem + sizeof(T) * xstride * R);     // [R][npair]
  __shared__ uint64_t s_P[R], s_M[R];
  __shared__ uint32_t s_sa[R];
  const size_t ia = blockIdx.x;
  const size_t chunk0 = (size_t)blockIdx.y * NT * kSlots;
  double acc[kSlots];
#pragma unroll
  for (int k = 0; k < kSlots; ++k) acc[k] = 0.0;
  const uint64_t e0 = a_off[ia];
  const int ns = (int)a_nsing[ia];
  for (int k0 = 0; k0 < ns; k0 += R) {
    const int nr = min(R, ns - k0);
    __syncthreads();
    if ((int)threadIdx.x < nr) {
      const uint64_t e = e0 + k0 + threadIdx.x;
      const uint32_t inf = a_info[e];
      s_P[threadIdx.x] = prefix_parity(astr[a_ket[e]]);
      s_M[threadIdx.x] = a_omask[e];
      s_sa[threadIdx.x] = inf >> 31;
    }
    for (int rr = 0; rr < nr; ++rr) {
      const uint64_t e = e0 + k0 + rr;
      const T* xrow = X + (size_t)a_ket[e] * nb;
      T* dst = xs + (size_t)rr * xstride;
      for (size_t t = threadIdx.x; t < nb; t += NT) dst[t] = xrow[t];
      const size_t pq = (a_info[e] >> 12) & 0xfffu;
      V* er = erow + (size_t)rr * npair;
      for (int t = threadIdx.x; t < npair; t += NT) er[t] = eri[pair2_index(pq, (size_t)t)];
    }
    __syncthreads();
    uint64_t P[R], M[R];
    uint32_t sa[R];
#pragma unroll
    for (int rr = 0; rr < R; ++rr) {
      P[rr] = rr < nr ? s_P[rr] : 0ull;
      M[rr] = rr < nr ? s_M[rr] : 0ull;
      sa[rr] = rr < nr ? s_sa[rr] : 0u;
    }
#pragma unroll
    for (int k = 0; k < kSlots; ++k) {
      const size_t idx = snake_index(chunk0, k, NT, threadIdx.x);
      if (idx >= nb) continue;
      const uint32_t ib = b_order[idx];
      const uint64_t bI = bstr[ib];
      uint32_t base[R];
#pragma unroll
      for (int rr = 0; rr < R; ++rr) base[rr] = sa[rr] ^ (uint32_t)popc64(bI & M[rr]);
      const uint64_t m0 = b_off[ib], m1 = m0 + b_nsing[ib];
      double s = acc[k];
      uint64_t next = m0 < m1 ? __ldg(b_rec + m0) : 0ull;
      for (uint64_t m = m0; m < m1; ++m) {
        const uint64_t rec = next;
        if (m + 1 < m1) next = __ldg(b_rec + m + 1);
        const uint32_t jb = rec_ket(rec);
        const uint32_t pq = (uint32_t)((rec >> 16) & 0xfffu);
        const uint32_t lo = (uint32_t)((rec >> 28) & 63u), hi = (uint32_t)((rec >> 34) & 63u);
        const uint32_t sb = (uint32_t)(rec >> 40);
#pragma unroll
        for (int rr = 0; rr < R; ++rr) {
          if (rr < nr) {
            const uint32_t par = base[rr] ^ sb ^ (uint32_t)((P[rr] >> hi) ^ (P[rr] >> lo));
            const double v = (double)erow[(size_t)rr * npair + pq];
            s = fma(flip_sign(v, par), (double)xs[(size_t)rr * xstride + jb], s);
          }
        }
      }
      acc[k] = s;
    }
  }
#pragma unroll
  for (int k = 0; k < kSlots; ++k) {
    const size_t idx = snake_index(chunk0, k, NT, threadIdx.x);
    if (idx < nb) {
      const uint32_t ib = b_order[idx];
      Y[ia * nb + ib] += acc[k];
    }
  }
}

// Alpha single x beta single, v5: the v2 staging scheme with the beta-single
// records read in SELL-32 layout. Warp w of the CTA owns slices w, 63-w,
// 64+w, ... (a snake over the length-sorted slices, so warps get equal work);
// lane l of a slice owns bra beta string order[32s+l]. Every record load of a
// warp is one contiguous 256-byte read; padded records contribute zero.
template <typename T, int R, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT)
sigma_ab_v5_kernel(const T* __restrict__ X, size_t nb, const uint64_t* __restrict__ astr,
                   const uint64_t* __restrict__ bstr, const uint64_t* __restrict__ a_off,
                   const uint32_t* __restrict__ a_nsing, const uint32_t* __restrict__ a_ket,
                   const uint32_t* __restrict__ a_info, const uint64_t* __restrict__ a_omask,
                   const uint64_t* __restrict__ sell, const uint64_t* __restrict__ soff,
                   const uint32_t* __restrict__ slen, size_t nslice, const uint32_t* __restrict__ b_order,
                   const typename Prec<T>::V* __restrict__ eri, int npair, size_t xstride,
                   double* __restrict__ Y) {
  using V = typename Prec<T>::V;
  constexpr int kWarps = NT / 32;
  constexpr int kSlices = 8192 / NT;  // slices per warp per CTA (32*kWarps*kSlices = 8192 strings)
  extern __shared__ __align__(16) unsigned char smem[];
  T* xs = reinterpret_cast<T*>(smem);
  V* erow = reinterpret_cast<V*>(smem + sizeof(T) * xstride * R);
  __shared__ uint64_t s_P[R], s_M[R];
  __shared__ uint32_t s_sa[R];
  const size_t ia = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t slice0 = (size_t)blockIdx.y * kWarps * kSlices;
  auto slice_of = [&](int k) -> size_t {
    return slice0 + (size_t)k * kWarps + ((k & 1) ? (kWarps - 1 - warp) : warp);
  };
  uint64_t bI[kSlices];
  double acc[kSlices];
#pragma unroll
  for (int k = 0; k < kSlices; ++k) {
    const size_t sl = slice_of(k);
    const size_t pos = sl * 32 + lane;
    bI[k] = (sl < nslice && pos < nb) ? bstr[b_order[pos]] : 0ull;
    acc[k] = 0.0;
  }
  const uint64_t e0 = a_off[ia];
  const int ns = (int)a_nsing[ia];
  for (int k0 = 0; k0 < ns; k0 += R) {
    const int nr = min(R, ns - k0);
    __syncthreads();
    if ((int)threadIdx.x < nr) {
      const uint64_t e = e0 + k0 + threadIdx.x;
      s_P[threadIdx.x] = prefix_parity(astr[a_ket[e]]);
      s_M[threadIdx.x] = a_omask[e];
      s_sa[threadIdx.x] = a_info[e] >> 31;
    }
    for (int rr = 0; rr < nr; ++rr) {
      const uint64_t e = e0 + k0 + rr;
      const T* xrow = X + (size_t)a_ket[e] * nb;
      T* dst = xs + (size_t)rr * xstride;
      for (size_t t = threadIdx.x; t < nb; t += NT) dst[t] = xrow[t];
      const size_t pq = (a_info[e] >> 12) & 0xfffu;
      V* er = erow + (size_t)rr * npair;
      for (int t = threadIdx.x; t < npair; t += NT) er[t] = eri[pair2_index(pq, (size_t)t)];
    }
    __syncthreads();
    uint64_t P[R], M[R];
    uint32_t sa[R];
#pragma unroll
    for (int rr = 0; rr < R; ++rr) {
      P[rr] = rr < nr ? s_P[rr] : 0ull;
      M[rr] = rr < nr ? s_M[rr] : 0ull;
      sa[rr] = rr < nr ? s_sa[rr] : 0u;
    }
#pragma unroll
    for (int k = 0; k < kSlices; ++k) {
      const size_t sl = slice_of(k);
      if (sl >= nslice) continue;
      uint32_t base[R];
#pragma unroll
      for (int rr = 0; rr < R; ++rr) base[rr] = sa[rr] ^ (uint32_t)popc64(bI[k] & M[rr]);
      const uint32_t len = slen[sl];
      const uint64_t* rp = sell + soff[sl] + lane;
      double s = acc[k];
      uint64_t next = len ? __ldg(rp) : 0ull;
      for (uint32_t m = 0; m < len; ++m) {
        const uint64_t rec = next;
        if (m + 1 < len) next = __ldg(rp + 32ull * (m + 1));
        const uint32_t jb = rec_ket(rec);
        const uint32_t pq = (uint32_t)((rec >> 16) & 0xfffu);
        const uint32_t lo = (uint32_t)((rec >> 28) & 63u), hi = (uint32_t)((rec >> 34) & 63u);
        const uint32_t sb = (uint32_t)(rec >> 40);
        const bool pad = (rec >> 41) & 1ull;
#pragma unroll
        for (int rr = 0; rr < R; ++rr) {
          if (rr < nr) {
            const uint32_t par = base[rr] ^ sb ^ (uint32_t)((P[rr] >> hi) ^ (P[rr] >> lo));
            const double v = pad ? 0.0 : (double)erow[(size_t)rr * npair + pq];
            s = fma(flip_sign(v, par), (double)xs[(size_t)rr * xstride + jb], s);
          }
        }
      }
      acc[k] = s;
    }
  }
#pragma unroll
  for (int k = 0; k < kSlices; ++k) {
    const size_t sl = slice_of(k);
    const size_t pos = sl * 32 + lane;
    if (sl < nslice && pos < nb) Y[ia * nb + b_order[pos]] += acc[k];
  }
}

// ---- double-buffered TMA staging ---------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Bounded wait: gives up when the phase has not completed after `limit_ns`
// nanoseconds of the global timer (or 2^26 polls, whichever comes first).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint64_t limit_ns) {
  const uint64_t t0 = global_ns();
  for (uint32_t it = 0; it < (1u << 26); ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 255u) == 255u && global_ns() - t0 > limit_ns) return false;
  }
  return false;
}
__device__ __forceinline__ void tma_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

constexpr uint64_t kWaitLimit = 2000000000ull;  // 2 s

// Alpha single x beta single, v4: as v2, with the R ket rows and integral
// rows of the next group of alpha singles loaded by TMA (cp.async.bulk, one
// issuing thread) into the second of two shared-memory buffers while the
// current group is computed. Requires 16-byte aligned rows (nb*sizeof(T) % 16
// == 0 and a 16-byte aligned X); the host checks this.
template <typename T, int R>
__global__ void __launch_bounds__(kAb2Threads, 1)
sigma_ab_v4_kernel(const T* __restrict__ X, size_t nb, const uint64_t* __restrict__ astr,
                   const uint64_t* __restrict__ bstr, const uint64_t* __restrict__ a_off,
                   const uint32_t* __restrict__ a_nsing, const uint32_t* __restrict__ a_ket,
                   const uint32_t* __restrict__ a_info, const uint64_t* __restrict__ a_omask,
                   const uint64_t* __restrict__ b_off, const uint32_t* __restrict__ b_nsing,
                   const uint64_t* __restrict__ b_rec, const uint32_t* __restrict__ b_order,
                   const typename Prec<T>::V* __restrict__ Vtab, size_t vstride, int* __restrict__ err,
                   double* __restrict__ Y) {
  using V = typename Prec<T>::V;
  extern __shared__ __align__(128) unsigned char smem[];
  const size_t xbytes = sizeof(T) * nb, vbytes = sizeof(V) * vstride;
  const size_t bufbytes = (size_t)R * (xbytes + vbytes);
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ int s_abort;
  const size_t ia = blockIdx.x;
  const size_t chunk0 = (size_t)blockIdx.y * kAb2Threads * kAb2Slots;
  const uint64_t e0 = a_off[ia];
  const int ns = (int)a_nsing[ia];
  const int ngroups = (ns + R - 1) / R;
  if (threadIdx.x == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_abort = 0;
  }
  __syncthreads();
  auto issue = [&](int g) {  // thread 0 only
    const int b = g & 1;
    const int nr = min(R, ns - g * R);
    unsigned char* buf = smem + (size_t)b * bufbytes;
    mbar_arrive_expect_tx(&bar[b], (uint32_t)(nr * (xbytes + vbytes)));
    for (int rr = 0; rr < nr; ++rr) {
      const uint64_t e = e0 + (uint64_t)g * R + rr;
      const size_t ja = a_ket[e];
      const size_t pq = (a_info[e] >> 12) & 0xfffu;
      tma_load_1d(buf + (size_t)rr * xbytes, X + ja * nb, (uint32_t)xbytes, &bar[b]);
      tma_load_1d(buf + (size_t)R * xbytes + (size_t)rr * vbytes, Vtab + pq * vstride, (uint32_t)vbytes, &bar[b]);
    }
  };
  if (threadIdx.x == 0) {
    if (ngroups > 0) issue(0);
    if (ngroups > 1) issue(1);
  }
  double acc[kAb2Slots];
#pragma unroll
  for (int k = 0; k < kAb2Slots; ++k) acc[k] = 0.0;
  int g_abort = -1;  // group whose wait timed out (the same in every thread)
  for (int g = 0; g < ngroups; ++g) {
    const int b = g & 1;
    const int nr = min(R, ns - g * R);
    if (!mbar_wait_bounded(&bar[b], (uint32_t)((g >> 1) & 1), kWaitLimit)) {
      atomicExch(err, kErrWatchdogAb);
      s_abort = 1;
    }
    __syncthreads();
    if (s_abort) { g_abort = g; break; }
    const T* xs = reinterpret_cast<const T*>(smem + (size_t)b * bufbytes);
    const V* erow = reinterpret_cast<const V*>(smem + (size_t)b * bufbytes + (size_t)R * xbytes);
    uint64_t P[R], M[R];
    uint32_t sa[R];
#pragma unroll
    for (int rr = 0; rr < R; ++rr) {
      const uint64_t e = e0 + (uint64_t)g * R + (rr < nr ? rr : 0);
      const uint32_t inf = __ldg(a_info + e);
      P[rr] = prefix_parity(__ldg(astr + __ldg(a_ket + e)));
      M[rr] = __ldg(a_omask + e);
      sa[rr] = inf >> 31;
    }
#pragma unroll
    for (int k = 0; k < kAb2Slots; ++k) {
      const size_t idx = snake_index(chunk0, k, kAb2Threads, threadIdx.x);
      if (idx >= nb) continue;
      const uint32_t ib = __ldg(b_order + idx);
      const uint64_t bI = __ldg(bstr + ib);
      uint32_t base[R];
#pragma unroll
      for (int rr = 0; rr < R; ++rr) base[rr] = sa[rr] ^ (uint32_t)popc64(bI & M[rr]);
      const uint64_t m0 = __ldg(b_off + ib), m1 = m0 + __ldg(b_nsing + ib);
      double s = acc[k];
      uint64_t next = m0 < m1 ? __ldg(b_rec + m0) : 0ull;
      for (uint64_t m = m0; m < m1; ++m) {
        const uint64_t rec = next;
        if (m + 1 < m1) next = __ldg(b_rec + m + 1);
        const uint32_t jb = rec_ket(rec);
        const uint32_t pq = (uint32_t)((rec >> 16) & 0xfffu);
        const uint32_t lo = (uint32_t)((rec >> 28) & 63u), hi = (uint32_t)((rec >> 34) & 63u);
        const uint32_t sb = (uint32_t)(rec >> 40);
#pragma unroll
        for (int rr = 0; rr < R; ++rr) {
          if (rr < nr) {
            const uint32_t par = base[rr] ^ sb ^ (uint32_t)((P[rr] >> hi) ^ (P[rr] >> lo));
            const double v = (double)erow[(size_t)rr * vstride + pq];
            s = fma(flip_sign(v, par), (double)xs[(size_t)rr * nb + jb], s);
          }
        }
      }
      acc[k] = s;
    }
    __syncthreads();  // buffer b is free again
    if (threadIdx.x == 0 && g + 2 < ngroups) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      issue(g + 2);
    }
  }
  if (g_abort >= 0) {
    // Leave no bulk copy in flight into this CTA's shared memory. The groups
    // still outstanding are g_abort (its wait timed out) and g_abort + 1 when
    // it was issued; group q completes phase (q >> 1) & 1 of barrier q & 1.
    // Groups before g_abort were all waited for, and g_abort + 2 was never
    // issued (issue(g + 2) follows a completed group g).
    if (threadIdx.x == 0)
      for (int q = g_abort; q < min(g_abort + 2, ngroups); ++q)
        mbar_wait_bounded(&bar[q & 1], (uint32_t)((q >> 1) & 1), kWaitLimit);
    return;
  }
#pragma unroll
  for (int k = 0; k < kAb2Slots; ++k) {
    const size_t idx = snake_index(chunk0, k, kAb2Threads, threadIdx.x);
    if (idx < nb) Y[ia * nb + b_order[idx]] += acc[k];
  }
}

constexpr int kAb3Threads = 256;
constexpr int kAb3Slots = 8;

// Alpha single x beta single, v3: no shared-memory staging and no barriers.
// One CTA per (bra alpha row ia, chunk of kAb3Threads*kAb3Slots beta strings
// of the list-length order). Each thread walks the alpha singles of ia in
// groups of R and, for each of its bra beta strings, the beta-single records;
// the ket values C[ja, jb] and the integrals (ai|bj) (row pq(a,i) of the
// unpacked table) are gathered through L1, where the R rows shared by the CTA
// stay resident.
template <typename T, int R>
__global__ void __launch_bounds__(kAb3Threads)
sigma_ab_v3_kernel(const T* __restrict__ X, size_t nb, const uint64_t* __restrict__ astr,
                   const uint64_t* __restrict__ bstr, const uint64_t* __restrict__ a_off,
                   const uint32_t* __restrict__ a_nsing, const uint32_t* __restrict__ a_ket,
                   const uint32_t* __restrict__ a_info, const uint64_t* __restrict__ a_omask,
                   const uint64_t* __restrict__ b_off, const uint32_t* __restrict__ b_nsing,
                   const uint64_t* __restrict__ b_rec, const uint32_t* __restrict__ b_order,
                   const typename Prec<T>::V* __restrict__ V, int npair, double* __restrict__ Y) {
  using VT = typename Prec<T>::V;
  const size_t ia = blockIdx.x;
  const size_t chunk0 = (size_t)blockIdx.y * kAb3Threads * kAb3Slots;
  uint32_t ibs[kAb3Slots];
  uint32_t bIlo[kAb3Slots], bIhi[kAb3Slots];
  double acc[kAb3Slots];
#pragma unroll
  for (int k = 0; k < kAb3Slots; ++k) {
    const size_t idx = chunk0 + (size_t)k * kAb3Threads + threadIdx.x;
    ibs[k] = idx < nb ? b_order[idx] : 0xffffffffu;
    const uint64_t b = idx < nb ? bstr[ibs[k]] : 0ull;
    bIlo[k] = (uint32_t)b;
    bIhi[k] = (uint32_t)(b >> 32);
    acc[k] = 0.0;
  }
  const uint64_t e0 = a_off[ia];
  const int ns = (int)a_nsing[ia];
  for (int k0 = 0; k0 < ns; k0 += R) {
    const int nr = min(R, ns - k0);
    const T* xr[R];
    const VT* vr[R];
    uint64_t P[R];
    uint32_t Mlo[R], Mhi[R], sa[R];
#pragma unroll
    for (int rr = 0; rr < R; ++rr) {
      const uint64_t e = e0 + k0 + (rr < nr ? rr : 0);
      const uint32_t inf = __ldg(a_info + e);
      const uint32_t ja = __ldg(a_ket + e);
      const uint64_t m = __ldg(a_omask + e);
      xr[rr] = X + (size_t)ja * nb;
      vr[rr] = V + (size_t)((inf >> 12) & 0xfffu) * (size_t)npair;
      P[rr] = prefix_parity(__ldg(astr + ja));
      Mlo[rr] = (uint32_t)m;
      Mhi[rr] = (uint32_t)(m >> 32);
      sa[rr] = inf >> 31;
    }
#pragma unroll
    for (int k = 0; k < kAb3Slots; ++k) {
      if (ibs[k] == 0xffffffffu) continue;
      const uint32_t ib = ibs[k];
      uint32_t base[R];
#pragma unroll
      for (int rr = 0; rr < R; ++rr) base[rr] = sa[rr] + and_parity(bIlo[k], bIhi[k], Mlo[rr], Mhi[rr]);
      const uint64_t m0 = __ldg(b_off + ib), m1 = m0 + __ldg(b_nsing + ib);
      double s = acc[k];
      uint64_t next = m0 < m1 ? __ldg(b_rec + m0) : 0ull;
      for (uint64_t m = m0; m < m1; ++m) {
        const uint64_t rec = next;
        if (m + 1 < m1) next = __ldg(b_rec + m + 1);
        const uint32_t jb = rec_ket(rec);
        const uint32_t pq = (uint32_t)((rec >> 16) & 0xfffu);
        const uint32_t lo = (uint32_t)((rec >> 28) & 63u), hi = (uint32_t)((rec >> 34) & 63u);
        const uint32_t sb = (uint32_t)(rec >> 40);
#pragma unroll
        for (int rr = 0; rr < R; ++rr) {
          if (rr < nr) {
            const uint32_t par = base[rr] + sb + (uint32_t)((P[rr] >> hi) ^ (P[rr] >> lo));
            const double v = (double)__ldg(vr[rr] + pq);
            s = fma(flip_sign(v, par), (double)__ldg(xr[rr] + jb), s);
          }
        }
      }
      acc[k] = s;
    }
  }
#pragma unroll
  for (int k = 0; k < kAb3Slots; ++k)
    if (ibs[k] != 0xffffffffu) Y[ia * nb + ibs[k]] += acc[k];
}

__global__ void unpack_eri_kernel(const double* __restrict__ eri, size_t npair, size_t vs, size_t vs32,
                                  double* __restrict__ V, float* __restrict__ V32) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npair * npair) return;
  const size_t r = t / npair, q = t % npair;
  const double v = eri[pair2_index(r, q)];
  V[r * vs + q] = v;
  V32[r * vs32 + q] = (float)v;
}

template <typename T>
__global__ void transpose_kernel(const T* __restrict__ in, size_t rows, size_t cols, T* __restrict__ out) {
  __shared__ T tile[32][33];
  const size_t c0 = (size_t)blockIdx.x * 32, r0 = (size_t)blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const size_t r = r0 + k, c = c0 + threadIdx.x;
    if (r < rows && c < cols) tile[k][threadIdx.x] = in[r * cols + c];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const size_t c = c0 + k, r = r0 + threadIdx.x;  // out row = c, out col = r
    if (r < rows && c < cols) out[c * rows + r] = tile[threadIdx.x][k];
  }
}

// S[ia, ib] = Y[ia, ib] + Yt[ib, ia], stored in T.
template <typename T>
__global__ void combine_transpose_kernel(const double* __restrict__ Y, const double* __restrict__ Yt,
                                         size_t na, size_t nb, T* __restrict__ S) {
  __shared__ double tile[32][33];
  const size_t ib0 = (size_t)blockIdx.x * 32, ia0 = (size_t)blockIdx.y * 32;
  // load Yt rows ib0.. (cols ia0..) transposed into tile[ia][ib]
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const size_t ib = ib0 + k, ia = ia0 + threadIdx.x;
    if (ib < nb && ia < na) tile[threadIdx.x][k] = Yt[ib * na + ia];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const size_t ia = ia0 + k, ib = ib0 + threadIdx.x;
    if (ia < na && ib < nb) S[ia * nb + ib] = (T)(Y[ia * nb + ib] + tile[k][threadIdx.x]);
  }
}

__global__ void g_table_kernel(const double* __restrict__ eri, int L, size_t npair, double* __restrict__ G,
                               float* __restrict__ G32) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npair * (size_t)L) return;
  const size_t pq = t / L;
  const int q = (int)(t % L);
  const double v = eri[pair2_index(pq, (size_t)pair_index(q, q))];
  G[t] = v;
  G32[t] = (float)v;
}

template <typename T, int VEC>
int launch_same(Ctx* c, const T* X, size_t nrow, size_t ncol, const uint64_t* other, const Conn& cn,
                const typename Prec<T>::V* val, const typename Prec<T>::V* G, const double* hii, double* Y,
                int kind) {
  dim3 grid((unsigned)nrow, (unsigned)((ncol + (size_t)kSameThreads * VEC - 1) / ((size_t)kSameThreads * VEC)));
  if (kind == 1) {
    sigma_same_v2_kernel<T, VEC <= 4 ? VEC : 4><<<grid, kSameThreads, 0, c->stream>>>(
        X, ncol, other, cn.off, cn.nsing, cn.ket, val, cn.omask, cn.info, G, c->L, hii, Y);
  } else {
    sigma_same_v4_kernel<T, VEC><<<grid, kSameThreads, 0, c->stream>>>(X, ncol, other, cn.off, cn.nsing, cn.ket, val,
                                                                        cn.spos, cn.info, G, c->L, hii, Y);
  }
  SBDX_LAUNCHED(c);
  return 0;
}

template <typename T>
int run_same(Ctx* c, const T* X, size_t nrow, size_t ncol, const uint64_t* other, const Conn& cn,
             const typename Prec<T>::V* val, const typename Prec<T>::V* G, const double* hii, double* Y) {
  // default: popcount kernel x4 for FP64, parity-table kernel x8 for FP32;
  // narrowed to the widest vector that divides the row and keeps 16-byte alignment
  const int code0 = c->tune[sizeof(T) == 8 ? 0 : 1].same_code;
  const int code = code0 > 0 ? code0 : (sizeof(T) == 8 ? 14 : 8);
  const int kind = code >= 10 ? 1 : 0;
  int vec = code % 10;
  const bool aligned = (reinterpret_cast<uintptr_t>(X) % 16) == 0;
  while (vec > 1 && (!aligned || ncol % vec != 0)) vec >>= 1;
  if (vec >= 8 && kind == 0) return launch_same<T, 8>(c, X, nrow, ncol, other, cn, val, G, hii, Y, kind);
  if (vec >= 4) return launch_same<T, 4>(c, X, nrow, ncol, other, cn, val, G, hii, Y, kind);
  if (vec == 2) return launch_same<T, 2>(c, X, nrow, ncol, other, cn, val, G, hii, Y, kind);
  return launch_same<T, 1>(c, X, nrow, ncol, other, cn, val, G, hii, Y, kind);
}

size_t ab2_smem_bytes(size_t nb, size_t tsz, size_t vsz, size_t npair, int R, size_t* stride) {
  const size_t per = 16 / tsz;
  const size_t xstride = (nb + per - 1) / per * per;
  if (stride) *stride = xstride;
  return (size_t)R * (tsz * xstride + vsz * npair);
}

template <typename T, int R>
int launch_ab2(Ctx* c, const T* X, size_t smem, size_t xstride, int threads) {
  using V = typename Prec<T>::V;
  const Conn& ca = c->conn[0];
  const Conn& cb = c->conn[1];
  const V* eri = std::is_same<T, double>::value ? (const V*)c->d_eri : (const V*)c->d_eri32;
  const size_t per_cta = 8192;
  dim3 grid((unsigned)c->na, (unsigned)((c->nb + per_cta - 1) / per_cta));
  if (threads == 512) {
    SBDX_CUDA(c, cudaFuncSetAttribute(sigma_ab_v2_kernel<T, R, 512>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kAbSmemBudget));
    sigma_ab_v2_kernel<T, R, 512><<<grid, 512, smem, c->stream>>>(
        X, c->nb, c->d_a, c->d_b, ca.off, ca.nsing, ca.ket, ca.info, ca.omask, cb.off, cb.nsing, cb.srec, cb.order,
        eri, (int)c->npair, xstride, c->d_y);
    SBDX_LAUNCHED(c);
    return 0;
  }
  SBDX_CUDA(c, cudaFuncSetAttribute(sigma_ab_v2_kernel<T, R, 1024>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kAbSmemBudget));
  sigma_ab_v2_kernel<T, R, 1024><<<grid, 1024, smem, c->stream>>>(
      X, c->nb, c->d_a, c->d_b, ca.off, ca.nsing, ca.ket, ca.info, ca.omask, cb.off, cb.nsing, cb.srec, cb.order, eri,
      (int)c->npair, xstride, c->d_y);
  SBDX_LAUNCHED(c);
  return 0;
}

template <typename T, int R>
int launch_ab3(Ctx* c, const T* X) {
  using V = typename Prec<T>::V;
  const Conn& ca = c->conn[0];
  const Conn& cb = c->conn[1];
  const V* Vt = std::is_same<T, double>::value ? (const V*)c->d_V : (const V*)c->d_V32;
  const size_t vs = std::is_same<T, double>::value ? c->vstride : c->vstride32;
  const size_t per_cta = (size_t)kAb3Threads * kAb3Slots;
  dim3 grid((unsigned)c->na, (unsigned)((c->nb + per_cta - 1) / per_cta));
  sigma_ab_v3_kernel<T, R><<<grid, kAb3Threads, 0, c->stream>>>(
      X, c->nb, c->d_a, c->d_b, ca.off, ca.nsing, ca.ket, ca.info, ca.omask, cb.off, cb.nsing, cb.srec, cb.order, Vt,
      (int)vs, c->d_y);
  SBDX_LAUNCHED(c);
  return 0;
}

template <typename T, int R>
int launch_ab4(Ctx* c, const T* X, size_t smem) {
  using V = typename Prec<T>::V;
  const Conn& ca = c->conn[0];
  const Conn& cb = c->conn[1];
  const V* Vt = std::is_same<T, double>::value ? (const V*)c->d_V : (const V*)c->d_V32;
  const size_t vs = std::is_same<T, double>::value ? c->vstride : c->vstride32;
  SBDX_CUDA(c, cudaFuncSetAttribute(sigma_ab_v4_kernel<T, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAbSmemBudget));
  const size_t per_cta = (size_t)kAb2Threads * kAb2Slots;
  dim3 grid((unsigned)c->na, (unsigned)((c->nb + per_cta - 1) / per_cta));
  sigma_ab_v4_kernel<T, R><<<grid, kAb2Threads, smem, c->stream>>>(
      X, c->nb, c->d_a, c->d_b, ca.off, ca.nsing, ca.ket, ca.info, ca.omask, cb.off, cb.nsing, cb.srec, cb.order, Vt,
      vs, c->d_err, c->d_y);
  SBDX_LAUNCHED(c);
  return 0;
}

// Double-buffered TMA variant when rows are 16-byte aligned and two buffers of
// at least one row fit; returns 1 (not launched) otherwise.
template <typename T>
int try_ab4(Ctx* c, const T* X, int rows_req) {
  using V = typename Prec<T>::V;
  const size_t xbytes = sizeof(T) * c->nb;
  const size_t vs = std::is_same<T, double>::value ? c->vstride : c->vstride32;
  const size_t vbytes = sizeof(V) * vs;
  if (xbytes % 16 != 0 || (reinterpret_cast<uintptr_t>(X) % 16) != 0) return 1;
  const size_t budget = 200 * 1024;
  int R = rows_req > 0 ? rows_req : 4;
  for (; R >= 1; --R)
    if (2 * (size_t)R * (xbytes + vbytes) <= budget) break;
  if (R < 1) return 1;
  const size_t smem = 2 * (size_t)R * (xbytes + vbytes);
  int rc;
  if (R >= 4) rc = launch_ab4<T, 4>(c, X, smem);
  else if (R == 3) rc = launch_ab4<T, 3>(c, X, smem);
  else if (R == 2) rc = launch_ab4<T, 2>(c, X, smem);
  else rc = launch_ab4<T, 1>(c, X, smem);
  return rc ? -rc : 0;
}

template <typename T, int R>
int launch_ab5(Ctx* c, const T* X, size_t smem, size_t xstride) {
  using V = typename Prec<T>::V;
  const Conn& ca = c->conn[0];
  const Conn& cb = c->conn[1];
  const V* eri = std::is_same<T, double>::value ? (const V*)c->d_eri : (const V*)c->d_eri32;
  constexpr int NT = 1024;
  SBDX_CUDA(c, cudaFuncSetAttribute(sigma_ab_v5_kernel<T, R, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kAbSmemBudget));
  const size_t slices_per_cta = 8192 / 32;
  dim3 grid((unsigned)c->na, (unsigned)((cb.nslice + slices_per_cta - 1) / slices_per_cta));
  sigma_ab_v5_kernel<T, R, NT><<<grid, NT, smem, c->stream>>>(
      X, c->nb, c->d_a, c->d_b, ca.off, ca.nsing, ca.ket, ca.info, ca.omask, cb.sell, cb.soff, cb.slen, cb.nslice,
      cb.order, eri, (int)c->npair, xstride, c->d_y);
  SBDX_LAUNCHED(c);
  return 0;
}

template <typename T>
int run_ab(Ctx* c, const T* X) {
  using V = typename Prec<T>::V;
  const int code0 = c->tune[sizeof(T) == 8 ? 0 : 1].ab_code;
  const int code = code0 > 0 ? code0 : (sizeof(T) == 8 ? 42 : 13);
  const int variant = code / 10;
  const int rows = code % 10 > 0 ? code % 10 : 2;
  if (variant == 2) {  // double-buffered TMA staging, when rows are 16-byte aligned
    const int rc = try_ab4<T>(c, X, rows);
    if (rc <= 0) return -rc;
  }
  if (variant == 0) {
    if (rows >= 4) return launch_ab3<T, 4>(c, X);
    if (rows == 3) return launch_ab3<T, 3>(c, X);
    if (rows == 2) return launch_ab3<T, 2>(c, X);
    return launch_ab3<T, 1>(c, X);
  }
  const int threads = variant == 3 ? 512 : 1024;
  const size_t budget = threads == 512 ? 110 * 1024 : 220 * 1024;
  int R = rows;
  size_t stride = 0, smem = 0;
  for (; R >= 1; --R) {
    smem = ab2_smem_bytes(c->nb, sizeof(T), sizeof(V), c->npair, R, &stride);
    if (smem <= budget) break;
  }
  if (R < 1) {
    c->err = "sigma: beta dimension too large for one shared-memory ket row";
    return 1;
  }
  if (variant == 4) {
    if (R >= 4) return launch_ab5<T, 4>(c, X, smem, stride);
    if (R == 3) return launch_ab5<T, 3>(c, X, smem, stride);
    if (R == 2) return launch_ab5<T, 2>(c, X, smem, stride);
    return launch_ab5<T, 1>(c, X, smem, stride);
  }
  if (R >= 4) return launch_ab2<T, 4>(c, X, smem, stride, threads);
  if (R == 3) return launch_ab2<T, 3>(c, X, smem, stride, threads);
  if (R == 2) return launch_ab2<T, 2>(c, X, smem, stride, threads);
  return launch_ab2<T, 1>(c, X, smem, stride, threads);
}

// ---- alpha-first sigma (v6) -----------------------------------------------------
//
// The sigma is evaluated in the alpha-first determinant ordering: with the
// +-1 basis phase phi (basis_phase), H C = phi o (H' (phi o C)) where every
// sign of H' is a pure same-spin sign. So the same-spin kernels need no
// opposite-spin parity per pair, and the alpha-beta sign is the product of the
// two same-spin signs stored with the connectivity. The opposite-spin Coulomb
// term of a single excitation, sum_{q in other} (pq|qq), is read from the
// per-string Coulomb tables (Ctx::d_Db, d_Dr, d_Da) instead of being summed per pair.
//   0. Xp = phi o X, Xpt = (phi o X)^T, Xk = Xp in lane order (phase_split_kernel)
//   1. alpha same-spin on Xp -> Y                     (sigma_same_*_kernel)
//   2. beta same-spin on Xpt -> Yt                    (sigma_same_*_kernel)
//   3. alpha x beta on Xk -> Yab                      (sigma_ab_kernel)
//   (steps 1 to 3 side by side; in the lean form of large problems, Ctx::lean, one
//   after another, step 3 on lanes written after step 2 and added to Y)
//   4. S = phi o (Y + Yab + Yt^T) + hii o X           (combine_phase_kernel)
// Step 1 includes the Coulomb terms of the alpha singles with the beta string,
// step 3 those of the beta singles with the alpha string (one more integral
// row per alpha string), so step 2 is a product with a constant sparse matrix.
// The unpacked alpha-beta kernels (codes 61-64) evaluate the pairs only, add
// them to Y, and leave both Coulomb terms to the same-spin kernels (Dt).

// 256 lanes of up to 32 rows of Xk, phi o X with its columns in the lane order
// of the packed alpha-beta kernel (vket: the ket string of each lane), so that
// kernel's loads are coalesced: one gather per element here instead of one per
// alpha single there. v: the thread's lane; x, o: the rows; s_pa: their strings'
// prefix parities.
template <typename T>
__device__ __forceinline__ void lane_rows(const T* __restrict__ x, size_t nb, int rows, size_t v, const uint64_t* s_pa,
                                          const uint64_t* __restrict__ bstr, const uint32_t* __restrict__ vket,
                                          T* __restrict__ o, size_t xs) {
  if (v >= xs) return;
  const size_t ib = vket[v];
  const uint64_t beta = bstr[ib];
#pragma unroll 8
  for (int k = 0; k < rows; ++k) {
    const T w = x[(size_t)k * nb + ib];
    o[(size_t)k * xs + v] = basis_phase(s_pa[k], beta) ? -w : w;
  }
}

// The lanes of all rows by themselves (the split kernel's, where Xk takes the
// room of vectors that are read in between).
template <typename T>
__global__ void __launch_bounds__(256)
lane_order_kernel(const T* __restrict__ X, size_t na, size_t nb, const uint64_t* __restrict__ astr,
                  const uint64_t* __restrict__ bstr, const uint32_t* __restrict__ vket, T* __restrict__ Xk, size_t xs) {
  __shared__ uint64_t s_pa[32];
  const size_t ia0 = (size_t)blockIdx.y * 32;
  if (threadIdx.x < 32) s_pa[threadIdx.x] = ia0 + threadIdx.x < na ? prefix_parity(astr[ia0 + threadIdx.x]) : 0ull;
  __syncthreads();
  lane_rows(X + ia0 * nb, nb, (int)min((size_t)32, na - ia0), (size_t)blockIdx.x * 256 + threadIdx.x, s_pa, bstr, vket,
            Xk + ia0 * xs, xs);
}

// Blocks ibx < ntx split one 32 x 32 tile; the further ones write lane_rows.
// *nonfinite (unless null) is set where X holds an infinity or NaN.
template <typename T>
__global__ void phase_split_kernel(const T* __restrict__ X, size_t na, size_t nb, const uint64_t* __restrict__ astr,
                                   const uint64_t* __restrict__ bstr, T* __restrict__ Xp, T* __restrict__ Xpt,
                                   size_t xsa, size_t xsb, const uint32_t* __restrict__ vket, T* __restrict__ Xk,
                                   size_t xs, int* nonfinite) {
  __shared__ T tile[32][33];
  __shared__ uint64_t s_pa[32], s_b[32];
  const size_t ntx = (nb + 31) / 32;
  const size_t ib0 = (size_t)blockIdx.x * 32, ia0 = (size_t)blockIdx.y * 32;
  const int tx = threadIdx.x;
  if (threadIdx.y == 0) {
    s_pa[tx] = ia0 + tx < na ? prefix_parity(astr[ia0 + tx]) : 0ull;
    s_b[tx] = ib0 + tx < nb ? bstr[ib0 + tx] : 0ull;
  }
  __syncthreads();
  if (blockIdx.x >= ntx) {
    lane_rows(X + ia0 * nb, nb, (int)min((size_t)32, na - ia0), (blockIdx.x - ntx) * 256 + threadIdx.y * 32 + tx, s_pa, bstr,
              vket, Xk + ia0 * xs, xs);
    return;
  }
  bool odd = false;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const size_t ia = ia0 + k, ib = ib0 + tx;
    if (ia < na && ib < nb) {
      T v = X[ia * nb + ib];
      odd |= !isfinite(v);
      if (basis_phase(s_pa[k], s_b[tx])) v = -v;
      Xp[ia * xsa + ib] = v;
      tile[k][tx] = v;
    }
  }
  if (odd && nonfinite != nullptr) *nonfinite = 1;
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const size_t ib = ib0 + k, ia = ia0 + tx;
    if (ia < na && ib < nb) Xpt[ib * xsb + ia] = tile[tx][k];
  }
}

// S[ia, ib] = phi(ia, ib) (Y[ia, ib] + Yab[ia, ib] + Yt[ib, ia]) + hii[ia, ib]
// X[ia, ib], stored in T; Y, Yab and Yt have row strides xsa, xsa and xsb. Yab
// is null where the alpha-beta kernel has added its part to Y; with kInPlace S
// itself holds it. *nonfinite (unless null) is cleared.
template <typename T, bool kInPlace>
__global__ void combine_phase_kernel(const double* __restrict__ Y, const double* __restrict__ Yab,
                                     const double* __restrict__ Yt, const double* __restrict__ hii,
                                     const T* __restrict__ X, size_t na, size_t nb, const uint64_t* __restrict__ astr,
                                     const uint64_t* __restrict__ bstr, T* S, size_t xsa, size_t xsb,
                                     int* nonfinite) {
  __shared__ double tile[32][33];
  __shared__ uint64_t s_pa[32], s_b[32];
  const size_t ib0 = (size_t)blockIdx.x * 32, ia0 = (size_t)blockIdx.y * 32;
  const int tx = threadIdx.x;
  if (threadIdx.y == 0) {
    s_pa[tx] = ia0 + tx < na ? prefix_parity(astr[ia0 + tx]) : 0ull;
    s_b[tx] = ib0 + tx < nb ? bstr[ib0 + tx] : 0ull;
  }
#pragma unroll 4
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const size_t ib = ib0 + k, ia = ia0 + tx;
    if (ib < nb && ia < na) tile[tx][k] = Yt[ib * xsb + ia];
  }
  if (nonfinite != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && tx == 0 && threadIdx.y == 0) *nonfinite = 0;
  __syncthreads();
#pragma unroll 4
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const size_t ia = ia0 + k, ib = ib0 + tx;
    if (ia < na && ib < nb) {
      double y = Y[ia * xsa + ib] + tile[k][tx];
      if constexpr (kInPlace) y += (double)S[ia * nb + ib];
      else if (Yab != nullptr) y += Yab[ia * xsa + ib];
      const double d = hii[ia * nb + ib] * (double)X[ia * nb + ib];
      S[ia * nb + ib] = (T)(basis_phase(s_pa[k], s_b[tx]) ? d - y : d + y);
    }
  }
}

// D[pq * stride + k] = sum over the orbitals q < L of string k of (pq|qq).
__global__ void coulomb_table_kernel(const double* __restrict__ G, int L, const uint64_t* __restrict__ s, size_t n,
                                     size_t stride, double* __restrict__ D, float* __restrict__ D32) {
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t pq = blockIdx.y;
  if (k >= n) return;
  const double* g = G + pq * (size_t)L;
  uint64_t bits = s[k] & range_mask(0, L);
  double v = 0.0;
  while (bits) {
    const int q = __ffsll((long long)bits) - 1;
    bits &= bits - 1;
    v += g[q];
  }
  D[pq * stride + k] = v;
  D32[pq * stride + k] = (float)v;
}

// The integrals over the pairs in use: row pq = (pq|pairs[t]), t < n.
__global__ void gather_pairs_kernel(const double* __restrict__ V, size_t vstride, const uint32_t* __restrict__ pairs,
                                    int n, size_t vs, size_t vs32, double* __restrict__ out, float* __restrict__ out32) {
  const size_t pq = blockIdx.x;
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    const double v = V[pq * vstride + pairs[t]];
    out[pq * vs + t] = v;
    out32[pq * vs32 + t] = (float)v;
  }
}

// The table by string: row k = sum over the orbitals p of string k of the
// integral row (pp|..) over npair pairs.
__global__ void coulomb_row_sum_kernel(const double* __restrict__ V, size_t npair, size_t vs, size_t vs32, int L,
                                       const uint64_t* __restrict__ s, double* __restrict__ D,
                                       float* __restrict__ D32) {
  const size_t k = blockIdx.x;
  const uint64_t bits = s[k] & range_mask(0, L);
  for (size_t t = threadIdx.x; t < npair; t += blockDim.x) {
    double v = 0.0;
    for (uint64_t m = bits; m; m &= m - 1) {
      const size_t p = (size_t)(__ffsll((long long)m) - 1);
      v += V[(p * (p + 1) / 2 + p) * vs + t];
    }
    D[k * vs + t] = v;
    D32[k * vs32 + t] = (float)v;
  }
}

// True in every thread of the last CTA to arrive for split entry q: the
// parts' partial rows are then visible to it. The counter returns to zero for
// the next launch.
__device__ __forceinline__ bool last_part(uint32_t* done, size_t q, uint32_t parts) {
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = atomicAdd(done + q, 1u) + 1 == parts;
    if (s_last) done[q] = 0;
  }
  __syncthreads();
  if (s_last) __threadfence();
  return s_last != 0;
}

// Row `row` of Y in columns c0 .. c0 + VEC - 1 as the sum of a split row's
// partial rows in slot order, by the last part to finish a strip. Partial row
// k of slot q is ypart row (first slot + q) * stride + k.
template <int VEC>
__device__ __forceinline__ void same_split_sum(const uint4* split, const uint32_t* slot_split, uint32_t* done,
                                               uint32_t slot, int k_rows, const double* ypart, size_t ldx, size_t c0,
                                               bool active, double* Y, size_t row) {
  const uint32_t q = slot_split[slot];
  const uint4 sp = split[q];
  if (!last_part(done, (size_t)q * gridDim.y + blockIdx.y, sp.z) || !active) return;
  double t[VEC];
#pragma unroll
  for (int v = 0; v < VEC; ++v) t[v] = 0.0;
#pragma unroll 4
  for (uint32_t p = 0; p < sp.z; ++p)
#pragma unroll
    for (int v = 0; v < VEC; ++v) t[v] += __ldcg(ypart + (size_t)(sp.y + p) * k_rows * ldx + c0 + v);
#pragma unroll
  for (int v = 0; v < VEC; ++v) Y[row * ldx + c0 + v] = t[v];
}

// Same-spin excitations in the alpha-first basis, VEC consecutive columns per
// thread; grid x = bra row (fastest: the resident CTAs share one column strip
// of the ket rows, which stays in L2), y = column strip. A CTA stages the
// entries of its row (ket, signed value, signed pair index) in shared memory;
// per pair a double costs one FMA and a single, when Dt is given, one add (the
// Coulomb table element of its column) and one FMA. X and Y rows have stride ldx, a multiple
// of VEC (padding columns up to ldx are computed and never read).
// Bound by the latency of the ket loads from L2: four entries' loads are
// issued before their products (written as one loop of single entries the
// compiler keeps two in flight: 8000 x 150 strings, 7 electrons in 58
// orbitals, FP64 alpha side 370 -> 296 us; 150 x 4000, 5 in 24, beta side 160
// -> 131 us; eight at a time 333 and 147 us).
template <typename T, int VEC>
__global__ void __launch_bounds__(kSameThreads)
sigma_same_v6_kernel(const T* __restrict__ X, size_t ncol, size_t ldx, const uint64_t* __restrict__ off,
                     const uint32_t* __restrict__ nsing, const uint32_t* __restrict__ ket,
                     const typename Prec<T>::V* __restrict__ val, const uint32_t* __restrict__ info,
                     const typename Prec<T>::V* __restrict__ Dt, size_t dstride,
                     const uint4* __restrict__ items, const uint4* __restrict__ split,
                     const uint32_t* __restrict__ slot_split, uint32_t* __restrict__ done, double* __restrict__ ypart,
                     double* __restrict__ Y) {
  __shared__ uint32_t s_ket[kSameThreads], s_pq[kSameThreads];
  __shared__ double s_val[kSameThreads];
  constexpr int kAhead = 4;
  const uint4 item = items[blockIdx.x];  // bra string, entry range, output row
  const size_t r = item.x;
  double* __restrict__ Yrow = item.w ? ypart + (size_t)(item.w - 1) * ldx : Y + r * ldx;
  const size_t c0 = ((size_t)blockIdx.y * kSameThreads + threadIdx.x) * VEC;
  const bool active = c0 < ncol;
  double acc[VEC];
#pragma unroll
  for (int v = 0; v < VEC; ++v) acc[v] = 0.0;
  const uint64_t beg = off[r] + item.y, end = off[r] + item.z, send = off[r] + nsing[r];
  const unsigned t = threadIdx.x;
  for (uint64_t base = beg; base < end; base += kSameThreads) {
    const int cnt = (int)min((uint64_t)kSameThreads, end - base);
    const int nsb = Dt != nullptr && send > base ? (int)min((uint64_t)cnt, send - base) : 0;
    __syncthreads();
    if ((int)t < cnt) {
      const uint64_t e = base + t;
      const uint32_t inf = info[e];
      const double v = (double)val[e];
      s_ket[t] = ket[e];
      s_val[t] = (inf >> 31) ? -v : v;
      s_pq[t] = ((inf >> 12) & 0xfffu) | (inf & kInfoNeg);
    }
    __syncthreads();
    if (!active) continue;
    auto single = [&](int e) {
      const uint32_t pqs = s_pq[e];
      const double hv = s_val[e];
      double x[VEC], d[VEC];
      VecIO<T, VEC>::load(X + (size_t)s_ket[e] * ldx + c0, x);
      VecIO<T, VEC>::load(Dt + (size_t)(pqs & 0xfffu) * dstride + c0, d);
#pragma unroll
      for (int v = 0; v < VEC; ++v) acc[v] = fma(hv + flip_sign(d[v], pqs >> 31), x[v], acc[v]);
    };
#pragma unroll 2
    for (int e = 0; e < nsb; ++e) single(e);
    int e = nsb;
    for (; e + kAhead <= cnt; e += kAhead) {  // the ket values of a run in flight together
      double x[kAhead][VEC];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) VecIO<T, VEC>::load(X + (size_t)s_ket[e + u] * ldx + c0, x[u]);
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
#pragma unroll
        for (int v = 0; v < VEC; ++v) acc[v] = fma(s_val[e + u], x[u][v], acc[v]);
    }
    for (; e < cnt; ++e) {
      double x[VEC];
      VecIO<T, VEC>::load(X + (size_t)s_ket[e] * ldx + c0, x);
#pragma unroll
      for (int v = 0; v < VEC; ++v) acc[v] = fma(s_val[e], x[v], acc[v]);
    }
  }
  if (active) {
#pragma unroll
    for (int v = 0; v < VEC; ++v) Yrow[c0 + v] = acc[v];
  }
  if (item.w) same_split_sum<VEC>(split, slot_split, done, item.w - 1, 1, ypart, ldx, c0, active, Y, r);
}

// FP32-storage variant of sigma_same_v6_kernel: products and short runs of up
// to kRun entries are summed in FP32, and each run's sum is added to the FP64
// row accumulator (one conversion per run and column instead of one per pair).
constexpr int kRun = 8;

template <int VEC> struct VecF;
template <> struct VecF<1> {
  static __device__ __forceinline__ void load(const float* p, float* o) { o[0] = __ldg(p); }
};
template <> struct VecF<2> {
  static __device__ __forceinline__ void load(const float* p, float* o) {
    const float2 v = __ldg(reinterpret_cast<const float2*>(p));
    o[0] = v.x; o[1] = v.y;
  }
};
template <> struct VecF<4> {
  static __device__ __forceinline__ void load(const float* p, float* o) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  }
};
template <> struct VecF<8> {
  static __device__ __forceinline__ void load(const float* p, float* o) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    const float4 w = __ldg(reinterpret_cast<const float4*>(p) + 1);
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; o[4] = w.x; o[5] = w.y; o[6] = w.z; o[7] = w.w;
  }
};

template <int VEC>
__global__ void __launch_bounds__(kSameThreads)
sigma_same_v6f_kernel(const float* __restrict__ X, size_t ncol, size_t ldx, const uint64_t* __restrict__ off,
                      const uint32_t* __restrict__ nsing, const uint32_t* __restrict__ ket,
                      const float* __restrict__ val, const uint32_t* __restrict__ info, const float* __restrict__ Dt,
                      size_t dstride, const uint4* __restrict__ items,
                      const uint4* __restrict__ split, const uint32_t* __restrict__ slot_split,
                      uint32_t* __restrict__ done, double* __restrict__ ypart, double* __restrict__ Y) {
  __shared__ uint32_t s_ket[kSameThreads], s_pq[kSameThreads];
  __shared__ float s_val[kSameThreads];
  const uint4 item = items[blockIdx.x];  // bra string, entry range, output row
  const size_t r = item.x;
  double* __restrict__ Yrow = item.w ? ypart + (size_t)(item.w - 1) * ldx : Y + r * ldx;
  const size_t c0 = ((size_t)blockIdx.y * kSameThreads + threadIdx.x) * VEC;
  const bool active = c0 < ncol;
  double acc[VEC];
#pragma unroll
  for (int v = 0; v < VEC; ++v) acc[v] = 0.0;
  const uint64_t beg = off[r] + item.y, end = off[r] + item.z, send = off[r] + nsing[r];
  const unsigned t = threadIdx.x;
  for (uint64_t base = beg; base < end; base += kSameThreads) {
    const int cnt = (int)min((uint64_t)kSameThreads, end - base);
    const int nsb = Dt != nullptr && send > base ? (int)min((uint64_t)cnt, send - base) : 0;
    __syncthreads();
    if ((int)t < cnt) {
      const uint64_t e = base + t;
      const uint32_t inf = info[e];
      const float v = val[e];
      s_ket[t] = ket[e];
      s_val[t] = (inf >> 31) ? -v : v;
      s_pq[t] = ((inf >> 12) & 0xfffu) | (inf & kInfoNeg);
    }
    __syncthreads();
    if (!active) continue;
    for (int e0 = 0; e0 < nsb; e0 += kRun) {  // singles: value + signed Coulomb-table element
      const int e1 = min(e0 + kRun, nsb);
      float pf[VEC];
#pragma unroll
      for (int v = 0; v < VEC; ++v) pf[v] = 0.f;
      for (int e = e0; e < e1; ++e) {
        const uint32_t pqs = s_pq[e];
        const float hv = s_val[e];
        float x[VEC], d[VEC];
        VecF<VEC>::load(X + (size_t)s_ket[e] * ldx + c0, x);
        VecF<VEC>::load(Dt + (size_t)(pqs & 0xfffu) * dstride + c0, d);
#pragma unroll
        for (int v = 0; v < VEC; ++v) pf[v] = fmaf(hv + ((pqs >> 31) ? -d[v] : d[v]), x[v], pf[v]);
      }
#pragma unroll
      for (int v = 0; v < VEC; ++v) acc[v] += (double)pf[v];
    }
    for (int e0 = nsb; e0 < cnt; e0 += kRun) {  // doubles
      const int e1 = min(e0 + kRun, cnt);
      float pf[VEC];
#pragma unroll
      for (int v = 0; v < VEC; ++v) pf[v] = 0.f;
#pragma unroll 4
      for (int e = e0; e < e1; ++e) {
        const float hv = s_val[e];
        float x[VEC];
        VecF<VEC>::load(X + (size_t)s_ket[e] * ldx + c0, x);
#pragma unroll
        for (int v = 0; v < VEC; ++v) pf[v] = fmaf(hv, x[v], pf[v]);
      }
#pragma unroll
      for (int v = 0; v < VEC; ++v) acc[v] += (double)pf[v];
    }
  }
  if (active) {
#pragma unroll
    for (int v = 0; v < VEC; ++v) Yrow[c0 + v] = acc[v];
  }
  if (item.w) same_split_sum<VEC>(split, slot_split, done, item.w - 1, 1, ypart, ldx, c0, active, Y, r);
}

// VEC consecutive elements in the storage type.
template <typename T, int VEC> struct LoadT;
template <int VEC> struct LoadT<double, VEC> {
  static __device__ __forceinline__ void load(const double* p, double* o) { VecIO<double, VEC>::load(p, o); }
};
template <int VEC> struct LoadT<float, VEC> {
  static __device__ __forceinline__ void load(const float* p, float* o) { VecF<VEC>::load(p, o); }
};

// Blocked same-spin products: CTA = (work item of SameBlocks, strip of
// columns). Every ket row strip of the block's union is loaded once and
// applied to all bra strings of the block with their signed values (zero
// where a string does not connect).

// Stages up to kSameThreads union entries (kets and values).
template <int ROWS, typename V>
__device__ __forceinline__ void stage_union(uint32_t* s_ket, V* s_val, const uint32_t* __restrict__ uket,
                                            const V* __restrict__ uval, uint64_t base, int cnt) {
  constexpr int kPer = 16 / sizeof(V);
  __syncthreads();
  if ((int)threadIdx.x < cnt) s_ket[threadIdx.x] = uket[base + threadIdx.x];
  const uint4* src = reinterpret_cast<const uint4*>(uval + base * ROWS);
  uint4* dst = reinterpret_cast<uint4*>(s_val);
  for (int i = threadIdx.x; i < cnt * ROWS / kPer; i += kSameThreads) dst[i] = src[i];
  __syncthreads();
}

// Y[r, c] += sum over the singles e of string r of s_e Dt[pq_e, c] X[ket_e, c]: the
// Coulomb terms that the blocked kernels leave out (the constant part of a
// single is in their unions). CTA = (string row0 + blockIdx.x, strip), 16 bytes of
// consecutive columns per thread, the loads of kAhead singles before their
// products. FP32: sums over kRun singles in FP32, then FP64. Reads two strips
// per single from L2 (19.7 GB at 8000 x 8000 strings, FP64). Inside the matrix
// kernel the same loads wait for the row with the most singles of eight, and
// their registers spill (8000 x 8000, FP64: 7.3 ms for both, 5.1 + 1.3 ms apart).
template <typename T>
__global__ void __launch_bounds__(kSameThreads, 4)
sigma_coulomb_kernel(const T* __restrict__ X, size_t ncol, size_t ldx, size_t row0, const uint64_t* __restrict__ off,
                     const uint32_t* __restrict__ nsing, const uint32_t* __restrict__ ket,
                     const uint32_t* __restrict__ info, const T* __restrict__ Dt, size_t dstride,
                     double* __restrict__ Y) {
  constexpr int PW = 16 / sizeof(T), kAhead = 4;
  __shared__ uint32_t s_ket[kSameThreads], s_pq[kSameThreads];
  const size_t r = row0 + blockIdx.x;
  const size_t c0 = ((size_t)blockIdx.y * kSameThreads + threadIdx.x) * PW;
  const uint64_t e0 = off[r];
  const int ns = (int)nsing[r];
  if (ns == 0) return;
  const bool active = c0 < ncol;
  double acc[PW];
#pragma unroll
  for (int v = 0; v < PW; ++v) acc[v] = 0.0;
  for (int base = 0; base < ns; base += kSameThreads) {
    const int cnt = min(kSameThreads, ns - base);
    __syncthreads();
    if ((int)threadIdx.x < cnt) {
      const uint32_t inf = info[e0 + base + threadIdx.x];
      s_ket[threadIdx.x] = ket[e0 + base + threadIdx.x];
      s_pq[threadIdx.x] = ((inf >> 12) & 0xfffu) | (inf & kInfoNeg);
    }
    __syncthreads();
    if (!active) continue;
    T pf[PW];
    for (int b0 = 0; b0 < cnt; b0 += kAhead) {
      T x[kAhead][PW], d[kAhead][PW];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int b = min(b0 + u, cnt - 1);
        LoadT<T, PW>::load(X + (size_t)s_ket[b] * ldx + c0, x[u]);
        LoadT<T, PW>::load(Dt + (size_t)(s_pq[b] & 0xfffu) * dstride + c0, d[u]);
      }
      if (b0 % kRun == 0)
#pragma unroll
        for (int v = 0; v < PW; ++v) pf[v] = (T)0;
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if (b0 + u < cnt) {
          const bool neg = (s_pq[b0 + u] >> 31) != 0;
#pragma unroll
          for (int v = 0; v < PW; ++v) pf[v] = fma(neg ? -d[u][v] : d[u][v], x[u][v], pf[v]);
        }
      if (b0 % kRun + kAhead == kRun || b0 + kAhead >= cnt)
#pragma unroll
        for (int v = 0; v < PW; ++v) acc[v] += (double)pf[v];
    }
  }
  if (!active) return;
#pragma unroll
  for (int v = 0; v < PW; v += 2) {
    double2* y = reinterpret_cast<double2*>(Y + r * ldx + c0 + v);
    double2 t = *y;
    t.x += acc[v];
    t.y += acc[v + 1];
    *y = t;
  }
}

// The blocked kernels multiply the zeros of a block's union too, and zero times
// an infinity is NaN: where the input holds one (*nonfinite), this kernel
// evaluates their rows again, string by string, so that it reaches the
// elements that the matrix connects it with and no others. Otherwise its CTAs end at once
// (2 us on a side stream beside products of 0.9 ms and more).
template <typename T>
__global__ void __launch_bounds__(kSameThreads)
sigma_same_nonfinite_kernel(const int* __restrict__ nonfinite, const T* __restrict__ X, size_t ncol, size_t ldx, size_t row0,
                            size_t nrow, const uint64_t* __restrict__ off, const uint32_t* __restrict__ nsing,
                            const uint32_t* __restrict__ ket, const typename Prec<T>::V* __restrict__ val,
                            const uint32_t* __restrict__ info, const typename Prec<T>::V* __restrict__ Dt, size_t dstride,
                            double* __restrict__ Y) {
  if (*nonfinite == 0) return;
  const size_t strips = (ncol + kSameThreads - 1) / kSameThreads;
  for (size_t w = blockIdx.x; w < nrow * strips; w += gridDim.x) {
    const size_t r = row0 + w / strips, c = w % strips * kSameThreads + threadIdx.x;
    if (c >= ncol) continue;
    double acc = 0.0;
    const uint64_t e0 = off[r], e1 = off[r + 1], send = Dt != nullptr ? e0 + nsing[r] : e0;
    for (uint64_t e = e0; e < e1; ++e) {
      const uint32_t inf = info[e];
      double v = (double)val[e];
      if (inf >> 31) v = -v;
      if (e < send) v += flip_sign((double)Dt[(size_t)((inf >> 12) & 0xfffu) * dstride + c], inf >> 31);
      acc = fma(v, (double)X[(size_t)ket[e] * ldx + c], acc);
    }
    Y[r * ldx + c] = acc;
  }
}

// FP64, eight strings per block: the strings times four union entries are the A
// operand of m8n8k4, four ket rows times eight columns its B operand, so the
// product is a dense (8 x entries)(entries x columns) sum on the FP64 tensor
// pipe. TMA bulk copies bring the strips of kMmaG entries and their values to
// shared memory, a ring of kMmaStages stages that the warps refill in turn. A
// warp owns 128 columns: lane l reads ket l & 3's columns 16 i + 2 (l >> 2) + {0,
// 1} in one 16-byte load per i, the operands of an even and an odd tile; it ends
// with string l >> 2, columns 16 i + 4 (l & 3) .. + 3. Rows in shared memory are
// 32 bytes longer than the strip, so the four kets that a quarter-warp reads
// lie in different banks. Bound: the FP64 tensor pipe (72% busy at 4800 x 4800);
// padding of the unions counts as work there. 8000 x 8000: 5.1 ms for the beta
// side, where CUDA-core products of four strings per block took 7.5 ms and of
// eight 6.0 ms (issue slots, 60% of the FP64 pipe); with the B operands loaded
// straight from global memory, a wavefront per ket and quarter-warp, 8.0 ms;
// with two stages 6.8 ms; with kMmaI = 4 (shorter strips, the A operands read
// twice as often) 5.5 ms.
constexpr int kMmaI = 8;  // loads, of two 8-column tiles each, per lane and four entries
constexpr int kMmaCols = 16 * kMmaI * (kSameThreads / 32), kMmaG = 32 / kMmaI, kMmaPitch = kMmaCols + 4;
constexpr size_t kMmaStageBytes = sizeof(double) * kMmaG * (kMmaPitch + kBlkRows64);
constexpr int kMmaStages = 3;

// Bounded wait by polls (each suspends the thread for a while in hardware).
__device__ __forceinline__ bool mbar_wait_polls(uint64_t* bar, uint32_t parity) {
  for (int it = 0; it < (1 << 20); ++it)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

__global__ void __launch_bounds__(kSameThreads, 2)
sigma_same_mma_kernel(const double* __restrict__ X, size_t ncol, size_t ldx,
                      const uint32_t* __restrict__ brows, const uint64_t* __restrict__ uoff,
                      const uint32_t* __restrict__ uket, const double* __restrict__ uval,
                      const uint4* __restrict__ items, const uint4* __restrict__ split,
                      const uint32_t* __restrict__ slot_split, uint32_t* __restrict__ done,
                      double* __restrict__ ypart, double* __restrict__ Y, int* __restrict__ err) {
  constexpr int ROWS = kBlkRows64, G = kMmaG, NS = kMmaStages, kWarps = kSameThreads / 32;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[NS], empty[NS];
  const uint4 item = items[blockIdx.x];  // block, union range, partial slot
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  // columns up to ncol rounded up to 8: the rows' padding, never another range's columns
  const size_t lim = (ncol + 7) & ~(size_t)7, s0 = (size_t)blockIdx.y * kMmaCols, cw = s0 + 16 * kMmaI * warp;
  const bool active = cw < ncol;  // warp-uniform
  const int n_stage = (int)((item.z - item.y) / G);  // the unions are padded to 8 entries
  const uint64_t beg = uoff[item.x] + item.y;
  const uint32_t r = brows[item.x * ROWS + g];
  if (threadIdx.x == 0) {
    for (int k = 0; k < NS; ++k) {
      mbar_init(&full[k], 1);
      mbar_init(&empty[k], kWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  // stage k's copies (G strips and their values) by one warp; kt: the lane's ket
  const uint32_t bytes = (uint32_t)(min((size_t)kMmaCols, lim - s0) * sizeof(double));
  constexpr uint32_t vbytes = G * ROWS * sizeof(double);
  auto tile = [&](int b) { return reinterpret_cast<double*>(smem + b * kMmaStageBytes); };
  auto fill_ket = [&](int k) { return lane < G ? __ldg(uket + beg + (uint64_t)k * G + lane) : 0u; };
  auto fill = [&](int k, int b, uint32_t kt) {
    if (lane == 0) mbar_arrive_expect_tx(&full[b], G * bytes + vbytes);
    __syncwarp();
    if (lane < G) tma_load_1d(tile(b) + (size_t)lane * kMmaPitch, X + (size_t)kt * ldx + s0, bytes, &full[b]);
    else if (lane == G) tma_load_1d(tile(b) + (size_t)G * kMmaPitch, uval + (beg + (uint64_t)k * G) * ROWS, vbytes, &full[b]);
  };
  if (warp == 0)
    for (int k = 0; k < min(NS, n_stage); ++k) fill(k, k, fill_ket(k));
  double acc[kMmaI][2][2];
#pragma unroll
  for (int i = 0; i < kMmaI; ++i) acc[i][0][0] = acc[i][0][1] = acc[i][1][0] = acc[i][1][1] = 0.0;
  int b = 0, last = NS - 1;  // buffers of stages k and k - 1
  uint32_t ph = 0, lph = 1;  // parities of their phases
  for (int k = 0; k < n_stage; ++k) {
    // warp k mod 8 refills the buffer of stage k - 1, which the others have
    // finished or are about to
    const bool mine = k > 0 && k - 1 + NS < n_stage && warp == (k & (kWarps - 1));
    const uint32_t kt = mine ? fill_ket(k - 1 + NS) : 0u;
    bool ok = mbar_wait_polls(&full[b], ph);
    if (ok) {
      if (active) {
        const double* x = tile(b) + (size_t)q * kMmaPitch + 16 * kMmaI * warp + 2 * g;
        const double* w = tile(b) + (size_t)G * kMmaPitch + lane;
#pragma unroll
        for (int u = 0; u < G / 4; ++u) {
          const double a = w[4 * ROWS * u];
          double2 xv[kMmaI];
#pragma unroll
          for (int i = 0; i < kMmaI; ++i) xv[i] = *reinterpret_cast<const double2*>(x + (size_t)4 * u * kMmaPitch + 16 * i);
#pragma unroll
          for (int i = 0; i < kMmaI; ++i) {
            dmma_m8n8k4(acc[i][0], a, xv[i].x);
            dmma_m8n8k4(acc[i][1], a, xv[i].y);
          }
        }
      }
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&empty[b])) : "memory");
      if (mine) ok = mbar_wait_polls(&empty[last], lph);
    }
    if (!__all_sync(0xffffffffu, ok)) {  // flag it; the copies in flight land before shared memory is given up
      if (lane == 0) atomicExch(err, kErrWatchdogSame);
      for (int j = k; j < min(k + NS, n_stage); ++j) mbar_wait_polls(&full[j % NS], (uint32_t)((j / NS) & 1));
      break;
    }
    if (mine) fill(k - 1 + NS, last, kt);
    last = b;
    lph = ph;
    if (++b == NS) { b = 0; ph ^= 1; }
  }
  bool on[kMmaI];
#pragma unroll
  for (int i = 0; i < kMmaI; ++i) on[i] = active && cw + 16 * i + 4 * q < lim;
  // columns 4 q .. 4 q + 3 of each i: {even tile, odd tile} x {0, 1}
  double* y = (item.w ? ypart + ((size_t)(item.w - 1) * ROWS + g) * ldx : Y + (size_t)r * ldx) + cw;
  if (item.w || r != kNoRow) {
#pragma unroll
    for (int i = 0; i < kMmaI; ++i)
      if (on[i]) {
        double2* o = reinterpret_cast<double2*>(y + 16 * i + 4 * q);
        o[0] = make_double2(acc[i][0][0], acc[i][1][0]);
        o[1] = make_double2(acc[i][0][1], acc[i][1][1]);
      }
  }
  if (item.w == 0) return;
  const uint32_t sq = slot_split[item.w - 1];
  const uint4 sp = split[sq];
  if (!last_part(done, (size_t)sq * gridDim.y + blockIdx.y, sp.z) || r == kNoRow) return;
  for (int i = 0; i < kMmaI; ++i) {
    const size_t c = cw + 16 * i + 4 * q;
    if (!on[i]) continue;
    double t[4] = {0.0, 0.0, 0.0, 0.0};
    for (uint32_t p = 0; p < sp.z; ++p) {
      const double2* o = reinterpret_cast<const double2*>(ypart + ((size_t)(sp.y + p) * ROWS + g) * ldx + c);
      const double2 u = __ldcg(o), v = __ldcg(o + 1);
      t[0] += u.x; t[1] += u.y; t[2] += v.x; t[3] += v.y;
    }
    double2* o = reinterpret_cast<double2*>(Y + (size_t)r * ldx + c);
    o[0] = make_double2(t[0], t[1]);
    o[1] = make_double2(t[2], t[3]);
  }
}

// FP32 storage, VEC columns per thread: products summed in FP32 over runs of
// kRun union entries (or of kRun singles), each run's sum added to the FP64
// row accumulator. The unions are padded to whole runs, so the run's ket
// strips are all loaded before the first product and no product is guarded.
// Four strings: a ket value is converted once for four products. Bound: issue
// slots (68% busy at 4800 x 4800) and L1 wavefronts (66%), the FMA pipe at 43%; the
// tensor pipe has no FP32 type without a loss of bits.
// 8000 x 8000: 3.3 ms for the beta side (4.4 ms with the singles in lists of
// their own and with guarded products; 4.3 ms with the strips brought by TMA).
template <int VEC>
__global__ void __launch_bounds__(kSameThreads, 3)
sigma_same_blkf_kernel(const float* __restrict__ X, size_t ncol, size_t ldx,
                       const uint32_t* __restrict__ brows, const uint64_t* __restrict__ uoff, const uint32_t* __restrict__ uket,
                       const float* __restrict__ uval, const uint4* __restrict__ items,
                       const uint4* __restrict__ split, const uint32_t* __restrict__ slot_split,
                       uint32_t* __restrict__ done, double* __restrict__ ypart, double* __restrict__ Y) {
  constexpr int ROWS = kBlkRows32;
  static_assert(kRun == 8 && ROWS == 4, "the unions are padded to runs of 8 entries of 4 values");
  __shared__ __align__(16) uint32_t s_ket[kSameThreads];
  __shared__ __align__(16) float s_val[kSameThreads * ROWS];
  const uint4 item = items[blockIdx.x];  // block, union range, partial slot
  const size_t c0 = ((size_t)blockIdx.y * kSameThreads + threadIdx.x) * VEC;
  const bool active = c0 < ncol;
  double acc[ROWS][VEC];
#pragma unroll
  for (int k = 0; k < ROWS; ++k)
#pragma unroll
    for (int v = 0; v < VEC; ++v) acc[k][v] = 0.0;
  const uint64_t ub = uoff[item.x];
  const uint64_t beg = ub + item.y, end = ub + item.z;
  const float* xc = X + c0;
  for (uint64_t base = beg; base < end; base += kSameThreads) {
    const int cnt = (int)min((uint64_t)kSameThreads, end - base);
    stage_union<ROWS>(s_ket, s_val, uket, uval, base, cnt);
    if (!active) continue;
#pragma unroll 1
    for (int e0 = 0; e0 < cnt; e0 += kRun) {
      float pf[ROWS][VEC], x[kRun][VEC];
      const uint4 k0 = *reinterpret_cast<const uint4*>(s_ket + e0), k1 = *reinterpret_cast<const uint4*>(s_ket + e0 + 4);
      const uint32_t kt[kRun] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
#pragma unroll
      for (int u = 0; u < kRun; ++u) VecF<VEC>::load(xc + (size_t)kt[u] * ldx, x[u]);
#pragma unroll
      for (int u = 0; u < kRun; ++u) {
        const float4 w4 = *reinterpret_cast<const float4*>(s_val + (e0 + u) * ROWS);
        const float w[ROWS] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
        for (int k = 0; k < ROWS; ++k)
#pragma unroll
          for (int v = 0; v < VEC; ++v) pf[k][v] = u == 0 ? w[k] * x[u][v] : fmaf(w[k], x[u][v], pf[k][v]);
      }
#pragma unroll
      for (int k = 0; k < ROWS; ++k)
#pragma unroll
        for (int v = 0; v < VEC; ++v) acc[k][v] += (double)pf[k][v];
    }
  }
  if (active) {
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const uint32_t r = brows[item.x * ROWS + k];
      if (item.w == 0 && r == kNoRow) continue;
      double* y = item.w ? ypart + ((size_t)(item.w - 1) * ROWS + k) * ldx + c0 : Y + (size_t)r * ldx + c0;
#pragma unroll
      for (int v = 0; v < VEC; ++v) y[v] = acc[k][v];
    }
  }
  if (item.w == 0) return;
  const uint32_t sq = slot_split[item.w - 1];
  const uint4 sp = split[sq];
  if (!last_part(done, (size_t)sq * gridDim.y + blockIdx.y, sp.z) || !active) return;
  for (int k = 0; k < ROWS; ++k) {
    const uint32_t r = brows[item.x * ROWS + k];
    if (r == kNoRow) continue;
    double t[VEC];
#pragma unroll
    for (int v = 0; v < VEC; ++v) t[v] = 0.0;
    for (uint32_t p = 0; p < sp.z; ++p)
#pragma unroll
      for (int v = 0; v < VEC; ++v) t[v] += __ldcg(ypart + ((size_t)(sp.y + p) * ROWS + k) * ldx + c0 + v);
#pragma unroll
    for (int v = 0; v < VEC; ++v) Y[(size_t)r * ldx + c0 + v] = t[v];
  }
}

constexpr int kAb6Threads = 1024;

// Alpha single x beta single in the alpha-first basis, balanced. One CTA per
// (bra alpha row ia, chunk of 1024*KS virtual rows of the balanced beta SELL).
// Per group of R alpha singles ja of ia: the ket rows Xp[ja, :] and the
// integral rows (ai|..) of the unpacked table are copied to shared memory with
// 16-byte loads; lane l of a warp owns virtual row 32s+l of slice s and walks
// its records (contiguous 256-byte warp reads), applying each to the R staged
// rows: sign = s_alpha(ia,ja) xor s_beta(ib,jb), both from the connectivity.
// Warp w owns slices w, 2*32-1-w, 2*32+w, ... (a snake over the length-sorted
// slices). Unsplit virtual rows add their sum to Y directly; split parts park
// theirs in shared memory and are added in slot order (deterministic). All
// split parts lie in chunk 0.
template <typename T, int R, int KS>
__global__ void __launch_bounds__(kAb6Threads, 1)
sigma_ab_v6_kernel(const T* __restrict__ Xp, size_t nb, size_t ldx, const uint64_t* __restrict__ a_off,
                   const uint32_t* __restrict__ a_nsing, const uint32_t* __restrict__ a_ket,
                   const uint32_t* __restrict__ a_info, const uint64_t* __restrict__ sell,
                   const uint64_t* __restrict__ soff, const uint32_t* __restrict__ slen, size_t nslice,
                   const uint32_t* __restrict__ vrow, const uint32_t* __restrict__ vslot, size_t nv,
                   const uint32_t* __restrict__ split_row, const uint32_t* __restrict__ split_slot, int nsplit,
                   const typename Prec<T>::V* __restrict__ Vt, size_t vstride, size_t xstride,
                   double* __restrict__ Y) {
  using V = typename Prec<T>::V;
  constexpr int kWarps = kAb6Threads / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  T* xs = reinterpret_cast<T*>(smem);                                               // [R][xstride]
  V* erow = reinterpret_cast<V*>(smem + sizeof(T) * xstride * R);                   // [R][vstride]
  double* part = reinterpret_cast<double*>(smem + sizeof(T) * xstride * R + sizeof(V) * vstride * R);
  __shared__ uint32_t s_sa[R];
  const size_t ia = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t slice0 = (size_t)blockIdx.y * kWarps * KS;
  auto slice_of = [&](int k) -> size_t {
    return slice0 + (size_t)k * kWarps + ((k & 1) ? (kWarps - 1 - warp) : warp);
  };
  double acc[KS];
#pragma unroll
  for (int k = 0; k < KS; ++k) acc[k] = 0.0;
  const uint64_t e0 = a_off[ia];
  const int ns = (int)a_nsing[ia];
  const size_t xv = (nb * sizeof(T) + 15) / 16;  // 16-byte vectors of a ket row (xstride and ldx cover the tail)
  const size_t ev = vstride * sizeof(V) / 16;   // 16-byte vectors of an integral row
  for (int k0 = 0; k0 < ns; k0 += R) {
    const int nr = min(R, ns - k0);
    __syncthreads();
    if ((int)threadIdx.x < nr) s_sa[threadIdx.x] = a_info[e0 + k0 + threadIdx.x] >> 31;
    for (int rr = 0; rr < nr; ++rr) {
      const uint64_t e = e0 + k0 + rr;
      const uint4* s4 = reinterpret_cast<const uint4*>(Xp + (size_t)a_ket[e] * ldx);
      uint4* d4 = reinterpret_cast<uint4*>(xs + (size_t)rr * xstride);
      for (size_t t = threadIdx.x; t < xv; t += kAb6Threads) d4[t] = __ldg(s4 + t);
      const uint4* v4 = reinterpret_cast<const uint4*>(Vt + (size_t)((a_info[e] >> 12) & 0xfffu) * vstride);
      uint4* ed = reinterpret_cast<uint4*>(erow + (size_t)rr * vstride);
      for (size_t t = threadIdx.x; t < ev; t += kAb6Threads) ed[t] = __ldg(v4 + t);
    }
    __syncthreads();
    uint32_t sa[R];
#pragma unroll
    for (int rr = 0; rr < R; ++rr) sa[rr] = rr < nr ? s_sa[rr] : 0u;
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      const size_t sl = slice_of(k);
      if (sl >= nslice) continue;
      const uint32_t len = slen[sl];
      const uint64_t* rp = sell + soff[sl] + lane;
      double s = acc[k];
      uint64_t next = len ? __ldg(rp) : 0ull;
      for (uint32_t m = 0; m < len; ++m) {
        const uint64_t rec = next;
        if (m + 1 < len) next = __ldg(rp + 32ull * (m + 1));
        const uint32_t jb = rec_ket(rec);
        const uint32_t pq = (uint32_t)((rec >> 16) & 0xfffu);
        const uint32_t sb = (uint32_t)(rec >> 40) & 1u;
        const bool pad = (rec >> 41) & 1ull;
#pragma unroll
        for (int rr = 0; rr < R; ++rr) {
          if (rr < nr) {
            const double v = pad ? 0.0 : (double)erow[(size_t)rr * vstride + pq];
            s = fma(flip_sign(v, sa[rr] ^ sb), (double)xs[(size_t)rr * xstride + jb], s);
          }
        }
      }
      acc[k] = s;
    }
  }
#pragma unroll
  for (int k = 0; k < KS; ++k) {
    const size_t sl = slice_of(k);
    const size_t pos = sl * 32 + lane;
    if (sl < nslice && pos < nv) {
      const uint32_t slot1 = vslot[pos];
      if (slot1 == 0) Y[ia * ldx + vrow[pos]] += acc[k];
      else part[slot1 - 1] = acc[k];
    }
  }
  if (blockIdx.y == 0 && nsplit > 0) {
    __syncthreads();
    for (int s = threadIdx.x; s < nsplit; s += kAb6Threads) {
      double t = 0.0;
      for (uint32_t j = split_slot[s]; j < split_slot[s + 1]; ++j) t += part[j];
      Y[ia * ldx + split_row[s]] += t;
    }
  }
}

// 16-byte packs of the packed alpha-beta kernel: element e of pack h of pair
// index pq (of the pairs in use) is the signed integral s_alpha(ja) (a i|pq) of alpha single
// h * kRows + e of the group.
template <typename T> struct RowPack;
template <> struct RowPack<double> {
  using P = double2;
  static constexpr int kRows = 2;
  static __device__ __forceinline__ void set(P& p, int e, double v) { if (e == 0) p.x = v; else p.y = v; }
  static __device__ __forceinline__ void dot(const P& a, const double* c, double (&t)[2]) {
    t[0] = fma(a.x, c[0], t[0]);
    t[1] = fma(a.y, c[1], t[1]);
  }
};
template <> struct RowPack<float> {
  using P = float4;
  static constexpr int kRows = 4;
  static __device__ __forceinline__ void set(P& p, int e, float v) {
    if (e == 0) p.x = v; else if (e == 1) p.y = v; else if (e == 2) p.z = v; else p.w = v;
  }
  // 4-term dots in FP32, summed in FP64
  static __device__ __forceinline__ void dot(const P& a, const float* c, double (&t)[2]) {
    const float u = fmaf(a.x, c[0], a.y * c[1]), v = fmaf(a.z, c[2], a.w * c[3]);
    t[0] += (double)(u + v);
  }
};

// Arguments of the packed alpha-beta kernel on one panel of bra strings.
template <typename T>
struct AbArgs {
  const T* Xk;       // na x xs: phi o C, columns in lane order
  size_t xs, ldx;    // ldx: row stride of the partial rows
  size_t ldy;        // row stride of Y
  bool add;          // Y += instead of Y =
  const uint64_t* a_off;
  const uint32_t *a_ns, *a_ket, *a_info;
  const T* Vt;       // integrals over the pairs in use, row stride vstride
  const T* Dr;       // [na] rows of the integral row of the alpha string itself, row stride vstride
  size_t vstride;
  int npair;
  uint32_t vstr;     // packs per staged integral row
  int max_packs, np, panel, nmain, nex, ny;
  const uint4* rec;
  const uint64_t* boff;
  const uint32_t *bsteps, *wsteps, *ex_row, *ex_off;
  const uint4 *items, *split;
  const uint32_t* slot_split;
  uint32_t* done;
  double *ypart, *Y;
  int* err;
};

// Order of the updates of y: one arrival per warp and window on an mbarrier. A
// warp waits for window w - 1 before it updates y in window w, so the integral
// gathers of window w run while slower warps finish window w - 1; with a full
// barrier per step the shared-memory pipe drains at each one. Phases end
// by arrivals of this CTA's own warps alone; the wait is bounded all the same.
__device__ __forceinline__ void step_init(uint32_t bar, uint32_t warps) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(warps) : "memory");
}
__device__ __forceinline__ void step_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void step_wait(uint32_t bar, uint32_t ph, int* err) {
  if (ph == 0) return;
  const uint32_t parity = (ph - 1) & 1u;
  for (int it = 0; it < (1 << 20); ++it) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return;
  }
  atomicExch(err, kErrWatchdogAb);  // gives up: the result is flagged, nothing waits for it
}

// Batches b0 .. b1 - 1 of one group of nr alpha singles held in NH packs.
template <typename T, int NT, int NH>
__device__ __forceinline__ void ab_sweep(const AbArgs<T>& a, const typename RowPack<T>::P* __restrict__ vs,
                                         double* __restrict__ y, const uint32_t* s_ket, int nr, int b0, int b1,
                                         uint32_t bar, uint32_t& ph) {
  using RP = RowPack<T>;
  constexpr int VR = RP::kRows, R = NH * VR;
  const int warp = threadIdx.x >> 5;
  T c[R];
  auto load_c = [&](int b) {
    const bool live = a.wsteps[b * (NT / 32) + warp] > 0;
    const T* xb = a.Xk + (size_t)b * NT + threadIdx.x;
#pragma unroll
    for (int r = 0; r < R; ++r) c[r] = (r < nr && live) ? __ldg(xb + (size_t)s_ket[r] * a.xs) : (T)0;
  };
  load_c(b0);
  for (int b = b0; b < b1; ++b) {
    const int steps = (int)a.bsteps[b];
    const int wst = (int)a.wsteps[b * (NT / 32) + warp];
    const uint4* rp = a.rec + a.boff[b] + threadIdx.x;
    uint4 cur = wst > 0 ? __ldg(rp) : make_uint4(kAbPad, kAbPad, kAbPad, kAbPad);
    bool more = b + 1 < b1;  // the next batch's ket values are still to be loaded
    for (int m0 = 0; m0 < steps; m0 += 4) {
      if (m0 < wst) {
        const uint4 nxt = m0 + 4 < wst ? __ldg(rp + (size_t)(m0 / 4 + 1) * NT) : cur;
        const uint32_t recs[4] = {cur.x, cur.y, cur.z, cur.w};
#pragma unroll
        for (int w0 = 0; w0 < 4; w0 += kAbWindow) {
          if (m0 + w0 >= steps) break;
          double t[kAbWindow][2];
#pragma unroll
          for (int q = 0; q < kAbWindow; ++q) {
            t[q][0] = t[q][1] = 0.0;
            if (m0 + w0 + q < wst) {  // warp-uniform
              const typename RP::P* v = vs + (recs[w0 + q] & 0xfffu);
#pragma unroll
              for (int h = 0; h < NH; ++h) RP::dot(v[(size_t)h * a.vstr], c + h * VR, t[q]);
            }
          }
          if (more && m0 + w0 + kAbWindow >= wst) {  // this batch's values are used up
            load_c(b + 1);
            more = false;
          }
          step_wait(bar, ph, a.err);  // the previous window's updates of y are done
#pragma unroll
          for (int q = 0; q < kAbWindow; ++q) {
            const uint32_t rec = recs[w0 + q];
            if (m0 + w0 + q < wst && !(rec & kAbPad)) {
              double* yp = y + ((rec >> 12) & 0xffffu);
              *yp += flip_sign(t[q][0] + t[q][1], rec >> 31);
            }
          }
          __syncwarp();
          if ((threadIdx.x & 31) == 0) step_arrive(bar);
          ++ph;
        }
        cur = nxt;
      } else {
        if (more) {
          load_c(b + 1);
          more = false;
        }
        for (int w0 = 0; w0 < 4 && m0 + w0 < steps; w0 += kAbWindow) {
          step_wait(bar, ph, a.err);
          if ((threadIdx.x & 31) == 0) step_arrive(bar);
          ++ph;
        }
      }
    }
    if (more) load_c(b + 1);  // a batch without steps
  }
}

// Alpha single x beta single in the alpha-first basis. One CTA per work item:
// a bra alpha string, or a range of its singles and of the schedule's batches
// (AbItems).
// Per group of up to kAbPacks * kRows alpha singles (ja_r, pq_r, s_r) of the
// item, the signed integral rows s_r (pq_r|..) are staged in shared memory as
// 16-byte packs; a thread owns one ket string jb at a time, with C'[ja_r, jb]
// of the whole group in registers, and walks jb's singles (ib <- jb, rs, s):
// y[ib] += s * sum_r s_r (pq_r|rs) C'[ja_r, jb], y in shared memory. The
// Coulomb terms of the beta singles with the alpha string ride along as one
// more "single" ja = ia whose integral row is Dr. The
// schedule (AbPlan) never lets two threads of a window of steps update the same
// slot, so the updates need no atomics and have one summation order.
//
// Bound: the shared-memory pipe. Staging integrals instead of ket rows lets a
// group hold 10 (FP64) or 20 (FP32) alpha singles instead of the 2 or 4 whose
// ket rows of 8000 strings fit, and replaces the ket gather of every pair by
// registers: per record of a group one 16-byte gather per pack and one
// read-add-write of y, against two 16-byte gathers per pack. The pipe is 78% busy
// at 8000 x 8000 (62% at 613 x 1187). 8000 x 8000: 17.4 -> 13.6 ms FP64, 9.6 ->
// 8.4 ms FP32. Measured and not taken: a barrier per step instead of the
// mbarrier (13.8 against 12.9 ms at the time), ket strings sorted by string or
// pair indices spread over the banks by the schedule (no change), the Coulomb
// terms of the alpha singles here (5.5 ms more), the first ket values loaded
// before the integrals are staged (no change FP64, 0.2 ms more FP32).
template <typename T, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) sigma_ab_kernel(const AbArgs<T> a) {
  using RP = RowPack<T>;
  using P = typename RP::P;
  constexpr int VR = RP::kRows;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t s_ket[kAbPacks * 4], s_pq[kAbPacks * 4];
  __shared__ __align__(8) uint64_t s_bar;
  const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&s_bar);
  uint32_t ph = 0;  // windows finished by this warp
  if (threadIdx.x == 0) step_init(bar, NT / 32);
  const uint4 item = a.items[blockIdx.x];
  const size_t ia = item.x;
  double* y = reinterpret_cast<double*>(smem);                        // [ny]
  P* vs = reinterpret_cast<P*>(smem + (((size_t)a.ny * 8 + 15) & ~(size_t)15));  // [packs][vstr]
  for (int i = threadIdx.x; i < a.ny; i += NT) y[i] = 0.0;
  const uint64_t e0 = a.a_off[ia];
  const int first = (int)(item.y & 0xffffu), n = (int)(item.y >> 16) - first, ns = (int)a.a_ns[ia];
  const int b0 = (int)(item.z & 0xffffu), b1 = (int)(item.z >> 16);
  const int rmax = a.max_packs * VR;
  const int ng = (n + rmax - 1) / rmax;
  const int per = ng > 0 ? ((n + ng - 1) / ng + VR - 1) / VR * VR : VR;  // balanced groups of whole packs
  for (int k0 = 0; k0 < n; k0 += per) {
    const int nr = min(per, n - k0), nh = (nr + VR - 1) / VR;
    const int nd = min(nr, ns - first - k0);  // the rest (at most one) is the string itself
    __syncthreads();  // the integrals of the group before are no longer read
    if ((int)threadIdx.x < nh * VR) {
      uint32_t ket = (uint32_t)ia, pqs = 0;
      if ((int)threadIdx.x < nd) {
        const uint64_t ent = e0 + first + k0 + threadIdx.x;
        const uint32_t inf = a.a_info[ent];
        ket = a.a_ket[ent];
        pqs = ((inf >> 12) & 0xfffu) | (inf & kInfoNeg);
      }
      s_ket[threadIdx.x] = ket;
      s_pq[threadIdx.x] = pqs;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < a.npair; t += NT) {
#pragma unroll
      for (int h = 0; h < kAbPacks; ++h) {
        if (h >= nh) break;
        P p;
#pragma unroll
        for (int e = 0; e < VR; ++e) {
          const int r = h * VR + e;
          const uint32_t pqs = s_pq[r];
          const T* row = r < nd ? a.Vt + (size_t)(pqs & 0xfffu) * a.vstride : a.Dr + ia * a.vstride;
          const T v = r < nr ? __ldg(row + t) : (T)0;
          RP::set(p, e, (pqs >> 31) ? -v : v);
        }
        vs[(size_t)h * a.vstr + t] = p;
      }
    }
    __syncthreads();
    switch (nh) {
      case 1: ab_sweep<T, NT, 1>(a, vs, y, s_ket, nr, b0, b1, bar, ph); break;
      case 2: ab_sweep<T, NT, 2>(a, vs, y, s_ket, nr, b0, b1, bar, ph); break;
      case 3: ab_sweep<T, NT, 3>(a, vs, y, s_ket, nr, b0, b1, bar, ph); break;
      case 4: ab_sweep<T, NT, 4>(a, vs, y, s_ket, nr, b0, b1, bar, ph); break;
      default: ab_sweep<T, NT, 5>(a, vs, y, s_ket, nr, b0, b1, bar, ph); break;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < a.nex; e += NT) {  // extra slots of crowded strings, in slot order
    double t = y[a.ex_row[e]];
    for (uint32_t j = a.ex_off[e]; j < a.ex_off[e + 1]; ++j) t += y[a.nmain + j];
    y[a.ex_row[e]] = t;
  }
  if (a.nex > 0) __syncthreads();
  auto col = [&](int i) -> size_t { return a.np == 1 ? (size_t)i : (size_t)(i / 4) * 4 * a.np + 4 * a.panel + i % 4; };
  double* __restrict__ Yrow = a.Y + ia * a.ldy;
  if (item.w == 0) {
    for (int i = threadIdx.x; i < a.nmain; i += NT) {
      const size_t k = col(i);
      Yrow[k] = a.add ? Yrow[k] + y[i] : y[i];
    }
    return;
  }
  // a part of a split string: its partial row; the last part to finish adds all in slot order
  double* mine = a.ypart + (size_t)(item.w - 1) * a.ldx;
  for (int i = threadIdx.x; i < a.nmain; i += NT) mine[col(i)] = y[i];
  const uint32_t sp = a.slot_split[item.w - 1];
  const uint4 s = a.split[sp];
  if (!last_part(a.done, sp, s.z)) return;
  const double* part = a.ypart + (size_t)s.y * a.ldx;
  for (int i = threadIdx.x; i < a.nmain; i += NT) {
    const size_t k = col(i);
    double t = 0.0;
    for (uint32_t q = 0; q < s.z; ++q) t += __ldcg(part + (size_t)q * a.ldx + k);
    Yrow[k] = a.add ? Yrow[k] + t : t;
  }
}

template <typename T, int NT, int MINB>
int launch_ab(Ctx* c, const AbArgs<T>& args, size_t n_item, size_t smem) {
  SBDX_CUDA(c, cudaFuncSetAttribute(sigma_ab_kernel<T, NT, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kAbSmemBudget));
  sigma_ab_kernel<T, NT, MINB><<<(unsigned)n_item, NT, smem, c->stream>>>(args);
  SBDX_LAUNCHED(c);
  return 0;
}

// The alpha-beta product of Xk over the rows of the work items (the alpha
// connectivity's, or those of a row range, Ctx::range_conn) into Y, row stride
// ldy, or added to it.
template <typename T>
int run_ab_packed(Ctx* c, const Conn* items, const T* Xk, double* Y, size_t ldy, bool add) {
  const Conn& ca = c->conn[0];
  const bool f64 = std::is_same<T, double>::value;
  const AbItems& it = (items ? *items : ca).ab[f64 ? 0 : 1];
  if (it.n == 0) return 0;
  const AbPlan& P = c->ab;
  for (size_t q = 0; q < P.panels.size(); ++q) {
    const AbPanel& p = P.panels[q];
    AbArgs<T> a{};
    a.Xk = Xk;
    a.xs = P.xs;
    a.ldx = c->xsa;
    a.ldy = ldy;
    a.add = add;
    a.a_off = ca.off;
    a.a_ns = ca.nsing;
    a.a_ket = ca.ket;
    a.a_info = ca.info;
    a.Dr = f64 ? (const T*)c->d_Dr : (const T*)c->d_Dr32;
    a.Vt = f64 ? (const T*)P.V : (const T*)P.V32;
    a.vstride = f64 ? P.vstride : P.vstride32;
    a.npair = P.npu;
    a.vstr = P.vstr;
    a.max_packs = P.packs;
    a.np = P.np;
    a.panel = (int)q;
    a.nmain = p.nmain;
    a.nex = p.nex;
    a.ny = p.ny;
    a.rec = reinterpret_cast<const uint4*>(p.rec);
    a.boff = p.boff;
    a.bsteps = p.bsteps;
    a.wsteps = p.wsteps;
    a.ex_row = p.ex_row;
    a.ex_off = p.ex_off;
    a.items = it.item;
    a.split = it.split;
    a.slot_split = it.slot;
    a.done = it.done;
    a.ypart = it.ypart;
    a.Y = Y;
    a.err = c->d_err;
    const size_t smem = (((size_t)p.ny * 8 + 15) & ~(size_t)15) + 16 * (size_t)a.max_packs * P.vstr;
    int rc;
    if (P.threads == 256) rc = launch_ab<T, 256, 4>(c, a, it.n, smem);
    else if (P.threads == 512) rc = launch_ab<T, 512, 2>(c, a, it.n, smem);
    else rc = launch_ab<T, 1024, 1>(c, a, it.n, smem);
    if (rc) return rc;
  }
  return 0;
}

template <typename T, int VEC>
int launch_same_v6(Ctx* c, const T* X, size_t ncol, size_t ldx, const Conn& cn, const typename Prec<T>::V* val,
                   const typename Prec<T>::V* Dt, size_t dstride, double* Y) {
  if (cn.n_same_item == 0) return 0;
  dim3 grid((unsigned)cn.n_same_item,
            (unsigned)((ncol + (size_t)kSameThreads * VEC - 1) / ((size_t)kSameThreads * VEC)));
  if constexpr (std::is_same<T, float>::value) {
    sigma_same_v6f_kernel<VEC><<<grid, kSameThreads, 0, c->stream>>>(
        X, ncol, ldx, cn.off, cn.nsing, cn.ket, val, cn.info, Dt, dstride, cn.same_item, cn.same_split,
        cn.same_slot, cn.same_done, cn.same_ypart, Y);
  } else {
    sigma_same_v6_kernel<T, VEC><<<grid, kSameThreads, 0, c->stream>>>(
        X, ncol, ldx, cn.off, cn.nsing, cn.ket, val, cn.info, Dt, dstride, cn.same_item, cn.same_split,
        cn.same_slot, cn.same_done, cn.same_ypart, Y);
  }
  SBDX_LAUNCHED(c);
  return 0;
}

int launch_same_blk(Ctx* c, int, const double* X, size_t ncol, size_t ldx, const SameBlocks& B, double* Y) {
  constexpr size_t smem = kMmaStageBytes * kMmaStages;
  SBDX_CUDA(c, cudaFuncSetAttribute(sigma_same_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const dim3 grid((unsigned)B.n_item, (unsigned)((ncol + kMmaCols - 1) / kMmaCols));
  sigma_same_mma_kernel<<<grid, kSameThreads, smem, c->stream>>>(X, ncol, ldx, B.rows, B.uoff, B.uket, B.uval, B.item,
                                                                 B.split, B.slot, B.done, B.ypart, Y, c->d_err);
  SBDX_LAUNCHED(c);
  return 0;
}

template <int VEC>
int launch_same_blkf(Ctx* c, const float* X, size_t ncol, size_t ldx, const SameBlocks& B, double* Y) {
  const dim3 grid((unsigned)B.n_item, (unsigned)((ncol + (size_t)kSameThreads * VEC - 1) / ((size_t)kSameThreads * VEC)));
  sigma_same_blkf_kernel<VEC><<<grid, kSameThreads, 0, c->stream>>>(X, ncol, ldx, B.rows, B.uoff, B.uket, B.uval32, B.item,
                                                                    B.split, B.slot, B.done, B.ypart, Y);
  SBDX_LAUNCHED(c);
  return 0;
}

int launch_same_blk(Ctx* c, int vec, const float* X, size_t ncol, size_t ldx, const SameBlocks& B, double* Y) {
  if (vec >= 4) return launch_same_blkf<4>(c, X, ncol, ldx, B, Y);
  if (vec == 2) return launch_same_blkf<2>(c, X, ncol, ldx, B, Y);
  return launch_same_blkf<1>(c, X, ncol, ldx, B, Y);
}

constexpr int kStrings64 = 22;  // the one-string kernel that serves FP64 best

// Same-spin codes: 21, 22, 24, 28 = 1, 2, 4, 8 columns per thread of the
// one-string kernels, narrowed to the widest vector that divides the row
// stride and keeps 16-byte alignment (the internal vectors have strides
// padded to 8 elements, so only a misaligned base narrows). 31, 32, 34, 38:
// the blocked kernels, whose FP64 form has one shape (128 columns per warp) and
// whose FP32 form takes up to 4 columns per thread.
template <typename T>
int run_same_v6(Ctx* c, const Tune& tune, const T* X, size_t ncol, size_t ldx, const Conn& cn, size_t row0, size_t nrow,
                const typename Prec<T>::V* val, const typename Prec<T>::V* Dt, size_t dstride, double* Y) {
  int code = tune.same_code;
  if (tune.by_size && std::is_same<T, double>::value && ncol < kBlkMinCols64) code = kStrings64;
  int vec = code % 10;
  const bool aligned = (reinterpret_cast<uintptr_t>(X) % 16) == 0;
  while (vec > 1 && (!aligned || ldx % vec != 0 || (Dt != nullptr && dstride % vec != 0))) vec >>= 1;
  if (code / 10 == 3 && cn.blk[0].nblk > 0 && aligned && nrow > 0) {
    const int rc = launch_same_blk(c, vec, X, ncol, ldx, cn.blk[std::is_same<T, double>::value ? 0 : 1], Y);
    if (rc) return rc;
    if (Dt != nullptr) {  // the singles' Coulomb terms
      constexpr size_t cols = (size_t)kSameThreads * 16 / sizeof(T);
      const dim3 grid((unsigned)nrow, (unsigned)((ncol + cols - 1) / cols));
      sigma_coulomb_kernel<T><<<grid, kSameThreads, 0, c->stream>>>(X, ncol, ldx, row0, cn.off, cn.nsing, cn.ket, cn.info,
                                                                    Dt, dstride, Y);
      SBDX_LAUNCHED(c);
    }
    sigma_same_nonfinite_kernel<T><<<148, kSameThreads, 0, c->stream>>>(c->d_nonfinite, X, ncol, ldx, row0, nrow, cn.off,
                                                                        cn.nsing, cn.ket, val, cn.info, Dt, dstride, Y);
    SBDX_LAUNCHED(c);
    return 0;
  }
  if (vec >= 8) return launch_same_v6<T, 8>(c, X, ncol, ldx, cn, val, Dt, dstride, Y);
  if (vec >= 4) return launch_same_v6<T, 4>(c, X, ncol, ldx, cn, val, Dt, dstride, Y);
  if (vec == 2) return launch_same_v6<T, 2>(c, X, ncol, ldx, cn, val, Dt, dstride, Y);
  return launch_same_v6<T, 1>(c, X, ncol, ldx, cn, val, Dt, dstride, Y);
}

template <typename T, int R, int KS>
int launch_ab_v6(Ctx* c, const T* Xp, size_t smem, size_t xstride) {
  using V = typename Prec<T>::V;
  const Conn& ca = c->conn[0];
  const Conn& cb = c->conn[1];
  const bool f64 = std::is_same<T, double>::value;
  const V* Vt = f64 ? (const V*)c->d_V : (const V*)c->d_V32;
  const size_t vs = f64 ? c->vstride : c->vstride32;
  SBDX_CUDA(c, cudaFuncSetAttribute(sigma_ab_v6_kernel<T, R, KS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kAbSmemBudget));
  const size_t per_cta = (size_t)(kAb6Threads / 32) * KS;  // slices
  const SellPanel& bp = cb.bal;
  dim3 grid((unsigned)c->na, (unsigned)((bp.nslice + per_cta - 1) / per_cta));
  if (grid.y == 0) grid.y = 1;
  sigma_ab_v6_kernel<T, R, KS><<<grid, kAb6Threads, smem, c->stream>>>(
      Xp, c->nb, c->xsa, ca.off, ca.nsing, ca.ket, ca.info, bp.sell, bp.soff, bp.slen, bp.nslice, bp.vrow, bp.vslot,
      bp.nv,
      bp.split_row, bp.split_slot, bp.nsplit, Vt, vs, xstride, c->d_y);
  SBDX_LAUNCHED(c);
  return 0;
}

template <typename T, int R>
int launch_ab_v6_ks(Ctx* c, const T* Xp, size_t smem, size_t xstride) {
  const int ks = c->conn[1].bal.slices_per_warp;
  if (ks >= 16) return launch_ab_v6<T, R, 16>(c, Xp, smem, xstride);
  if (ks >= 12) return launch_ab_v6<T, R, 12>(c, Xp, smem, xstride);
  return launch_ab_v6<T, R, 8>(c, Xp, smem, xstride);
}

// v6 alpha-beta codes: 61-64 = 1-4 staged alpha singles per group, narrowed
// until the ket rows, integral rows and split slots fit in shared memory.
template <typename T>
int run_ab_v6(Ctx* c, int code, const T* Xp) {
  using V = typename Prec<T>::V;
  const bool f64 = std::is_same<T, double>::value;
  const size_t vs = f64 ? c->vstride : c->vstride32;
  const size_t per = 16 / sizeof(T);
  const size_t xstride = (c->nb + per - 1) / per * per;
  const size_t budget = kAbSmemBudget;  // dynamic part; the static part is a few bytes
  const size_t extra = sizeof(double) * (size_t)c->conn[1].bal.nslot;
  int R = code % 10 > 0 ? code % 10 : 2;
  size_t smem = 0;
  for (; R >= 1; --R) {
    smem = (size_t)R * (sizeof(T) * xstride + sizeof(V) * vs) + extra;
    if (smem <= budget) break;
  }
  if (R < 1) {
    c->err = "sigma: beta dimension too large for one shared-memory ket row";
    return 1;
  }
  if (R >= 4) return launch_ab_v6_ks<T, 4>(c, Xp, smem, xstride);
  if (R == 3) return launch_ab_v6_ks<T, 3>(c, Xp, smem, xstride);
  if (R == 2) return launch_ab_v6_ks<T, 2>(c, Xp, smem, xstride);
  return launch_ab_v6_ks<T, 1>(c, Xp, smem, xstride);
}

// Xk of all rows.
template <typename T>
int launch_lanes(Ctx* c, const T* X, T* Xk) {
  const size_t xs = c->ab.xs;
  const dim3 grid((unsigned)((xs + 255) / 256), (unsigned)((c->na + 31) / 32));
  lane_order_kernel<T><<<grid, 256, 0, c->stream>>>(X, c->na, c->nb, c->d_a, c->d_b, c->ab.vket, Xk, xs);
  SBDX_LAUNCHED(c);
  return 0;
}

// The alpha-beta product of the items' rows (code 71): into d_yab from the
// lanes that the split wrote, or, lean, added to d_y from lanes in the room of
// d_xp and d_xt, once the same-spin products have read those.
template <typename T>
int run_ab_71(Ctx* c, const T* X, const Conn* items = nullptr) {
  if (!c->lean) return run_ab_packed<T>(c, items, reinterpret_cast<const T*>(c->d_xk), c->d_yab, c->xsa, false);
  T* xk = reinterpret_cast<T*>(c->d_xp);
  const int rc = launch_lanes<T>(c, X, xk);
  return rc ? rc : run_ab_packed<T>(c, items, xk, c->d_y, c->xsa, true);
}

// Phase split of the rows [a0, a0 + nr) (X: the whole input), with their
// lane-order copy when the packed alpha-beta kernel reads it beside the others.
template <typename T>
int launch_split(Ctx* c, const T* X, size_t a0, size_t nr, T* xp, T* xpt, bool lanes, int* nonfinite) {
  const size_t nb = c->nb, xs = lanes && !c->lean ? c->ab.xs : 0;
  const dim3 grid((unsigned)((nb + 31) / 32 + (xs + 255) / 256), (unsigned)((nr + 31) / 32));
  phase_split_kernel<T><<<grid, dim3(32, 8), 0, c->stream>>>(
      X + a0 * nb, nr, nb, c->d_a + a0, c->d_b, xp + a0 * c->xsa, xpt + a0, c->xsa, c->xsb, c->ab.vket,
      reinterpret_cast<T*>(c->d_xk) + a0 * xs, xs, nonfinite);
  SBDX_LAUNCHED(c);
  return 0;
}

// S (row 0 = alpha string a0) of the rows [a0, a0 + nr); X: the whole input.
// in_place: S holds the alpha-beta part; otherwise d_yab does after code 71,
// or d_y. last: nothing reads the input's flag after this.
template <typename T>
int launch_combine(Ctx* c, const T* X, size_t a0, size_t nr, T* S, bool packed, bool in_place = false, bool last = true) {
  const size_t nb = c->nb;
  const dim3 grid((unsigned)((nb + 31) / 32), (unsigned)((nr + 31) / 32));
  auto go = [&](auto kernel) {
    kernel<<<grid, dim3(32, 8), 0, c->stream>>>(c->d_y + a0 * c->xsa, packed && !c->lean ? c->d_yab + a0 * c->xsa : nullptr,
                                                c->d_yt + a0, c->d_hii + a0 * nb, X + a0 * nb, nr, nb, c->d_a + a0, c->d_b,
                                                S, c->xsa, c->xsb, last ? c->d_nonfinite : nullptr);
  };
  if (in_place) go(combine_phase_kernel<T, true>);
  else go(combine_phase_kernel<T, false>);
  SBDX_LAUNCHED(c);
  return 0;
}

bool same_alpha_first(int code) { return (code > 20 && code < 30) || (code > 30 && code < 40); }

bool is_v6(const Tune& t) {
  return same_alpha_first(t.same_code) && ((t.ab_code > 60 && t.ab_code < 70) || t.ab_code == 71);
}

// Runs launches of the context on its side streams, so that a small problem's
// three products, none of which fills the GPU, overlap (FP64 275 x 275 strings:
// 72.5 us per sigma one after another, 49.5 us side by side; 2000 x 2000: 1324
// and 1210 us; 8000 x 8000 unchanged within 1%): fork() makes both follow
// the context stream, on(k) directs the next launches to side stream k, main()
// back, join() makes the context stream follow both.
struct SideBySide {
  Ctx* c;
  cudaStream_t home;
  explicit SideBySide(Ctx* ctx) : c(ctx), home(ctx->stream) {}
  ~SideBySide() { c->stream = home; }
  int fork() {
    SBDX_CUDA(c, cudaEventRecord(c->fork, home));
    for (cudaStream_t s : c->side) SBDX_CUDA(c, cudaStreamWaitEvent(s, c->fork, 0));
    return 0;
  }
  void on(int k) { c->stream = c->side[k]; }
  void main() { c->stream = home; }
  int join() {
    c->stream = home;
    for (int k = 0; k < 2; ++k) {
      SBDX_CUDA(c, cudaEventRecord(c->join[k], c->side[k]));
      SBDX_CUDA(c, cudaStreamWaitEvent(home, c->join[k], 0));
    }
    return 0;
  }
};

template <typename T>
int run_sigma_v6(Ctx* c, const Tune& tune, const T* X, T* S) {
  using V = typename Prec<T>::V;
  const size_t na = c->na, nb = c->nb;
  const bool f64 = std::is_same<T, double>::value;
  const Conn& ca = c->conn[0];
  const Conn& cb = c->conn[1];
  const V* valA = f64 ? (const V*)ca.val : (const V*)ca.val32;
  const V* valB = f64 ? (const V*)cb.val : (const V*)cb.val32;
  const V* Db = f64 ? (const V*)c->d_Db : (const V*)c->d_Db32;
  const V* Da = f64 ? (const V*)c->d_Da : (const V*)c->d_Da32;
  T* xp = reinterpret_cast<T*>(c->d_xp);
  T* xpt = reinterpret_cast<T*>(c->d_xt);
  auto mark = [&](int k) {
    if (c->profiling) cudaEventRecord(c->ev[k], c->stream);
  };
  int rc = 0;
  mark(0);
  if ((rc = launch_split<T>(c, X, 0, na, xp, xpt, tune.ab_code == 71, c->d_nonfinite))) return rc;
  // the beta singles' Coulomb terms: in the packed alpha-beta kernel, or in the
  // same-spin kernels beside an unpacked one
  const bool packed = tune.ab_code == 71;
  const V* DtA = Db;
  const V* DtB = packed ? nullptr : Da;
  if (packed && !c->lean && !c->profiling) {
    SideBySide f(c);
    if ((rc = f.fork())) return rc;
    f.on(0);
    rc = run_same_v6<T>(c, tune, xp, nb, c->xsa, ca, 0, na, valA, DtA, c->db_stride, c->d_y);
    f.on(1);
    if (!rc) rc = run_same_v6<T>(c, tune, xpt, na, c->xsb, cb, 0, nb, valB, DtB, c->da_stride, c->d_yt);
    f.main();
    if (!rc) rc = run_ab_71<T>(c, X);
    const int rj = f.join();
    if (rc || rj) return rc ? rc : rj;
    return launch_combine<T>(c, X, 0, na, S, true);
  }
  mark(1);
  if ((rc = run_same_v6<T>(c, tune, xp, nb, c->xsa, ca, 0, na, valA, DtA, c->db_stride, c->d_y)))
    return rc;
  mark(2);
  if ((rc = run_same_v6<T>(c, tune, xpt, na, c->xsb, cb, 0, nb, valB, DtB, c->da_stride, c->d_yt)))
    return rc;
  mark(3);
  if ((rc = packed ? run_ab_71<T>(c, X) : run_ab_v6<T>(c, tune.ab_code, xp))) return rc;
  mark(4);
  if ((rc = launch_combine<T>(c, X, 0, na, S, packed))) return rc;
  mark(5);
  if (c->profiling) {
    // reported in the phase order alpha same-spin, transpose (here the phase
    // split), beta same-spin, alpha-beta, combine
    const int from[kSigmaPhases] = {1, 0, 2, 3, 4};
    SBDX_CUDA(c, cudaEventSynchronize(c->ev[5]));
    for (int k = 0; k < kSigmaPhases; ++k) {
      float ms = 0.f;
      SBDX_CUDA(c, cudaEventElapsedTime(&ms, c->ev[from[k]], c->ev[from[k] + 1]));
      c->phase_ms[k] += ms;
    }
    ++c->phase_calls;
  }
  return 0;
}

template <typename T>
int run_sigma_v5(Ctx* c, const T* X, T* S) {
  using V = typename Prec<T>::V;
  const size_t na = c->na, nb = c->nb;
  const Conn& ca = c->conn[0];
  const Conn& cb = c->conn[1];
  const V* valA = std::is_same<T, double>::value ? (const V*)ca.val : (const V*)ca.val32;
  const V* valB = std::is_same<T, double>::value ? (const V*)cb.val : (const V*)cb.val32;
  const V* G = std::is_same<T, double>::value ? (const V*)c->d_G : (const V*)c->d_G32;
  T* xt = reinterpret_cast<T*>(c->d_xt);
  auto mark = [&](int k) {
    if (c->profiling) cudaEventRecord(c->ev[k], c->stream);
  };
  int rc = 0;
  mark(0);
  // 1. alpha excitations + diagonal -> Y
  if ((rc = run_same<T>(c, X, na, nb, c->d_b, ca, valA, G, c->d_hii, c->d_y))) return rc;
  mark(1);
  // 2. C -> C^T
  {
    dim3 grid((unsigned)((nb + 31) / 32), (unsigned)((na + 31) / 32));
    transpose_kernel<T><<<grid, dim3(32, 8), 0, c->stream>>>(X, na, nb, xt);
    SBDX_LAUNCHED(c);
  }
  mark(2);
  // 3. beta excitations on C^T -> Yt
  if ((rc = run_same<T>(c, xt, nb, na, c->d_a, cb, valB, G, nullptr, c->d_yt))) return rc;
  mark(3);
  // 4. alpha single x beta single -> Y +=
  if ((rc = run_ab<T>(c, X))) return rc;
  mark(4);
  // 5. S = Y + Yt^T
  {
    dim3 grid((unsigned)((nb + 31) / 32), (unsigned)((na + 31) / 32));
    combine_transpose_kernel<T><<<grid, dim3(32, 8), 0, c->stream>>>(c->d_y, c->d_yt, na, nb, S);
    SBDX_LAUNCHED(c);
  }
  mark(5);
  if (c->profiling) {
    SBDX_CUDA(c, cudaEventSynchronize(c->ev[5]));
    for (int k = 0; k < kSigmaPhases; ++k) {
      float ms = 0.f;
      SBDX_CUDA(c, cudaEventElapsedTime(&ms, c->ev[k], c->ev[k + 1]));
      c->phase_ms[k] += ms;
    }
    ++c->phase_calls;
  }
  return 0;
}

// Default launch codes: the alpha-first kernels; the blocked same-spin kernels
// above a size where the grid of their blocks still fills the GPU and the
// strings of a block share excitations, the one-string-per-CTA kernel below it.
// Measured on both sides of the lines (alpha and beta same-spin, us): FP64,
// 2000 x 2000: 278 and 205 blocked, 368 and 370 by strings; FP32, 613 x 1187:
// 97 and 44 blocked, 58 and 47 by strings. In FP64 the blocked kernel gives a
// warp 128 columns of a strip of 1024, so a product with few columns (the other
// spin's strings, or the rows of a range) leaves most warps idle: 7 electrons
// in 58 orbitals, us, blocked / by strings: 100 columns of 20000 strings 2345 /
// 1097, 250 of 8000 560 / 374, 400 of 8000 615 / 574, 500 of 5000 314 / 350.
Tune default_tune(const Ctx* c, bool f64) {
  const size_t D = c->na * c->nb;
  if (f64) return D >= kBlkMinDets64 ? Tune{34, 71, true} : Tune{kStrings64, 71, true};
  return D >= kBlkMinDets32 ? Tune{34, 71, true} : Tune{24, 71, true};
}

Tune effective_tune(const Ctx* c, bool f64) {
  Tune t = c->tune[f64 ? 0 : 1];
  const Tune d = default_tune(c, f64);
  const bool v6 = same_alpha_first(t.same_code) || (t.ab_code > 60 && t.ab_code < 70) ||
                  t.ab_code == 71 || (t.same_code == 0 && t.ab_code == 0);
  if (v6) {
    if (t.same_code == 0) t.same_code = d.same_code, t.by_size = true;
    if (t.ab_code == 0) t.ab_code = d.ab_code;
  }
  return t;
}

template <typename T>
int run_sigma(Ctx* c, const T* X, T* S) {
  const Tune t = effective_tune(c, std::is_same<T, double>::value);
  if (is_v6(t)) return run_sigma_v6<T>(c, t, X, S);
  return run_sigma_v5<T>(c, X, S);
}

// Output rows [a0, a1) of the alpha-first sigma (one shard of the alpha
// strings; the reference's bra block of a rank, chemistry/tpb/mult.h:429-432).
// The phase split covers the whole input (every ket row may be read); the
// alpha same-spin and alpha-beta kernels run the range's work items
// (Ctx::range_conn); the beta same-spin kernel runs on the range's columns of
// the transposed input (its output and Coulomb-table columns offset by a0,
// a multiple of 8 so that the vector loads stay aligned); the combine writes
// the range's rows into S, whose row 0 is alpha string a0.
template <typename T>
int run_sigma_rows(Ctx* c, const Tune& tune, const T* X, T* S, size_t a0, size_t a1) {
  using V = typename Prec<T>::V;
  const size_t na = c->na, nb = c->nb, nr = a1 - a0;
  const bool f64 = std::is_same<T, double>::value;
  const Conn& ca = c->conn[0];
  const Conn& cb = c->conn[1];
  const Conn& rc_items = c->range_conn;
  Conn ra = ca;  // the alpha lists with the range's same-spin work items
  for (int q = 0; q < 2; ++q) ra.blk[q] = rc_items.blk[q];
  ra.same_item = rc_items.same_item;
  ra.n_same_item = rc_items.n_same_item;
  ra.same_split = rc_items.same_split;
  ra.same_slot = rc_items.same_slot;
  ra.same_done = rc_items.same_done;
  ra.n_same_split = rc_items.n_same_split;
  ra.n_same_part = rc_items.n_same_part;
  ra.same_ypart = rc_items.same_ypart;
  const V* valA = f64 ? (const V*)ca.val : (const V*)ca.val32;
  const V* valB = f64 ? (const V*)cb.val : (const V*)cb.val32;
  const V* Db = f64 ? (const V*)c->d_Db : (const V*)c->d_Db32;
  T* xp = reinterpret_cast<T*>(c->d_xp);
  T* xpt = reinterpret_cast<T*>(c->d_xt);
  auto mark = [&](int k) {
    if (c->profiling) cudaEventRecord(c->ev[k], c->stream);
  };
  int rc = 0;
  mark(0);
  if ((rc = launch_split<T>(c, X, 0, na, xp, xpt, true, c->d_nonfinite))) return rc;
  mark(1);
  if (nr == 0) return 0;
  if ((rc = run_same_v6<T>(c, tune, xp, nb, c->xsa, ra, a0, nr, valA, Db, c->db_stride, c->d_y)))
    return rc;
  mark(2);
  if ((rc = run_same_v6<T>(c, tune, xpt + a0, nr, c->xsb, cb, 0, nb, valB, (const V*)nullptr, 0, c->d_yt + a0)))
    return rc;
  mark(3);
  if ((rc = run_ab_71<T>(c, X, &rc_items))) return rc;
  mark(4);
  if ((rc = launch_combine<T>(c, X, a0, nr, S, true))) return rc;
  mark(5);
  if (c->profiling) {  // the phase order of run_sigma_v6
    const int from[kSigmaPhases] = {1, 0, 2, 3, 4};
    SBDX_CUDA(c, cudaEventSynchronize(c->ev[5]));
    for (int k = 0; k < kSigmaPhases; ++k) {
      float ms = 0.f;
      SBDX_CUDA(c, cudaEventElapsedTime(&ms, c->ev[from[k]], c->ev[from[k] + 1]));
      c->phase_ms[k] += ms;
    }
    ++c->phase_calls;
  }
  return 0;
}

}  // namespace

// The Coulomb tables of the alpha-first sigma (Ctx::d_Db, d_Dr).
int build_coulomb_tables(Ctx* c) {
  c->db_stride = pad8(c->nb);
  const size_t nb_el = c->npair * c->db_stride;
  SBDX_CUDA(c, dev_alloc(c, &c->d_Db, sizeof(double) * nb_el));
  SBDX_CUDA(c, dev_alloc(c, &c->d_Db32, sizeof(float) * nb_el));
  AbPlan& P = c->ab;
  SBDX_CUDA(c, dev_alloc(c, &P.V, sizeof(double) * c->npair * P.vstride));
  SBDX_CUDA(c, dev_alloc(c, &P.V32, sizeof(float) * c->npair * P.vstride32));
  SBDX_CUDA(c, dev_alloc(c, &c->d_Dr, sizeof(double) * c->na * P.vstride));
  SBDX_CUDA(c, dev_alloc(c, &c->d_Dr32, sizeof(float) * c->na * P.vstride32));
  SBDX_CUDA(c, cudaMemsetAsync(c->d_Db, 0, sizeof(double) * nb_el, c->stream));
  SBDX_CUDA(c, cudaMemsetAsync(c->d_Db32, 0, sizeof(float) * nb_el, c->stream));
  const dim3 gb((unsigned)((c->nb + 255) / 256), (unsigned)c->npair);
  coulomb_table_kernel<<<gb, 256, 0, c->stream>>>(c->d_G, c->L, c->d_b, c->nb, c->db_stride, c->d_Db, c->d_Db32);
  SBDX_LAUNCHED(c);
  gather_pairs_kernel<<<(unsigned)c->npair, 256, 0, c->stream>>>(c->d_V, c->vstride, P.pairs, P.npu, P.vstride,
                                                                  P.vstride32, P.V, P.V32);
  SBDX_LAUNCHED(c);
  coulomb_row_sum_kernel<<<(unsigned)c->na, 256, 0, c->stream>>>(P.V, (size_t)P.npu, P.vstride, P.vstride32, c->L, c->d_a,
                                                                 c->d_Dr, c->d_Dr32);
  SBDX_LAUNCHED(c);
  return 0;
}

int ensure_coulomb_a(Ctx* c) {
  if (c->d_Da) return 0;
  c->da_stride = pad8(c->na);
  const size_t na_el = c->npair * c->da_stride;
  SBDX_CUDA(c, dev_alloc(c, &c->d_Da32, sizeof(float) * na_el));
  SBDX_CUDA(c, cudaMemsetAsync(c->d_Da32, 0, sizeof(float) * na_el, c->stream));
  double* Da = nullptr;
  SBDX_CUDA(c, dev_alloc(c, &Da, sizeof(double) * na_el));
  c->d_Da = Da;
  SBDX_CUDA(c, cudaMemsetAsync(c->d_Da, 0, sizeof(double) * na_el, c->stream));
  const dim3 ga((unsigned)((c->na + 255) / 256), (unsigned)c->npair);
  coulomb_table_kernel<<<ga, 256, 0, c->stream>>>(c->d_G, c->L, c->d_a, c->na, c->da_stride, c->d_Da, c->d_Da32);
  SBDX_LAUNCHED(c);
  return 0;
}

int phase_vectors(Ctx* c, const double* W) {
  return launch_split<double>(c, W, 0, c->na, reinterpret_cast<double*>(c->d_xp), reinterpret_cast<double*>(c->d_xt), false, nullptr);
}

int build_g_table(Ctx* c) {
  const size_t n = c->npair * (size_t)c->L;
  dev_free(c, c->d_G);
  dev_free(c, c->d_G32);
  c->d_G = nullptr;
  c->d_G32 = nullptr;
  SBDX_CUDA(c, dev_alloc(c, &c->d_G, sizeof(double) * n));
  SBDX_CUDA(c, dev_alloc(c, &c->d_G32, sizeof(float) * n));
  g_table_kernel<<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(c->d_eri, c->L, c->npair, c->d_G, c->d_G32);
  SBDX_LAUNCHED(c);
  const size_t nv = c->npair * c->npair;
  c->vstride = (c->npair + 1) / 2 * 2;
  c->vstride32 = (c->npair + 3) / 4 * 4;
  dev_free(c, c->d_V);
  dev_free(c, c->d_V32);
  c->d_V = nullptr;
  c->d_V32 = nullptr;
  SBDX_CUDA(c, dev_alloc(c, &c->d_V, sizeof(double) * c->npair * c->vstride));
  SBDX_CUDA(c, dev_alloc(c, &c->d_V32, sizeof(float) * c->npair * c->vstride32));
  SBDX_CUDA(c, cudaMemsetAsync(c->d_V, 0, sizeof(double) * c->npair * c->vstride, c->stream));
  SBDX_CUDA(c, cudaMemsetAsync(c->d_V32, 0, sizeof(float) * c->npair * c->vstride32, c->stream));
  unpack_eri_kernel<<<(unsigned)((nv + 255) / 256), 256, 0, c->stream>>>(c->d_eri, c->npair, c->vstride,
                                                                           c->vstride32, c->d_V, c->d_V32);
  SBDX_LAUNCHED(c);
  return 0;
}

int ensure_sigma_scratch(Ctx* c) {
  c->xsa = pad8(c->nb);
  c->xsb = pad8(c->na);
  size_t n = std::max(c->na * c->xsa, c->nb * c->xsb);  // >= D
  if (!c->fork) {
    for (auto& x : c->side) SBDX_CUDA(c, cudaStreamCreateWithFlags(&x, cudaStreamNonBlocking));
    for (auto& e : c->join) SBDX_CUDA(c, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    SBDX_CUDA(c, cudaEventCreateWithFlags(&c->fork, cudaEventDisableTiming));
  }
  // One request (6 vectors of 72 MB by themselves take 2 ms to allocate), and
  // nothing is cleared: a padding column enters only the products' padding
  // columns, which nobody reads.
  c->lean = c->na * c->nb >= kLeanDets;
  if (c->lean) n = std::max(n, (c->na * c->ab.xs + 1) / 2);  // two vectors hold the lanes
  n = (n + 15) / 16 * 16;
  const size_t want = c->lean ? 4 * n : 5 * n + c->na * c->ab.xs;
  if (!c->d_scratch || c->scratch_size < want) {
    free_sigma_scratch(c);
    SBDX_CUDA(c, dev_alloc(c, &c->d_scratch, sizeof(double) * want));
    c->scratch_size = want;
  }
  c->d_xp = c->d_scratch;
  c->d_xt = c->d_scratch + n;
  c->d_y = c->d_scratch + 2 * n;
  c->d_yt = c->d_scratch + 3 * n;
  c->d_yab = c->lean ? nullptr : c->d_scratch + 4 * n;
  c->d_xk = c->lean ? nullptr : c->d_scratch + 5 * n;
  return 0;
}

void free_sigma_scratch(Ctx* c) {
  clear_sigma_graphs(c);
  dev_free(c, c->d_scratch);
  c->d_scratch = c->d_y = c->d_yt = c->d_yab = nullptr;
  c->d_xt = c->d_xp = c->d_xk = nullptr;
  c->scratch_size = 0;
}

// Autotuner: for each precision, time the candidate kernel variants and launch
// shapes on the current problem (one warm-up and two timed sigmas each, CUDA
// events between the phases, scratch input vectors) and keep the fastest
// same-spin and alpha-beta choice separately.
int autotune(Ctx* c) {
  int rc = 0;
  clear_sigma_graphs(c);
  if (!c->have_conn && (rc = build_connectivity(c))) return rc;
  if (!c->have_hii && (rc = diag_terms(c))) return rc;
  if ((rc = ensure_sigma_scratch(c)) || (rc = ensure_sell(c)) || (rc = ensure_coulomb_a(c))) return rc;
  const size_t D = c->na * c->nb;
  void *X = nullptr, *S = nullptr;
  SBDX_CUDA(c, pool_alloc(c, &X, sizeof(double) * D));
  SBDX_CUDA(c, pool_alloc(c, &S, sizeof(double) * D));
  SBDX_CUDA(c, cudaMemsetAsync(X, 0, sizeof(double) * D, c->stream));
  const bool prof0 = c->profiling;
  if (!c->ev[0])
    for (auto& e : c->ev) SBDX_CUDA(c, cudaEventCreate(&e));
  c->profiling = true;
  // one code per kernel and launch shape: the blocked FP64 kernel has one, and
  // the FP32 one takes at most 4 columns per thread
  const std::vector<int> same_cand[2] = {{34, 24, 28, 22}, {34, 32, 24, 28, 22}};
  const int ab_cand[] = {71, 62, 61, 63, 64};
  for (int prec = 0; prec < 2 && rc == 0; ++prec) {
    const Tune saved = c->tune[prec];
    auto measure = [&](int same, int ab, double* same_ms, double* ab_ms) -> int {
      c->tune[prec].same_code = same;
      c->tune[prec].ab_code = ab;
      int r2 = prec == 0 ? run_sigma<double>(c, (const double*)X, (double*)S)
                         : run_sigma<float>(c, (const float*)X, (float*)S);
      if (r2) return r2;
      for (double& x : c->phase_ms) x = 0.0;
      c->phase_calls = 0;
      for (int k = 0; k < 2 && r2 == 0; ++k)
        r2 = prec == 0 ? run_sigma<double>(c, (const double*)X, (double*)S)
                       : run_sigma<float>(c, (const float*)X, (float*)S);
      *same_ms = c->phase_ms[0] + c->phase_ms[2];
      *ab_ms = c->phase_ms[3];
      return r2;
    };
    int best_same = 0, best_ab = 0;
    double t_same = 1e300, t_ab = 1e300;
    for (int sc : same_cand[prec]) {
      double sm = 0, ab = 0;
      if ((rc = measure(sc, ab_cand[0], &sm, &ab))) break;
      if (sm < t_same) { t_same = sm; best_same = sc; }
    }
    for (int ac : ab_cand) {
      if (rc) break;
      double sm = 0, ab = 0;
      if ((rc = measure(best_same, ac, &sm, &ab))) break;
      if (ab < t_ab) { t_ab = ab; best_ab = ac; }
    }
    if (rc) { c->tune[prec] = saved; break; }
    c->tune[prec].same_code = best_same;
    c->tune[prec].ab_code = best_ab;
  }
  c->profiling = prof0;
  for (double& x : c->phase_ms) x = 0.0;
  c->phase_calls = 0;
  cudaFreeAsync(X, c->stream);
  cudaFreeAsync(S, c->stream);
  pool_trim(c);
  if (rc) return rc;
  SBDX_CUDA(c, cudaStreamSynchronize(c->stream));
  return 0;
}

void clear_sigma_graphs(Ctx* c) {
  for (auto& g : c->graphs) cudaGraphExecDestroy(g.exec);
  c->graphs.clear();
}

namespace {

int run_sigma_any(Ctx* c, int precision, const void* X, void* S) {
  if (precision == 0) return run_sigma<double>(c, (const double*)X, (double*)S);
  return run_sigma<float>(c, (const float*)X, (float*)S);
}

// Replays the captured graph of this (precision, X, S), capturing it first.
// Returns -1 (nothing launched) when capture is not possible here, so that
// the caller runs the sigma directly.
int sigma_graph(Ctx* c, int precision, const void* X, void* S) {
  for (const auto& g : c->graphs)
    if (g.precision == precision && g.X == X && g.S == S) {
      SBDX_CUDA(c, cudaGraphLaunch(g.exec, c->stream));
      c->launches += g.kernels;
      return 0;
    }
  if (c->graphs.size() >= 96) clear_sigma_graphs(c);
  const unsigned long long before = c->launches;
  if (cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  const int rc = run_sigma_any(c, precision, X, S);
  cudaGraph_t graph = nullptr;
  const cudaError_t e = cudaStreamEndCapture(c->stream, &graph);
  const unsigned long long kernels = c->launches - before;
  c->launches = before;
  if (rc != 0 || e != cudaSuccess || graph == nullptr) {
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    return rc != 0 ? rc : -1;
  }
  cudaGraphExec_t exec = nullptr;
  const cudaError_t ei = cudaGraphInstantiate(&exec, graph, 0);
  cudaGraphDestroy(graph);
  if (ei != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  c->graphs.push_back({precision, X, S, exec, kernels});
  SBDX_CUDA(c, cudaGraphLaunch(exec, c->stream));
  c->launches += kernels;
  return 0;
}

}  // namespace

int sigma_rows_device(Ctx* c, int precision, const void* X, void* S, size_t a0, size_t a1) {
  if (a0 > a1 || a1 > c->na) {
    c->err = "sigma_rows: need a0 <= a1 <= na";
    return SBDX_ERR_ARG;
  }
  if (a0 % 8 != 0 && a0 != a1) {
    c->err = "sigma_rows: the first row must be a multiple of 8";
    return SBDX_ERR_ARG;
  }
  if (precision != 0 && precision != 1) {
    c->err = "sigma_rows: precision must be SBDX_FP64 or SBDX_FP32";
    return SBDX_ERR_ARG;
  }
  if (precision == 0 && c->stored.val != nullptr) {
    c->err = "sigma_rows: a row range is evaluated on the fly; release the stored Hamiltonian first";
    return SBDX_ERR_STATE;
  }
  if (!c->have_conn) {
    int rc = build_connectivity(c);
    if (rc) return rc;
  }
  if (!c->have_hii) {
    int rc = diag_terms(c);
    if (rc) return rc;
  }
  int rc = ensure_sigma_scratch(c);
  if (rc) return rc;
  const bool f64 = precision == 0;
  Tune t = effective_tune(c, f64);
  if (!is_v6(t)) t = default_tune(c, f64);  // the row range runs the alpha-first kernels
  if (!c->have_range || c->range_a0 != a0 || c->range_a1 != a1) {
    if ((rc = build_row_range(c, a0, a1))) return rc;
  }
  if (f64) return run_sigma_rows<double>(c, t, static_cast<const double*>(X), static_cast<double*>(S), a0, a1);
  return run_sigma_rows<float>(c, t, static_cast<const float*>(X), static_cast<float*>(S), a0, a1);
}

int sigma_device(Ctx* c, int precision, const void* X, void* S) {
  if (!c->have_conn) {
    int rc = build_connectivity(c);
    if (rc) return rc;
  }
  if (!c->have_hii) {
    int rc = diag_terms(c);
    if (rc) return rc;
  }
  int rc = ensure_sigma_scratch(c);
  if (rc) return rc;
  if (precision != 0 && precision != 1) {
    c->err = "sigma: precision must be SBDX_FP64 or SBDX_FP32";
    return 1;
  }
  if (precision == 0 && c->stored.val != nullptr)
    return stored_sigma(c, static_cast<const double*>(X), static_cast<double*>(S));
  if (effective_tune(c, precision == 0).ab_code != 71 && ((rc = ensure_sell(c)) || (rc = ensure_coulomb_a(c)))) return rc;
  if (c->use_graphs && !c->profiling && c->stream != nullptr) {
    rc = sigma_graph(c, precision, X, S);
    if (rc >= 0) return rc;
    c->use_graphs = false;  // capture unavailable: plain launches from now on
  }
  return run_sigma_any(c, precision, X, S);
}

// ---- the host-buffer sigma, copies overlapped with the kernels ----------------
//
// S = H C from host C to host S in chunks of alpha rows, each one contiguous
// block of both vectors (alpha-major layout). A copy stream brings chunk i in
// while the context stream runs, for every chunk that has arrived, the phase
// split of its rows and the beta same-spin product on its columns of the
// transpose (which read that chunk only). Once every chunk is in, the context
// stream runs the alpha-beta product of all rows (it reads any ket row), then
// per chunk the alpha same-spin work items of its rows and the combine of its
// rows; the copy stream takes each finished chunk out while the next one
// computes. Exposed: the first chunk's copy in, the last chunk's beta same-spin
// product and the last chunk's copy out.

namespace {

// Automatic chunk count: three from kIoMinDets determinants, one more for each
// kIoChunkDets, kIoMaxChunks at most. More chunks expose less of the copies but
// cost launches and the tails of the chunked kernels. Page-locked buffers, us
// with 1, 3, 4, 6 and 8 chunks: 2.25 M determinants 1317, 1245, 1267, 1408,
// 1613; 6.25 M 3430, 3107, 3078, 3044, 3274; 16 M 9598, 8658, 8451, 8382, 8631;
// 64 M (4, 6, 8, 12) 41.4, 40.7, 40.6 and 43 ms.
constexpr size_t kIoMinDets = size_t(2) << 20, kIoChunkDets = size_t(4) << 20;
// Pageable copies block the host, so more chunks only cost there (2.25 M: 2461
// against 2545, 11.6 M: 28.8 against 29.8 ms): one for each 8 M.
constexpr int kIoMinChunks = 3, kIoMaxChunks = 8;

bool page_locked(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost;
}

int io_chunk_count(const Ctx* c, bool locked) {
  if (c->io_chunks_req == 1) return 1;
  const size_t D = c->na * c->nb;
  int k = c->io_chunks_req;
  if (k < 2) {
    const size_t n = locked ? (D < kIoMinDets ? 1 : kIoMinChunks + D / kIoChunkDets)
                            : (D + kIoChunkDets) / (2 * kIoChunkDets);
    k = (int)std::min<size_t>(kIoMaxChunks, n);
  }
  k = std::min<int>(k, (int)(c->na / 8));  // at least 8 rows per chunk
  return std::max(k, 1);
}

// chunk boundaries for K chunks: equal row counts, multiples of 8
std::vector<size_t> io_bounds_for(const Ctx* c, int K) {
  const size_t na = c->na;
  std::vector<size_t> b{0};
  for (int i = 1; i < K; ++i) {
    const size_t x = na * (size_t)i / (size_t)K / 8 * 8;
    if (x > b.back() && x < na) b.push_back(x);
  }
  b.push_back(na);
  return b;
}

void free_chunks(Ctx* c, IoChunks& io) {
  for (auto& r : io.items) free_range_items(c, r);
  for (auto e : io.events)
    if (e) cudaEventDestroy(e);
  io = IoChunks{};
}

int build_io_chunks(Ctx* c, IoChunks& io, const std::vector<size_t>& bounds) {
  free_chunks(c, io);
  const size_t n = bounds.size() - 1;
  io.items.resize(n);
  for (size_t i = 0; i < n; ++i) {
    const int rc = build_range_items(c, bounds[i], bounds[i + 1], io.items[i], true);
    if (rc) return rc;
  }
  if (!c->io_copy) SBDX_CUDA(c, cudaStreamCreateWithFlags(&c->io_copy, cudaStreamNonBlocking));
  io.events.assign(2 * n + 2, nullptr);
  for (auto& e : io.events) SBDX_CUDA(c, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  io.bounds = bounds;  // last: a build that failed part way leaves no bounds, so the next call rebuilds
  return 0;
}

}  // namespace

void free_io_chunks(Ctx* c) {
  for (IoChunks& io : c->io) free_chunks(c, io);
  if (c->io_copy) cudaStreamDestroy(c->io_copy);
  c->io_copy = nullptr;
}

int sigma_host(Ctx* c, const double* hC, double* hS) {
  const size_t na = c->na, nb = c->nb, D = na * nb;
  int rc;
  if (!c->have_conn && (rc = build_connectivity(c))) return rc;
  if (!c->have_hii && (rc = diag_terms(c))) return rc;
  if ((rc = ensure_sigma_scratch(c))) return rc;
  double* din = static_cast<double*>(c->d_io_in);
  double* dout = static_cast<double*>(c->d_io_out);
  const Tune t = effective_tune(c, true);
  const bool locked = page_locked(hC) && page_locked(hS);
  const int K = io_chunk_count(c, locked);
  const bool pipe = K >= 2 && c->stored.val == nullptr && is_v6(t) && t.ab_code == 71 && !c->profiling;
  if (!pipe) {  // one copy in, the sigma, one copy out
    SBDX_CUDA(c, cudaMemcpyAsync(din, hC, sizeof(double) * D, cudaMemcpyHostToDevice, c->stream));
    if ((rc = sigma_device(c, SBDX_FP64, din, dout))) return rc;
    SBDX_CUDA(c, cudaMemcpyAsync(hS, dout, sizeof(double) * D, cudaMemcpyDeviceToHost, c->stream));
    return 0;
  }
  const std::vector<size_t> want = io_bounds_for(c, K);
  IoChunks& io = c->io[locked ? 1 : 0];  // a caller may use both kinds of buffers in turn
  if (want != io.bounds) {
    if ((rc = build_io_chunks(c, io, want))) return rc;
  }
  const std::vector<size_t>& b = io.bounds;
  const size_t n = b.size() - 1;
  cudaEvent_t* ev = io.events.data();  // [0, n): chunk in; [n, 2n): chunk out ready; 2n: start; 2n + 1: end
  const Conn& ca = c->conn[0];
  const Conn& cb = c->conn[1];
  double* xp = static_cast<double*>(c->d_xp);
  double* xpt = static_cast<double*>(c->d_xt);
  // the copies in follow whatever the context stream was doing
  SBDX_CUDA(c, cudaEventRecord(ev[2 * n], c->stream));
  SBDX_CUDA(c, cudaStreamWaitEvent(c->io_copy, ev[2 * n], 0));
  for (size_t i = 0; i < n; ++i) {
    const size_t off = b[i] * nb, len = (b[i + 1] - b[i]) * nb;
    SBDX_CUDA(c, cudaMemcpyAsync(din + off, hC + off, sizeof(double) * len, cudaMemcpyHostToDevice, c->io_copy));
    SBDX_CUDA(c, cudaEventRecord(ev[i], c->io_copy));
  }
  for (size_t i = 0; i < n; ++i) {  // per arrived chunk: phase split, beta same-spin on its columns
    const size_t a0 = b[i], nr = b[i + 1] - b[i];
    SBDX_CUDA(c, cudaStreamWaitEvent(c->stream, ev[i], 0));
    if ((rc = launch_split<double>(c, din, a0, nr, xp, xpt, true, c->d_nonfinite))) return rc;
    if ((rc = run_same_v6<double>(c, t, xpt + a0, nr, c->xsb, cb, 0, nb, cb.val, (const double*)nullptr, 0,
                                  c->d_yt + a0)))
      return rc;
  }
  // the alpha-beta product of all rows in one launch (its work items keep
  // the whole grid busy, longest first), then per chunk the alpha same-spin
  // items of its rows and the combine
  if (!c->lean) {
    rc = run_ab_71<double>(c, din);
  } else {  // the lanes take the room of d_xt and d_y, and the result that of the output
    if ((rc = launch_lanes<double>(c, din, xpt))) return rc;
    rc = run_ab_packed<double>(c, nullptr, xpt, dout, nb, false);
  }
  if (rc) return rc;
  for (size_t i = 0; i < n; ++i) {
    const size_t a0 = b[i], nr = b[i + 1] - b[i];
    const Conn& it = io.items[i];
    Conn ra = ca;
    for (int q = 0; q < 2; ++q) ra.blk[q] = it.blk[q];
    ra.same_item = it.same_item;
    ra.n_same_item = it.n_same_item;
    ra.same_split = it.same_split;
    ra.same_slot = it.same_slot;
    ra.same_done = it.same_done;
    ra.n_same_split = it.n_same_split;
    ra.n_same_part = it.n_same_part;
    ra.same_ypart = it.same_ypart;
    if ((rc = run_same_v6<double>(c, t, xp, nb, c->xsa, ra, a0, nr, ca.val, c->d_Db, c->db_stride, c->d_y)))
      return rc;
    if ((rc = launch_combine<double>(c, din, a0, nr, dout + a0 * nb, true, c->lean, i + 1 == n))) return rc;
    SBDX_CUDA(c, cudaEventRecord(ev[n + i], c->stream));
  }
  for (size_t i = 0; i < n; ++i) {  // each chunk out as soon as it is ready
    const size_t off = b[i] * nb, len = (b[i + 1] - b[i]) * nb;
    SBDX_CUDA(c, cudaStreamWaitEvent(c->io_copy, ev[n + i], 0));
    SBDX_CUDA(c, cudaMemcpyAsync(hS + off, dout + off, sizeof(double) * len, cudaMemcpyDeviceToHost, c->io_copy));
  }
  SBDX_CUDA(c, cudaEventRecord(ev[2 * n + 1], c->io_copy));
  SBDX_CUDA(c, cudaStreamWaitEvent(c->stream, ev[2 * n + 1], 0));  // the call's work ends on the context stream
  return 0;
}

}  // namespace sbdx
