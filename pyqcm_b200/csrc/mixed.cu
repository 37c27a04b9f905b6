// Symmetry-adapted (mixed) basis Hamiltonian on the device: see mixed.hpp.
#include "mixed.hpp"

#include <algorithm>
#include <cmath>
#include <mutex>

#include "kernels.cuh"
#include "options.hpp"
#include "qed_b200.h"

namespace qed {

MixedTerms mixed_terms(const Model &m, const std::map<std::string, double> &value) {
  const int n = m.n_orb;
  auto mask = [n](int i) -> uint64_t { return i >= n ? (uint64_t)1 << (i - n + 32) : (uint64_t)1 << i; };
  std::map<std::pair<int, int>, double> off;
  std::map<uint64_t, double> diag;
  for (const auto &kv : value) {
    const Operator &op = *m.term.at(kv.first);
    for (const Element &e : op.elements) {
      const double x = kv.second * e.v;
      if (op.is_interaction) diag[mask(e.r) + mask(e.c)] += x;  // r == c doubles the bit, as the reference does
      else if (e.r == e.c) diag[mask(e.r)] += x;
      else off[{e.r, e.c}] += x;
    }
  }
  MixedTerms t;
  for (const auto &kv : off) {
    if (kv.second == 0.0) continue;
    t.r.push_back(kv.first.first);
    t.c.push_back(kv.first.second);
    t.v.push_back(kv.second);
  }
  for (const auto &kv : diag) {
    if (kv.second == 0.0) continue;
    t.dmask.push_back(kv.first);
    t.dval.push_back(kv.second);
  }
  return t;
}

namespace {

constexpr int kMarkTile = 4096;   // factorized states per block of the mark scan
constexpr int kMarkThreads = 256; // 16 states per thread

__constant__ uint32_t c_mbinom[33][33];  // C(n, k), n, k <= 32

struct OffTerms {
  int n;
  const int *r, *c;
  const double *v;
};

// colex rank of an L-bit string: sum over its set bits p_1 < p_2 < ... of C(p_i, i)
__device__ __forceinline__ uint32_t colex_rank(uint32_t s) {
  uint32_t rank = 0;
  int i = 1;
  while (s) {
    const int p = __ffs(s) - 1;
    rank += c_mbinom[p][i++];
    s &= s - 1;
  }
  return rank;
}

__device__ __forceinline__ uint64_t orb_mask(int i, int n) {
  return i >= n ? (uint64_t)1 << (i - n + 32) : (uint64_t)1 << i;
}

__global__ void k_mixed_mark(SymGroup G, int irrep, const uint32_t *__restrict__ ustr, uint32_t du,
                             const uint32_t *__restrict__ dstr, uint64_t nf, uint8_t *__restrict__ lenf) {
  for (uint64_t f = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; f < nf; f += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t b = (uint64_t)ustr[f % du] | ((uint64_t)dstr[f / du] << 32);
    const RepMap m = sym_representative(G, b, irrep);
    lenf[f] = (m.length > 0 && m.rep == b) ? (uint8_t)m.length : (uint8_t)0;
  }
}

// Per tile of kMarkTile factorized states: how many are basis states.
__global__ void __launch_bounds__(kMarkThreads) k_mixed_tile_count(const uint8_t *__restrict__ lenf, uint64_t nf,
                                                                   uint32_t *__restrict__ tile_count) {
  const uint64_t base = (uint64_t)blockIdx.x * kMarkTile;
  uint32_t c = 0;
  for (int k = threadIdx.x; k < kMarkTile; k += kMarkThreads) {
    const uint64_t f = base + k;
    if (f < nf && lenf[f]) ++c;
  }
  __shared__ uint32_t red[kMarkThreads / 32];
  for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t s = 0;
    for (int w = 0; w < kMarkThreads / 32; ++w) s += red[w];
    tile_count[blockIdx.x] = s;
  }
}

// Writes the basis in factorized order: each thread takes 16 consecutive
// states of the tile, the block scans the per-thread counts.
__global__ void __launch_bounds__(kMarkThreads) k_mixed_scatter(const uint8_t *__restrict__ lenf, uint64_t nf,
                                                                const uint64_t *__restrict__ tile_off,
                                                                const uint32_t *__restrict__ ustr, uint32_t du,
                                                                const uint32_t *__restrict__ dstr,
                                                                int32_t *__restrict__ fmap,
                                                                uint64_t *__restrict__ states,
                                                                uint8_t *__restrict__ len) {
  constexpr int per = kMarkTile / kMarkThreads;
  const uint64_t f0 = (uint64_t)blockIdx.x * kMarkTile + (uint64_t)threadIdx.x * per;
  uint32_t c = 0;
  for (int k = 0; k < per; ++k)
    if (f0 + k < nf && lenf[f0 + k]) ++c;
  __shared__ uint32_t scan[kMarkThreads];
  scan[threadIdx.x] = c;
  __syncthreads();
  for (int o = 1; o < kMarkThreads; o <<= 1) {  // inclusive Hillis-Steele scan
    const uint32_t add = threadIdx.x >= o ? scan[threadIdx.x - o] : 0u;
    __syncthreads();
    scan[threadIdx.x] += add;
    __syncthreads();
  }
  uint64_t idx = tile_off[blockIdx.x] + scan[threadIdx.x] - c;
  for (int k = 0; k < per; ++k) {
    const uint64_t f = f0 + k;
    if (f >= nf) break;
    const uint8_t l = lenf[f];
    if (!l) {
      fmap[f] = -1;
      continue;
    }
    fmap[f] = (int32_t)idx;
    states[idx] = (uint64_t)ustr[f % du] | ((uint64_t)dstr[f / du] << 32);
    len[idx] = l;
    ++idx;
  }
}

// Row J's off-diagonal entries: count (fill == false) or write them.
template <bool fill>
__global__ void k_mixed_rows(SymGroup G, int irrep, OffTerms t, const uint64_t *__restrict__ states,
                             const uint8_t *__restrict__ len, uint64_t D, const int32_t *__restrict__ fmap,
                             uint32_t du, uint32_t *__restrict__ count, const uint64_t *__restrict__ row_ptr,
                             uint32_t *__restrict__ col, double *__restrict__ val) {
  const int n = G.N;
  for (uint64_t J = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; J < D; J += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t b = states[J];
    const double lj = (double)len[J];
    uint32_t k = 0;
    uint64_t out = fill ? row_ptr[J] : 0;
    for (int e = 0; e < t.n; ++e) {
      const uint64_t mc = orb_mask(t.c[e], n), mr = orb_mask(t.r[e], n);
      if (!(b & mc) || (b & mr)) continue;  // Pauli: c_c needs the orbital, c+_r an empty one
      const uint64_t lo = mc < mr ? mc : mr, hi = mc < mr ? mr : mc;
      const int sign = (__popcll(b & (hi - (lo << 1))) & 1) ? -1 : 1;
      const RepMap m = sym_representative(G, b - mc + mr, irrep);
      if (m.length == 0) continue;
      const uint64_t f = (uint64_t)colex_rank((uint32_t)m.rep) + (uint64_t)du * colex_rank((uint32_t)(m.rep >> 32));
      const int32_t K = fmap[f];
      if (K < 0) continue;
      if (fill) {
        col[out] = (uint32_t)K;
        val[out] = (m.phase ? -1.0 : 1.0) * t.v[e] * sign * sqrt(lj / (double)len[K]);
        ++out;
      } else {
        ++k;
      }
    }
    if (!fill) count[J] = k;
  }
}

__global__ void k_mixed_diag(const uint64_t *__restrict__ states, uint64_t D, const uint64_t *__restrict__ dmask,
                             const double *__restrict__ dval, int nd, double *__restrict__ dg) {
  for (uint64_t J = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; J < D; J += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t b = states[J];
    double d = 0.0;
    for (int k = 0; k < nd; ++k)
      if ((b & dmask[k]) == dmask[k]) d += dval[k];
    dg[J] = d;
  }
}

// Where a row's off-diagonal entries come from. CsrRows: the stored matrix
// (each lane takes every eighth stored entry). OtfRows: computed on the fly,
// with no stored matrix (each lane takes every eighth one-body element and
// evaluates it on the row's state exactly as k_mixed_rows does: Pauli test,
// fermion sign, representative of the image, its basis index, phase and
// orbit-length factor), for sectors whose matrix would not fit or when asked.
struct CsrRows {
  const uint64_t *row_ptr;
  const uint32_t *col;
  const double *val;
  __device__ __forceinline__ double lane_sum(uint64_t J, int lane, const double *__restrict__ x) const {
    double s = 0.0;
    const uint64_t a = row_ptr[J], e = row_ptr[J + 1];
    for (uint64_t k = a + lane; k < e; k += 8) s += val[k] * __ldg(x + col[k]);
    return s;
  }
};

struct OtfRows {
  SymGroup G;
  int irrep;
  OffTerms t;
  const uint64_t *states;
  const uint8_t *len;
  const int32_t *fmap;
  uint32_t du;
  __device__ __forceinline__ double lane_sum(uint64_t J, int lane, const double *__restrict__ x) const {
    const int n = G.N;
    const uint64_t b = states[J];
    const double lj = (double)len[J];
    double s = 0.0;
    for (int e = lane; e < t.n; e += 8) {
      const uint64_t mc = orb_mask(t.c[e], n), mr = orb_mask(t.r[e], n);
      if (!(b & mc) || (b & mr)) continue;
      const uint64_t lo = mc < mr ? mc : mr, hi = mc < mr ? mr : mc;
      const int sign = (__popcll(b & (hi - (lo << 1))) & 1) ? -1 : 1;
      const RepMap m = sym_representative(G, b - mc + mr, irrep);
      if (m.length == 0) continue;
      const uint64_t f = (uint64_t)colex_rank((uint32_t)m.rep) + (uint64_t)du * colex_rank((uint32_t)(m.rep >> 32));
      const int32_t K = fmap[f];
      if (K < 0) continue;
      s += (m.phase ? -1.0 : 1.0) * t.v[e] * sign * sqrt(lj / (double)len[K]) * __ldg(x + K);
    }
    return s;
  }
};

// y = H x: eight lanes per row stride over its entries, then a shuffle sum. A
// warp takes four consecutive rows per pass; the loop bound is the warp's first
// row, the same for all its lanes, so every shuffle sees the whole warp.
template <class Rows>
__global__ void k_mixed_spmv(const Rows R, const double *__restrict__ dg, const double *__restrict__ x,
                             double *__restrict__ y, uint64_t D) {
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 7;
  const int group = (threadIdx.x & 31) >> 3;
  for (uint64_t J0 = warp * 4; J0 < D; J0 += n_warps * 4) {
    const uint64_t J = J0 + group;
    double s = 0.0;
    if (J < D) s = R.lane_sum(J, lane, x);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    if (J < D && lane == 0) y[J] = dg[J] * x[J] + s;
  }
}

// One ground-state Lanczos step on the mixed basis: w = H v - beta v_prev with
// the per-block partial sums of <v, w> at partials[block * ld] (the layout the
// factorized path's reductions use), rows as in k_mixed_spmv.
template <class Rows>
__global__ void __launch_bounds__(256) k_mixed_lanczos_w(const Rows R, const double *__restrict__ dg,
                                                         const double *__restrict__ v,
                                                         const double *__restrict__ vprev,
                                                         const double *__restrict__ beta_dev,
                                                         double *__restrict__ w, uint64_t D,
                                                         double *__restrict__ partials, int ld) {
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 7;
  const int group = (threadIdx.x & 31) >> 3;
  const double beta = *beta_dev;
  double acc = 0.0;
  for (uint64_t J0 = warp * 4; J0 < D; J0 += n_warps * 4) {
    const uint64_t J = J0 + group;
    double s = 0.0;
    if (J < D) s = R.lane_sum(J, lane, v);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    if (J < D && lane == 0) {
      const double vj = v[J];
      const double wj = dg[J] * vj + s - beta * vprev[J];
      w[J] = wj;
      acc += vj * wj;
    }
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  __shared__ double red[8];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += red[k];
    partials[(size_t)blockIdx.x * ld] = t;
  }
}

// y = xs H x - sum_k c_k z_k with the reductions of the factorized column pass
// (block partials at partials[block * Reducer::kMaxRed + i]); rows as in
// k_mixed_spmv. *skip != 0: the whole call does nothing.
template <class Rows>
__global__ void __launch_bounds__(256) k_mixed_full(const Rows R, const double *__restrict__ dg,
                                                    const double *__restrict__ x, double xs, double *y, uint64_t D,
                                                    SubList sub, int red_mask, double *partials, const int *skip) {
  if (skip && *skip) return;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 7;
  const int group = (threadIdx.x & 31) >> 3;
  double red[3] = {0.0, 0.0, 0.0};
  for (uint64_t J0 = warp * 4; J0 < D; J0 += n_warps * 4) {
    const uint64_t J = J0 + group;
    double s = 0.0;
    if (J < D) s = R.lane_sum(J, lane, x);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    if (J < D && lane == 0) {
      const double xj = x[J];
      double yj = xs * (dg[J] * xj + s);
      for (int k = 0; k < sub.n; ++k) yj -= (sub.cdev ? sub.cdev[k] : sub.c[k]) * sub.z[k][J];
      y[J] = yj;
      red[0] += xs * xj * yj;
      red[1] += yj * yj;
      red[2] += xs * xs * xj * xj;
    }
  }
  if (!red_mask) return;
  __shared__ double sm[3][8];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double v = red[i];
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sm[i][threadIdx.x >> 5] = v;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += sm[threadIdx.x][k];
    partials[(size_t)blockIdx.x * Reducer::kMaxRed + threadIdx.x] = t;
  }
}

// ---- packed matrix ----------------------------------------------------------
//
// What bounds the CSR product is the 12 bytes per entry (2x7 ladder with both
// mirrors, 2.9e6 states, 98e6 entries: 1.2 GB, 331 us = 3.6 TB/s); the packed
// form moves 4 and gathers better (see the times at launch_packed).

constexpr uint32_t kPadCode = 255;
constexpr int kPackedThreads = 256;

// Amplitude classes of the off-diagonal terms.
struct PackTerms {
  int n, n_up, nlog;    // terms, the up-spin ones first; log2 of the group order
  const int *r, *c;
  const uint8_t *cls;   // class | 128 where the amplitude is negative
};

// Images of every string of one spin under every group element: index of the
// permuted string | phase (units of pi / g, mod 2 g) << 24, at img[e * dim + i].
__global__ void k_sym_images(SymGroup G, const uint32_t *__restrict__ str, uint32_t dim, uint32_t *__restrict__ img) {
  const uint64_t n = (uint64_t)dim * G.g;
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < n; t += (uint64_t)gridDim.x * blockDim.x) {
    const int e = (int)(t / dim);
    int ph = 0;
    const uint32_t b = sym_apply_half(G, e, str[t - (uint64_t)e * dim], ph);
    img[t] = colex_rank(b) | (uint32_t)(ph % (2 * G.g)) << 24;
  }
}

// Hops that the Pauli principle allows from state b (images that vanish in the
// irrep included: their slots stay padded).
__device__ __forceinline__ bool hop_allowed(uint64_t b, uint64_t mc, uint64_t mr) { return (b & mc) && !(b & mr); }

// up[s] and width[s] = the largest up-spin hop count among the 32 rows of slice s,
// and that plus the largest down-spin one (one warp each)
__global__ void __launch_bounds__(256) k_pack_width(int N, PackTerms t, const uint64_t *__restrict__ states,
                                                    uint64_t D, uint64_t nslices, uint8_t *__restrict__ up,
                                                    uint32_t *__restrict__ width) {
  const uint64_t sl = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  if (sl >= nslices) return;
  const uint64_t J = sl * 32 + (threadIdx.x & 31);
  unsigned ku = 0, kd = 0;
  if (J < D) {
    const uint64_t b = states[J];
    for (int e = 0; e < t.n; ++e) {
      const bool has = hop_allowed(b, orb_mask(t.c[e], N), orb_mask(t.r[e], N));
      if (e < t.n_up) ku += has;
      else kd += has;
    }
  }
  ku = __reduce_max_sync(0xffffffffu, ku);
  kd = __reduce_max_sync(0xffffffffu, kd);
  if ((threadIdx.x & 31) == 0) {
    up[sl] = (uint8_t)ku;
    width[sl] = ku + kd;
  }
}

// off[0 .. n] = exclusive sums of width[0 .. n); one CTA of 1024 threads
__global__ void __launch_bounds__(1024) k_scan_widths(const uint32_t *__restrict__ width, uint64_t n,
                                                      uint64_t *__restrict__ off) {
  __shared__ uint64_t warp_sum[32];
  uint64_t carry = 0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (uint64_t base = 0; base < n; base += 1024) {
    const uint64_t i = base + threadIdx.x;
    uint64_t v = i < n ? width[i] : 0;
    const uint64_t own = v;
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    if (lane == 31) warp_sum[w] = v;
    __syncthreads();
    uint64_t before = 0, all = 0;
    for (int q = 0; q < 32; ++q) {
      if (q < w) before += warp_sum[q];
      all += warp_sum[q];
    }
    if (i < n) off[i] = carry + before + v - own;
    carry += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) off[n] = carry;
}

// Row J's entries, the matrix elements of k_mixed_rows. The representative of a
// hopped state comes from the strings' image tables: the smallest factorized
// index over the group (the order of the indices is that of the states), its
// phase, and the stabiliser's order, as sym_representative finds them. A thread
// per row; *nnz counts the entries.
template <bool wide>
__global__ void __launch_bounds__(128) k_pack_rows(SymGroup G, int irrep, PackTerms t,
                                                   const uint32_t *__restrict__ img_up,
                                                   const uint32_t *__restrict__ img_dn, uint32_t du, uint32_t dd,
                                                   const uint64_t *__restrict__ states,
                                                   const uint8_t *__restrict__ len, uint64_t D,
                                                   const int32_t *__restrict__ fmap, const uint64_t *__restrict__ off,
                                                   const uint8_t *__restrict__ up, uint8_t *__restrict__ row_up,
                                                   uint32_t *__restrict__ ent, uint8_t *__restrict__ code,
                                                   unsigned long long *nnz) {
  const uint64_t J = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t sl = J >> 5;
  const int N = G.N, gm = 2 * G.g - 1;  // g is a power of two
  uint32_t found = 0;
  if (sl * 32 < D) {
    const uint64_t s0 = off[sl], s1 = off[sl + 1], su = s0 + up[sl];
    const int lane = threadIdx.x & 31;
    uint64_t k = s0;
    auto pad_to = [&](uint64_t end) {
      for (; k < end; ++k) {
        const uint64_t at = k * 32 + lane;
        ent[at] = wide ? 0u : kPadCode << 24;
        if (wide) code[at] = (uint8_t)kPadCode;
      }
    };
    if (J < D) {
      const uint64_t b = states[J];
      const uint32_t u = colex_rank((uint32_t)b), d = colex_rank((uint32_t)(b >> 32));
      const int lj = __ffs((int)len[J]) - 1;
      for (int e = 0; e < t.n; ++e) {
        if (e == t.n_up) {
          row_up[J] = (uint8_t)(k - s0);
          pad_to(su);
        }
        const uint64_t mc = orb_mask(t.c[e], N), mr = orb_mask(t.r[e], N);
        if (!hop_allowed(b, mc, mr)) continue;
        const uint64_t lo = mc < mr ? mc : mr, hi = mc < mr ? mr : mc;
        int neg = __popcll(b & (hi - (lo << 1))) & 1;
        const uint64_t nb = b - mc + mr;
        const bool down = (mc >> 32) != 0;
        const uint32_t u2 = down ? u : colex_rank((uint32_t)nb), d2 = down ? colex_rank((uint32_t)(nb >> 32)) : d;
        const uint32_t f0 = u2 + du * d2;  // below 2^31
        uint32_t rep = f0;
        int ph = 0, h = 1;
        bool null = false;
        for (int q = 1; q < G.g; ++q) {
          const uint32_t a = __ldg(img_up + (uint64_t)q * du + u2), c = __ldg(img_dn + (uint64_t)q * dd + d2);
          const uint32_t f = (a & 0xffffffu) + du * (c & 0xffffffu);
          const int pq = (int)((a >> 24) + (c >> 24) + 2 * G.phi[q][irrep]) & gm;
          if (f == f0) {
            ++h;
            if (pq != 0 && (2 * G.g) % pq == 0) null = true;
          }
          if (f < rep) {
            rep = f;
            ph = pq;
          }
        }
        if (null) continue;
        const int32_t K = fmap[rep];
        if (K < 0) continue;
        const int lk = __ffs(G.g / h) - 1;
        const uint8_t cls = t.cls[e];
        neg ^= (ph != 0) ^ (cls >> 7);
        const uint32_t cd = (uint32_t)((((cls & 127) * (2 * t.nlog + 1)) + (lj - lk + t.nlog)) * 2 + neg);
        const uint64_t at = k * 32 + lane;
        if (wide) {
          ent[at] = (uint32_t)K;
          code[at] = (uint8_t)cd;
        } else {
          ent[at] = (uint32_t)K | cd << 24;
        }
        ++k;
        ++found;
      }
    }
    pad_to(s1);
  }
  found = __reduce_add_sync(0xffffffffu, found);
  if ((threadIdx.x & 31) == 0 && found) atomicAdd(nnz, (unsigned long long)found);
}

// What a packed product does with a row's sum: the three epilogues of the CSR
// kernels above; out(b, i, t) takes sum i of virtual block b.
struct EpiSpmv {
  static constexpr int kRed = 0;
  const double *dg, *x;
  double *y;
  __device__ bool off() const { return false; }
  __device__ __forceinline__ void row(uint64_t J, double s, double *) const { y[J] = dg[J] * x[J] + s; }
  __device__ __forceinline__ void out(uint64_t, int, double) const {}
};

struct EpiLanczos {
  static constexpr int kRed = 1;
  const double *dg, *v, *vprev, *beta;
  double *w, *partials;
  int ld;
  __device__ bool off() const { return false; }
  __device__ __forceinline__ void row(uint64_t J, double s, double *red) const {
    const double vj = v[J];
    const double wj = dg[J] * vj + s - *beta * vprev[J];
    w[J] = wj;
    red[0] += vj * wj;
  }
  __device__ __forceinline__ void out(uint64_t b, int, double t) const { partials[(size_t)b * ld] = t; }
};

struct EpiFull {
  static constexpr int kRed = 3;
  const double *dg, *x;
  double xs;
  double *y;
  SubList sub;
  int red_mask;
  double *partials;
  const int *skip;
  __device__ bool off() const { return skip && *skip; }
  __device__ __forceinline__ void row(uint64_t J, double s, double *red) const {
    const double xj = x[J];
    double yj = xs * (dg[J] * xj + s);
    for (int k = 0; k < sub.n; ++k) yj -= (sub.cdev ? sub.cdev[k] : sub.c[k]) * sub.z[k][J];
    y[J] = yj;
    red[0] += xs * xj * yj;
    red[1] += yj * yj;
    red[2] += xs * xs * xj * xj;
  }
  __device__ __forceinline__ void out(uint64_t b, int i, double t) const {
    if (red_mask) partials[(size_t)b * Reducer::kMaxRed + i] = t;
  }
};

// Every sum is taken in the order of the CSR kernels (eight lanes per row, 256
// threads per block of 32 rows), so that both give the same bits - the solver's
// recurrences stop at thresholds that last digits can tip (HvOperator::keep_order):
// a row keeps the eight partial sums of its entries k mod 8 (entry j of the down
// part is entry row_up + j of the row) and adds them as the shuffles did; virtual
// block b of `nb` owns the slices b, b + nb, ... and adds its rows as block b did.
// A lane per row; W warps share a virtual block's slice, slots w, w + W, ... of each
// part (between the parts the partial sums change hands in shared memory).
//
// Bound by latency (offsets -> entries -> gathers) where a sector has a slice or
// two per warp, by the gathers where it has many: a warp's first entries of both
// parts are requested together, before the up part's gathers.
template <int W> struct PackedBatch {
  static constexpr int Q = 8 / W;                                  // partial sums of a warp
  static constexpr int R = W == 4 ? 3 : 4;  // rounds of eight slots per batch
};
template <int W, bool wide>
__device__ __forceinline__ void packed_entries(const PackedView &P, uint64_t k, uint64_t s1, int lane,
                                               uint32_t (&e)[PackedBatch<W>::Q * PackedBatch<W>::R],
                                               uint32_t (&c)[PackedBatch<W>::Q * PackedBatch<W>::R]) {
#pragma unroll
  for (int q = 0; q < PackedBatch<W>::Q * PackedBatch<W>::R; ++q) {
    const bool in = k + q * W < s1;
    const uint64_t at = (k + q * W) * 32 + lane;
    e[q] = in ? __ldcs(P.ent + at) : kPadCode << 24;
    c[q] = wide ? (in ? (uint32_t)__ldcs(P.code + at) : kPadCode) : e[q] >> 24;
  }
}
template <int W, bool wide>
__device__ __forceinline__ void packed_apply(const double *__restrict__ x, const double *values,
                                             const uint32_t (&e)[PackedBatch<W>::Q * PackedBatch<W>::R],
                                             const uint32_t (&c)[PackedBatch<W>::Q * PackedBatch<W>::R],
                                             double (&acc)[PackedBatch<W>::Q]) {
  constexpr int Q = PackedBatch<W>::Q, N = Q * PackedBatch<W>::R;
  double xv[N];
#pragma unroll
  for (int q = 0; q < N; ++q) xv[q] = c[q] != kPadCode ? __ldg(x + (wide ? e[q] : e[q] & 0xffffffu)) : 0.0;
#pragma unroll
  for (int q = 0; q < N; ++q) acc[q % Q] = fma(values[c[q]], xv[q], acc[q % Q]);  // values[255] = 0
}
// slots k, k + W, ... of a part, the first batch of entries already there
template <int W, bool wide>
__device__ __forceinline__ void packed_part(const PackedView &P, const double *__restrict__ x, const double *values,
                                            uint64_t k, uint64_t s1, int lane,
                                            uint32_t (&e)[PackedBatch<W>::Q * PackedBatch<W>::R],
                                            uint32_t (&c)[PackedBatch<W>::Q * PackedBatch<W>::R],
                                            double (&acc)[PackedBatch<W>::Q]) {
  constexpr int kStep = 8 * PackedBatch<W>::R;
  packed_apply<W, wide>(x, values, e, c, acc);
  for (k += kStep; k < s1; k += kStep) {
    packed_entries<W, wide>(P, k, s1, lane, e, c);
    packed_apply<W, wide>(x, values, e, c, acc);
  }
}

template <int W, bool wide, class Epi>
__global__ void __launch_bounds__(kPackedThreads) k_packed(const PackedView P, const double *__restrict__ x,
                                                           uint64_t D, uint64_t nslices, uint64_t nb, const Epi epi) {
  pdl_begin();
  if (epi.off()) return;
  constexpr int kWarps = kPackedThreads / 32, kBlocks = kWarps / W, Q = 8 / W;
  __shared__ double values[256];
  __shared__ double part[kBlocks][8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, w = warp % W, own = warp / W;
  values[threadIdx.x] = P.values[threadIdx.x];
  __syncthreads();
  const uint64_t vb = (uint64_t)blockIdx.x * kBlocks + own;
  double red[Epi::kRed > 0 ? Epi::kRed : 1] = {};
  for (uint64_t base = 0; base < nslices; base += nb) {
    const uint64_t sl = base + vb, J = sl * 32 + lane;
    const bool on = vb < nb && sl < nslices;
    uint64_t s0 = 0, su = 0, s1 = 0;
    int first = 0;
    constexpr int kBatch = Q * PackedBatch<W>::R;
    uint32_t eu[kBatch], cu[kBatch], ed[kBatch], cd[kBatch];
    double acc[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) acc[q] = 0.0;
    if (on) {
      s0 = P.off[sl];
      s1 = P.off[sl + 1];
      su = s0 + P.up[sl];
      first = J < D ? P.row_up[J] : 0;
      packed_entries<W, wide>(P, s0 + w, su, lane, eu, cu);
      packed_entries<W, wide>(P, su + w, s1, lane, ed, cd);
      packed_part<W, wide>(P, x, values, s0 + w, su, lane, eu, cu, acc);
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) part[own][w + q * W][lane] = acc[q];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) acc[q] = part[own][(first + w + q * W) & 7][lane];
    if (on) packed_part<W, wide>(P, x, values, su + w, s1, lane, ed, cd, acc);
#pragma unroll
    for (int q = 0; q < Q; ++q) part[own][(first + w + q * W) & 7][lane] = acc[q];
    __syncthreads();
    if (w == 0 && on && J < D) {
      double p[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) p[q] = part[own][q][lane];
      epi.row(J, ((p[0] + p[4]) + (p[2] + p[6])) + ((p[1] + p[5]) + (p[3] + p[7])), red);
    }
    __syncthreads();  // part is read before the next slice
  }
  if (Epi::kRed > 0 && w == 0 && vb < nb) {
#pragma unroll
    for (int i = 0; i < Epi::kRed; ++i) {
      double v = red[i];  // rows 4 k .. 4 k + 3 were one warp of block vb
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      double t = 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k) t += __shfl_sync(0xffffffffu, v, 4 * k);
      if (lane == 0) epi.out(vb, i, t);
    }
  }
}

// y = H x for callers outside the recurrences: the same entries, summed as they
// come by one lane per row, W warps per slice. Half the time of the ordered form on
// large sectors (no exchange between the parts, one accumulator, six entries in
// flight whatever the part).
template <int W, bool wide>
__global__ void __launch_bounds__(kPackedThreads) k_packed_free(const PackedView P, const double *__restrict__ x,
                                                                uint64_t D, uint64_t nslices,
                                                                const double *__restrict__ dg, double *y) {
  constexpr int kWarps = kPackedThreads / 32, kPer = kWarps / W, kDeep = 6;
  __shared__ double values[256];
  __shared__ double part[W > 1 ? kWarps : 1][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  values[threadIdx.x] = P.values[threadIdx.x];
  __syncthreads();
  for (uint64_t base = (uint64_t)blockIdx.x * kPer; base < nslices; base += (uint64_t)gridDim.x * kPer) {
    const uint64_t sl = base + warp / W;
    double acc = 0.0;
    if (sl < nslices) {
      const uint64_t s1 = P.off[sl + 1];
      for (uint64_t k = P.off[sl] + warp % W; k < s1; k += (uint64_t)W * kDeep) {
        uint32_t e[kDeep], c[kDeep];
#pragma unroll
        for (int q = 0; q < kDeep; ++q) {
          const bool in = k + q * W < s1;
          const uint64_t at = (k + q * W) * 32 + lane;
          e[q] = in ? __ldcs(P.ent + at) : kPadCode << 24;
          c[q] = wide ? (in ? (uint32_t)__ldcs(P.code + at) : kPadCode) : e[q] >> 24;
        }
        double xv[kDeep];
#pragma unroll
        for (int q = 0; q < kDeep; ++q) xv[q] = c[q] != kPadCode ? __ldg(x + (wide ? e[q] : e[q] & 0xffffffu)) : 0.0;
#pragma unroll
        for (int q = 0; q < kDeep; ++q) acc += values[c[q]] * xv[q];
      }
    }
    if (W > 1) {
      part[warp][lane] = acc;
      __syncthreads();
      if (warp % W == 0)
        for (int q = 1; q < W; ++q) acc += part[warp + q][lane];
    }
    const uint64_t J = sl * 32 + lane;
    if (warp % W == 0 && J < D) y[J] = dg[J] * x[J] + acc;
    if (W > 1) __syncthreads();  // part is read before the next slices
  }
}

struct OrbCoef {
  double c[kMaxSymOrb];
};

// basis index of state b in a sector: through the colex ranks of its two words
__device__ __forceinline__ int32_t mixed_index(const int32_t *fmap, uint32_t du, uint64_t b) {
  return fmap[(uint64_t)colex_rank((uint32_t)b) + (uint64_t)du * colex_rank((uint32_t)(b >> 32))];
}

// phi[J] = (c+ psi)[J]: the target state J carries the created particle; each
// occupied orbital a of the orbital's support, emptied, gives a source state
// whose representative (in the source irrep) holds the amplitude.
__global__ void k_mixed_create(SymGroup G, int r_src, int r_tgt, int spin, int n_sites, OrbCoef cf,
                               const uint64_t *__restrict__ tstates, const uint8_t *__restrict__ tlen, uint64_t Dt,
                               const int32_t *__restrict__ sfmap, uint32_t sdu, const uint8_t *__restrict__ slen,
                               const double *__restrict__ psi, double *__restrict__ phi) {
  const int N = G.N;
  for (uint64_t J = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; J < Dt; J += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t b = tstates[J];
    const double lj = (double)tlen[J];
    double acc = 0.0;
    for (int a = 0; a < n_sites; ++a) {
      if (cf.c[a] == 0.0) continue;
      const uint64_t m = orb_mask(a + spin * N, N);
      if (!(b & m)) continue;
      const RepMap rm = sym_representative(G, b ^ m, r_src);
      if (rm.length == 0) continue;
      const int32_t I = mixed_index(sfmap, sdu, rm.rep);
      if (I < 0) continue;
      int ph = rm.phase + ((__popcll(b & (m - 1)) & 1) ? G.g : 0);
      ph %= 2 * G.g;
      acc += (ph == 0 ? 1.0 : -1.0) * cf.c[a] * sqrt(lj / (double)rm.length) * psi[I];
    }
    phi[J] = acc;
  }
}

// phi[J] = (c psi)[J]: every source state b' whose orbital a, emptied, lands in
// J's orbit is b' = h(J) + a for a group element h (each distinct image h(J)
// once) and an orbital a that h(J) leaves empty; b' contributes when it is its
// own representative in the source irrep.
__global__ void k_mixed_destroy(SymGroup G, int r_src, int r_tgt, int spin, int n_sites, OrbCoef cf,
                                const uint64_t *__restrict__ tstates, uint64_t Dt, const int32_t *__restrict__ sfmap,
                                uint32_t sdu, const uint8_t *__restrict__ slen, const double *__restrict__ psi,
                                double *__restrict__ phi) {
  const int N = G.N;
  for (uint64_t J = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; J < Dt; J += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t bj = tstates[J];
    uint64_t seen[kMaxGroup];
    int nseen = 0;
    double acc = 0.0;
    for (int h = 0; h < G.g; ++h) {
      int q;
      const uint64_t sh = sym_apply(G, h, 0, bj, q);
      bool dup = false;
      for (int k = 0; k < nseen; ++k) dup |= seen[k] == sh;
      if (dup) continue;
      seen[nseen++] = sh;
      for (int a = 0; a < n_sites; ++a) {
        if (cf.c[a] == 0.0) continue;
        const uint64_t m = orb_mask(a + spin * N, N);
        if (sh & m) continue;
        const uint64_t bs = sh | m;  // the source state
        const RepMap rs = sym_representative(G, bs, r_src);
        if (rs.length == 0 || rs.rep != bs) continue;
        const int32_t I = mixed_index(sfmap, sdu, bs);
        if (I < 0) continue;
        const RepMap rt = sym_representative(G, sh, r_tgt);  // rep bj; its phase and length
        if (rt.length == 0) continue;
        int ph = rt.phase + ((__popcll(bs & (m - 1)) & 1) ? G.g : 0);
        ph %= 2 * G.g;
        acc += (ph == 0 ? 1.0 : -1.0) * cf.c[a] * sqrt((double)slen[I] / (double)rt.length) * psi[I];
      }
    }
    phi[J] = acc;
  }
}

unsigned grid_for(uint64_t n, int threads) {
  static const int sms = [] {
    int dev = 0, v = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  }();
  const uint64_t want = (n + threads - 1) / threads;
  const uint64_t cap = (uint64_t)sms * 16;
  return (unsigned)(want < 1 ? 1 : (want > cap ? cap : want));
}

void upload_binomials() {
  static std::once_flag once;
  std::call_once(once, [] {
    uint32_t h[33][33] = {};
    for (int n = 0; n <= 32; ++n)
      for (int k = 0; k <= n; ++k) h[n][k] = (uint32_t)binom(n, k);
    QED_CUDA(cudaMemcpyToSymbol(c_mbinom, h, sizeof(h)));
    QED_CUDA(cudaDeviceSynchronize());
  });
}

}  // namespace

MixedHamiltonian::MixedHamiltonian(const SymmetryGroup &G, const MixedTerms &t, int irrep, int n_up, int n_dn,
                                   cudaStream_t s) {
  const int N = G.tab.N;
  if (irrep < 0 || irrep >= G.g()) fail(QED_ERR_ARGUMENT, "irrep out of range");
  if (n_up < 0 || n_dn < 0 || n_up > N || n_dn > N) fail(QED_ERR_ARGUMENT, "bad sector for the mixed basis");
  upload_binomials();
  const uint64_t du = binom(N, n_up), dd = binom(N, n_dn), nf = du * dd;
  if (du > 0xffffffffull || dd > 0xffffffffull || nf > 0x7fffffffull)
    fail(QED_ERR_UNSUPPORTED, "sector too large for the mixed-basis index map");
  this->irrep = irrep;
  this->n_up = n_up;
  this->n_dn = n_dn;
  this->du = (uint32_t)du;
  this->dd = (uint32_t)dd;
  group = G.tab;
  DevBuf<uint32_t> us(du), ds(dd);
  launch_unrank(N, n_up, (uint32_t)du, us.p, s);
  launch_unrank(N, n_dn, (uint32_t)dd, ds.p, s);
  DevBuf<uint8_t> lenf(nf);
  k_mixed_mark<<<grid_for(nf, 256), 256, 0, s>>>(G.tab, irrep, us.p, (uint32_t)du, ds.p, nf, lenf.p);
  QED_LAUNCH();
  const uint64_t ntiles = (nf + kMarkTile - 1) / kMarkTile;
  DevBuf<uint32_t> tcount(ntiles);
  k_mixed_tile_count<<<(unsigned)ntiles, kMarkThreads, 0, s>>>(lenf.p, nf, tcount.p);
  QED_LAUNCH();
  std::vector<uint32_t> htc(ntiles);
  tcount.download(htc.data(), ntiles, s);
  QED_CUDA(cudaStreamSynchronize(s));
  std::vector<uint64_t> toff(ntiles);
  uint64_t total = 0;
  for (uint64_t k = 0; k < ntiles; ++k) {
    toff[k] = total;
    total += htc[k];
  }
  D = total;
  DevBuf<uint64_t> dtoff;
  dtoff.upload(toff, s);
  states.alloc(D);
  len.alloc(D);
  fmap.alloc(nf);
  k_mixed_scatter<<<(unsigned)ntiles, kMarkThreads, 0, s>>>(lenf.p, nf, dtoff.p, us.p, (uint32_t)du, ds.p, fmap.p,
                                                            states.p, len.p);
  QED_LAUNCH();
  dg.alloc(D);
  if (D == 0) {
    row_ptr.alloc(1);
    const uint64_t zero = 0;
    row_ptr.upload(&zero, 1, s);
    QED_CUDA(cudaStreamSynchronize(s));
    return;
  }
  term_r.upload(t.r, s);
  term_c.upload(t.c, s);
  term_v.upload(t.v, s);
  n_terms = (int)t.r.size();
  const OffTerms ot{n_terms, term_r.p, term_c.p, term_v.p};
  DevBuf<uint64_t> dm;
  DevBuf<double> dv;
  dm.upload(t.dmask, s);
  dv.upload(t.dval, s);
  k_mixed_diag<<<grid_for(D, 256), 256, 0, s>>>(states.p, D, dm.p, dv.p, (int)t.dmask.size(), dg.p);
  QED_LAUNCH();
  if (pack(t, us.p, ds.p, s)) return;
  DevBuf<uint32_t> cnt(D);
  k_mixed_rows<false><<<grid_for(D, 128), 128, 0, s>>>(G.tab, irrep, ot, states.p, len.p, D, fmap.p, (uint32_t)du,
                                                       cnt.p, nullptr, nullptr, nullptr);
  QED_LAUNCH();
  std::vector<uint32_t> hc(D);
  cnt.download(hc.data(), D, s);
  QED_CUDA(cudaStreamSynchronize(s));
  std::vector<uint64_t> rp(D + 1);
  rp[0] = 0;
  for (size_t J = 0; J < D; ++J) rp[J + 1] = rp[J] + hc[J];
  nnz = rp[D];
  // the stored matrix (12 bytes per entry + the row pointers) or, above the
  // size budget or when asked, entries recomputed at every product; sectors
  // that may be diagonalised in full keep the stored form
  const double csr_bytes = 12.0 * (double)nnz + 8.0 * (double)(D + 1);
  on_the_fly = (long)D >= opt_int("max_dim_full") &&
               (opt_bool("mixed_on_the_fly") || csr_bytes > opt_double("mixed_csr_max_gb") * 1e9);
  if (!on_the_fly) {
    row_ptr.upload(rp, s);
    col.alloc(nnz);
    val.alloc(nnz);
    if (nnz)
      k_mixed_rows<true><<<grid_for(D, 128), 128, 0, s>>>(G.tab, irrep, ot, states.p, len.p, D, fmap.p,
                                                          (uint32_t)du, nullptr, row_ptr.p, col.p, val.p);
    QED_LAUNCH();
  }
  QED_CUDA(cudaStreamSynchronize(s));
}

// Builds the packed form where it applies (see mixed.hpp); false: nothing done.
bool MixedHamiltonian::pack(const MixedTerms &t, const uint32_t *ustr, const uint32_t *dstr, cudaStream_t s) {
  const int g = group.g, N = group.N;
  if ((long)D < opt_int("max_dim_full") || opt_bool("mixed_on_the_fly") || (opt_int("mixed_variant") & 1)) return false;
  if ((g & (g - 1)) || du >= (1u << 24) || dd >= (1u << 24) || t.r.empty()) return false;
  int nlog = 0;
  while ((1 << nlog) < g) ++nlog;
  std::vector<double> amp;  // classes of equal |amplitude|
  std::vector<uint8_t> cls;
  for (size_t e = 0; e < t.r.size(); ++e) {
    const double a = std::fabs(t.v[e]);
    const size_t k = std::find(amp.begin(), amp.end(), a) - amp.begin();
    if (k == amp.size()) amp.push_back(a);
    if (k >= 127) return false;
    cls.push_back((uint8_t)(k | (t.v[e] < 0.0 ? 128 : 0)));
  }
  // up-spin hops, then down-spin ones, none between the spins: the order of t
  int n_up = 0;
  while (n_up < n_terms && t.r[n_up] < N) ++n_up;
  for (int e = 0; e < n_terms; ++e)
    if ((t.r[e] < N) != (e < n_up) || (t.c[e] < N) != (e < n_up)) return false;
  if (n_up == 0 || n_up == n_terms || n_up > 255) return false;
  const int nr = 2 * nlog + 1;
  if (amp.size() * nr * 2 > kPadCode) return false;
  std::vector<double> hv(256, 0.0);
  for (size_t k = 0; k < amp.size(); ++k)
    for (int q = 0; q < nr; ++q) {  // sqrt(len_J / len_K) = sqrt(2^(q - nlog))
      const double v = amp[k] * std::sqrt(std::ldexp(1.0, q - nlog));
      hv[(k * nr + q) * 2] = v;
      hv[(k * nr + q) * 2 + 1] = -v;
    }
  DevBuf<uint8_t> dcls;
  dcls.upload(cls, s);
  values.upload(hv, s);
  const PackTerms pt{n_terms, n_up, nlog, term_r.p, term_c.p, dcls.p};
  const uint64_t nslices = (D + 31) / 32;
  DevBuf<uint32_t> width(nslices);
  slice_off.alloc(nslices + 1);
  slice_up.alloc(nslices);
  k_pack_width<<<(unsigned)((nslices * 32 + 255) / 256), 256, 0, s>>>(N, pt, states.p, D, nslices, slice_up.p, width.p);
  QED_LAUNCH();
  k_scan_widths<<<1, 1024, 0, s>>>(width.p, nslices, slice_off.p);
  QED_LAUNCH();
  uint64_t slots = 0;
  QED_CUDA(cudaMemcpyAsync(&slots, slice_off.p + nslices, sizeof(slots), cudaMemcpyDeviceToHost, s));
  QED_CUDA(cudaStreamSynchronize(s));
  const bool wide = D > (1u << 24) || (opt_int("mixed_variant") & 2);
  if ((wide ? 5.0 : 4.0) * 32.0 * (double)slots > opt_double("mixed_csr_max_gb") * 1e9) {
    slice_off.release();
    slice_up.release();
    values.release();
    return false;
  }
  DevBuf<uint32_t> iu((size_t)g * du), id((size_t)g * dd);
  k_sym_images<<<grid_for((uint64_t)g * du, 256), 256, 0, s>>>(group, ustr, du, iu.p);
  QED_LAUNCH();
  k_sym_images<<<grid_for((uint64_t)g * dd, 256), 256, 0, s>>>(group, dstr, dd, id.p);
  QED_LAUNCH();
  row_up.alloc(D);
  ent.alloc(32 * slots);
  if (wide) code.alloc(32 * slots);
  DevBuf<unsigned long long> dn(1);
  QED_CUDA(cudaMemsetAsync(dn.p, 0, dn.bytes(), s));
  auto rows = wide ? k_pack_rows<true> : k_pack_rows<false>;
  rows<<<(unsigned)((D + 127) / 128), 128, 0, s>>>(group, irrep, pt, iu.p, id.p, du, dd, states.p, len.p, D, fmap.p,
                                                   slice_off.p, slice_up.p, row_up.p, ent.p, code.p, dn.p);
  QED_LAUNCH();
  unsigned long long n = 0;
  dn.download(&n, 1, s);
  QED_CUDA(cudaStreamSynchronize(s));
  nnz = n;
  packed = true;
  return true;
}

namespace {
CsrRows csr_rows(const MixedHamiltonian &H) { return CsrRows{H.row_ptr.p, H.col.p, H.val.p}; }
OtfRows otf_rows(const MixedHamiltonian &H) {
  return OtfRows{H.group, H.irrep, OffTerms{H.n_terms, H.term_r.p, H.term_c.p, H.term_v.p}, H.states.p, H.len.p,
                 H.fmap.p, H.du};
}

// nb virtual blocks (those of the CSR kernels where there are sums to keep in
// order), W warps each: enough that the launch has about 32 warps per SM.
template <int W, class Epi>
void launch_packed_w(const MixedHamiltonian &H, const double *x, const Epi &epi, unsigned nb, cudaStream_t s) {
  const uint64_t nslices = (H.D + 31) / 32;
  const unsigned per = kPackedThreads / 32 / W, grid = (nb + per - 1) / per;
  if (H.code.p)
    launch_pdl(H.D, k_packed<W, true, Epi>, grid, kPackedThreads, 0, s, H.packed_view(), x, H.D, nslices, nb, epi);
  else
    launch_pdl(H.D, k_packed<W, false, Epi>, grid, kPackedThreads, 0, s, H.packed_view(), x, H.D, nslices, nb, epi);
  QED_LAUNCH();
}
template <class Epi>
int launch_packed(const MixedHamiltonian &H, const double *x, const Epi &epi, unsigned nb, cudaStream_t s) {
  if (nb >= 148 * 3) launch_packed_w<4>(H, x, epi, nb, s);
  else launch_packed_w<8>(H, x, epi, nb, s);
  return (int)nb;
}

template <int W> void launch_packed_free_w(const MixedHamiltonian &H, const double *x, double *y, cudaStream_t s) {
  const uint64_t nslices = (H.D + 31) / 32, per = kPackedThreads / 32 / W;
  const unsigned grid = (unsigned)std::min<uint64_t>((nslices + per - 1) / per, 148 * 16);
  if (H.code.p)
    k_packed_free<W, true><<<grid, kPackedThreads, 0, s>>>(H.packed_view(), x, H.D, nslices, H.dg.p, y);
  else
    k_packed_free<W, false><<<grid, kPackedThreads, 0, s>>>(H.packed_view(), x, H.D, nslices, H.dg.p, y);
  QED_LAUNCH();
}
// Warps per slice: about 24 slices per SM fill it with one warp each.
void launch_packed_free(const MixedHamiltonian &H, const double *x, double *y, cudaStream_t s) {
  const uint64_t nslices = (H.D + 31) / 32;
  if (nslices >= 148 * 24) launch_packed_free_w<1>(H, x, y, s);
  else if (nslices >= 148 * 16) launch_packed_free_w<2>(H, x, y, s);
  else if (nslices >= 148 * 3) launch_packed_free_w<4>(H, x, y, s);
  else launch_packed_free_w<8>(H, x, y, s);
}
}  // namespace

int MixedHamiltonian::lanczos_w(const double *v, const double *vprev, const double *beta_dev, double *w,
                                double *partials, int ld, int max_blocks, cudaStream_t s) const {
  unsigned nb = grid_for(D * 8, 256);
  if (nb > (unsigned)max_blocks) nb = (unsigned)max_blocks;
  if (packed) return launch_packed(*this, v, EpiLanczos{dg.p, v, vprev, beta_dev, w, partials, ld}, nb, s);
  if (on_the_fly)
    k_mixed_lanczos_w<<<nb, 256, 0, s>>>(otf_rows(*this), dg.p, v, vprev, beta_dev, w, D, partials, ld);
  else
    k_mixed_lanczos_w<<<nb, 256, 0, s>>>(csr_rows(*this), dg.p, v, vprev, beta_dev, w, D, partials, ld);
  QED_LAUNCH();
  return (int)nb;
}

void MixedHamiltonian::apply(const double *x, double *y, cudaStream_t s) const {
  if (D && packed)
    launch_packed_free(*this, x, y, s);
  else
    apply_ordered(x, y, s);
}

void MixedHamiltonian::apply_ordered(const double *x, double *y, cudaStream_t s) const {
  if (!D) return;
  if (packed) {
    launch_packed(*this, x, EpiSpmv{dg.p, x, y}, (unsigned)std::min<uint64_t>((D + 31) / 32, 148 * 256), s);
    return;
  }
  if (on_the_fly)
    k_mixed_spmv<<<grid_for(D * 8, 256), 256, 0, s>>>(otf_rows(*this), dg.p, x, y, D);
  else
    k_mixed_spmv<<<grid_for(D * 8, 256), 256, 0, s>>>(csr_rows(*this), dg.p, x, y, D);
  QED_LAUNCH();
}

int MixedHamiltonian::apply_full(const double *x, double xs, double *y, const SubList &sub, int red_mask,
                                 Reducer &r, cudaStream_t s, const int *skip) const {
  if (!D) return 0;
  unsigned nb = grid_for(D * 8, 256);
  if (red_mask && nb > (unsigned)r.max_blocks) nb = (unsigned)r.max_blocks;
  if (packed) return launch_packed(*this, x, EpiFull{dg.p, x, xs, y, sub, red_mask, r.partials, skip}, nb, s);
  if (on_the_fly)
    k_mixed_full<<<nb, 256, 0, s>>>(otf_rows(*this), dg.p, x, xs, y, D, sub, red_mask, r.partials, skip);
  else
    k_mixed_full<<<nb, 256, 0, s>>>(csr_rows(*this), dg.p, x, xs, y, D, sub, red_mask, r.partials, skip);
  QED_LAUNCH();
  return (int)nb;
}

std::vector<double> MixedHamiltonian::dense(cudaStream_t s) const {
  if (on_the_fly || packed) fail(QED_ERR_INTERNAL, "dense form of a mixed Hamiltonian without CSR");
  std::vector<uint64_t> rp(D + 1);
  std::vector<uint32_t> c(nnz);
  std::vector<double> v(nnz), d(D), out(D * D, 0.0);
  row_ptr.download(rp.data(), D + 1, s);
  if (nnz) {
    col.download(c.data(), nnz, s);
    val.download(v.data(), nnz, s);
  }
  dg.download(d.data(), D, s);
  QED_CUDA(cudaStreamSynchronize(s));
  for (size_t J = 0; J < D; ++J) {
    out[J + D * J] += d[J];
    for (uint64_t k = rp[J]; k < rp[J + 1]; ++k) out[J + D * c[k]] += v[k];
  }
  return out;
}

void mixed_cdag(const MixedHamiltonian &src, const MixedHamiltonian &tgt, int pm, int spin, int n_sites,
                const double *coef, const double *psi, double *phi, cudaStream_t s) {
  if (!tgt.D) return;
  if (n_sites > kMaxSymOrb) fail(QED_ERR_UNSUPPORTED, "more than 32 sites");
  OrbCoef cf{};
  for (int a = 0; a < n_sites; ++a) cf.c[a] = coef[a];
  if (pm == 1)
    k_mixed_create<<<grid_for(tgt.D, 128), 128, 0, s>>>(src.group, src.irrep, tgt.irrep, spin, n_sites, cf,
                                                        tgt.states.p, tgt.len.p, tgt.D, src.fmap.p, src.du, src.len.p,
                                                        psi, phi);
  else
    k_mixed_destroy<<<grid_for(tgt.D, 128), 128, 0, s>>>(src.group, src.irrep, tgt.irrep, spin, n_sites, cf,
                                                         tgt.states.p, tgt.D, src.fmap.p, src.du, src.len.p, psi,
                                                         phi);
  QED_LAUNCH();
}

}  // namespace qed
