// Lattice sums over wavevectors: the integrand of the self-energy functional
// and the projected CPT Green function (see kernels.cuh for the contracts).
//
// Both kernels factorise one small dense complex matrix per (frequency w,
// wavevector k), A = +-(V(k) G(iw) - 1) with
//   V(k) = V0 + sum_e v_e exp(2 pi i k.R_e) at (r_e, c_e)   (set_V, src_qcm/CPT.cpp:22-64).
// A matrix of dimension N (a template argument, 1..16) belongs to N lanes of a
// warp, lane r holding row r in registers; a warp works on 32 / N matrices at
// once and a CTA on one frequency. V0 G - 1 does not depend on k: the CTA forms
// it once in shared memory, and a lane only adds its own elements' rows,
//   row r += sum_{e: r_e = r} v_e exp(2 pi i k.R_e) G[c_e, :],
// N multiplications per element instead of the N^3 of the whole product (the
// elements couple neighbouring super cells: two or three per boundary site).
// Gaussian elimination with partial pivoting then needs no row exchanges: the
// pivot lane is the largest |re| + |im| among the lanes not used yet (one
// redux.sync over the matrix's lanes) and its row goes round by shuffles.
//
// What bounds it: the FP64 pipe (elimination, divisions, phases) and the
// shuffles (4 per broadcast complex entry, one warp instruction per cycle and
// SM). On a B200, 64 x 4096 matrices of dimension 10: 293 us, and 1537 us with
// one thread per matrix holding V, V G and the factors in local memory; the
// averages of 64 x 1024 matrices of dimension 4: 17 us, and 354 us in 64 CTAs of
// 64 threads.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.hpp"
#include "kernels.cuh"

namespace qed {

namespace {

constexpr int kLatThreads = 128;
constexpr int kLatWarps = kLatThreads / 32;
constexpr int kLatMaxN = 16;

struct LatticeTerms {
  const int *row;    // elements of matrix row r: row[r] .. row[r + 1]
  const int *col;
  const double *R;   // 3 per element
  const double *v;   // complex
  int nkx, nky, nkz;
  double off;        // grid point i sits at (i + off) / nk
};

struct Cplx {
  double x, y;
};

__device__ __forceinline__ Cplx cmul(Cplx a, Cplx b) { return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
__device__ __forceinline__ Cplx shfl(Cplx a, int src) {
  return {__shfl_sync(0xffffffffu, a.x, src), __shfl_sync(0xffffffffu, a.y, src)};
}

// G of one frequency and +-(V0 G - 1) in shared memory, rows padded to N + 1
// entries so that lanes reading different rows hit different banks.
template <int N> struct LatticeTile {
  static constexpr int kLd = N + 1;
  double2 g[N * kLd], w[N * kLd];

  // sign = 1: V0 G - 1, sign = -1: 1 - V0 G; G and V0 column-major
  __device__ void load(const double *__restrict__ G, const double *__restrict__ V0, double sign) {
    for (int t = threadIdx.x; t < N * N; t += blockDim.x)
      g[(t % N) * kLd + t / N] = make_double2(G[2 * t], G[2 * t + 1]);
    __syncthreads();
    for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
      const int r = t % N, b = t / N;
      double sr = (r == b) ? -1.0 : 0.0, si = 0.0;
      for (int c = 0; c < N; ++c) {
        const double xr = V0[2 * (r + N * c)], xi = V0[2 * (r + N * c) + 1];
        const double2 y = g[c * kLd + b];
        sr += xr * y.x - xi * y.y;
        si += xr * y.y + xi * y.x;
      }
      w[r * kLd + b] = make_double2(sign * sr, sign * si);
    }
    __syncthreads();
  }

  // row r of +-(V(k) G - 1)
  __device__ __forceinline__ void row(const LatticeTerms &t, unsigned long long kid, int r, double sign,
                                      Cplx (&a)[N]) const {
    unsigned ix, iy, iz;
    const unsigned nz = (unsigned)t.nkz, ny = (unsigned)t.nky;
    if (kid <= 0xffffffffull) {  // 32-bit divisions unless the grid is larger
      const unsigned k = (unsigned)kid, q = k / nz;
      iz = k - q * nz;
      ix = q / ny;
      iy = q - ix * ny;
    } else {
      const unsigned long long q = kid / nz;
      iz = (unsigned)(kid - q * nz);
      ix = (unsigned)(q / ny);
      iy = (unsigned)(q - (unsigned long long)ix * ny);
    }
    const double kx = (ix + t.off) / t.nkx, ky = (iy + t.off) / t.nky, kz = (iz + t.off) / t.nkz;
#pragma unroll
    for (int b = 0; b < N; ++b) {
      const double2 v = w[r * kLd + b];
      a[b] = {v.x, v.y};
    }
    const int e1 = __ldg(t.row + r + 1);
    for (int e = __ldg(t.row + r); e < e1; ++e) {
      double s, c;
      sincospi(2.0 * (kx * __ldg(t.R + 3 * e) + ky * __ldg(t.R + 3 * e + 1) + kz * __ldg(t.R + 3 * e + 2)), &s, &c);
      const double vr = sign * __ldg(t.v + 2 * e), vi = sign * __ldg(t.v + 2 * e + 1);
      const Cplx p = {vr * c - vi * s, vr * s + vi * c};
      const double2 *gr = g + __ldg(t.col + e) * kLd;
#pragma unroll
      for (int b = 0; b < N; ++b) {
        const double2 y = gr[b];
        a[b].x += p.x * y.x - p.y * y.y;
        a[b].y += p.x * y.y + p.y * y.x;
      }
    }
  }
};

// The pivot lane (within the matrix's lanes `mask`) of one elimination step:
// the largest |re| + |im| among the lanes with `open` set. The key is the high
// word of that double (monotonic for values >= 0) with the lane in the last
// four bits, so pivots equal to 1 part in 2^16 are told apart by lane only.
__device__ __forceinline__ int pivot_lane(unsigned mask, bool open, Cplx v, int r) {
  const unsigned hi = (unsigned)__double2hiint(fabs(v.x) + fabs(v.y));
  return (int)(__reduce_max_sync(mask, open ? (0x80000000u | (hi & ~15u) | (unsigned)r) : 0u) & 15u);
}

// Per frequency (blockIdx.y) and CTA: the sum over its wavevectors of
// log |det(V(k) G - 1)|. per_warp: wavevector batches of one warp.
template <int N>
__global__ void __launch_bounds__(kLatThreads) k_sef_logdet(const double *__restrict__ G,
                                                            const double *__restrict__ V0, LatticeTerms terms,
                                                            unsigned long long nk, int per_warp, double *partials) {
  constexpr int GW = 32 / N;  // matrices per warp
  __shared__ LatticeTile<N> tile;
  __shared__ double red[kLatWarps];
  const int iw = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  tile.load(G + 2 * (size_t)iw * N * N, V0, 1.0);
  const int grp = min(lane / N, GW - 1);  // lanes past the last whole matrix repeat it, without a say in the pivots
  const bool mine = lane < GW * N;
  const int base = grp * N, r = mine ? lane - base : 0;
  const unsigned mask = mine ? ((1u << N) - 1u) << base : (0xffffffffu << (GW * N));
  double sum = 0.0;
  const unsigned long long k0 = ((unsigned long long)blockIdx.x * kLatWarps + warp) * per_warp * GW + grp;
  for (int it = 0; it < per_warp; ++it) {
    const unsigned long long kid = k0 + (unsigned long long)it * GW;
    const bool valid = kid < nk;
    if (!__any_sync(0xffffffffu, valid)) break;
    Cplx a[N];
    tile.row(terms, valid ? kid : 0, r, 1.0, a);
    bool open = true;
    Cplx piv = {1.0, 0.0};
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int p = pivot_lane(mask, open, a[j], r);
      const int src = base + p;
      const Cplx pv = shfl(a[j], src);
      const double d = pv.x * pv.x + pv.y * pv.y;
      const double rd = d > 0.0 ? 1.0 / d : 0.0;  // a zero pivot: log 0 below, nothing eliminated
      if (r == p) {
        piv = pv;
        open = false;
      }
      Cplx l = cmul(a[j], Cplx{pv.x * rd, -pv.y * rd});
      if (!open) l = {0.0, 0.0};
#pragma unroll
      for (int c = j + 1; c < N; ++c) {
        const Cplx q = shfl(a[c], src);
        a[c].x -= l.x * q.x - l.y * q.y;
        a[c].y -= l.x * q.y + l.y * q.x;
      }
    }
    if (valid && mine) sum += log(hypot(piv.x, piv.y));
  }
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
  if (lane == 0) red[warp] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < kLatWarps; ++w) s += red[w];
    partials[(size_t)iw * gridDim.x + blockIdx.x] = s;
  }
}

// Per frequency (blockIdx.y) and CTA: the sum over its wavevectors of
// (1 - V(k) G)^{-1}, by Gauss-Jordan elimination in place. With pivot rows p_j
// left where they are, lane p_j ends with row j of the inverse, its column c
// holding the inverse's column p_c; every matrix slot of the CTA adds into its
// own N x N accumulator in shared memory, and the slots are added in order.
template <int N>
__global__ void __launch_bounds__(kLatThreads) k_cpt_partial(const double *__restrict__ G,
                                                             const double *__restrict__ V0, LatticeTerms terms,
                                                             unsigned long long nk, int per_warp, double *partials) {
  constexpr int GW = 32 / N;
  __shared__ LatticeTile<N> tile;
  __shared__ double2 acc[kLatWarps * GW][N * N];
  const int iw = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double2 *flat = &acc[0][0];
  for (int t = threadIdx.x; t < kLatWarps * GW * N * N; t += blockDim.x) flat[t] = make_double2(0.0, 0.0);
  tile.load(G + 2 * (size_t)iw * N * N, V0 + 2 * (size_t)iw * N * N, -1.0);
  const int grp = min(lane / N, GW - 1);
  const bool mine = lane < GW * N;
  const int base = grp * N, r = mine ? lane - base : 0;
  const unsigned mask = mine ? ((1u << N) - 1u) << base : (0xffffffffu << (GW * N));
  double2 *out = acc[warp * GW + grp];
  const unsigned long long k0 = ((unsigned long long)blockIdx.x * kLatWarps + warp) * per_warp * GW + grp;
  for (int it = 0; it < per_warp; ++it) {
    const unsigned long long kid = k0 + (unsigned long long)it * GW;
    const bool valid = kid < nk;
    if (!__any_sync(0xffffffffu, valid)) break;
    Cplx a[N];
    tile.row(terms, valid ? kid : 0, r, -1.0, a);
    int row = -1;                  // the inverse's row this lane ends with
    unsigned long long perm = 0;   // p_c in bits 4 c ..
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int p = pivot_lane(mask, row < 0, a[j], r);
      const int src = base + p;
      const Cplx pv = shfl(a[j], src);
      const double rd = 1.0 / (pv.x * pv.x + pv.y * pv.y);
      const Cplx inv = {pv.x * rd, -pv.y * rd};
      const bool self = r == p;
      if (self) row = j;
      perm |= (unsigned long long)p << (4 * j);
      const Cplx f = a[j];
#pragma unroll
      for (int c = 0; c < N; ++c) {
        if (c == j) continue;
        const Cplx q = cmul(shfl(a[c], src), inv);
        if (self) {
          a[c] = q;
        } else {
          a[c].x -= f.x * q.x - f.y * q.y;
          a[c].y -= f.x * q.y + f.y * q.x;
        }
      }
      const Cplx fi = cmul(f, inv);
      a[j] = self ? inv : Cplx{-fi.x, -fi.y};
    }
    if (valid && mine) {
#pragma unroll
      for (int c = 0; c < N; ++c) {  // lanes own different rows: no two touch one entry
        double2 &o = out[row * N + (int)((perm >> (4 * c)) & 15u)];
        o.x += a[c].x;
        o.y += a[c].y;
      }
    }
    __syncwarp();  // the rows change hands between lanes at the next wavevector
  }
  __syncthreads();
  double *dst = partials + 2 * ((size_t)iw * gridDim.x + blockIdx.x) * N * N;
  for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
    double sr = 0.0, si = 0.0;
    for (int s = 0; s < kLatWarps * GW; ++s) {
      sr += acc[s][t].x;
      si += acc[s][t].y;
    }
    dst[2 * t] = sr;
    dst[2 * t + 1] = si;
  }
}

// Gproj[w] = G(iw) (sum over the CTAs of the inverses, in order) / nk,
// column-major; the inverses are row-major.
__global__ void k_cpt_reduce(int n, int nblk, double nk, const double *__restrict__ G,
                             const double *__restrict__ partials, double *Gproj) {
  __shared__ double2 s[kLatMaxN * kLatMaxN];
  const int iw = blockIdx.x, nn = n * n;
  for (int t = threadIdx.x; t < nn; t += blockDim.x) {
    double sr = 0.0, si = 0.0;
    for (int q = 0; q < nblk; ++q) {
      const double *p = partials + 2 * ((size_t)iw * nblk + q) * nn;
      sr += p[2 * t];
      si += p[2 * t + 1];
    }
    s[t] = make_double2(sr, si);
  }
  __syncthreads();
  const double *g = G + 2 * (size_t)iw * nn;
  for (int t = threadIdx.x; t < nn; t += blockDim.x) {
    const int a = t % n, b = t / n;
    double xr = 0.0, xi = 0.0;
    for (int c = 0; c < n; ++c) {
      const double gr = g[2 * (a + n * c)], gi = g[2 * (a + n * c) + 1];
      const double2 y = s[c * n + b];
      xr += gr * y.x - gi * y.y;
      xi += gr * y.y + gi * y.x;
    }
    Gproj[2 * ((size_t)iw * nn + t)] = xr / nk;
    Gproj[2 * ((size_t)iw * nn + t) + 1] = xi / nk;
  }
}

// Wavevector batches per warp: as many as leave about eight CTAs per SM over
// all frequencies (forming V0 G costs a CTA about N batches' work), at most 16.
int batches_per_warp(int n, int nw, unsigned long long nk) {
  const unsigned long long per = (unsigned long long)kLatWarps * (32 / n);
  const unsigned long long all = (nk + per - 1) / per * (unsigned long long)std::max(nw, 1);
  return (int)std::min<unsigned long long>(16, std::max<unsigned long long>(1, all / (148 * 8)));
}

using LatticeFn = void (*)(const double *, const double *, LatticeTerms, unsigned long long, int, double *);
const LatticeFn kLogdet[kLatMaxN] = {k_sef_logdet<1>,  k_sef_logdet<2>,  k_sef_logdet<3>,  k_sef_logdet<4>,
                                     k_sef_logdet<5>,  k_sef_logdet<6>,  k_sef_logdet<7>,  k_sef_logdet<8>,
                                     k_sef_logdet<9>,  k_sef_logdet<10>, k_sef_logdet<11>, k_sef_logdet<12>,
                                     k_sef_logdet<13>, k_sef_logdet<14>, k_sef_logdet<15>, k_sef_logdet<16>};
const LatticeFn kCpt[kLatMaxN] = {k_cpt_partial<1>,  k_cpt_partial<2>,  k_cpt_partial<3>,  k_cpt_partial<4>,
                                  k_cpt_partial<5>,  k_cpt_partial<6>,  k_cpt_partial<7>,  k_cpt_partial<8>,
                                  k_cpt_partial<9>,  k_cpt_partial<10>, k_cpt_partial<11>, k_cpt_partial<12>,
                                  k_cpt_partial<13>, k_cpt_partial<14>, k_cpt_partial<15>, k_cpt_partial<16>};

}  // namespace

int lattice_blocks(int n, int nw, long nk) {
  if (n < 1 || n > kLatMaxN) fail(QED_ERR_UNSUPPORTED, "lattice sums: Green function dimension above 16");
  const unsigned long long per =
      (unsigned long long)kLatWarps * (32 / n) * (unsigned long long)batches_per_warp(n, nw, (unsigned long long)nk);
  return (int)(((unsigned long long)nk + per - 1) / per);
}

void launch_sef_logdet(int n, int nw, const double *G, const double *V0, const int *row, const int *col,
                       const double *eR, const double *ev, int nkx, int nky, int nkz, double *partials,
                       cudaStream_t s) {
  const long nk = (long)nkx * nky * nkz;
  const int nblk = lattice_blocks(n, nw, nk);
  if (nw <= 0 || nk <= 0) return;
  if (nw > 65535) fail(QED_ERR_ARGUMENT, "SEF grid integrand: more than 65535 frequencies");
  const LatticeTerms t{row, col, eR, ev, nkx, nky, nkz, 0.0};
  kLogdet[n - 1]<<<dim3(nblk, nw), kLatThreads, 0, s>>>(G, V0, t, (unsigned long long)nk,
                                                         batches_per_warp(n, nw, nk), partials);
  QED_LAUNCH();
}

void launch_cpt_projected(int n, int nw, const double *G, const double *V0, const int *row, const int *col,
                          const double *eR, const double *ev, int nkx, int nky, int nkz, double off,
                          double *partials, double *Gproj, cudaStream_t s) {
  const long nk = (long)nkx * nky * nkz;
  const int nblk = lattice_blocks(n, std::min(nw, 65535), nk);
  if (nw <= 0 || nk <= 0) return;
  const LatticeTerms t{row, col, eR, ev, nkx, nky, nkz, off};
  for (int w0 = 0; w0 < nw; w0 += 65535) {  // the grid's second dimension ends there
    const int m = std::min(nw - w0, 65535);
    const size_t o = 2 * (size_t)w0 * n * n;
    kCpt[n - 1]<<<dim3(nblk, m), kLatThreads, 0, s>>>(G + o, V0 + o, t, (unsigned long long)nk,
                                                       batches_per_warp(n, std::min(nw, 65535), nk),
                                                       partials + o * nblk);
    QED_LAUNCH();
  }
  k_cpt_reduce<<<nw, 256, 0, s>>>(n, nblk, (double)nk, G, partials, Gproj);
  QED_LAUNCH();
}

}  // namespace qed
