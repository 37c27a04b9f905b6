// Lattice sums over wavevectors: the integrand of the self-energy functional
// and the projected CPT Green function (see kernels.cuh for the contracts).
//
// Both kernels factorise one small dense complex matrix per (frequency w,
// wavevector k), A = +-(V(k) G(iw) - 1) with
//   V(k) = V0 + sum_e v_e exp(2 pi i k.R_e) at (r_e, c_e)   (set_V, src_qcm/CPT.cpp:22-64).
// A matrix of dimension N (a template argument, 1..16) belongs to N lanes of a
// warp, lane r holding row r in registers; a warp works on 32 / N matrices at
// once and a CTA on one frequency. V0 G does not depend on k: the CTA forms
// it once in shared memory, and a lane only adds its own elements' rows,
//   row r += sum_{e: r_e = r} v_e exp(2 pi i k.R_e) G[c_e, :],
// N multiplications per element instead of the N^3 of the whole product (the
// elements couple neighbouring super cells: two or three per boundary site). Many
// elements in a row (long-range hops) are summed per entry of V(k) beforehand, once
// for all frequencies (STORED; the rule and both sides stand at stored_entries). The 1 is
// subtracted last, per wavevector: V0 G is small against it, and the rounding of
// V0 G - 1, formed once, would be the same for all wavevectors and stay in their mean
// (30 cases of dimension 2 to 12 against 80-bit values: 1.5e-15 so, 4.5e-16 now, 1.2e-15
// with V(k) G - 1 formed per wavevector; 221 us a kernel so, 234 now).
// Gaussian elimination with partial pivoting then needs no row exchanges: the
// pivot lane is the largest |re| + |im| among the lanes not used yet (a
// maximum passed round the matrix's lanes) and its row goes round by shuffles.
//
// What bounds it: the shuffles (4 per broadcast complex entry; the pipe they
// share with shared memory is busy 53 % of the time) and the latency of the
// elimination's serial chain (22 warps per SM, two instructions per cycle).
// On a B200, 64 x 4096 matrices of dimension 10: 234 us, and 1537 us with one
// thread per matrix holding V, V G and the factors in local memory; the averages
// of 64 x 1024 matrices of dimension 4: 19 us, and 354 us in 64 CTAs of 64
// threads. On the way: a sincospi per element and wavevector, divisions and a
// redux.sync per elimination step 293 us; the phase table and fewer registers
// 272 us; Newton-Raphson reciprocals and fused multiply-adds 254 us; the pivot
// search by shuffles 216 to 221 us; the 1 per wavevector 234 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.hpp"
#include "kernels.cuh"
#include "reciprocal.cuh"

namespace qed {

namespace {

constexpr int kLatThreads = 128;
constexpr int kLatWarps = kLatThreads / 32;
constexpr int kLatMaxN = 16;
constexpr int lattice_ctas(int n) { return n <= 6 ? 8 : (n <= 10 ? 6 : (n <= 13 ? 5 : 4)); }

// Grids of at most this many points along the three directions together keep
// exp(2 pi i j / nk) of every direction in shared memory (6 KB): a phase is then
// two or three products instead of a sincospi (about as many FP64 instructions
// as one row of dimension 10). Larger grids evaluate sincospi.
constexpr int kPhaseTable = 384;

struct LatticeTerms {
  const int *row;               // elements (or stored entries) of matrix row r: row[r] .. row[r + 1]
  const LatticeElement *el;
  const double2 *vk;            // stored entries of V(k), k slowest, entries' columns
  const int *col;
  int entries;
  int nk0, nk1, nk2;            // grid, the largest direction last
  unsigned magic0, magic1, magic2;  // ceil(2^32 / nk): j mod nk by a multiplication, for j < nk^2
  bool table;
};

struct Cplx {
  double x, y;
};

__device__ __forceinline__ Cplx cmul(Cplx a, Cplx b) {
  return {fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x)};
}
// a -= l q
__device__ __forceinline__ void csub(Cplx &a, Cplx l, Cplx q) {
  a.x = fma(-l.x, q.x, fma(l.y, q.y, a.x));
  a.y = fma(-l.x, q.y, fma(-l.y, q.x, a.y));
}
__device__ __forceinline__ Cplx shfl(Cplx a, int src) {
  return {__shfl_sync(0xffffffffu, a.x, src), __shfl_sync(0xffffffffu, a.y, src)};
}

// A point of the grid, advanced along its last direction.
struct GridPoint {
  unsigned i0, i1, i2;
  __device__ GridPoint(const LatticeTerms &t, unsigned long long kid) {
    const unsigned long long q = kid / (unsigned)t.nk2;
    i2 = (unsigned)(kid - q * (unsigned)t.nk2);
    i0 = (unsigned)(q / (unsigned)t.nk1);
    i1 = (unsigned)(q - (unsigned long long)i0 * (unsigned)t.nk1);
  }
  __device__ __forceinline__ void advance(const LatticeTerms &t, unsigned n) {
    i2 += n;
    while (i2 >= (unsigned)t.nk2) {  // past the grid's end it starts over: those points are not used
      i2 -= t.nk2;
      if (++i1 == (unsigned)t.nk1) {
        i1 = 0;
        if (++i0 == (unsigned)t.nk0) i0 = 0;
      }
    }
  }
};

// G of one frequency and +-V0 G in shared memory, rows padded to N + 1
// entries so that lanes reading different rows hit different banks.
template <int N> struct LatticeTile {
  static constexpr int kLd = N + 1;
  double2 g[N * kLd], w[N * kLd];

  // w = sign V0 G; G and V0 column-major
  __device__ void load(const double *__restrict__ G, const double *__restrict__ V0, double sign) {
    for (int t = threadIdx.x; t < N * N; t += blockDim.x)
      g[(t % N) * kLd + t / N] = make_double2(G[2 * t], G[2 * t + 1]);
    __syncthreads();
    for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
      const int r = t % N, b = t / N;
      double sr = 0.0, si = 0.0;
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

  // row r of +-(V(k) G - 1) at grid point (i0, i1, i2); ph: the phase table, or unused
  template <bool STORED>
  __device__ __forceinline__ void row(const LatticeTerms &t, const double2 *ph, const GridPoint &k, int e, int e1,
                                      int r, double sign, Cplx (&a)[N]) const {
#pragma unroll
    for (int b = 0; b < N; ++b) {
      const double2 v = w[r * kLd + b];
      a[b] = {v.x, v.y};
    }
    if (STORED) {
      const double2 *vk = t.vk + (((size_t)k.i0 * t.nk1 + k.i1) * t.nk2 + k.i2) * t.entries;
#pragma unroll 2
      for (; e < e1; ++e) {
        const double2 v = __ldg(vk + e);
        const double2 *gr = g + __ldg(t.col + e) * kLd;
        const Cplx p = {-sign * v.x, -sign * v.y};
#pragma unroll
        for (int b = 0; b < N; ++b) {
          const double2 y = gr[b];
          csub(a[b], p, Cplx{y.x, y.y});
        }
      }
    } else {
      for (; e < e1; ++e) {
        const double2 v = __ldg(&t.el[e].v);
        const int4 m = __ldg(&t.el[e].where);  // column, R
        Cplx p = {sign * v.x, sign * v.y};
        if (t.table) {
          auto turn = [&](unsigned j, int nk, unsigned magic, const double2 *tab) {
            const double2 f = tab[j - (unsigned)nk * __umulhi(j, magic)];
            p = cmul(p, Cplx{f.x, f.y});
          };
          if (t.nk0 > 1) turn(k.i0 * (unsigned)m.y, t.nk0, t.magic0, ph);
          if (t.nk1 > 1) turn(k.i1 * (unsigned)m.z, t.nk1, t.magic1, ph + t.nk0);
          turn(k.i2 * (unsigned)m.w, t.nk2, t.magic2, ph + t.nk0 + t.nk1);
        } else {
          auto part = [](unsigned i, int R, int nk) {
            return (double)((unsigned long long)i * (unsigned)R % (unsigned)nk) / nk;
          };
          double s, c;
          sincospi(2.0 * (part(k.i0, m.y, t.nk0) + part(k.i1, m.z, t.nk1) + part(k.i2, m.w, t.nk2)), &s, &c);
          p = cmul(p, Cplx{c, s});
        }
        const double2 *gr = g + m.x * kLd;
        p = {-p.x, -p.y};
#pragma unroll
        for (int b = 0; b < N; ++b) {
          const double2 y = gr[b];
          csub(a[b], p, Cplx{y.x, y.y});
        }
      }
    }
#pragma unroll
    for (int b = 0; b < N; ++b)
      if (b == r) a[b].x -= sign;
  }
};

// The entries of V(k) that have elements, for every wavevector: out[k * entries + i], by
// L lanes each (a grid of few entries has too few threads otherwise, each with a chain
// of sincospi: one entry of 64 elements on 256 wavevectors 100 us with one lane).
template <int L>
__global__ void __launch_bounds__(128) k_lattice_entries(LatticeTerms t, const int *__restrict__ start,
                                                         unsigned long long n, double2 *out) {
  const unsigned lane = threadIdx.x % L;
  const unsigned long long all = (n + 128 / L - 1) / (128 / L) * (128 / L);  // whole CTAs, for the shuffles
  for (unsigned long long q = blockIdx.x * (128ull / L) + threadIdx.x / L; q < all; q += gridDim.x * (128ull / L)) {
    const unsigned long long kid = min(q, n - 1) / (unsigned)t.entries;
    const int i = (int)(min(q, n - 1) - kid * (unsigned)t.entries);
    const GridPoint k(t, kid);
    auto part = [](unsigned j, int R, int nk) {
      return (double)((unsigned long long)j * (unsigned)R % (unsigned)nk) / nk;
    };
    double sr = 0.0, si = 0.0;
    for (int e = start[i] + lane; e < start[i + 1]; e += L) {
      const double2 v = __ldg(&t.el[e].v);
      const int4 m = __ldg(&t.el[e].where);
      double s, c;
      sincospi(2.0 * (part(k.i0, m.y, t.nk0) + part(k.i1, m.z, t.nk1) + part(k.i2, m.w, t.nk2)), &s, &c);
      sr += v.x * c - v.y * s;
      si += v.x * s + v.y * c;
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
      sr += __shfl_xor_sync(0xffffffffu, sr, o);
      si += __shfl_xor_sync(0xffffffffu, si, o);
    }
    if (lane == 0 && q < n) out[q] = make_double2(sr, si);
  }
}

// The CTA's phase table (visible after the next barrier).
__device__ __forceinline__ void fill_phases(const LatticeTerms &t, double2 *ph) {
  if (!t.table) return;
  for (int i = threadIdx.x; i < t.nk0 + t.nk1 + t.nk2; i += blockDim.x) {
    const int j1 = i - t.nk0, j2 = j1 - t.nk1;
    const double turn = j1 < 0 ? (double)i / t.nk0 : (j2 < 0 ? (double)j1 / t.nk1 : (double)j2 / t.nk2);
    double s, c;
    sincospi(2.0 * turn, &s, &c);
    ph[i] = make_double2(c, s);
  }
}

// The pivot lane of one elimination step among a matrix's N lanes: the largest
// |re| + |im| among those with `open` set. The key is the high word of that
// double (monotonic for values >= 0) with the lane in the last four bits, so
// pivots equal to 1 part in 2^16 are told apart by lane only. The maximum goes
// round the lanes in steps of 1, 2, 4, ... (a maximum may count a lane twice, so
// N need not be a power of two); redux.sync with a mask per matrix took longer.
template <int N> struct PivotRing {
  static constexpr int kRounds = N > 8 ? 4 : (N > 4 ? 3 : (N > 2 ? 2 : N - 1));
  int from[kRounds > 0 ? kRounds : 1];
  __device__ PivotRing(int base, int r) {
#pragma unroll
    for (int o = 0; o < kRounds; ++o) from[o] = base + (r + (1 << o)) % N;
  }
  __device__ __forceinline__ int lane(bool open, Cplx v, int r) const {
    const unsigned hi = (unsigned)__double2hiint(fabs(v.x) + fabs(v.y));
    unsigned key = open ? (0x80000000u | (hi & ~15u) | (unsigned)r) : 0u;
#pragma unroll
    for (int o = 0; o < kRounds; ++o) key = max(key, __shfl_sync(0xffffffffu, key, from[o]));
    return (int)(key & 15u);
  }
};

// Per frequency (blockIdx.y) and CTA: the sum over its wavevectors of
// log |det(V(k) G - 1)|. per_warp: wavevector batches of one warp.
template <int N, bool STORED>
__global__ void __launch_bounds__(kLatThreads, lattice_ctas(N)) k_sef_logdet(const double *__restrict__ G,
                                                            const double *__restrict__ V0, LatticeTerms terms,
                                                            unsigned long long nk, int per_warp, double *partials) {
  constexpr int GW = 32 / N;  // matrices per warp
  __shared__ LatticeTile<N> tile;
  __shared__ double2 ph[kPhaseTable];
  __shared__ double red[kLatWarps];
  const int iw = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (!STORED) fill_phases(terms, ph);
  tile.load(G + 2 * (size_t)iw * N * N, V0, 1.0);
  const int grp = min(lane / N, GW - 1);  // lanes past the last whole matrix repeat it, without a say in the pivots
  const bool mine = lane < GW * N;
  const int base = grp * N, r = mine ? lane - base : 0;
  const PivotRing<N> ring(base, r);
  // sum of the pivots' log |.|: half the log of the product of |.|^2, kept as a
  // mantissa in [1, 2) and an exponent, so that a lane takes one logarithm in all
  double sum = 0.0, prod = 1.0;
  int expo = 0;
  const unsigned long long k0 = ((unsigned long long)blockIdx.x * kLatWarps + warp) * per_warp * GW + grp;
  GridPoint k(terms, k0 < nk ? k0 : 0);
  const int e0 = mine ? __ldg(terms.row + r) : 0, e1 = mine ? __ldg(terms.row + r + 1) : 0;
  for (int it = 0; it < per_warp; ++it, k.advance(terms, GW)) {
    const unsigned long long kid = k0 + (unsigned long long)it * GW;
    const bool valid = kid < nk;
    if (!__any_sync(0xffffffffu, valid)) break;
    Cplx a[N];
    tile.template row<STORED>(terms, ph, k, e0, e1, r, 1.0, a);
    bool open = true;
    Cplx piv = {1.0, 0.0};
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int p = ring.lane(open, a[j], r);
      const int src = base + p;
      const Cplx pv = shfl(a[j], src);
      const double d = pv.x * pv.x + pv.y * pv.y;
      const double rd = d > 0.0 ? reciprocal(d) : 0.0;  // a zero pivot: log 0 below, nothing eliminated
      if (r == p) {
        piv = pv;
        open = false;
      }
      Cplx l = cmul(a[j], Cplx{pv.x * rd, -pv.y * rd});
      if (!open) l = {0.0, 0.0};
#pragma unroll
      for (int c = j + 1; c < N; ++c) {
        const Cplx q = shfl(a[c], src);
        csub(a[c], l, q);
      }
    }
    if (valid && mine) {
      const double d = piv.x * piv.x + piv.y * piv.y;
      if (d > 1e-290 && d < 1e290) {
        prod *= d;
        const int e = ((__double2hiint(prod) >> 20) & 0x7ff) - 1023;
        expo += e;
        prod = __hiloint2double(__double2hiint(prod) - (e << 20), __double2loint(prod));
      } else {  // zero (log 0), not a number, or a square out of range
        sum += log(hypot(piv.x, piv.y));
      }
    }
  }
  sum += 0.5 * (log(prod) + expo * 0.69314718055994530942);
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
template <int N, bool STORED>
__global__ void __launch_bounds__(kLatThreads, lattice_ctas(N)) k_cpt_partial(const double *__restrict__ G,
                                                             const double *__restrict__ V0, LatticeTerms terms,
                                                             unsigned long long nk, int per_warp, double *partials) {
  constexpr int GW = 32 / N;
  __shared__ LatticeTile<N> tile;
  __shared__ double2 ph[kPhaseTable];
  __shared__ double2 acc[kLatWarps * GW][N * N];
  const int iw = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (!STORED) fill_phases(terms, ph);
  double2 *flat = &acc[0][0];
  for (int t = threadIdx.x; t < kLatWarps * GW * N * N; t += blockDim.x) flat[t] = make_double2(0.0, 0.0);
  tile.load(G + 2 * (size_t)iw * N * N, V0 + 2 * (size_t)iw * N * N, -1.0);
  const int grp = min(lane / N, GW - 1);
  const bool mine = lane < GW * N;
  const int base = grp * N, r = mine ? lane - base : 0;
  const PivotRing<N> ring(base, r);
  double2 *out = acc[warp * GW + grp];
  const unsigned long long k0 = ((unsigned long long)blockIdx.x * kLatWarps + warp) * per_warp * GW + grp;
  GridPoint k(terms, k0 < nk ? k0 : 0);
  const int e0 = mine ? __ldg(terms.row + r) : 0, e1 = mine ? __ldg(terms.row + r + 1) : 0;
  for (int it = 0; it < per_warp; ++it, k.advance(terms, GW)) {
    const unsigned long long kid = k0 + (unsigned long long)it * GW;
    const bool valid = kid < nk;
    if (!__any_sync(0xffffffffu, valid)) break;
    Cplx a[N];
    tile.template row<STORED>(terms, ph, k, e0, e1, r, -1.0, a);
    int row = -1;                  // the inverse's row this lane ends with
    unsigned long long perm = 0;   // p_c in bits 4 c ..
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int p = ring.lane(row < 0, a[j], r);
      const int src = base + p;
      const Cplx pv = shfl(a[j], src);
      const double rd = reciprocal(pv.x * pv.x + pv.y * pv.y);
      const Cplx inv = {pv.x * rd, -pv.y * rd};
      const bool self = r == p;
      if (self) row = j;
      perm |= (unsigned long long)p << (4 * j);
      const Cplx f = a[j];
#pragma unroll
      for (int c = 0; c < N; ++c) {
        if (c == j) continue;
        const Cplx q = cmul(shfl(a[c], src), inv);
        if (self) a[c] = q;
        else csub(a[c], f, q);
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
  __shared__ double2 s[kLatMaxN * kLatMaxN], part[256];
  const int iw = blockIdx.x, nn = n * n;
  // nn entries by `slices` strided shares of the CTAs' sums (256 threads)
  const int slices = max(1, (int)blockDim.x / nn), entry = threadIdx.x % nn, slice = threadIdx.x / nn;
  if (slice < slices) {
    double sr = 0.0, si = 0.0;
#pragma unroll 4
    for (int q = slice; q < nblk; q += slices) {
      const double *p = partials + 2 * (((size_t)iw * nblk + q) * nn + entry);
      sr += p[0];
      si += p[1];
    }
    part[threadIdx.x] = make_double2(sr, si);
  }
  __syncthreads();
  if (threadIdx.x < nn) {
    double2 t = part[threadIdx.x];
    for (int q = 1; q < slices; ++q) {
      t.x += part[q * nn + threadIdx.x].x;
      t.y += part[q * nn + threadIdx.x].y;
    }
    s[threadIdx.x] = t;
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

// Wavevector batches per warp: as many as leave about eight CTAs per SM over all
// frequencies (forming V0 G costs a CTA about N batches' work), at most 8, where the
// CTAs' start is a few per cent of their work. Beyond that the grid has CTAs enough,
// and more batches only bound their number: at most kLatMaxBlocks per frequency, or
// 32 per SM over all of them, since each leaves a partial sum of n^2 entries in memory
// (100 frequencies of dimension 16 on 128^3 wavevectors: 27 MB; at 8 batches 13 GB).
// The time is the same: 64 frequencies, 128^2 wavevectors, dimension 10, whole calls:
// 971 and 1769 us (log det, inverse), at 8 batches 983 and 1798; dimension 16: 2430
// and 6865, 2505 and 6815.
constexpr unsigned long long kLatCtas = 148 * 8, kLatMaxBlocks = 64;
int batches_per_warp(int n, int nw, unsigned long long nk) {
  const unsigned long long per = (unsigned long long)kLatWarps * (32 / n), w = (unsigned long long)std::max(nw, 1);
  const unsigned long long one = (nk + per - 1) / per;  // CTAs per frequency at one batch per warp
  const unsigned long long few = std::min<unsigned long long>(8, std::max<unsigned long long>(1, one * w / kLatCtas));
  const unsigned long long most = std::max(kLatMaxBlocks, 4 * kLatCtas / w);
  return (int)std::max(few, (one + most - 1) / most);
}

using LatticeFn = void (*)(const double *, const double *, LatticeTerms, unsigned long long, int, double *);
// The terms of a sum, with the stored entries formed on s where the view has them.
LatticeTerms lattice_terms(const LatticeView &el, const int (&nk)[3], cudaStream_t s) {
  auto magic = [](int nk) { return nk > 1 ? (unsigned)((0x100000000ull + nk - 1) / (unsigned)nk) : 0u; };
  const LatticeTerms t = {el.row, el.el, reinterpret_cast<const double2 *>(el.vk), el.col, el.entries, nk[0], nk[1],
                          nk[2], magic(nk[0]), magic(nk[1]), magic(nk[2]), (long)nk[0] + nk[1] + nk[2] <= kPhaseTable};
  if (el.entries) {
    const unsigned long long n = (unsigned long long)nk[0] * nk[1] * nk[2] * (unsigned)el.entries;
    const int lanes = n < 65536 ? 16 : 1;
    const unsigned grid = (unsigned)std::min<unsigned long long>((n * lanes + 127) / 128, 148 * 32);
    (lanes == 16 ? k_lattice_entries<16> : k_lattice_entries<1>)<<<grid, 128, 0, s>>>(
        t, el.start, n, reinterpret_cast<double2 *>(el.vk));
    QED_LAUNCH();
  }
  return t;
}

template <bool STORED> struct LatticeFns {
  static constexpr LatticeFn logdet[kLatMaxN] = {
      k_sef_logdet<1, STORED>,  k_sef_logdet<2, STORED>,  k_sef_logdet<3, STORED>,  k_sef_logdet<4, STORED>,
      k_sef_logdet<5, STORED>,  k_sef_logdet<6, STORED>,  k_sef_logdet<7, STORED>,  k_sef_logdet<8, STORED>,
      k_sef_logdet<9, STORED>,  k_sef_logdet<10, STORED>, k_sef_logdet<11, STORED>, k_sef_logdet<12, STORED>,
      k_sef_logdet<13, STORED>, k_sef_logdet<14, STORED>, k_sef_logdet<15, STORED>, k_sef_logdet<16, STORED>};
  static constexpr LatticeFn cpt[kLatMaxN] = {
      k_cpt_partial<1, STORED>,  k_cpt_partial<2, STORED>,  k_cpt_partial<3, STORED>,  k_cpt_partial<4, STORED>,
      k_cpt_partial<5, STORED>,  k_cpt_partial<6, STORED>,  k_cpt_partial<7, STORED>,  k_cpt_partial<8, STORED>,
      k_cpt_partial<9, STORED>,  k_cpt_partial<10, STORED>, k_cpt_partial<11, STORED>, k_cpt_partial<12, STORED>,
      k_cpt_partial<13, STORED>, k_cpt_partial<14, STORED>, k_cpt_partial<15, STORED>, k_cpt_partial<16, STORED>};
};

}  // namespace

int lattice_blocks(int n, int nw, long nk) {
  if (n < 1 || n > kLatMaxN) fail(QED_ERR_UNSUPPORTED, "lattice sums: Green function dimension above 16");
  const unsigned long long per =
      (unsigned long long)kLatWarps * (32 / n) * (unsigned long long)batches_per_warp(n, nw, (unsigned long long)nk);
  return (int)(((unsigned long long)nk + per - 1) / per);
}

void launch_sef_logdet(int n, int nw, const double *G, const double *V0, const LatticeView &el, const int (&nk3)[3], double *partials,
                       cudaStream_t s) {
  const long nk = (long)nk3[0] * nk3[1] * nk3[2];
  const int nblk = lattice_blocks(n, nw, nk);
  if (nw <= 0 || nk <= 0) return;
  if (nw > 65535) fail(QED_ERR_ARGUMENT, "SEF grid integrand: more than 65535 frequencies");
  const LatticeTerms t = lattice_terms(el, nk3, s);
  (el.entries ? LatticeFns<true>::logdet : LatticeFns<false>::logdet)[n - 1]<<<dim3(nblk, nw), kLatThreads, 0, s>>>(G, V0, t, (unsigned long long)nk,
                                                         batches_per_warp(n, nw, nk), partials);
  QED_LAUNCH();
}

void launch_cpt_projected(int n, int nw, const double *G, const double *V0, const LatticeView &el, const int (&nk3)[3], double *partials, double *Gproj, cudaStream_t s) {
  const long nk = (long)nk3[0] * nk3[1] * nk3[2];
  const int nblk = lattice_blocks(n, std::min(nw, 65535), nk);
  if (nw <= 0 || nk <= 0) return;
  const LatticeTerms t = lattice_terms(el, nk3, s);
  for (int w0 = 0; w0 < nw; w0 += 65535) {  // the grid's second dimension ends there
    const int m = std::min(nw - w0, 65535);
    const size_t o = 2 * (size_t)w0 * n * n;
    (el.entries ? LatticeFns<true>::cpt : LatticeFns<false>::cpt)[n - 1]<<<dim3(nblk, m), kLatThreads, 0, s>>>(G + o, V0 + o, t, (unsigned long long)nk,
                                                       batches_per_warp(n, std::min(nw, 65535), nk),
                                                       partials + o * nblk);
    QED_LAUNCH();
  }
  k_cpt_reduce<<<nw, 256, 0, s>>>(n, nblk, (double)nk, G, partials, Gproj);
  QED_LAUNCH();
}

}  // namespace qed
