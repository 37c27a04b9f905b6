// One-launch H.v for small sectors (see launch_hv_fused).
//
// The two-pass kernels (kernels.cu) read and write y twice and launch twice; on a
// sector of up to 10^5 states the launches, the serial chain count -> entry ->
// value -> gather of each pass, and a grid of one or two rows per CTA are what
// they cost, not bytes. Here a work item is NV rows by a chunk of up strings. The
// item's rows are staged in shared memory (NV values side by side, so that an up
// hop is one table entry and one wide gather for all of them), the rows' down
// hops come as gathers from L2 that are contiguous over the CTA, and the
// diagonal, the up hops, the down hops, the subtractions and the reductions are
// one pass over the item. Up-hop entries are loaded kAhead at a time, before the
// item's rows arrive for the first string.
//
// Bound by latency (launch, tables and rows, gathers; one wave of CTAs). Measured
// against the two passes on a B200, H x with its dot products (each with the 2.3
// us of their final sum): 4900 states 7.0 against 12.5 us, 63504 states 8.6
// against 16.7, 312312 states (3432 x 91) 20.5 against 25.8.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.hpp"
#include "hv_device.cuh"
#include "kernels.cuh"

namespace qed {

namespace {

constexpr int kFusedThreads = 512;
constexpr int kFusedHops = 256;  // at most 255 hops per string
constexpr int kAhead = 4;        // up-hop entries loaded ahead

struct DnHop {
  double v;
  uint32_t off;  // target row x dim_up
  uint32_t pad;
};

template <int NV> struct Values {
  double v[NV];
};

// NV values at st, as wide loads (st is 16-byte aligned for NV >= 2)
template <int NV> __device__ __forceinline__ Values<NV> staged(const double *st) {
  Values<NV> t;
  if constexpr (NV == 1) {
    t.v[0] = st[0];
  } else {
#pragma unroll
    for (int c = 0; c < NV; c += 2) {
      const double2 d = *reinterpret_cast<const double2 *>(st + c);
      t.v[c] = d.x;
      t.v[c + 1] = d.y;
    }
  }
  return t;
}

// The tables of an up string, with its first kAhead entries.
struct UpString {
  int cnt = 0;
  uint32_t bits = 0, e[kAhead];
  double diag = 0.0;
  __device__ __forceinline__ void load(const SpinTable &t, uint32_t u, uint32_t u1) {
    if (u >= u1) return;
    cnt = t.cnt[u];
    bits = t.bits[u];
    diag = t.diag[u];
#pragma unroll
    for (int q = 0; q < kAhead; ++q)
      if (q < t.width) e[q] = __ldg(t.ell + (size_t)q * t.dim + u);
  }
};

template <int NV>
__global__ void __launch_bounds__(kFusedThreads, 2)
    k_hv_fused(const __grid_constant__ HvOperator op, const double *x, double xs, double *y,
               const __grid_constant__ SubList sub, int red_mask, double *partials, uint32_t chunk, uint32_t nchunk) {
  if (op.skip && *op.skip) return;
  extern __shared__ __align__(16) double st[];
  __shared__ double vup[256], vdn[256];
  __shared__ __align__(16) DnHop hop[NV][kFusedHops];
  __shared__ int nhop[NV];
  const uint32_t du = op.up.dim, dd = op.dn.dim, T = blockDim.x;
  const uint32_t nrg = (dd + NV - 1) / NV, nitem = nrg * nchunk;
  for (uint32_t i = threadIdx.x; i < (uint32_t)op.up.nvals; i += T) vup[i] = op.up.vals[i];
  for (uint32_t i = threadIdx.x; i < (uint32_t)op.dn.nvals; i += T) vdn[i] = op.dn.vals[i];
  double red[3] = {0.0, 0.0, 0.0};
  for (uint32_t item = blockIdx.x; item < nitem; item += gridDim.x) {
    const uint32_t d0 = (item / nchunk) * NV, u0 = (item % nchunk) * chunk, u1 = min(du, u0 + chunk);
    if (item != blockIdx.x) __syncthreads();  // the previous item is done with the staged rows
    // this thread's first string: table data that does not depend on x
    uint32_t u = u0 + threadIdx.x;
    UpString cur;
    cur.load(op.up, u, u1);
    // the rows' down hops: entries past a row's count may hold anything and are not used
    for (uint32_t j = threadIdx.x; j < (uint32_t)(NV * op.dn.width); j += T) {
      const uint32_t r = j / (uint32_t)op.dn.width, k = j - r * (uint32_t)op.dn.width, d = d0 + r;
      if (d < dd) hop[r][k].off = __ldg(op.dn.ell + (size_t)k * dd + d);
    }
    if (threadIdx.x < NV) nhop[threadIdx.x] = d0 + threadIdx.x < dd ? (int)op.dn.cnt[d0 + threadIdx.x] : 0;
    for (uint32_t i = threadIdx.x; i < du; i += T) {
      double t[NV];
#pragma unroll
      for (int c = 0; c < NV; ++c) {
        t[c] = d0 + c < dd ? __ldg(x + (size_t)(d0 + c) * du + i) : 0.0;
      }
      if constexpr (NV == 1) {
        st[i] = t[0];
      } else {
#pragma unroll
        for (int c = 0; c < NV; c += 2)
          *reinterpret_cast<double2 *>(st + (size_t)i * NV + c) = make_double2(t[c], t[c + 1]);
      }
    }
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < (uint32_t)(NV * op.dn.width); j += T) {
      const uint32_t r = j / (uint32_t)op.dn.width, k = j - r * (uint32_t)op.dn.width;
      if (k >= (uint32_t)nhop[r]) continue;
      const uint32_t h = hop[r][k].off;
      hop[r][k] = DnHop{vdn[h & 255u], (h >> 8) * du, 0u};
    }
    uint32_t dnb[NV];
    double ddn[NV];
#pragma unroll
    for (int r = 0; r < NV; ++r) {
      dnb[r] = d0 + r < dd ? op.dn.bits[d0 + r] : 0u;
      ddn[r] = d0 + r < dd ? op.dn.diag[d0 + r] : 0.0;
    }
    __syncthreads();
    while (u < u1) {
      double acc[NV];
      {
        const Values<NV> x0 = staged<NV>(st + (size_t)u * NV);
#pragma unroll
        for (int c = 0; c < NV; ++c) {
          acc[c] = (cur.diag + ddn[c] + inter_term(op.inter, cur.bits, dnb[c])) * x0.v[c];
        }
      }
      // up hops, kAhead entries in flight while the previous ones gather
      for (int k = 0; k < cur.cnt; k += kAhead) {
        uint32_t f[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
          f[q] = cur.e[q];
          if (k + kAhead + q < cur.cnt) cur.e[q] = __ldg(op.up.ell + (size_t)(k + kAhead + q) * du + u);
        }
#pragma unroll
        for (int q = 0; q < kAhead; ++q)
          if (k + q < cur.cnt) {
            const Values<NV> t = staged<NV>(st + (size_t)(f[q] >> 8) * NV);
            const double v = vup[f[q] & 255u];
#pragma unroll
            for (int c = 0; c < NV; ++c) acc[c] += v * t.v[c];
          }
      }
      UpString nxt;  // the next string's table data travel during the down hops
      nxt.load(op.up, u + T, u1);
      const double *xu = x + u;
#pragma unroll
      for (int r = 0; r < NV; ++r) {
        const int n = nhop[r];
#pragma unroll 4
        for (int k = 0; k < n; ++k) {
          const DnHop h = hop[r][k];
          acc[r] += h.v * __ldg(xu + h.off);
        }
      }
#pragma unroll
      for (int c = 0; c < NV; ++c) {
        if (d0 + c >= dd) break;
        const size_t I = (size_t)(d0 + c) * du + u;
        double a = acc[c] * xs;
        for (int s = 0; s < sub.n; ++s) a -= (sub.cdev ? sub.cdev[s] : sub.c[s]) * sub.z[s][I];
        y[I] = a;
        if (red_mask) {
          const double xv = xs * st[(size_t)u * NV + c];
          red[0] += xv * a;
          red[1] += a * a;
          red[2] += xv * xv;
        }
      }
      u += T;
      cur = nxt;
    }
  }
  if (red_mask) block_reduce_store<3>(red, partials, 3);
}

using FusedFn = void (*)(HvOperator, const double *, double, double *, SubList, int, double *, uint32_t, uint32_t);

int fused_sms() {
  static const int n = [] {
    int dev = 0, c = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev);
    return c > 0 ? c : 148;
  }();
  return n;
}

constexpr uint32_t kFusedMaxRow = 4096;  // up strings: every chunk stages whole rows
constexpr size_t kFusedSmemMax = 2 * kFusedMaxRow * sizeof(double);

struct FusedPlan {
  int nv;  // rows per work item
  uint32_t chunk, nchunk, items, threads;
};

// Chunks of the up strings: at most four per row group (each stages the whole
// rows), enough of them that every SM gets about three work items.
void plan_chunks(const HvOperator &op, int rows, FusedPlan &p) {
  const uint32_t du = op.up.dim, nrg = (op.dn.dim + rows - 1) / rows, want = 3u * (uint32_t)fused_sms();
  const uint32_t nchunk = std::max(1u, std::min({(want + nrg - 1) / nrg, 4u, du / 64u}));
  p.chunk = (du + nchunk - 1) / nchunk;
  p.nchunk = (du + p.chunk - 1) / p.chunk;
  p.items = nrg * p.nchunk;
  const uint32_t turns = (p.chunk + kFusedThreads - 1) / kFusedThreads;
  p.threads = std::min<uint32_t>(kFusedThreads, ((p.chunk + turns - 1) / turns + 31) / 32 * 32);
}

// Rows per work item: two share table entries, one keeps the SMs full (sectors of
// 213444 states: 11.9 and 10.3 us for 1 and 2 rows, 11.7 for 4). With rows of at most
// kFusedMaxRow strings both fit shared memory.
FusedPlan plan_fused(const HvOperator &op) {
  const uint64_t D = (uint64_t)op.up.dim * op.dn.dim;
  FusedPlan p;
  p.nv = D >= 150000 && op.dn.dim >= 2 ? 2 : 1;
  plan_chunks(op, p.nv, p);
  return p;
}

FusedFn fused_fn(int nv) { return nv == 2 ? k_hv_fused<2> : k_hv_fused<1>; }

void set_fused_attributes() {
  static const bool once = [] {
    for (int nv : {1, 2})
      QED_CUDA(cudaFuncSetAttribute(fused_fn(nv), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFusedSmemMax));
    return true;
  }();
  (void)once;
}

int grid_of(const FusedPlan &p) { return (int)std::min<uint32_t>(p.items, 8u * (uint32_t)fused_sms()); }

}  // namespace

bool fused_applies(const HvOperator &op) {
  const uint64_t D = (uint64_t)op.up.dim * op.dn.dim;
  return D <= kFusedMaxStates && op.up.dim <= kFusedMaxRow;
}

int fused_grid(const HvOperator &op) { return grid_of(plan_fused(op)); }

int launch_hv_fused(const HvOperator &op, const double *x, double xs, double *y, const SubList &sub, int red_mask,
                    Reducer &r, cudaStream_t s) {
  set_fused_attributes();
  const FusedPlan p = plan_fused(op);
  int grid = grid_of(p);
  if (red_mask && grid > r.max_blocks) grid = r.max_blocks;
  fused_fn(p.nv)<<<grid, p.threads, (size_t)op.up.dim * p.nv * sizeof(double), s>>>(op, x, xs, y, sub, red_mask,
                                                                                    r.partials, p.chunk, p.nchunk);
  QED_LAUNCH();
  return grid;
}

}  // namespace qed
