// Two-pass H.v in tiles of eight rows or columns, for half bases that fit shared
// memory eight vectors wide (see launch_hv_tile).
//
// A pass takes one spin's hops. Its work item is a tile: all strings of that spin
// by eight strings of the other one (eight rows of x for the up hops, eight
// columns for the down hops), staged in shared memory with cp.async as [string][8].
// A warp works on eight strings at once, a lane on one string and two of the eight
// vectors: one table entry (the same for the four lanes of a string), one value
// from shared memory and one 16-byte gather serve two states, the four lanes of a
// string read 64 contiguous bytes, and lanes wait only for the longest of eight
// neighbouring strings. The column pass writes y = xs (down hops) x; the row pass
// adds the rest and takes the reductions.
//
// What bounds it: the shared-memory pipe (about 10 wavefronts per entry and warp:
// 5 to 6 of the gather, 4 of them unavoidable, 2 of the table, 1 to 2 of the
// value) and, below about 150 tiles, latency: launch, staging, hops and stores of
// one CTA per SM follow one another (issue slots are 36 % busy in the column pass
// of 924 x 924 states). The row pass therefore starts under the column pass
// (programmatic launch) and waits before it reads y.
//
// Measured on a B200 with the dot products and their final sum, against the forms
// it replaces there (k_hv_rows2 + k_hv_cols2, or k_hv_rows16 + k_hv_cols16w for
// two hopping magnitudes and an even row): 462 x 462 10.5 against 18.2 us, 924 x
// 924 with eight bath orbitals 22.0 against 24.8, of the 3x4 cluster with t' 29.5
// against 39.5, 2002 x 2002 100 against 108, 3432 x 3432 of the 2x7 cluster 293
// against 336, of the 14-site chain 201 against 251.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.hpp"
#include "hv_device.cuh"
#include "kernels.cuh"

namespace qed {

namespace {

constexpr int kTile = 8;           // vectors per tile
constexpr size_t kTileSmemMax = (kTileMaxDim + 1) * kTile * sizeof(double);
static_assert(kTileSmemMax <= 224 * 1024, "the largest tile and the values fit one CTA");

__device__ __forceinline__ void cp_async8(void *dst, const void *src, bool on) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(on ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(on ? 16 : 0)
               : "memory");
}

// A group's step count and first entries, loaded one group ahead of their use
// (more entries ahead cost shared-memory bandwidth for short lists: two steps
// ahead took 1.05x, four 1.3x the time).
struct TileGroup {
  const uint4 *p;
  uint32_t steps;
  uint4 w;
  __device__ __forceinline__ void load(const SpinTable &t, uint32_t g, uint32_t g1, uint32_t s) {
    steps = 0;
    if (g >= g1) return;
    steps = __ldg(t.tile_steps + g);
    p = t.tile_ent + (size_t)g * t.tile_max * 8 + s;
    w = __ldg(p);  // an empty group has a step of padding, if the table has any step
  }
};

__device__ __forceinline__ double2 lds2(uint32_t a) {
  double2 v;
  asm("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ double lds1(uint32_t a) {
  double v;
  asm("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
// The two entries of one step: (a0, a1) += value x the pair of the target's row.
__device__ __forceinline__ void hop_step(uint4 w, uint32_t st, uint32_t vals, double &a0, double &a1) {
  const double2 g = lds2(st + w.x), h = lds2(st + w.z);
  const double v = lds1(vals + w.y), u = lds1(vals + w.w);
  a0 = fma(v, g.x, a0);
  a1 = fma(v, g.y, a1);
  a0 = fma(u, h.x, a0);
  a1 = fma(u, h.y, a1);
}

// ROW: the row pass (up hops) on rows 8 tile ..; else the column pass (down hops)
// on columns 8 tile ... VEC: columns come in 16-byte pairs (dim_up even, vectors
// aligned).
template <bool ROW, bool VEC>
__global__ void __launch_bounds__(1024, 1) k_hv_tile(const __grid_constant__ HvOperator op,
                                                     const double *__restrict__ x, double xs, double *y,
                                                     const __grid_constant__ SubList sub, int red_mask,
                                                     double *partials, uint32_t ntile, uint32_t nchunk) {
  if (op.skip && *op.skip) return;
  extern __shared__ __align__(16) double tile[];
  __shared__ double vals[256];
  const SpinTable &t = ROW ? op.up : op.dn;
  const uint32_t du = op.up.dim, n = t.dim, m = ROW ? op.dn.dim : du;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const uint32_t s = lane >> 2, q = lane & 3;
  for (uint32_t i = threadIdx.x; i < (uint32_t)t.nvals; i += blockDim.x) vals[i] = t.vals[i];
  const uint32_t per = ((n + nchunk - 1) / nchunk + 7) / 8 * 8;  // strings per chunk
  double red[3] = {0.0, 0.0, 0.0};
  for (uint32_t item = blockIdx.x; item < ntile * nchunk; item += gridDim.x) {
    const uint32_t o0 = (item / nchunk) * kTile, c0 = (item % nchunk) * per, c1 = min(n, c0 + per);
    if (c0 >= n) continue;
    if (item != blockIdx.x) __syncthreads();  // the previous tile has been read
    if (threadIdx.x < kTile) tile[(size_t)n * kTile + threadIdx.x] = 0.0;  // the target of padding entries
    for (uint32_t idx = threadIdx.x; idx < 4 * n; idx += blockDim.x) {
      const uint32_t i = idx >> 2, o = o0 + 2 * (idx & 3);
      double *dst = tile + 2 * (size_t)idx;
      const bool on0 = o < m, on1 = o + 1 < m;
      if (ROW) {
        const double *src = x + (size_t)(on0 ? o : 0) * du + i;
        cp_async8(dst, src, on0);
        cp_async8(dst + 1, on1 ? src + du : x, on1);
      } else {
        const double *src = x + (size_t)i * du + (on0 ? o : 0);
        if (VEC) {
          cp_async16(dst, src, on0);
        } else {
          cp_async8(dst, src, on0);
          cp_async8(dst + 1, on1 ? src + 1 : x, on1);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    // the first strings' tables and this lane's two vectors while x arrives
    uint32_t i = c0 + warp * 8 + s;
    const uint32_t g1 = (c1 + 7) / 8;
    TileGroup cur;
    cur.load(t, (i - s) / 8, g1, s);
    const uint32_t oa = o0 + 2 * q, ob = oa + 1;
    const size_t ia = (size_t)oa * du, ib = ia + du;  // rows oa and ob (row pass)
    uint32_t bits0 = 0, bits1 = 0;
    double dg0 = 0.0, dg1 = 0.0;
    if (ROW) {
      if (oa < m) {
        bits0 = op.dn.bits[oa];
        dg0 = op.dn.diag[oa];
      }
      if (ob < m) {
        bits1 = op.dn.bits[ob];
        dg1 = op.dn.diag[ob];
      }
    }
    if (!ROW) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (ROW) asm volatile("griddepcontrol.wait;" ::: "memory");  // the column pass's y
    const double2 *st = reinterpret_cast<const double2 *>(tile) + q;  // this lane's pair of string 0
    const uint32_t sta = (uint32_t)__cvta_generic_to_shared(st), va = (uint32_t)__cvta_generic_to_shared(vals);
    for (; i - s < c1; i += nwarp * 8) {
      const bool on = i < c1;
      double y0 = 0.0, y1 = 0.0, dup = 0.0;
      uint32_t ub = 0;
      if (ROW && on) {  // used after the hops
        if (oa < m) y0 = y[ia + i];
        if (ob < m) y1 = y[ib + i];
        dup = t.diag[i];
        ub = t.bits[i];
      }
      TileGroup nxt;
      nxt.load(t, (i - s) / 8 + nwarp, g1, s);
      double a0 = 0.0, a1 = 0.0;
      const uint4 *p = cur.p + 8;
      if (cur.steps) hop_step(cur.w, sta, va, a0, a1);
#pragma unroll 4
      for (uint32_t j = 1; j < cur.steps; ++j, p += 8) hop_step(__ldg(p), sta, va, a0, a1);  // uniform over the warp
      if (on) {
        if (ROW) {
          const double2 g = st[i * 4];
          double r0 = y0 + xs * (a0 + (dup + dg0 + inter_term(op.inter, ub, bits0)) * g.x);
          double r1 = y1 + xs * (a1 + (dup + dg1 + inter_term(op.inter, ub, bits1)) * g.y);
          for (int z = 0; z < sub.n; ++z) {
            const double c = sub.cdev ? sub.cdev[z] : sub.c[z];
            if (oa < m) r0 -= c * sub.z[z][ia + i];
            if (ob < m) r1 -= c * sub.z[z][ib + i];
          }
          if (oa < m) y[ia + i] = r0;
          if (ob < m) y[ib + i] = r1;
          if (red_mask) {  // rows past the end hold zeros
            if (oa >= m) r0 = 0.0;
            if (ob >= m) r1 = 0.0;
            const double x0 = xs * g.x, x1 = xs * g.y;
            red[0] += x0 * r0 + x1 * r1;
            red[1] += r0 * r0 + r1 * r1;
            red[2] += x0 * x0 + x1 * x1;
          }
        } else {
          double *yp = y + (size_t)i * du + oa;
          if (VEC) {
            if (oa < m) *reinterpret_cast<double2 *>(yp) = make_double2(xs * a0, xs * a1);
          } else {
            if (oa < m) yp[0] = xs * a0;
            if (ob < m) yp[1] = xs * a1;
          }
        }
      }
      cur = nxt;
    }
  }
  if (ROW && red_mask) block_reduce_store<3>(red, partials, 3);
}

using TileFn = void (*)(HvOperator, const double *, double, double *, SubList, int, double *, uint32_t, uint32_t);

int tile_sms() {
  static const int n = [] {
    int dev = 0, c = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev);
    return c > 0 ? c : 148;
  }();
  return n;
}

struct TilePlan {
  uint32_t ntile, nchunk, grid, threads;
  size_t smem;
};

// n strings of the pass's spin, m of the other. Tiles are split into
// chunks of strings (each staging the whole tile) when there are too few of them.
TilePlan plan_tiles(uint32_t n, uint32_t m) {
  TilePlan p;
  p.ntile = (m + kTile - 1) / kTile;
  p.smem = (size_t)(n + 1) * kTile * sizeof(double);
  const uint32_t sms = (uint32_t)tile_sms();
  p.nchunk = std::max(1u, std::min({sms / std::max(1u, p.ntile), n / 128u, 4u}));
  const uint32_t items = p.ntile * p.nchunk;
  p.grid = std::min(items, 8u * sms);
  // one CTA per SM by shared memory or by number: as many warps as it can hold
  const uint32_t strings = (n + p.nchunk - 1) / p.nchunk;
  p.threads = (p.smem > 100 * 1024 || items <= sms) ? 1024 : 512;
  p.threads = std::min(p.threads, std::max(64u, (strings + 7) / 8 * 32));
  return p;
}

void set_tile_attributes() {
  static const bool once = [] {
    for (TileFn f : {(TileFn)k_hv_tile<true, false>, (TileFn)k_hv_tile<false, false>, (TileFn)k_hv_tile<false, true>})
      QED_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmemMax));
    return true;
  }();
  (void)once;
}

}  // namespace

// Work of a pass's fullest SM over an even share of it.
double tile_unevenness(uint32_t n, uint32_t m) {
  const TilePlan p = plan_tiles(n, m);
  const uint32_t sms = (uint32_t)tile_sms(), items = p.ntile * p.nchunk;
  return (double)((items + sms - 1) / sms) * sms * kTile / ((double)m * p.nchunk);
}

// Where the tiled form is the faster one, from 812 sectors of 11 to 28 sites against the
// two-pass and staged kernels. Below kTileAlwaysStates they gain 1.0 to 2.0x (but for
// 0.93x at 2925 x 351 with six hops a string at most). Above, tiles that leave most SMs idle in a last wave lose: 171 tiles on 148 SMs at 1365 x
// 1365 states 49 to 68 us against 46 to 62, 1365 x 3003 110 to 151 against 101 to 139.
// For rows of even length that takes an almost empty wave in both passes (mean
// unevenness 1.78 0.94x, 1.61 1.01x). For odd ones, whose columns are read and written 8
// bytes at a time, an unevenness of 1.3 (1.18 gains up to 1.4x, 1.34 0.95x), and vectors
// that leave L2 (3003 x 2002 states 1.15x, 3003 x 3432 0.88x).
bool tile_sizes(uint32_t du, uint32_t dd) {
  constexpr uint64_t kTileAlwaysStates = 1700000, kTileOddStates = 8000000;
  const uint64_t D = (uint64_t)du * dd;
  if (std::min(du, dd) < kTileMinDim || std::max(du, dd) > kTileMaxDim || D < kTileMinStates) return false;
  if (D < kTileAlwaysStates) return true;
  const double uneven = 0.5 * (tile_unevenness(du, dd) + tile_unevenness(dd, du));
  return du % 2 == 0 ? uneven < 1.7 : uneven < 1.25 && D < kTileOddStates;
}

bool tile_applies(const HvOperator &op) {
  return op.up.tile_max && op.dn.tile_max && tile_sizes(op.up.dim, op.dn.dim);
}

int tile_grid(const HvOperator &op) { return (int)plan_tiles(op.up.dim, op.dn.dim).grid; }

int launch_hv_tile(const HvOperator &op, const double *x, double xs, double *y, const SubList &sub, int red_mask,
                   Reducer &r, cudaStream_t s) {
  set_tile_attributes();
  const bool vec = op.up.dim % 2 == 0 && !(((uintptr_t)x | (uintptr_t)y) & 15u);
  const SubList none{};
  const TilePlan pc = plan_tiles(op.dn.dim, op.up.dim);
  const TileFn col = vec ? (TileFn)k_hv_tile<false, true> : (TileFn)k_hv_tile<false, false>;
  col<<<pc.grid, pc.threads, pc.smem, s>>>(op, x, xs, y, none, 0, nullptr, pc.ntile, pc.nchunk);
  QED_LAUNCH();
  TilePlan pr = plan_tiles(op.up.dim, op.dn.dim);
  if (red_mask && pr.grid > (uint32_t)r.max_blocks) pr.grid = (uint32_t)r.max_blocks;
  // the row pass may start while the column pass runs (it waits before it reads y)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(pr.grid);
  cfg.blockDim = dim3(pr.threads);
  cfg.dynamicSmemBytes = pr.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  QED_CUDA(cudaLaunchKernelEx(&cfg, (TileFn)k_hv_tile<true, false>, op, x, xs, y, sub, red_mask, r.partials, pr.ntile,
                              pr.nchunk));
  return (int)pr.grid;
}

}  // namespace qed
