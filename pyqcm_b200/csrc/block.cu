// Dense block kernels of the block form of the band-Lanczos recurrence
// (block_lanczos_qmatrix, solver.cpp). A block is p <= 16 separate FP64 vectors
// of D states (pointer arrays, so the start vectors form a block without a
// copy).
//
// k_bl_simple (odd dimensions, misaligned vectors): Y = a Y + s1 X1 M1 (M1 p x p,
// row-major), or (X1 M1) M2, then optionally the per-CTA partials of L^T Y for L =
// the updated Y or another block. One thread per state: the thread loads its state's p values of each block (coalesced
// across the warp), forms the update with M1 broadcast from shared memory and
// stores the result. The Gram matrix runs on the FP64 tensor cores: each warp
// copies its 32 states of L and Y into shared memory (rows padded to 20
// doubles, so the fragment reads are free of bank conflicts) and accumulates
// L^T Y with mma.sync m8n8k4 (A = L^T: row = vector, column = state; B = Y:
// row = state, column = vector), 2 x 2 tiles of 8 x 8 for p > 8.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.hpp"
#include "kernels.cuh"

namespace qed {

namespace {

constexpr int kBlThreads = 256;
constexpr int kBlWarps = kBlThreads / 32;
constexpr int kStageLd = 20;  // padded row of one state's 16 values in shared memory

__device__ __forceinline__ void mma_f64(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

template <int P>
__global__ void __launch_bounds__(kBlThreads, 1) k_bl_simple(size_t D, int p, double a, BlockOut Y, double s1,
                                                          BlockIn X1, const double *__restrict__ M1,
                                                          const double *__restrict__ M2, bool keep, int gram,
                                                          BlockIn L, double *partials) {
  constexpr int NT = P / 8;  // 8 x 8 tiles per side
  // dynamic shared memory: M1, M2, then per warp the two staged 32-state panels
  // (reused for the cross-warp sum of the Gram partials at the end)
  extern __shared__ double smem_bl[];
  double *m1 = smem_bl, *m2 = smem_bl + P * P;
  double *stage = smem_bl + 2 * P * P;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool upd = X1.v[0] != nullptr;
  for (int t = threadIdx.x; t < P * P; t += blockDim.x) {
    const int i = t / P, c = t % P;
    m1[t] = (upd && i < p && c < p) ? M1[i * p + c] : 0.0;
    m2[t] = (M2 && i < p && c < p) ? M2[i * p + c] : 0.0;
  }
  __syncthreads();
  double acc[NT * NT][2];
#pragma unroll
  for (int q = 0; q < NT * NT; ++q) acc[q][0] = acc[q][1] = 0.0;
  double *sl = stage + (size_t)warp * 2 * 32 * kStageLd, *sy = sl + 32 * kStageLd;
  const size_t stride = (size_t)gridDim.x * kBlThreads;
  for (size_t I0 = (size_t)blockIdx.x * kBlThreads + warp * 32; I0 < D; I0 += stride) {
    const size_t I = I0 + lane;
    const bool valid = I < D;
    double y[P];
#pragma unroll
    for (int c = 0; c < P; ++c) y[c] = (valid && c < p && a != 0.0) ? a * Y.v[c][I] : 0.0;
    if (upd) {
      double x[P];
#pragma unroll
      for (int i = 0; i < P; ++i) x[i] = (valid && i < p) ? X1.v[i][I] : 0.0;
#pragma unroll
      for (int c = 0; c < P; ++c) {
        double t = 0.0;
#pragma unroll
        for (int i = 0; i < P; ++i) t = fma(x[i], m1[i * P + c], t);
        y[c] = fma(s1, t, y[c]);
      }
      if (M2) {
#pragma unroll
        for (int i = 0; i < P; ++i) x[i] = y[i];
#pragma unroll
        for (int c = 0; c < P; ++c) {
          double t = 0.0;
#pragma unroll
          for (int i = 0; i < P; ++i) t = fma(x[i], m2[i * P + c], t);
          y[c] = t;
        }
      }
    }
    if (keep && valid && (upd || a != 1.0)) {  // a pure Gram (a = 1, no update) leaves Y as it is
#pragma unroll
      for (int c = 0; c < P; ++c)
        if (c < p) Y.v[c][I] = y[c];
    }
    if (gram) {
#pragma unroll
      for (int c = 0; c < P; ++c) {
        const double l = gram == 1 ? y[c] : ((valid && c < p) ? L.v[c][I] : 0.0);
        sl[lane * kStageLd + c] = l;
        sy[lane * kStageLd + c] = y[c];
      }
      __syncwarp();
#pragma unroll
      for (int k0 = 0; k0 < 32; k0 += 4) {
        const int st = (k0 + (lane & 3)) * kStageLd + (lane >> 2);
        double af[NT], bf[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          af[t] = sl[st + 8 * t];
          bf[t] = sy[st + 8 * t];
        }
#pragma unroll
        for (int mt = 0; mt < NT; ++mt)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) mma_f64(acc[mt * NT + nt][0], acc[mt * NT + nt][1], af[mt], bf[nt]);
      }
      __syncwarp();  // the stage is read before the next states overwrite it
    }
  }
  if (!gram) return;
  __syncthreads();  // every warp is done with its panels: they now hold the partial Grams
  double *red = stage;  // [warp][P * P]
  // C fragment: row lane >> 2, columns 2 (lane & 3) + {0, 1} of each tile
#pragma unroll
  for (int mt = 0; mt < NT; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int j = 0; j < 2; ++j)
        red[warp * P * P + (mt * 8 + (lane >> 2)) * P + nt * 8 + 2 * (lane & 3) + j] = acc[mt * NT + nt][j];
  __syncthreads();
  for (int t = threadIdx.x; t < p * p; t += blockDim.x) {
    const int i = t / p, c = t % p;
    double s = 0.0;
    for (int w = 0; w < kBlWarps; ++w) s += red[w * P * P + i * P + c];
    partials[(size_t)blockIdx.x * p * p + t] = s;
  }
}

// ---- pipelined tensor-core form -------------------------------------------
//
// Each warp streams tiles of 32 consecutive states. A tile's p values of each
// block it reads (X1, Y unless a = 0, L for gram 2) arrive as panels in shared
// memory by cp.async (16-byte chunks), the next tiles' while this one computes. A
// panel is laid out [vector][state], P rows (p rounded up to a multiple of four, the
// rows from p on stay zero) of kPanelLd = 36 doubles, so that every fragment read
// below hits 16 distinct 8-byte bank slots per half-warp. The update runs as FP64
// mma: C (8 states x 8 vectors) = a Y + (X1 tile) (s1 M1 tile), M1's fragments held
// in registers; C goes back into the Y panel (the X1 panel if a = 0), with M2 through
// a second product; the Gram fragments read the panels, and the result goes out with
// coalesced 16-byte stores. Rows and columns of a Gram tile from P on hold copies
// of others and are not used.
//
// The grid, two CTAs of four warps per SM, fixes the order of the Gram sums and is
// kept. With two warps per scheduler the kernel is bound by the instructions of a
// tile and their latency, not by memory (ncu: 554 a tile at 0.4 per cycle and
// scheduler, L2 at a fifth of its rate, with P = 8 for p = 4 and addresses formed anew
// for each chunk), hence a kernel per combination of blocks, pointers kept per
// lane, a path without range checks for whole tiles, and no barrier between the four
// products of a tile. For 731,808 states and p = 4: 10.3 us reading one block, 13.9 two,
// 15.4 three, where the former kernel took 24 us on average.
constexpr int kPanelLd = 36;
constexpr int kPipeWarps = 4;
constexpr int kPipeThreads = 32 * kPipeWarps;
constexpr size_t kPipeSmem = 112 * 1024;  // per CTA, two CTAs per SM

// Stages of panels that two CTAs per SM have room for
__host__ __device__ constexpr int pipe_stages(int P, int npanel) {
  const int fit = (int)(kPipeSmem / ((size_t)kPipeWarps * npanel * P * kPanelLd * sizeof(double)));
  return fit > 4 ? 4 : fit;
}
__host__ __device__ constexpr size_t pipe_smem(int P, int npanel) {
  const size_t panels = (size_t)kPipeWarps * pipe_stages(P, npanel) * npanel * P * kPanelLd * sizeof(double);
  const size_t grams = (size_t)kPipeWarps * 256 * sizeof(double);
  return panels > grams ? panels : grams;
}
static_assert(pipe_stages(16, 3) >= 2, "a stage to compute on and one in flight");

__device__ __forceinline__ void cp_async16(void *dst, const void *src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// A block's vectors as one lane copies them: chunk q = lane + 32 r of a tile holds
// vector q / 16, states 2 (q % 16) and 2 (q % 16) + 1 of the tile.
template <int P, class T>
struct LaneRows {
  T *v[P / 2];
  template <class B>
  __device__ __forceinline__ LaneRows(const B &V, int p, int lane) {
#pragma unroll
    for (int r = 0; r < P / 2; ++r) {  // lanes 0-15 vector 2r, lanes 16-31 vector 2r + 1
      T *w = (lane >> 4) ? V.v[2 * r + 1] : V.v[2 * r];
      v[r] = 2 * r + (lane >> 4) < p ? w + 2 * (lane & 15) : nullptr;
    }
  }
  // into a panel (dst: the lane's place in it), zero-filled past D
  __device__ __forceinline__ void load(double *dst, size_t I0, size_t D, int lane) const {
    if (I0 + 32 <= D) {
#pragma unroll
      for (int r = 0; r < P / 2; ++r)
        if (v[r]) cp_async16(dst + 2 * r * kPanelLd, v[r] + I0, 16);
    } else {
      const size_t I = I0 + 2 * (lane & 15);  // D is even: a chunk is all in or all out
#pragma unroll
      for (int r = 0; r < P / 2; ++r)
        if (v[r]) cp_async16(dst + 2 * r * kPanelLd, I < D ? v[r] + I0 : v[r] - 2 * (lane & 15), I < D ? 16 : 0);
    }
  }
  __device__ __forceinline__ void store(const double *src, size_t I0, size_t D, int lane) const {
    const bool in = I0 + 2 * (lane & 15) < D;
#pragma unroll
    for (int r = 0; r < P / 2; ++r)
      if (v[r] && in)
        *reinterpret_cast<double2 *>(v[r] + I0) = *reinterpret_cast<const double2 *>(src + 2 * r * kPanelLd);
  }
};

// UPD: X1 M1 is added; RDY: Y is read (a != 0); USEL: Gram matrix with L (gram 2)
template <int P, bool UPD, bool RDY, bool USEL>
__global__ void __launch_bounds__(kPipeThreads) k_bl_pipe(size_t D, int p, double a, BlockOut Y, double s1,
                                                          BlockIn X1, const double *__restrict__ M1,
                                                          const double *__restrict__ M2, bool keep, int gram,
                                                          BlockIn L, double *partials) {
  pdl_begin();
  constexpr int NT = (P + 7) / 8;  // 8-vector tiles
  constexpr int KS = P / 4;        // k steps of the update
  constexpr int PANEL = P * kPanelLd;
  constexpr int NP = (int)UPD + (int)RDY + (int)USEL;
  constexpr int S = pipe_stages(P, NP);
  constexpr int OUT = UPD && RDY ? PANEL : 0;  // the panel of Y, X1's if Y is not read
  extern __shared__ double smem_pipe[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool change = UPD || a != 1.0;
  double *base = smem_pipe + warp * (S * NP * PANEL);
  for (int i = lane; i < S * NP * PANEL; i += 32) base[i] = 0.0;
  __syncwarp();
  const LaneRows<P, const double> xin(X1, UPD ? p : 0, lane), lin(L, USEL ? p : 0, lane);
  const LaneRows<P, double> yio(Y, p, lane);
  const int mine = (lane >> 4) * kPanelLd + 2 * (lane & 15);  // the lane's chunk in a panel
  // M1, M2 as B fragments: row k = input vector, column n = output vector
  double bm[KS][NT], bm2[KS][NT];
#pragma unroll
  for (int ks = 0; ks < KS; ++ks)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const int i = 4 * ks + (lane & 3), c = 8 * nt + (lane >> 2);
      bm[ks][nt] = (UPD && i < p && c < p) ? s1 * M1[i * p + c] : 0.0;
      bm2[ks][nt] = (UPD && M2 && i < p && c < p) ? M2[i * p + c] : 0.0;
    }
  const int xrow = (lane & 3) * kPanelLd + (lane >> 2);      // A fragment: vector, state
  const int crow = 2 * (lane & 3) * kPanelLd + (lane >> 2);  // C fragment: first vector, state
  int grow[NT];                                              // Gram fragments: vector, state
#pragma unroll
  for (int u = 0; u < NT; ++u) {
    const int v = 8 * u + (lane >> 2);
    grow[u] = (v < P ? v : v - 4) * kPanelLd + (lane & 3);
  }
  double g[NT * NT][2];
#pragma unroll
  for (int q = 0; q < NT * NT; ++q) g[q][0] = g[q][1] = 0.0;
  const size_t ntile = (D + 31) / 32;
  const size_t nw = (size_t)gridDim.x * kPipeWarps;
  const size_t t0 = (size_t)blockIdx.x * kPipeWarps + warp;
  auto issue = [&](size_t tt, double *panels) {
    if (tt < ntile) {
      if (UPD) xin.load(panels + mine, tt * 32, D, lane);
      if (RDY) yio.load(panels + OUT + mine, tt * 32, D, lane);
      if (USEL) lin.load(panels + (NP - 1) * PANEL + mine, tt * 32, D, lane);
    }
    cp_async_commit();  // one group per tile, empty past the end
  };
#pragma unroll
  for (int q = 0; q < S - 1; ++q) issue(t0 + q * nw, base + q * NP * PANEL);
  double *cur = base, *ahead = base + (S - 1) * NP * PANEL;
  for (size_t t = t0; t < ntile; t += nw) {
    issue(t + (S - 1) * nw, ahead);
    cp_async_wait<S - 1>();
    __syncwarp();
    double *X = cur, *Yp = cur + OUT;
    if (change) {
      // C = a Y + X (s1 M1), 4 tiles of 8 states x NT tiles of 8 vectors
      double c[4][NT][2];
#pragma unroll
      for (int mt = 0; mt < 4; ++mt) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int j = 0; j < 2; ++j)
            c[mt][nt][j] =
                RDY && 8 * nt + 2 * (lane & 3) < P ? a * Yp[crow + (8 * nt + j) * kPanelLd + 8 * mt] : 0.0;
        if (UPD) {
#pragma unroll
          for (int ks = 0; ks < KS; ++ks) {
            const double af = X[xrow + 4 * ks * kPanelLd + 8 * mt];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) mma_f64(c[mt][nt][0], c[mt][nt][1], af, bm[ks][nt]);
          }
        }
      }
      auto put = [&]() {
        __syncwarp();  // every lane has read its fragments
#pragma unroll
        for (int mt = 0; mt < 4; ++mt)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int j = 0; j < 2; ++j)
              if (8 * nt + 2 * (lane & 3) < P) Yp[crow + (8 * nt + j) * kPanelLd + 8 * mt] = c[mt][nt][j];
        __syncwarp();
      };
      put();
      if (UPD && M2) {
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) c[mt][nt][0] = c[mt][nt][1] = 0.0;
#pragma unroll
          for (int ks = 0; ks < KS; ++ks) {
            const double af = Yp[xrow + 4 * ks * kPanelLd + 8 * mt];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) mma_f64(c[mt][nt][0], c[mt][nt][1], af, bm2[ks][nt]);
          }
        }
        put();
      }
    }
    if (gram) {
      // G += L^T Y' over the tile's 32 states
      const double *Lp = USEL ? cur + (NP - 1) * PANEL : Yp;
#pragma unroll
      for (int k0 = 0; k0 < 32; k0 += 4) {
        double af[NT], bf[NT];
#pragma unroll
        for (int u = 0; u < NT; ++u) {
          bf[u] = Yp[grow[u] + k0];
          af[u] = USEL ? Lp[grow[u] + k0] : bf[u];
        }
#pragma unroll
        for (int mt = 0; mt < NT; ++mt)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) mma_f64(g[mt * NT + nt][0], g[mt * NT + nt][1], af[mt], bf[nt]);
      }
    }
    if (change && keep) yio.store(Yp + mine, t * 32, D, lane);
    __syncwarp();  // the stage is free for a later tile
    ahead = cur;
    cur += NP * PANEL;
    if (cur == base + S * NP * PANEL) cur = base;
  }
  if (!gram) return;
  __syncthreads();
  double *red = smem_pipe;  // [warp][16 * 16], over the panels (all warps are done with them)
#pragma unroll
  for (int mt = 0; mt < NT; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int j = 0; j < 2; ++j)
        red[warp * 256 + (mt * 8 + (lane >> 2)) * 16 + nt * 8 + 2 * (lane & 3) + j] = g[mt * NT + nt][j];
  __syncthreads();
  for (int u = threadIdx.x; u < p * p; u += blockDim.x) {
    const int i = u / p, c = u % p;
    double s = 0.0;
    for (int w = 0; w < kPipeWarps; ++w) s += red[w * 256 + i * 16 + c];
    partials[(size_t)blockIdx.x * p * p + u] = s;
  }
}

template <int P, bool UPD, bool RDY, bool USEL, class... A>
void launch_pipe(size_t D, int grid, cudaStream_t s, A &&...args) {
  constexpr size_t smem = pipe_smem(P, (int)UPD + (int)RDY + (int)USEL);
  static const bool attr = [] {
    QED_CUDA(cudaFuncSetAttribute(k_bl_pipe<P, UPD, RDY, USEL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem));
    return true;
  }();
  (void)attr;
  launch_pdl(D, k_bl_pipe<P, UPD, RDY, USEL>, grid, kPipeThreads, smem, s, D, args...);
}

template <int P, class... A>
void launch_pipe_for(bool upd, bool rdy, bool usel, A &&...args) {
  if (upd && rdy) usel ? launch_pipe<P, true, true, true>(args...) : launch_pipe<P, true, true, false>(args...);
  else if (upd) usel ? launch_pipe<P, true, false, true>(args...) : launch_pipe<P, true, false, false>(args...);
  else usel ? launch_pipe<P, false, true, true>(args...) : launch_pipe<P, false, true, false>(args...);
}

}  // namespace

int launch_bl_update(size_t D, int p, double a, const BlockOut &Y, double s1, const BlockIn &X1, const double *M1,
                     int gram, const BlockIn &L, double *partials, int max_blocks, cudaStream_t s, const double *M2,
                     bool keep) {
  if (p < 1 || p > 16) fail(QED_ERR_ARGUMENT, "block update: block size outside [1, 16]");
  if (!D) return 0;
  static const int sms = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 148;
  }();
  const size_t want = (D + kBlThreads - 1) / kBlThreads;
  int grid = (int)std::min<size_t>(want, (size_t)sms * 2);
  if (gram && grid > max_blocks) grid = max_blocks;
  grid = std::max(grid, 1);
  // the pipelined form needs 16-byte aligned vectors (D even, aligned bases) and
  // something to read
  bool pipe = D % 2 == 0 && (a != 0.0 || X1.v[0]);
  for (int c = 0; c < p; ++c) {
    if ((uintptr_t)Y.v[c] & 15u) pipe = false;
    if (X1.v[0] && ((uintptr_t)X1.v[c] & 15u)) pipe = false;
    if (gram == 2 && ((uintptr_t)L.v[c] & 15u)) pipe = false;
  }
  if (pipe) {
    const size_t tiles = (D + 31) / 32;
    // two CTAs per SM fit (shared memory); the warps stride over the tiles
    int g2 = (int)std::min<size_t>((tiles + kPipeWarps - 1) / kPipeWarps, (size_t)sms * 2);
    if (gram && g2 > max_blocks) g2 = max_blocks;
    g2 = std::max(g2, 1);
    const bool upd = X1.v[0] != nullptr, rdy = a != 0.0, usel = gram == 2;
    if (p <= 4) launch_pipe_for<4>(upd, rdy, usel, D, g2, s, p, a, Y, s1, X1, M1, M2, keep, gram, L, partials);
    else if (p <= 8) launch_pipe_for<8>(upd, rdy, usel, D, g2, s, p, a, Y, s1, X1, M1, M2, keep, gram, L, partials);
    else if (p <= 12) launch_pipe_for<12>(upd, rdy, usel, D, g2, s, p, a, Y, s1, X1, M1, M2, keep, gram, L, partials);
    else launch_pipe_for<16>(upd, rdy, usel, D, g2, s, p, a, Y, s1, X1, M1, M2, keep, gram, L, partials);
    return g2;
  }
  auto smem = [](int P) { return (size_t)(2 * P * P + kBlWarps * 2 * 32 * kStageLd) * sizeof(double); };
  static const bool attr = [&] {
    QED_CUDA(cudaFuncSetAttribute(k_bl_simple<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem(8)));
    QED_CUDA(cudaFuncSetAttribute(k_bl_simple<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem(16)));
    return true;
  }();
  (void)attr;
  if (p <= 8)
    k_bl_simple<8><<<grid, kBlThreads, smem(8), s>>>(D, p, a, Y, s1, X1, M1, M2, keep, gram, L, partials);
  else
    k_bl_simple<16><<<grid, kBlThreads, smem(16), s>>>(D, p, a, Y, s1, X1, M1, M2, keep, gram, L, partials);
  QED_LAUNCH();
  return grid;
}

}  // namespace qed
