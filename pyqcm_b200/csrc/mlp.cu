// Surrogate network for VCA: a multilayer perceptron n_in -> W -> W -> W -> 1
// with GELU activations, trained by Adam on data this solver generates
// (Potthoff functional values at points of the variational parameters).
//
// Arithmetic: weights and activations enter the matrix products in BF16 on
// the tensor cores with FP32 accumulation; biases, pre-activations, gradients,
// the loss and Adam's master weights and moments are FP32. Every matrix
// product is one tcgen05 kernel (128 x BN tiles accumulated in tensor memory,
// operands staged in shared memory); sizes are padded to multiples of 16 (the
// input width to 16 with zero columns).
//
// One training step (forward, backward, Adam) is a fixed sequence of kernels
// on the network's stream; the steps of an epoch are captured once into a
// CUDA graph and replayed, the epoch's shuffled data being gathered into the
// same device buffers before each replay.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <random>
#include <string>
#include <type_traits>
#include <vector>

#include "common.hpp"
#include "qed_b200.h"

typedef __nv_bfloat16 bf16;

namespace qed {
namespace {

inline int pad16(int x) { return (x + 15) / 16 * 16; }

// ---- matrix products on the 5th-generation tensor cores (tcgen05) ----------
//
// One CTA of 256 threads computes a 128 x bn tile of C = A B^T (A: M x K, B: N x K,
// bf16) into a TMEM accumulator (fp32, 128 lanes x bn columns). K goes in rounds of
// 64 through kUmmaStages stages of shared memory, filled with cp.async in the
// canonical layouts without swizzle, so that an operand may be contiguous along K
// or along its own rows (the products of the backward pass, which sum over the
// batch or read W transposed): core matrices of 128 contiguous bytes, eight rows
// of eight K-elements, or eight K of eight row elements. The rounds' loads are in
// flight together; one elected thread issues a round's four 128 x bn x 16
// tcgen05.mma (kind::f16, bf16 inputs, fp32 accumulation) and commits them to the
// stage's mbarrier, on which the threads wait (bounded) before the stage is filled
// again. The epilogue reads the accumulator back with tcgen05.ld (warps w and w + 4
// hold lanes 32 w .. 32 w + 31) and finishes the layer: bias and GELU, or GELU'.
//
// At 256 x 256 x 256 (0.03 GFLOP) the latency of one chain - load, multiply, read
// back - is all there is: a training step was 32 launches with four-CTA products
// whose rounds waited for one another, 210 us for a batch of 256; with the rounds
// in flight, 32-column tiles, no transposes and the elementwise work in the
// epilogues it is eight launches and 61 us, 54 with each launch beginning as its
// predecessor ends. Every sum keeps its
// order, so that both train to the same bits.

constexpr int kUmmaM = 128;       // rows of a tile = TMEM lanes (cta_group::1)
constexpr int kUmmaBK = 64;       // K elements staged per round
constexpr int kUmmaMaxBN = 128;   // columns of a tile
constexpr int kUmmaThreads = 256;
constexpr int kUmmaStages = 4;
constexpr size_t kUmmaTileBytes = (size_t)kUmmaM * kUmmaBK * 2;
// Dynamic shared memory: kUmmaStages of both tiles. At least 72 KB, so that at most
// three CTAs share an SM (3 x 128 TMEM columns <= 512).
inline size_t umma_smem(int bn) {
  return std::max<size_t>(72 * 1024, kUmmaStages * (kUmmaTileBytes + (size_t)bn * kUmmaBK * 2));
}

// Set when a bounded wait for the tensor core gave up; read by the host.
__device__ int g_mlp_wait_timeout = 0;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor (sm_100 format): start address, leading and
// stride byte offsets (all >> 4), descriptor version 1 at bit 46, no swizzle.
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: fp32 D (bits 4-5 = 1), bf16 A and B (bits
// 7-9 and 10-12 = 1), bits 15 and 16 set for an A or B contiguous along its rows,
// N >> 3 at bit 17, M >> 4 at bit 24.
__device__ __forceinline__ uint32_t umma_idesc_bf16(int m, int n, int a_mn, int b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}

// Waits for phase `parity` of the mbarrier; gives up after about two seconds.
__device__ __forceinline__ bool umma_wait(uint64_t *bar, uint32_t parity) {
  const uint32_t a = smem_u32(bar);
  uint64_t t0 = 0;
  for (uint32_t it = 0;; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 255u) == 0) {
      uint64_t t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (it == 0) t0 = t;
      else if (t - t0 > 2000000000ull) {
        atomicExch(&g_mlp_wait_timeout, 1);
        return false;
      }
    }
  }
}

// An operand tile in shared memory: `rows` (a multiple of 16) rows by one round of
// K. mn: the source is K x rows with the rows contiguous.
struct UmmaTile {
  uint32_t lbo, sbo;  // byte strides of the core matrices (descriptor meaning)
  __device__ UmmaTile(int rows, int mn) : lbo(mn ? (uint32_t)rows / 8 * 128 : 128u), sbo(mn ? 128u : 1024u) {}
  __device__ uint32_t step() const { return 2 * lbo; }  // 16 K further
};

// Stages rows [r0, r0 + rows) x K-elements [k0, k0 + kc) of a bf16 operand
// (leading dimension ld); rows at or past `total` are zero-filled.
__device__ __forceinline__ void umma_stage(uint32_t sdst, const bf16 *src, int ld, int mn, int r0, int rows,
                                           int total, int k0, int kc) {
  if (!mn) {
    for (int c = threadIdx.x; c < rows * (kUmmaBK / 8); c += kUmmaThreads) {
      const int r = c >> 3, q = c & 7;
      if (8 * q >= kc) continue;
      const bool in = r0 + r < total;
      cp_async16(sdst + (uint32_t)(r >> 3) * 1024u + (uint32_t)q * 128u + (uint32_t)(r & 7) * 16u,
                 src + (size_t)(in ? r0 + r : 0) * ld + k0 + 8 * q, in ? 16 : 0);
    }
  } else {
    const int across = rows >> 3;
    for (int c = threadIdx.x; c < across * kc; c += kUmmaThreads) {
      const int k = c / across, q = c - k * across;
      const bool in = r0 + 8 * q < total;
      cp_async16(sdst + ((uint32_t)(k >> 3) * across + (uint32_t)q) * 128u + (uint32_t)(k & 7) * 16u,
                 src + (size_t)(k0 + k) * ld + (in ? r0 + 8 * q : 0), in ? 16 : 0);
    }
  }
}

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// One product and what its epilogue does with C (fp32, row-major, ldc):
//   kStore:    C
//   kForward:  C += bias; H = bf16(GELU(C))
//   kBackward: C *= GELU'(Z); H = bf16(C)
enum { kStore, kForward, kBackward };
struct GemmJob {
  int M = 0, N = 0, K = 0;
  const bf16 *A = nullptr, *B = nullptr;
  int lda = 0, ldb = 0, a_mn = 0, b_mn = 0;
  float *C = nullptr;
  int ldc = 0, epi = kStore;
  const float *bias = nullptr, *Z = nullptr;
  bf16 *H = nullptr;
  int bn = 16, tiles_n = 0, tiles = 0;
};

__device__ void umma_tile(const GemmJob &j, int tile, unsigned char *sm) {
  __shared__ __align__(8) uint64_t bar[kUmmaStages];
  __shared__ uint32_t tslot;
  const uint32_t sa = smem_u32(sm), sb = sa + kUmmaStages * (uint32_t)kUmmaTileBytes;
  const uint32_t b_bytes = (uint32_t)j.bn * kUmmaBK * 2;
  const int m0 = tile / j.tiles_n * kUmmaM, n0 = tile % j.tiles_n * j.bn;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ncols = j.bn <= 32 ? 32u : j.bn <= 64 ? 64u : 128u;  // a power of two >= 32
  const int rounds = (j.K + kUmmaBK - 1) / kUmmaBK;
  auto fill = [&](int r) {
    const int k0 = r * kUmmaBK, kc = min(kUmmaBK, j.K - k0), st = r % kUmmaStages;
    umma_stage(sa + st * (uint32_t)kUmmaTileBytes, j.A, j.lda, j.a_mn, m0, kUmmaM, j.M, k0, kc);
    umma_stage(sb + st * b_bytes, j.B, j.ldb, j.b_mn, n0, j.bn, j.N, k0, kc);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tslot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (threadIdx.x == 32) {
    for (int st = 0; st < kUmmaStages; ++st)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar[st])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // the previous launch's results from here on (tensor memory is taken before the
  // next launch may begin, so no two launches' tiles wait for one another's)
  pdl_begin();
  for (int r = 0; r < min(kUmmaStages, rounds); ++r) fill(r);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tslot;
  const uint32_t idesc = umma_idesc_bf16(kUmmaM, j.bn, j.a_mn, j.b_mn);
  const UmmaTile ta(kUmmaM, j.a_mn), tb(j.bn, j.b_mn);
  bool ok = true;
  for (int r = 0; r < rounds && ok; ++r) {
    const int st = r % kUmmaStages, kc = min(kUmmaBK, j.K - r * kUmmaBK);
    switch (min(rounds, r + kUmmaStages) - (r + 1)) {  // rounds that may still be in flight
      case 0: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
      case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
      case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
      default: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // visible to the tensor core's reads
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int kk = 0; kk < kc / 16; ++kk) {
        const uint64_t ad = umma_smem_desc(sa + st * (uint32_t)kUmmaTileBytes + ta.step() * (uint32_t)kk, ta.lbo, ta.sbo);
        const uint64_t bd = umma_smem_desc(sb + st * b_bytes + tb.step() * (uint32_t)kk, tb.lbo, tb.sbo);
        const uint32_t acc = (r > 0 || kk > 0) ? 1u : 0u;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
            : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(&bar[st]))
                   : "memory");
    }
    if (r + kUmmaStages < rounds) {  // the MMAs have read the stage: fill it again
      ok = __syncthreads_and(umma_wait(&bar[st], (uint32_t)(r / kUmmaStages) & 1u));
      if (ok) fill(r + kUmmaStages);
    } else if (r + 1 == rounds) {  // the last commit covers every MMA
      ok = __syncthreads_and(umma_wait(&bar[st], (uint32_t)(r / kUmmaStages) & 1u));
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (ok) {
    const int row = m0 + (warp & 3) * 32 + lane;
    for (int c0 = (warp >> 2) * 16; c0 < j.bn; c0 += 32) {
      uint32_t v[16];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
          "%14, %15}, [%16];"
          : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
            "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
          : "r"(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      const int n = n0 + c0;  // N and n are multiples of 16: the chunk is inside or outside as a whole
      if (row < j.M && n < j.N) {
        const size_t at = (size_t)row * j.ldc + n;
        float c[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) c[q] = 0.0f + __uint_as_float(v[q]);
        if (j.epi == kForward) {
#pragma unroll
          for (int q = 0; q < 16; ++q) c[q] = c[q] + j.bias[n + q];
        } else if (j.epi == kBackward) {
#pragma unroll
          for (int q = 0; q < 16; ++q) c[q] = c[q] * gelu_grad(j.Z[at + q]);
        }
#pragma unroll
        for (int q = 0; q < 16; q += 4)
          *reinterpret_cast<float4 *>(j.C + at + q) = make_float4(c[q], c[q + 1], c[q + 2], c[q + 3]);
        if (j.epi != kStore) {
          __align__(16) bf16 h[16];
#pragma unroll
          for (int q = 0; q < 16; ++q) h[q] = __float2bfloat16_rn(j.epi == kForward ? gelu(c[q]) : c[q]);
          reinterpret_cast<uint4 *>(j.H + at)[0] = reinterpret_cast<const uint4 *>(h)[0];
          reinterpret_cast<uint4 *>(j.H + at)[1] = reinterpret_cast<const uint4 *>(h)[1];
        }
      }
    }
  } else {
    for (int st = 0; st < kUmmaStages; ++st)  // commits still in flight have their bounded chance to land
      if (st < rounds) umma_wait(&bar[st], (uint32_t)((rounds - 1 - st) / kUmmaStages) & 1u);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
}

// out[f] = sum_b w[b] X[b][f] over rows b in order (w null: 1), F columns of an
// fp32 or bf16 matrix: a CTA takes 32 columns, stages 256 rows at a time in shared
// memory and a thread per column adds them up (the order of the sums is the rows',
// so only the loads can be spread).
struct ColJob {
  int rows = 0, F = 0;
  const float *X = nullptr;
  const bf16 *Xh = nullptr;
  const float *w = nullptr;
  float *out = nullptr;
  int ctas = 0;  // 0: no job
};
constexpr int kColRows = 256;

__device__ void column_sums(const ColJob &j, int cta, float *sm) {
  pdl_begin();
  const int f0 = cta * 32, lane = threadIdx.x & 31, f = f0 + lane;
  float *wr = sm + kColRows * 32;
  float s = 0.0f;
  for (int b0 = 0; b0 < j.rows; b0 += kColRows) {
    const int n = min(kColRows, j.rows - b0);
    if (b0) __syncthreads();
    constexpr int kWarps = kUmmaThreads / 32, kPer = kColRows / kWarps;
    float v[kPer];  // every load of the block of rows before the first store
    const size_t at = (size_t)(b0 + (int)(threadIdx.x >> 5)) * j.F + f;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const bool in = f < j.F && (int)(threadIdx.x >> 5) + q * kWarps < n;
      const size_t a = at + (size_t)q * kWarps * j.F;
      v[q] = !in ? 0.0f : (j.Xh ? __bfloat162float(j.Xh[a]) : j.X[a]);
    }
#pragma unroll
    for (int q = 0; q < kPer; ++q) sm[((threadIdx.x >> 5) + q * kWarps) * 32 + lane] = v[q];
    if ((int)threadIdx.x < n) wr[threadIdx.x] = j.w ? j.w[b0 + threadIdx.x] : 1.0f;
    __syncthreads();
    if (threadIdx.x < 32 && f < j.F) {
#pragma unroll 16
      for (int r = 0; r < n; ++r) s = fmaf(sm[r * 32 + lane], wr[r], s);
    }
  }
  if (threadIdx.x < 32 && f < j.F) j.out[f] = s;
}

// The products and column sums of one stage of the network (all independent).
struct StageJobs {
  GemmJob g[2];
  ColJob c[3];
};
__global__ void __launch_bounds__(kUmmaThreads) k_mlp_stage(const __grid_constant__ StageJobs jobs) {
  extern __shared__ __align__(1024) unsigned char sm[];
  int cta = blockIdx.x;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (cta < jobs.g[i].tiles) {
      umma_tile(jobs.g[i], cta, sm);
      return;
    }
    cta -= jobs.g[i].tiles;
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if (cta < jobs.c[i].ctas) {
      column_sums(jobs.c[i], cta, reinterpret_cast<float *>(sm));
      return;
    }
    cta -= jobs.c[i].ctas;
  }
}

void umma_setup() {
  static bool done = false;  // the attribute is per function, once per process is enough
  if (!done) {
    QED_CUDA(cudaFuncSetAttribute(k_mlp_stage, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)umma_smem(kUmmaMaxBN)));
    done = true;
  }
}

// Fails the call if a product's bounded wait for the tensor core gave up since
// the last check (the flag is cleared for the next call).
void check_umma_wait(cudaStream_t s) {
  int flag = 0;
  QED_CUDA(cudaStreamSynchronize(s));
  QED_CUDA(cudaMemcpyFromSymbol(&flag, g_mlp_wait_timeout, sizeof(int)));
  if (flag) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_mlp_wait_timeout, &zero, sizeof(int));
    fail(QED_ERR_CUDA, "mlp: a tensor-core product timed out waiting for its MMAs");
  }
}

// The product C = A B^T of one stage: checked, with its tile width - the widest
// that still gives every SM a tile, at least 32 columns (256 x 256 x 256 in 16
// tiles of 32 columns; 4 of 128 left 144 SMs idle).
GemmJob gemm_job(int M, int N, int K, const bf16 *A, int lda, bool a_mn, const bf16 *B, int ldb, bool b_mn, float *C,
                 int ldc) {
  if (M <= 0 || N <= 0 || K <= 0 || K % 16 || N % 16 || lda % 8 || ldb % 8)
    fail(QED_ERR_ARGUMENT, "mlp: tensor-core product needs K and N multiples of 16 and 16-byte rows");
  GemmJob j;
  j.M = M;
  j.N = N;
  j.K = K;
  j.A = A;
  j.lda = lda;
  j.a_mn = a_mn;
  j.B = B;
  j.ldb = ldb;
  j.b_mn = b_mn;
  j.C = C;
  j.ldc = ldc;
  const int tiles_m = (M + kUmmaM - 1) / kUmmaM;
  j.bn = std::min(N, kUmmaMaxBN);
  while (j.bn >= 64 && j.bn % 32 == 0 && tiles_m * ((N + j.bn - 1) / j.bn) < 148) j.bn /= 2;
  j.tiles_n = (N + j.bn - 1) / j.bn;
  j.tiles = tiles_m * j.tiles_n;
  return j;
}

ColJob col_job(int rows, int F, const float *X, const bf16 *Xh, const float *w, float *out) {
  return {rows, F, X, Xh, w, out, (F + 31) / 32};
}

void run_stage(const StageJobs &jobs, cudaStream_t s) {
  size_t smem = (kColRows * 32 + kColRows) * sizeof(float);
  int grid = 0;
  for (const GemmJob &j : jobs.g) {
    if (j.tiles) smem = std::max(smem, umma_smem(j.bn));
    grid += j.tiles;
  }
  for (const ColJob &j : jobs.c) grid += j.ctas;
  launch_pdl(0, k_mlp_stage, grid, kUmmaThreads, smem, s, jobs);
}

// The output layer, one warp per row b: y = sum_k H[b][k] w[k] + b0 (fp32
// accumulation) and, with targets, the loss terms (y - t)^2 / n, dy = 2 (y - t) / n
// and dZ[b][k] = dy w[k] GELU'(Z[b][k]) (fp32 and bf16 copies). step, if given, is
// the optimiser's step count, advanced here once per training step.
__global__ void k_head(int rows, int F, const bf16 *H, const bf16 *w, const float *b0, float *y, const float *t,
                       float *dy, float *loss_terms, const float *Z, float *dZ, bf16 *dZh, int *step) {
  pdl_begin();
  if (step && blockIdx.x == 0 && threadIdx.x == 0) *step += 1;
  const int b = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x % 32;
  if (b >= rows) return;
  float s = 0.0f;
  for (int k = lane; k < F; k += 32) s += __bfloat162float(H[(size_t)b * F + k]) * __bfloat162float(w[k]);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const float yb = s + b0[0];
  if (lane == 0) y[b] = yb;
  if (!t) return;
  const float d = yb - t[b];
  const float g = 2.0f * d / rows;
  if (lane == 0) {
    dy[b] = g;
    loss_terms[b] = d * d / rows;
  }
  for (int k = lane; k < F; k += 32) {
    const size_t at = (size_t)b * F + k;
    const float z = g * __bfloat162float(w[k]) * gelu_grad(Z[at]);
    dZ[at] = z;
    dZh[at] = __float2bfloat16_rn(z);
  }
}

// Adam (Kingma & Ba 2015, Algorithm 1) on fp32 master weights; the step count
// lives on the device so that a captured step can be replayed.
__global__ void k_adam(int n, float *w, const float *g, float *m, float *v, bf16 *wh, const int *step, float lr,
                       float b1, float b2, float eps, const unsigned char *mask) {
  pdl_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (mask && !mask[i]) return;  // padding stays zero
  const int t = *step;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.0f - b1) * gi;
  const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float mh = mi / (1.0f - powf(b1, (float)t)), vh = vi / (1.0f - powf(b2, (float)t));
  const float wi = w[i] - lr * mh / (sqrtf(vh) + eps);
  w[i] = wi;
  if (wh) wh[i] = __float2bfloat16_rn(wi);
}

__global__ void k_to_bf16(int n, const float *x, bf16 *y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = __float2bfloat16_rn(x[i]);
}

// gather rows (and pad the input width with zeros): X[b][0..n_in) -> Xp[b][0..ld)
__global__ void k_gather(int rows, int n_in, int ld, const float *X, const float *T, const int *perm, bf16 *Xp,
                         float *Tp) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= rows) return;
  const int src = perm ? perm[b] : b;
  for (int j = 0; j < ld; ++j) Xp[(size_t)b * ld + j] = __float2bfloat16_rn(j < n_in ? X[(size_t)src * n_in + j] : 0.0f);
  if (T) Tp[b] = T[src];
}

// CTAs of a kernel with a thread per element
inline int blocks_for(size_t n, int threads = 256) { return (int)std::max<size_t>((n + threads - 1) / threads, 1); }

}  // namespace

// ------------------------------------------------------------------ network --

struct MLP {
  int n_in = 0, k_in = 0, W = 0, L = 3;  // L hidden layers of width W
  cudaStream_t s = nullptr;
  // parameters (fp32 master) in one buffer: W1 [W][k_in], b1 [W], W2 [W][W], b2, W3 [W][W], b3, w4 [W], b4 [1]
  std::vector<size_t> off;  // offsets of the 8 parameter blocks
  size_t n_par = 0;
  DevBuf<float> p, g, m, v;
  DevBuf<bf16> ph;              // bf16 copy for the products
  DevBuf<unsigned char> mask;   // 0 on the input-width padding of W1
  DevBuf<int> step;
  // activations for a batch of `cap` rows
  int cap = 0;
  DevBuf<bf16> X, H[3], dZh[3];
  DevBuf<float> T, Z[3], dZ[3], y, dy, lt;
  DevBuf<int> perm;
  DevBuf<float> data_x, data_t;
  int n_data = 0;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int graph_batch = 0, graph_steps = 0;
  float graph_lr = 0.0f;

  ~MLP() {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    if (s) {
      cudaStreamSynchronize(s);
      cudaStreamDestroy(s);
    }
  }

  float *P(int i) { return p.p + off[i]; }
  bf16 *Ph(int i) { return ph.p + off[i]; }
  float *Gr(int i) { return g.p + off[i]; }

  void init(int nin, int width, uint64_t seed) {
    if (nin < 1 || nin > 16) fail(QED_ERR_ARGUMENT, "mlp: input width must be in [1, 16]");
    if (width < 16 || width % 16) fail(QED_ERR_ARGUMENT, "mlp: hidden width must be a positive multiple of 16");
    n_in = nin;
    k_in = pad16(nin);
    W = width;
    QED_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    umma_setup();
    const size_t sizes[8] = {(size_t)W * k_in, (size_t)W, (size_t)W * W, (size_t)W, (size_t)W * W, (size_t)W,
                             (size_t)W, 16};
    off.resize(8);
    size_t o = 0;
    for (int i = 0; i < 8; ++i) {
      off[i] = o;
      o += (sizes[i] + 15) / 16 * 16;  // 32-byte aligned blocks for the bf16 tiles
    }
    n_par = o;
    // He-style uniform init for the weights, zero biases (seeded)
    std::vector<float> h(n_par, 0.0f);
    std::vector<unsigned char> mk(n_par, 1);
    std::mt19937_64 rng(seed);
    auto fill = [&](int blk, int rows, int cols, int fan_in, int ld) {
      std::uniform_real_distribution<float> U(-1.0f, 1.0f);
      const float a = std::sqrt(3.0f / (float)fan_in);
      for (int r = 0; r < rows; ++r)
        for (int c = 0; c < ld; ++c) {
          const size_t i = off[blk] + (size_t)r * ld + c;
          if (c < cols) h[i] = a * U(rng);
          else mk[i] = 0;
        }
    };
    fill(0, W, n_in, n_in, k_in);
    fill(2, W, W, W, W);
    fill(4, W, W, W, W);
    fill(6, 1, W, W, W);
    for (size_t i = off[7] + 1; i < n_par; ++i) mk[i] = 0;
    p.alloc(n_par);
    g.alloc(n_par);
    m.alloc(n_par);
    v.alloc(n_par);
    ph.alloc(n_par);
    mask.alloc(n_par);
    step.alloc(1);
    QED_CUDA(cudaMemcpyAsync(p.p, h.data(), n_par * sizeof(float), cudaMemcpyHostToDevice, s));
    QED_CUDA(cudaMemcpyAsync(mask.p, mk.data(), n_par, cudaMemcpyHostToDevice, s));
    QED_CUDA(cudaMemsetAsync(g.p, 0, n_par * sizeof(float), s));
    QED_CUDA(cudaMemsetAsync(m.p, 0, n_par * sizeof(float), s));
    QED_CUDA(cudaMemsetAsync(v.p, 0, n_par * sizeof(float), s));
    QED_CUDA(cudaMemsetAsync(step.p, 0, sizeof(int), s));
    sync_bf16();
  }

  void sync_bf16() {
    k_to_bf16<<<blocks_for(n_par), 256, 0, s>>>((int)n_par, p.p, ph.p);
    QED_LAUNCH();
    QED_CUDA(cudaStreamSynchronize(s));
  }

  void reserve(int rows) {
    rows = pad16(rows);
    if (rows <= cap) return;
    if (exec) {
      cudaGraphExecDestroy(exec);
      exec = nullptr;
    }
    if (graph) {
      cudaGraphDestroy(graph);
      graph = nullptr;
    }
    cap = rows;
    X.alloc((size_t)cap * k_in);
    T.alloc(cap);
    for (int l = 0; l < 3; ++l) {
      H[l].alloc((size_t)cap * W);
      dZh[l].alloc((size_t)cap * W);
      Z[l].alloc((size_t)cap * W);
      dZ[l].alloc((size_t)cap * W);
    }
    y.alloc(cap);
    dy.alloc(cap);
    lt.alloc(cap);
  }

  // hidden layers on rows [0, rows) of X (bf16, padded)
  void hidden(int rows) {
    for (int l = 0; l < 3; ++l) {
      const int kin = l ? W : k_in;
      StageJobs st;
      GemmJob &j = st.g[0];
      j = gemm_job(rows, W, kin, l ? H[l - 1].p : X.p, kin, false, Ph(2 * l), kin, false, Z[l].p, W);
      j.epi = kForward;
      j.bias = P(2 * l + 1);
      j.H = H[l].p;
      run_stage(st, s);
    }
  }

  // y = network output
  void forward(int rows) {
    hidden(rows);
    launch_pdl(0, k_head, (rows * 32 + 255) / 256, 256, 0, s, rows, W, H[2].p, Ph(6), P(7), y.p, nullptr, nullptr, nullptr,
                                                  nullptr, nullptr, nullptr, nullptr);
    QED_LAUNCH();
  }

  // forward and the gradients of the mean squared error over rows [0, rows) into g.
  // Three launches forward, the output layer, and one per layer backward: dW_l =
  // dZ_l^T prev, db_l and dZ_{l-1} = dZ_l W_l GELU'(Z_{l-1}) all read dZ_l only.
  void gradients(int rows, bool training) {
    hidden(rows);
    launch_pdl(0, k_head, (rows * 32 + 255) / 256, 256, 0, s, rows, W, H[2].p, Ph(6), P(7), y.p, T.p, dy.p, lt.p, Z[2].p,
                                                  dZ[2].p, dZh[2].p, training ? step.p : nullptr);
    QED_LAUNCH();
    for (int l = 2; l >= 0; --l) {
      const int kin = l ? W : k_in;
      StageJobs st;
      if (l > 0) {
        GemmJob &j = st.g[0];
        j = gemm_job(rows, W, W, dZh[l].p, W, false, Ph(2 * l), W, true, dZ[l - 1].p, W);
        j.epi = kBackward;
        j.Z = Z[l - 1].p;
        j.H = dZh[l - 1].p;
      }
      st.g[1] = gemm_job(W, kin, rows, dZh[l].p, W, true, l ? H[l - 1].p : X.p, kin, true, Gr(2 * l), kin);
      st.c[0] = col_job(rows, W, dZ[l].p, nullptr, nullptr, Gr(2 * l + 1));
      if (l == 2) {  // the output layer's weights and bias
        st.c[1] = col_job(rows, W, nullptr, H[2].p, dy.p, Gr(6));
        st.c[2] = col_job(rows, 1, dy.p, nullptr, nullptr, Gr(7));
      }
      run_stage(st, s);
    }
  }

  void adam(float lr) {
    launch_pdl(0, k_adam, blocks_for(n_par), 256, 0, s, (int)n_par, p.p, g.p, m.p, v.p, ph.p, step.p, lr, 0.9f, 0.999f,
                                              1e-8f, mask.p);
    QED_LAUNCH();
  }

  void load_rows(int rows, const float *hx, const float *ht) {
    reserve(rows);
    DevBuf<float> dx((size_t)rows * n_in), dt(ht ? rows : 1);
    dx.upload(hx, (size_t)rows * n_in, s);
    if (ht) dt.upload(ht, rows, s);
    k_gather<<<(rows + 255) / 256, 256, 0, s>>>(rows, n_in, k_in, dx.p, ht ? dt.p : nullptr, nullptr, X.p, T.p);
    QED_LAUNCH();
    QED_CUDA(cudaStreamSynchronize(s));
  }
};

}  // namespace qed

using qed::MLP;

namespace {
thread_local std::string t_mlp_err;

template <class F> int mlp_guarded(F &&f) {
  try {
    f();
    return QED_OK;
  } catch (const qed::Error &e) {
    t_mlp_err = e.what();
    return e.code;
  } catch (const std::exception &e) {
    t_mlp_err = e.what();
    return QED_ERR_INTERNAL;
  }
}
}  // namespace

extern "C" {

int qed_mlp_last_error(char *buf, int len) {
  if (buf && len > 0) {
    std::strncpy(buf, t_mlp_err.c_str(), (size_t)len - 1);
    buf[len - 1] = 0;
  }
  return (int)t_mlp_err.size();
}

int qed_mlp_create(int n_in, int width, unsigned long long seed, void **handle) {
  return mlp_guarded([&] {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) qed::fail(QED_ERR_NO_DEVICE, "mlp: no CUDA device available");
    auto h = std::make_unique<MLP>();
    h->init(n_in, width, seed);
    *handle = h.release();
  });
}

void qed_mlp_destroy(void *handle) { delete static_cast<MLP *>(handle); }

int qed_mlp_num_params(void *handle, long *n) {
  return mlp_guarded([&] { *n = (long)static_cast<MLP *>(handle)->n_par; });
}

int qed_mlp_get_params(void *handle, float *out) {
  return mlp_guarded([&] {
    MLP &h = *static_cast<MLP *>(handle);
    QED_CUDA(cudaMemcpyAsync(out, h.p.p, h.n_par * sizeof(float), cudaMemcpyDeviceToHost, h.s));
    QED_CUDA(cudaStreamSynchronize(h.s));
  });
}

int qed_mlp_set_params(void *handle, const float *in) {
  return mlp_guarded([&] {
    MLP &h = *static_cast<MLP *>(handle);
    QED_CUDA(cudaMemcpyAsync(h.p.p, in, h.n_par * sizeof(float), cudaMemcpyHostToDevice, h.s));
    h.sync_bf16();
  });
}

int qed_mlp_layout(void *handle, long *offsets) {
  return mlp_guarded([&] {
    MLP &h = *static_cast<MLP *>(handle);
    for (int i = 0; i < 8; ++i) offsets[i] = (long)h.off[i];
    offsets[8] = h.k_in;
  });
}

int qed_mlp_forward(void *handle, int rows, const float *x, float *y) {
  return mlp_guarded([&] {
    MLP &h = *static_cast<MLP *>(handle);
    if (rows <= 0) return;
    h.load_rows(rows, x, nullptr);
    h.forward(qed::pad16(rows));
    QED_CUDA(cudaMemcpyAsync(y, h.y.p, rows * sizeof(float), cudaMemcpyDeviceToHost, h.s));
    qed::check_umma_wait(h.s);
  });
}

int qed_mlp_gradients(void *handle, int rows, const float *x, const float *t, float *grads, float *loss) {
  return mlp_guarded([&] {
    MLP &h = *static_cast<MLP *>(handle);
    if (rows <= 0 || rows % 16) qed::fail(QED_ERR_ARGUMENT, "mlp: gradient batches are a positive multiple of 16 rows");
    h.load_rows(rows, x, t);
    h.gradients(rows, false);
    std::vector<float> lt(rows);
    QED_CUDA(cudaMemcpyAsync(grads, h.g.p, h.n_par * sizeof(float), cudaMemcpyDeviceToHost, h.s));
    QED_CUDA(cudaMemcpyAsync(lt.data(), h.lt.p, rows * sizeof(float), cudaMemcpyDeviceToHost, h.s));
    qed::check_umma_wait(h.s);
    double L = 0.0;
    for (float v : lt) L += v;
    *loss = (float)L;
  });
}

int qed_mlp_train(void *handle, int rows, const float *x, const float *t, int epochs, int batch, float lr,
                  unsigned long long seed, float *epoch_loss) {
  return mlp_guarded([&] {
    MLP &h = *static_cast<MLP *>(handle);
    if (batch <= 0 || batch % 16) qed::fail(QED_ERR_ARGUMENT, "mlp: batch must be a positive multiple of 16");
    const int steps = rows / batch;
    if (steps < 1) qed::fail(QED_ERR_ARGUMENT, "mlp: fewer rows than one batch");
    const int used = steps * batch;
    h.reserve(used);
    h.data_x.alloc((size_t)rows * h.n_in);
    h.data_t.alloc(rows);
    h.perm.alloc(used);
    h.data_x.upload(x, (size_t)rows * h.n_in, h.s);
    h.data_t.upload(t, rows, h.s);
    // one epoch = `steps` optimiser steps on consecutive batches of the gathered rows
    if (!h.exec || h.graph_batch != batch || h.graph_steps != steps || h.graph_lr != lr) {
      if (h.exec) cudaGraphExecDestroy(h.exec);
      if (h.graph) cudaGraphDestroy(h.graph);
      h.exec = nullptr;
      h.graph = nullptr;
      QED_CUDA(cudaStreamSynchronize(h.s));
      QED_CUDA(cudaStreamBeginCapture(h.s, cudaStreamCaptureModeThreadLocal));
      bf16 *X0 = h.X.p;
      float *T0 = h.T.p;
      try {
        for (int st = 0; st < steps; ++st) {
          h.X.p = X0 + (size_t)st * batch * h.k_in;  // views into the gathered rows
          h.T.p = T0 + (size_t)st * batch;
          h.gradients(batch, true);
          h.adam(lr);
        }
      } catch (...) {
        h.X.p = X0;
        h.T.p = T0;
        cudaGraph_t broken = nullptr;
        cudaStreamEndCapture(h.s, &broken);
        if (broken) cudaGraphDestroy(broken);
        throw;
      }
      h.X.p = X0;
      h.T.p = T0;
      cudaError_t e = cudaStreamEndCapture(h.s, &h.graph);
      if (e != cudaSuccess) qed::fail(QED_ERR_CUDA, std::string("mlp: graph capture failed: ") + cudaGetErrorString(e));
      QED_CUDA(cudaGraphInstantiate(&h.exec, h.graph, 0));
      h.graph_batch = batch;
      h.graph_steps = steps;
      h.graph_lr = lr;
    }
    std::mt19937_64 rng(seed);
    std::vector<int> perm(rows);
    std::vector<float> lt(used);
    for (int ep = 0; ep < epochs; ++ep) {
      for (int i = 0; i < rows; ++i) perm[i] = i;
      std::shuffle(perm.begin(), perm.end(), rng);
      h.perm.upload(perm.data(), used, h.s);
      qed::k_gather<<<(used + 255) / 256, 256, 0, h.s>>>(used, h.n_in, h.k_in, h.data_x.p, h.data_t.p, h.perm.p,
                                                         h.X.p, h.T.p);
      QED_LAUNCH();
      QED_CUDA(cudaGraphLaunch(h.exec, h.s));
      if (epoch_loss) {  // the loss terms of the last batch of the epoch
        QED_CUDA(cudaMemcpyAsync(lt.data(), h.lt.p, batch * sizeof(float), cudaMemcpyDeviceToHost, h.s));
        qed::check_umma_wait(h.s);
        double L = 0.0;
        for (int i = 0; i < batch; ++i) L += lt[i];
        epoch_loss[ep] = (float)L;
      }
    }
    qed::check_umma_wait(h.s);
  });
}

int qed_mlp_tensor_product(int M, int N, int K, const uint16_t *A, const uint16_t *B, float *C) {
  return mlp_guarded([&] {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) qed::fail(QED_ERR_NO_DEVICE, "mlp: no CUDA device available");
    if (M <= 0 || N <= 0 || K <= 0 || K % 16 || N % 16)
      qed::fail(QED_ERR_ARGUMENT, "mlp: tensor product needs positive M and K, N multiples of 16");
    cudaStream_t s = nullptr;
    QED_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct Guard {
      cudaStream_t s;
      ~Guard() {
        cudaStreamSynchronize(s);
        cudaStreamDestroy(s);
      }
    } guard{s};
    qed::umma_setup();
    qed::DevBuf<bf16> a((size_t)M * K), b((size_t)N * K);
    qed::DevBuf<float> c((size_t)M * N);
    QED_CUDA(cudaStreamSynchronize(qed::alloc_stream()));  // the allocations are usable on s
    a.upload(reinterpret_cast<const bf16 *>(A), (size_t)M * K, s);
    b.upload(reinterpret_cast<const bf16 *>(B), (size_t)N * K, s);
    qed::StageJobs st;
    st.g[0] = qed::gemm_job(M, N, K, a.p, K, false, b.p, K, false, c.p, N);
    qed::run_stage(st, s);
    c.download(C, (size_t)M * N, s);
    qed::check_umma_wait(s);
  });
}

}  // extern "C"
