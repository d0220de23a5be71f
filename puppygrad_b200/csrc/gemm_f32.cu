// FP32 products of more rows than the decode kernels take, on the FMA units: out[m, n] = x[m, k] . w[n, k]^T.
#include <algorithm>

#include "device_util.cuh"
#include "kernels.cuh"

namespace pg {
namespace {

// A CTA makes a BM x BN tile; a thread TM x TN of it, rows BM / TM and columns BN / TN apart, with two partial sums per
// output (even and odd k) so that one instruction does two multiply-adds. Both operands lie in shared memory as they lie
// in HBM, k contiguous, four k at a time in one 16-byte read: rows are BK + 4 floats apart, which puts eight neighbouring rows
// on different banks. A ring of three stages is filled by 16-byte asynchronous copies. k may be shared out over a cluster
// (third grid dimension): the CTAs leave their sums in shared memory and each adds a slice of the tile in rank order.
//
// Bound by the FMA pipe (72 TFLOP/s nominal) where the tiles fill the chip (2048 x 4096 x 1024: 62% of its cycles, waits for it
// are the first of the stalls), else by the latency of the k loop (64 x 2304 x 768: 24%): that is what the small tiles and the shares
// of k are for.
template <int BM, int BN, int TM, int TN>
struct F32Tile {
  static constexpr int BK = 32, STRIDE = BK + 4, STAGES = 3;
  static constexpr int TY = BM / TM, TX = BN / TN, THREADS = TY * TX;
  static constexpr int STAGE_FLOATS = (BM + BN) * STRIDE;
  static constexpr size_t SMEM = STAGES * STAGE_FLOATS * sizeof(float);
  static_assert(BM * (BN + 1) <= STAGES * STAGE_FLOATS, "the sums of a tile reuse the ring");
};

__device__ __forceinline__ void copy16_or_zero(float* dst, const float* src, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

// tanh-GELU in the reference's evaluation order (src/models/cpu.rs:145-150)
__device__ __forceinline__ float gelu_tanh(float x) { return 0.5f * x * (1.0f + tanhf(0.7978846f * (x + 0.044715f * x * x * x))); }

template <int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__((F32Tile<BM, BN, TM, TN>::THREADS)) gemm_f32_kernel(LinearArgs a, int epi, int splits) {
  using T = F32Tile<BM, BN, TM, TN>;
  constexpr int BK = T::BK, STRIDE = T::STRIDE, TX = T::TX, TY = T::TY, THREADS = T::THREADS;
  extern __shared__ __align__(16) float ring[];
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int tiles_n = (a.n + BN - 1) / BN, n0 = (int)blockIdx.x % tiles_n * BN, m0 = (int)blockIdx.x / tiles_n * BM, rank = blockIdx.z;
  // this CTA's share of k, in whole blocks of BK
  const int blocks = (a.k + BK - 1) / BK, per = (blocks + splits - 1) / splits;
  const int first = rank * per, count = max(0, min(blocks, first + per) - first);

  auto fetch = [&](int block, int stage) {
    float* s = ring + stage * T::STAGE_FLOATS;
    const int k0 = (first + block) * BK;
#pragma unroll
    for (int i = tid; i < (BM + BN) * (BK / 4); i += THREADS) {
      const int r = i / (BK / 4), c = (i % (BK / 4)) * 4;
      const bool is_x = r < BM;
      const int row = is_x ? m0 + r : n0 + r - BM;
      const bool ok = k0 + c < a.k && row < (is_x ? a.m : a.n);  // k is a multiple of four: a 16-byte piece is whole or absent
      const float* src = (is_x ? a.x : a.w) + (ok ? (size_t)row * a.k + k0 + c : 0);
      copy16_or_zero(s + r * STRIDE + c, src, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  unsigned long long acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

  for (int b = 0; b < T::STAGES - 1; ++b) {
    if (b < count) fetch(b, b);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int b = 0; b < count; ++b) {
    asm volatile("cp.async.wait_group %0;" ::"n"(T::STAGES - 2) : "memory");
    __syncthreads();  // block b has arrived; the stage that is filled next was read in the last round
    const int next = b + T::STAGES - 1;
    if (next < count) fetch(next, next % T::STAGES);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    const float* xs = ring + (b % T::STAGES) * T::STAGE_FLOATS + ty * STRIDE;
    const float* ws = ring + (b % T::STAGES) * T::STAGE_FLOATS + (BM + tx) * STRIDE;
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      ulonglong2 xv[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) xv[i] = *reinterpret_cast<const ulonglong2*>(xs + i * TY * STRIDE + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(ws + j * TX * STRIDE + k);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fma2(xv[i].x, wv.x, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fma2(xv[i].y, wv.y, acc[i][j]);
      }
    }
  }

  auto finish = [&](int m, int n, float v) {
    if (m >= a.m || n >= a.n) return;
    if (a.bias) v += a.bias[n];
    if (epi == EPI_GELU) v = gelu_tanh(v);
    const size_t at = (size_t)m * a.n + n;
    if (epi == EPI_RESID) v += a.resid[at];
    a.out[at] = v;
  };
  if (splits == 1) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        float lo, hi;
        unpack2(acc[i][j], lo, hi);
        finish(m0 + i * TY + ty, n0 + j * TX + tx, lo + hi);
      }
    return;
  }
  __syncthreads();  // every warp is done with the ring
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      float lo, hi;
      unpack2(acc[i][j], lo, hi);
      ring[(i * TY + ty) * (BN + 1) + j * TX + tx] = lo + hi;
    }
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const unsigned base = (unsigned)__cvta_generic_to_shared(ring);
  for (int e = rank * THREADS + tid; e < BM * BN; e += splits * THREADS) {
    const int r = e / BN, c = e % BN;
    float v = 0.f;
    for (int q = 0; q < splits; ++q) {
      unsigned addr;
      float part;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(base + (r * (BN + 1) + c) * 4), "r"(q));
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(part) : "r"(addr) : "memory");
      v += part;
    }
    finish(m0 + r, n0 + c, v);
  }
  // nobody's shared memory goes away while another CTA reads it
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int BM, int BN, int TM, int TN>
cudaError_t launch_tile(const LinearArgs& a, int epi, int splits, cudaStream_t s) {
  using T = F32Tile<BM, BN, TM, TN>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((a.n + BN - 1) / BN) * (unsigned)((a.m + BM - 1) / BM), 1, splits);  // rows alone may be more than y holds
  cfg.blockDim = dim3(T::THREADS);
  cfg.dynamicSmemBytes = T::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = splits;
  cfg.attrs = attr;
  cfg.numAttrs = splits > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, gemm_f32_kernel<BM, BN, TM, TN>, a, epi, splits);
}

template <int BM, int BN, int TM, int TN>
cudaError_t allow_smem() {
  return cudaFuncSetAttribute(gemm_f32_kernel<BM, BN, TM, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)F32Tile<BM, BN, TM, TN>::SMEM);
}

}  // namespace

cudaError_t init_gemm_f32_attributes() {
  cudaError_t e = allow_smem<32, 64, 4, 4>();
  if (e == cudaSuccess) e = allow_smem<64, 64, 8, 4>();
  return e;
}

// Tiles of 32 rows up to 128 rows, of 64 above: at 128 rows both take the same time (n 2304, k 768: 25.5 and 26.6 us; n 4096,
// k 1024: 45.3 and 43.0 us), at 64 rows the small one is ahead (18.5 and 19.2; 28.7 and 28.0 us), at 256 the large one (37.2 and
// 35.2; 73.1 and 70.7 us). A 128 x 128 tile was not faster at any size up to 2048 rows (179 and 180 us; 455 and 399 us).
// k is halved while that leaves no more than four (64 rows: two and a half) CTAs per SM: n 768, k 3072, 32 rows took
// 92 / 49 / 28.7 / 18.5 us with 1 / 2 / 4 / 8 shares. The 128 x 128 x 8 tiles of one CTA each that were here before took 242 us
// per product of GPT-2 small at 32 rows (mean of the four) and 30 TFLOP/s at 8192.
cudaError_t launch_gemm_f32_tiles(const LinearArgs& a, int epilogue, cudaStream_t s) {
  if (a.m <= 0 || a.n <= 0) return cudaSuccess;
  auto shares = [&](int bm, long long most) {
    const long long tiles = (long long)((a.m + bm - 1) / bm) * ((a.n + 63) / 64);
    int sp = 1;
    while (sp < 8 && tiles * sp * 2 <= most && a.k >= sp * 2 * 64) sp *= 2;
    return sp;
  };
  if (a.m <= 128) return launch_tile<32, 64, 4, 4>(a, epilogue, shares(32, 4 * 148), s);
  return launch_tile<64, 64, 8, 4>(a, epilogue, shares(64, 5 * 148 / 2), s);
}

}  // namespace pg
