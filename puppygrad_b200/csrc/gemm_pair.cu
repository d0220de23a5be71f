// FP32-grade products of prompt rows on the FP16 tensor cores (sm_100a).
//
// A value v of a matrix with scale s (a power of two) is kept as a pair of FP16 numbers: hi = fp16(v s) and
// lo = fp16((v s - hi) 2^11), 22 and more significant bits. The product of two such matrices is
//
//   x . w = (sum hi_x hi_w + 2^-11 sum (hi_x lo_w + lo_x hi_w)) / (s_x s_w)
//
// with FP32 sums in tensor memory; the lo.lo term is below FP32 rounding. Three FP16 products at twice the TF32 rate, and half
// the bytes per value of the FP32 words that three TF32 products read. The scales put a bound of |v| at 2^14..2^15, so nothing
// overflows: the largest |w| of a matrix, and for activations what a LayerNorm, a convex combination of value rows or a
// product of a LayerNorm's row can reach (pair_scale, set when the weights are loaded). Everything within 2^-28 of the bound
// keeps its 22 bits; below that the error stays under 2^-50 of the bound. Whether that takes anything from a model is found out
// when it is loaded: how well pairs hold the rows of its weights (launch_pair_fit), and whether a bound is out of proportion to
// what the other columns can reach (PAIR_SPREAD). A model that fails either, or has weights that are not finite, goes without pairs.
// Splitting FP32 into FP16 parts with a scaled rest: Ootomo and Yokota, "Recovering single precision accuracy from Tensor Cores
// while surpassing the FP32 theoretical peak performance", 2022.
#include <cuda_fp16.h>

#include <algorithm>
#include <cfloat>
#include <cmath>

#include "kernels.cuh"
#include "pair.cuh"
#include "tc_common.cuh"

namespace pg {
namespace {

constexpr int PK = 64;   // FP16 elements per k block: one 128-byte swizzle row
constexpr int PBN = 128; // columns of an output tile
constexpr int PAIR_DRAIN = 8, PAIR_THREADS = (2 + PAIR_DRAIN) * 32;  // epilogue warps, two per quarter of the tensor-memory lanes

// EXACT_W: the weights are BF16 values that their hi parts hold, the lo parts are not read (PAIR_FIT_HI).
template <bool EXACT_W>
struct PairSmem {
  static constexpr int TILE_BYTES = TILE_M * PK * 2;  // 16 KB; 128 rows of weights are a tile too
  static constexpr int TILES = EXACT_W ? 3 : 4, STAGES = EXACT_W ? 4 : 3;
  static constexpr int STAGE_BYTES = TILES * TILE_BYTES;  // x hi, x lo, w hi, w lo
  static constexpr int EPI_BYTES = PAIR_DRAIN * 32 * 33 * 4;  // one padded 32x32 transpose tile per epilogue warp
  static constexpr size_t BYTES = (size_t)STAGES * STAGE_BYTES + EPI_BYTES + 1024 /*align*/ + 256 /*barriers*/;
};

// The weights lie in blocks of 128 rows x 64 values, hi tile and then (unless EXACT_W) lo tile, k block after k block, row tile after
// row tile (launch_tile_pairs): one box per block, and the same copy serves the decode step (gemm_chain.cu).
//
// Persistent over 128 x 128 output tiles (column tiles of one row panel are neighbours, so the activation panel is reused
// from L2). Warp 0 loads by TMA, one thread of warp 1 issues the MMAs, warps 2..9 drain, half of a tile's columns each.
// Tensor memory holds two buffers of two accumulators, so that a tile is drained while the next one is multiplied: the tensor core
// adds with truncation, a bias that grows with the MMAs into one accumulator, so the hi.hi products have one of their own and the
// small terms another. hi_x times the hi and the lo weight tile, which lie next to each other, is one MMA of N = 256 into both.
// Four warps did not drain a tile with GELU while the next one was multiplied: 8192 x 3072 x 768 with GELU 126.6 us with four and
// 96.2 with eight, 8192 x 768 x 768 36.1 and 32.5; 8192 x 4096 x 1024 with GELU 170.6 and 149.6.
//
// Bound by the tensor pipe where k is long: 82% of its active cycles at 8192 x 4800 x 1600; 66% at 8192 x 2304 x 768, where L2 (38%)
// and shared memory (28% of its reads, 23% of its writes) are no nearer their limits. Mean of a layer's four products, useful
// TFLOP/s (a third of the FP16 rate is 530): 8192 rows of GPT-2 small 343 (three TF32 products of FP32 words: 184), 16384 rows of
// GPT-2 XL 448 (207). Relative error against 64 bits of 16384 x 4800 x 1600: 1.9e-6.
template <bool EXACT_W>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
    tc_gemm_pair_kernel(const __grid_constant__ CUtensorMap map_xh, const __grid_constant__ CUtensorMap map_xl,
                        const __grid_constant__ CUtensorMap map_w, PairGemmArgs a) {
  using S = PairSmem<EXACT_W>;
  constexpr int TILE = S::TILE_BYTES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* epi_tiles = reinterpret_cast<float*>(base + (size_t)S::STAGES * S::STAGE_BYTES);
  uint64_t* full = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(epi_tiles) + S::EPI_BYTES);
  uint64_t* empty = full + S::STAGES;
  uint64_t* d_full = empty + S::STAGES;  // [2]: accumulator buffer holds a finished tile
  uint64_t* d_empty = d_full + 2;        // [2]: the epilogue warps have read it
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(d_empty + 2);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_n = (a.n + PBN - 1) / PBN, tiles = tiles_n * ((a.m + TILE_M - 1) / TILE_M);
  const int nkb = (a.k + PK - 1) / PK;
  // Reductions of more than 56 k blocks (224 MMAs into the hi.hi accumulator) are cut into chunks that the epilogue adds in
  // FP32, round to nearest, because of the truncation above. Not with GELU (not additive; its product has k = n_embd <= 4096).
  const int nchunk = a.epilogue == EPI_GELU ? 1 : (nkb + 55) / 56;
  const int kc = (nkb + nchunk - 1) / nchunk;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&d_full[i], 1);
      mbar_init(&d_empty[i], PAIR_DRAIN);
    }
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, 4 * PBN);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      RingCursor c;
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int n0 = (tile % tiles_n) * PBN, m0 = (tile / tiles_n) * TILE_M;
        for (int kb = 0; kb < nkb; ++kb, c.next(S::STAGES)) {  // chunk boundaries do not matter to the operand stream
          uint64_t* bar = &full[c.stage];
          ok = mbar_wait(&empty[c.stage], c.parity ^ 1, failed, a.error_flag, 1);
          if (!ok) break;
          uint8_t* st = base + (size_t)c.stage * S::STAGE_BYTES;
          mbar_expect_tx(bar, S::STAGE_BYTES);
          tma_load_2d(st, &map_xh, kb * PK, m0, bar);
          tma_load_2d(st + TILE, &map_xl, kb * PK, m0, bar);
          tma_load_2d(st + 2 * TILE, &map_w, 0, ((n0 / TILE_M) * nkb + kb) * ((EXACT_W ? 1 : 2) * TILE_M), bar);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = umma_idesc_f16(TILE_M, PBN), idesc_both = umma_idesc_f16(TILE_M, 2 * PBN);
      RingCursor c;
      uint32_t ti = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x)
        for (int kb0 = 0; kb0 < nkb && ok; kb0 += kc, ++ti) {
          const int kb1 = min(nkb, kb0 + kc);
          const uint32_t buf = ti & 1;
          if (ti >= 2) ok = mbar_wait(&d_empty[buf], ((ti >> 1) - 1) & 1, failed, a.error_flag, 4);
          if (!ok) break;
          tc_fence_after();
          const uint32_t tmem_d = tmem_base + buf * (2 * PBN), tmem_s = tmem_d + PBN;
          for (int kb = kb0; kb < kb1; ++kb, c.next(S::STAGES)) {
            ok = mbar_wait(&full[c.stage], c.parity, failed, a.error_flag, 2);
            if (!ok) break;
            tc_fence_after();
            const uint64_t xh = umma_desc_sw128(base + (size_t)c.stage * S::STAGE_BYTES), xl = xh + (TILE >> 4), wh = xl + (TILE >> 4);
#pragma unroll
            for (int k = 0; k < PK / 16; ++k) {
              const uint64_t o = (uint64_t)(k * 2);
              const uint32_t more = (kb != kb0) || k != 0;
              umma_bf16_ss(tmem_d, xh + o, wh + o, EXACT_W ? idesc : idesc_both, more);
              umma_bf16_ss(tmem_s, xl + o, wh + o, idesc, EXACT_W ? more : 1);
            }
            umma_commit(&empty[c.stage]);
          }
          if (ok) umma_commit(&d_full[buf]);
        }
    }
  } else {
    // TMEM lane = output row, but a row-per-thread store touches 32 cache lines per instruction: every 32x32 block goes
    // through a padded shared-memory tile and leaves column-per-lane (pairs: two columns per lane, two rows at a time).
    const int q = warp & 3, first_col = (warp - 2) / 4 * (PBN / 2);
    float* tile = epi_tiles + (warp - 2) * (32 * 33);
    uint32_t ti = 0;
    bool ok = true;
    for (int tile_id = blockIdx.x; tile_id < tiles && ok; tile_id += gridDim.x)
      for (int ch = 0; ch < nchunk && ok; ++ch, ++ti) {
        const bool first = ch == 0;
        const int n0 = (tile_id % tiles_n) * PBN, m0 = (tile_id / tiles_n) * TILE_M + q * 32;
        const uint32_t buf = ti & 1, tmem_d = tmem_base + buf * (2 * PBN) + ((uint32_t)(q * 32) << 16);
        ok = mbar_wait(&d_full[buf], (ti >> 1) & 1, failed, a.error_flag, 3);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int c0 = first_col; c0 < first_col + PBN / 2 && n0 + c0 < a.n; c0 += 32) {
          const int col = n0 + c0 + lane;
          // residual values (or what the chunks before left in `out`) are asked for before the accumulator is read: one
          // by one between the stores, which may alias them, each would cost a memory round trip
          float rv[32];
          const float* prev = first ? (a.epilogue == EPI_RESID ? a.resid : nullptr) : a.out;
          if (prev && col < a.n) {
#pragma unroll
            for (int rr = 0; rr < 32; ++rr) rv[rr] = m0 + rr < a.m ? prev[(size_t)(m0 + rr) * a.n + col] : 0.f;
          }
          const float bias = (a.bias && first && col < a.n) ? a.bias[col] : 0.f;
          float v[32], v2[32];
          tmem_ld32(tmem_d + (uint32_t)c0, v);
          tmem_ld32(tmem_d + (uint32_t)(PBN + c0), v2);
#pragma unroll
          for (int j = 0; j < 32; ++j) tile[lane * 33 + j] = fmaf(v2[j], PAIR_LO_INV, v[j]) * a.inv_x * a.inv_w;
          __syncwarp();
          if (a.out_hi) {
            const int cc = (lane & 15) * 2, half = lane >> 4;
            const float b0 = __shfl_sync(0xffffffffu, bias, cc), b1 = __shfl_sync(0xffffffffu, bias, cc + 1);
            if (n0 + c0 + cc < a.n) {  // n is even
#pragma unroll
              for (int rr = 0; rr < 32; rr += 2) {
                const int row = m0 + rr + half;
                if (row < a.m) {
                  float y0 = tile[(rr + half) * 33 + cc] + b0, y1 = tile[(rr + half) * 33 + cc + 1] + b1;
                  if (a.epilogue == EPI_GELU) {
                    y0 = gelu_ref(y0);
                    y1 = gelu_ref(y1);
                  }
                  const size_t at = (size_t)row * a.n + n0 + c0 + cc;
                  store_pair2(a.out_hi + at, a.out_lo + at, y0, y1, a.out_scale);
                }
              }
            }
          } else if (col < a.n) {
#pragma unroll
            for (int rr = 0; rr < 32; ++rr) {
              if (m0 + rr < a.m) {
                float r = tile[rr * 33 + lane] + bias;
                if (a.epilogue == EPI_GELU) r = gelu_ref(r);
                if (prev) r = rv[rr] + r;
                a.out[(size_t)(m0 + rr) * a.n + col] = r;
              }
            }
          }
          __syncwarp();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&d_empty[buf]);
      }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 4 * PBN);
}

__global__ void __launch_bounds__(256) make_pairs_kernel(const float4* __restrict__ x, uint16_t* hi, uint16_t* lo, size_t n4, float scale) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x)
    store_pair4(hi + 4 * i, lo + 4 * i, x[i], scale);
}

// One warp per 64-value piece of a weight row (rows up to the next multiple of 128 and k up to one of 64: zeros).
__global__ void __launch_bounds__(256) tile_pairs_kernel(const float* __restrict__ w, uint16_t* dst, int n, int k, int exact, float scale) {
  const int nkb = (k + PK - 1) / PK, lane = threadIdx.x & 31;
  const long long pieces = (long long)((n + TILE_M - 1) / TILE_M) * TILE_M * nkb;
  for (long long i = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); i < pieces; i += (long long)gridDim.x * 8) {
    const int row = (int)(i / nkb), kb = (int)(i - (long long)row * nkb), col = kb * PK + lane * 2;
    const float a = row < n && col < k ? w[(size_t)row * k + col] : 0.f, b = row < n && col + 1 < k ? w[(size_t)row * k + col + 1] : 0.f;
    uint32_t hi, lo;
    split_pair2(a, b, scale, hi, lo);
    const long long block = (long long)(row / TILE_M) * nkb + kb;
    uint32_t* at = reinterpret_cast<uint32_t*>(dst + (block * (exact ? 1 : 2) * TILE_M + row % TILE_M) * PK) + lane;
    at[0] = hi;
    if (!exact) at[TILE_M * PK / 2] = lo;
  }
}

// The largest |w| of a matrix [rows, cols], as a bit pattern that orders like the non-negative number it is, and the Euclidean norms
// of its rows (unless null). Values that are not finite do not count. One warp per row.
__global__ void __launch_bounds__(256) matrix_bounds_kernel(const float* __restrict__ w, int rows, int cols, unsigned* largest, float* norms) {
  const int lane = threadIdx.x & 31;
  float top = 0.f;
  for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8) {
    double sq = 0.0;
    for (int i = lane; i < cols; i += 32) {
      const float v = fabsf(w[(size_t)r * cols + i]);
      if (!isfinite(v)) continue;
      top = fmaxf(top, v);
      sq = fma((double)v, (double)v, sq);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if (norms && lane == 0) norms[r] = __double2float_ru(sqrt(sq));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
  if (lane == 0) atomicMax(largest, __float_as_uint(top));
}

// How well FP16 holds the rows of w * scale: the largest share of a row's squared length that is lost by hi parts alone and by
// pairs, as bit patterns (NaN, of a row with values that are not finite, comes out above all numbers). One warp per row.
__global__ void __launch_bounds__(256) pair_fit_kernel(const float* __restrict__ w, int rows, int cols, float scale, unsigned* out) {
  const int lane = threadIdx.x & 31;
  for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8) {
    double sq = 0.0, hi_off = 0.0, pair_off = 0.0;
    for (int i = lane; i < cols; i += 32) {
      const float v = w[(size_t)r * cols + i];
      uint32_t hi, lo;
      split_pair2(v, 0.f, scale, hi, lo);
      const double x = (double)v * scale, left = x - __half2float(__ushort_as_half((unsigned short)hi)),
                   rest = left - (double)__half2float(__ushort_as_half((unsigned short)lo)) * PAIR_LO_INV;
      sq = fma(x, x, sq);
      hi_off = fma(left, left, hi_off);
      pair_off = fma(rest, rest, pair_off);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sq += __shfl_xor_sync(0xffffffffu, sq, o);
      hi_off += __shfl_xor_sync(0xffffffffu, hi_off, o);
      pair_off += __shfl_xor_sync(0xffffffffu, pair_off, o);
    }
    if (lane == 0 && sq != 0.0) {
      atomicMax(out, __float_as_uint((float)(hi_off / sq)) & 0x7fffffffu);
      atomicMax(out + 1, __float_as_uint((float)(pair_off / sq)) & 0x7fffffffu);
    }
  }
}

int sm_count() {
  static const int n = [] {
    int dev = 0, v = 148;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) v = 148;
    return v;
  }();
  return n;
}

template <bool EXACT_W>
cudaError_t launch_pair(const PairGemmArgs& a, cudaStream_t s) {
  CUtensorMap xh, xl, w;
  const uint64_t w_rows = pair_tiled_halves(a.n, a.k, EXACT_W) / PK;
  if (!make_map_f16(&xh, a.x_hi, a.m, a.k, TILE_M) || !make_map_f16(&xl, a.x_lo, a.m, a.k, TILE_M) ||
      w_rows > 0x7fffffffull || !make_map_f16(&w, a.w, w_rows, PK, (EXACT_W ? 1 : 2) * TILE_M))
    return cudaErrorInvalidValue;
  const int tiles = ((a.n + PBN - 1) / PBN) * ((a.m + TILE_M - 1) / TILE_M);
  tc_gemm_pair_kernel<EXACT_W><<<std::min(tiles, sm_count()), PAIR_THREADS, PairSmem<EXACT_W>::BYTES, s>>>(xh, xl, w, a);
  return cudaGetLastError();
}

}  // namespace

bool pair_gemm_supported(int k) { return k > 0 && k % 32 == 0 && encode_fn() != nullptr; }

float pair_scale(double bound) {
  if (!(bound > 0.0)) return 1.f;
  const int e = 14 - std::ilogb(std::min(bound, (double)FLT_MAX));  // bound * 2^e in [2^14, 2^15); no FP32 value is above FLT_MAX
  return std::ldexp(1.f, std::min(120, e));
}

size_t pair_tiled_halves(int n, int k, bool exact) {
  return (size_t)((n + TILE_M - 1) / TILE_M) * ((k + PK - 1) / PK) * TILE_M * PK * (exact ? 1 : 2);
}

cudaError_t launch_tile_pairs(const float* w, uint16_t* dst, int n, int k, bool exact, float scale, cudaStream_t s) {
  tile_pairs_kernel<<<148 * 8, 256, 0, s>>>(w, dst, n, k, exact ? 1 : 0, scale);
  return cudaGetLastError();
}

cudaError_t launch_make_pairs(const float* x, uint16_t* hi, uint16_t* lo, size_t n, float scale, cudaStream_t s) {
  if (n % 4 != 0) return cudaErrorInvalidValue;
  const int blocks = (int)std::max<size_t>(1, std::min<size_t>((n / 4 + 255) / 256, 148 * 8));
  make_pairs_kernel<<<blocks, 256, 0, s>>>(reinterpret_cast<const float4*>(x), hi, lo, n / 4, scale);
  return cudaGetLastError();
}

cudaError_t launch_matrix_bounds(const float* w, int rows, int cols, unsigned* largest, float* norms, cudaStream_t s) {
  matrix_bounds_kernel<<<std::max(1, std::min((rows + 7) / 8, 148 * 8)), 256, 0, s>>>(w, rows, cols, largest, norms);
  return cudaGetLastError();
}

cudaError_t launch_pair_fit(const float* w, int rows, int cols, float scale, unsigned* out, cudaStream_t s) {
  pair_fit_kernel<<<std::max(1, std::min((rows + 7) / 8, 148 * 8)), 256, 0, s>>>(w, rows, cols, scale, out);
  return cudaGetLastError();
}

cudaError_t init_pair_gemm_attributes() {
  cudaError_t e = cudaFuncSetAttribute(tc_gemm_pair_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PairSmem<false>::BYTES);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(tc_gemm_pair_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PairSmem<true>::BYTES);
}

cudaError_t launch_tc_gemm_pair(const PairGemmArgs& a, cudaStream_t s) {
  if (a.m <= 0 || a.n <= 0) return cudaSuccess;
  if (!pair_gemm_supported(a.k) || !a.x_hi || !a.x_lo || !a.w || (!a.out && !a.out_hi)) return cudaErrorInvalidValue;
  if (a.out_hi && (a.n % 2 != 0 || !a.out_lo || a.epilogue == EPI_RESID || (a.epilogue != EPI_GELU && a.k > 56 * PK))) return cudaErrorInvalidValue;
  return a.w_exact ? launch_pair<true>(a, s) : launch_pair<false>(a, s);
}

}  // namespace pg
